"""State rows of newly admitted slots: any set of slots, one launch a state group."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def storage(slots, groups):
    from freetoken_b200.cache.storage import CacheStorage
    need = lambda shape, dtype: SimpleNamespace(shape=shape, dtype=dtype)
    manager = SimpleNamespace(paged_groups=[], max_slots=slots - 1, state_groups=[
        SimpleNamespace(stops=range(stops), need=need(shape, dtype)) for stops, shape, dtype in groups])
    s = CacheStorage(manager, torch.bfloat16, "cuda")
    for t in s.state:
        t.copy_(torch.arange(t.numel(), device="cuda").view(t.shape) % 100 + 1)
    return s


# rows of whole 16-byte pieces, longer than a launch's blocks take in one round, of odd lengths and one element
GROUPS = [(3, (8, 16), "float32"), (2, (300, 1024), "float32"), (4, (7, 3), "bfloat16"), (1, (1,), "int32"), (2, (5,), "float32")]


@pytest.mark.parametrize("slots,cleared", [(9, [4]), (9, [7, 0, 2, 5]), (40, list(range(0, 40, 2))), (300, list(range(299, 1, -2))),
                                           (9, [8, -9, 3, 3])])
def test_any_slots_in_one_launch_a_group(slots, cleared):
    from freetoken_b200.csrc import ops
    s = storage(slots, GROUPS)
    want = [t.clone() for t in s.state]
    for w in want:
        w[:, cleared] = 0
    before = ops.launch_count()
    s.clear_state(cleared)
    assert ops.launch_count() - before == len(GROUPS) * -(-len(cleared) // 128)
    assert all(torch.equal(t, w) for t, w in zip(s.state, want))


@pytest.mark.parametrize("cleared", [[9], [0, -10]])
def test_slots_outside_are_refused(cleared):
    s = storage(9, GROUPS[:1])
    kept = s.state[0].clone()
    with pytest.raises(IndexError):
        s.clear_state(cleared)
    assert torch.equal(s.state[0], kept)
