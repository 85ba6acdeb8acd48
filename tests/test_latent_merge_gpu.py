"""The merge of latent attention's splits: its rounds hold 1,024 splits, a launch may have any number."""

import pytest
import torch

from test_dizatar_gpu import ints, paged_rows

pytestmark = pytest.mark.gpu


# the last split of a round and the first of the next; splits that see no key, whole rounds of them before a window and
# behind the keys; 512 values and more: two pieces a thread
@pytest.mark.parametrize("d,rank,keys,window,splits", [
    (104, 88, 64 * 1024, None, 1024), (104, 88, 64 * 1025, None, 1025), (40, 24, 64 * 1100 + 5, None, 1101),
    (40, 24, 64 * 2100, 64 * 30, 2100), (24, 24, 700, None, 6142), (24, 24, 700, 100, 7000), (576, 568, 64 * 1030, None, 1030)])
def test_any_number_of_splits(monkeypatch, d, rank, keys, window, splits):
    from freetoken_b200.csrc import ops
    from freetoken_b200.parts.base import Workspace
    torch.manual_seed(splits)
    H, segs = 3, [(keys - 1, 1)]
    pages, table, rows, starts, pos0, _ = paged_rows(segs, 64, d)
    q = (torch.randn(1, H, d) * 0.5).to(torch.bfloat16)
    # every head sees two keys, one among the first and one among the last, at a score that leaves them most of the weight
    # (e^14 each beside up to e^12 of all others); their values differ
    for h in range(H):
        for at in ((keys - window if window else 0) + 5 + h, keys - 5 - h):
            side = torch.randn(d)
            row = q[0, h].float() * 14 * d ** 0.5 / q[0, h].float().square().sum()
            row += side - q[0, h].float() * (side @ q[0, h].float()) / q[0, h].float().square().sum()
            rows[0][at] = row.to(torch.bfloat16)
            pages[table[0, at // 64].long(), 0, at % 64] = rows[0][at].cuda()
    out = torch.full((1, H, rank), float("nan"), dtype=torch.bfloat16, device="cuda")
    monkeypatch.setattr(ops, "latent_splits", lambda tiles, max_kv_len, slots: (splits, 64))
    ops.attn_latent(q.cuda(), out, pages, ints([0]), ints([0]), starts, pos0, table, H, rank, d ** -0.5, window, keys,
                    Workspace("cuda"))
    seen = rows[0][keys - window if window else 0:].double()
    want = torch.softmax(q[0].double() @ seen.T * d ** -0.5, -1) @ seen[:, :rank]
    # bfloat16: probabilities and outputs to 2^-9 each
    assert float((out[0].double().cpu() - want).abs().max()) < 2 ** -7 * float(want.abs().max())
    ops.check_tc_status("cuda:0")
