"""How the decode attention's keys are divided, and on the GPU that every division gives the same rows."""

import pytest
import torch

from freetoken_b200.csrc import ops


@pytest.mark.parametrize("rows,heads,group,keys", [(1, 4, 4, 1024), (8, 4, 4, 1024), (8, 8, 6, 2100), (5, 8, 6, 2048), (64, 8, 6, 256),
                                                   (1, 1, 32, 63), (2, 8, 6, 65536)])
def test_splits_cover_the_keys_and_fit(rows, heads, group, keys):
    room = {2: 148, 3: 93, 4: 71, 5: 56, 6: 45, 7: 37, 8: 33}
    plain = ops.decode_splits(rows, heads, group, keys, 148, cluster_merge=True)
    splits, per = ops.decode_splits(rows, heads, group, keys, 148, cluster_merge=True, room=room)
    assert per % 64 == 0 and (splits - 1) * per < keys <= splits * per
    base = rows * heads * -(-group // 16)
    if plain[0] == 1 or plain[0] > ops.CLUSTER_SPLITS or base <= room[plain[0]] * 15 // 16:
        assert (splits, per) == plain
    elif splits in room:
        assert base <= room[splits] * 15 // 16 or base > 148


@pytest.mark.parametrize("rows,heads,group,keys", [(8, 4, 4, 1024), (1, 8, 12, 2048), (2, 1, 16, 8192), (1, 4, 4, 100)])
def test_a_cluster_that_finds_no_place_is_not_chosen(rows, heads, group, keys):
    def chosen(room):
        return ops.decode_splits(rows, heads, group, keys, 148, cluster_merge=True, room=room)[0]
    sizes = range(2, ops.CLUSTER_SPLITS + 1)
    free = ops.decode_splits(rows, heads, group, keys, 148, cluster_merge=True)[0]
    assert chosen({}) == chosen({size: 148 for size in sizes}) == free                # not known, and room for all
    for none in sizes:
        assert chosen({size: 148 * (size != none) for size in sizes}) != none
    assert chosen(dict.fromkeys(sizes, 0)) not in sizes


def test_sizes_that_are_refused_are_kept_apart_from_those_not_known(monkeypatch):
    answers = {2: 74, 3: 49, 4: 36, 5: 0, 6: -1, 7: 0, 8: -1}
    monkeypatch.setattr(ops, "_CLUSTER_ROOM", {})
    monkeypatch.setattr(ops.build, "load", lambda name: type("Library", (), {
        "ft_attn_decode_clusters": staticmethod(lambda d, size: answers[size])}))
    assert ops.cluster_room("cuda:0", 128) == {2: 74, 3: 49, 4: 36, 5: 0, 7: 0}


@pytest.mark.gpu
@pytest.mark.parametrize("window,chunk", [(None, 0), (100, 0), (128, 0), (63, 0), (None, 96), (200, 64), (1, 0)])
@pytest.mark.parametrize("D,page", [(128, 64), (64, 128), (32, 16)])
def test_every_division_gives_the_same_rows(monkeypatch, D, page, window, chunk):
    from test_kernels_gpu import DEV, rnd
    from freetoken_b200.parts.base import Workspace
    H, G, lens = 8, 2, [1, 64, 65, 200, 517]
    pages = [-(-n // page) for n in lens]
    width = max(pages)
    kv = rnd(2, sum(pages) + 1, G, page, D, dtype=torch.bfloat16, seed=1)
    table = torch.zeros(len(lens), width, dtype=torch.int32)
    at = 1
    for i, n in enumerate(pages):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    q = rnd(len(lens), H * D, dtype=torch.bfloat16, seed=2)
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    seg = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    options = ops.ScoreOptions(chunk=chunk, sink_value=0.5)
    want = torch.empty(len(lens), H * D)
    for i, n in enumerate(lens):
        keys, values = (kv[j, table[i].to(DEV).long()].transpose(1, 2).reshape(-1, G, D)[:n].double().cpu() for j in (0, 1))
        lo = max(0, n - window) if window else 0
        lo = max(lo, (n - 1) // chunk * chunk) if chunk else lo
        s = torch.einsum("hd,khd->hk", q[i].view(H, D).double().cpu(), keys[lo:].repeat_interleave(H // G, 1)) * D ** -0.5
        p = torch.softmax(torch.cat([s, torch.full((H, 1), 0.5, dtype=torch.float64)], 1), 1)[:, :-1]
        want[i] = torch.einsum("hk,khd->hd", p, values[lo:].repeat_interleave(H // G, 1)).flatten()
    real = ops.decode_splits
    seen = []
    for forced in (None, (1, 576), (3, 192), (5, 128), (9, 64)):
        def splits(rows, heads, group, keys, *a, **k):
            seen.append(keys)
            return real(rows, heads, group, keys, *a, **k) if forced is None else forced
        monkeypatch.setattr(ops, "decode_splits", splits)
        out = torch.empty_like(q)
        ops.attn_decode(q, out, kv, None, len(lens), pos, seg, table.to(DEV), H, G, D, D ** -0.5, window, max(lens), Workspace(DEV),
                        options=options)
        # probabilities and values are rounded to bfloat16 (2^-9 each) ahead of float32 sums, the result once more
        assert torch.allclose(out.float().cpu(), want, atol=0.02, rtol=0.02), forced
    reach = min([n for n in (window, chunk) if n], default=None)
    assert set(seen) == {min(max(lens), reach + 63) if reach else max(lens)}
