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


@pytest.mark.parametrize("ctas,behind,lets_in", [(48, 96, True), (52, 96, True), (53, 96, False), (64, 96, False), (64, 64, True),
                                                 (96, 64, False), (48, 128, False), (1, None, False), (147, 1, True), (148, 0, True)])
def test_what_stands_behind_decides_whether_it_is_let_in(ctas, behind, lets_in):
    assert ops.decode_lets_in(ctas, behind, 148) is lets_in


def test_sms_of_a_product_are_asked_once_and_kept_apart(monkeypatch):
    asked = []

    def answer(N, K, heads, rows):
        asked.append((N, K, heads, rows))
        return 2 ** 31 - 1 if K == 8 else N * heads // 16
    monkeypatch.setattr(ops, "_SKINNY_SMS", {})
    monkeypatch.setattr(ops.build, "load", lambda name: type("Library", (), {"ft_skinny_sms": staticmethod(answer)}))
    assert [ops.skinny_sms("cuda:0", rows, 64, 64) for rows in (1, 8, 9, 16, 32)] == [4] * 5
    assert ops.skinny_sms("cuda:1", 3, 64, 64) == 4 and ops.skinny_sms("cuda:0", 3, 64, 64, heads=4) == 16
    assert ops.skinny_sms("cuda:0", 3, 64, 8) is None and ops.skinny_sms("cuda:0", 4, 64, 8) is None
    assert asked == [(64, 64, 1, 8), (64, 64, 1, 16), (64, 64, 1, 32), (64, 64, 1, 8), (64, 64, 4, 8), (64, 8, 1, 8)]


def test_a_step_says_what_stands_behind_its_attention(monkeypatch):
    """The output projection of few rows, the gate's blocks, nothing where prompts' tiles come in between or the library takes
    the rows."""
    from types import SimpleNamespace

    from freetoken_b200.parts import attention, linear
    seen = []
    monkeypatch.setattr(ops, "attn_decode", lambda *a, sms_behind=None, **k: seen.append(sms_behind))
    monkeypatch.setattr(ops, "attn_decode_takes", lambda q, d: True)
    monkeypatch.setattr(ops, "attn_prefill", lambda *a, **k: None)
    monkeypatch.setattr(ops, "PREFILL_TC_MIN_SCORES", 1 << 60)
    monkeypatch.setattr(ops, "skinny_sms", lambda device, rows, N, K, heads=1: (rows, N, K, heads))
    core = attention.PagedSoftmaxCore()
    core.nq, core.nkv, core.d, core.scale = 8, 2, 64, 0.1
    q = torch.zeros(3, 512, dtype=torch.bfloat16)
    for tiles in (0, 2):
        plan = SimpleNamespace(host={"num_decode_rows": 3, "num_prefill_tiles": tiles, "prefill_scores": 0,
                                     "max_decode_kv_len": 64}, tensors={"tile_seg": None, "tile_q0": None})
        ctx = SimpleNamespace(plan=lambda part: plan, token_pos=None, token_seg=None, seg_q_start=None, seg_pos0=None,
                              workspace=None)
        core.attend(ctx, q, q, None, None, 40)
    assert seen == [40, None]
    w = torch.zeros(128, 512, dtype=torch.bfloat16)
    assert linear.sms_taken(q, w) == (3, 128, 512, 1)
    assert linear.sms_taken(torch.zeros(33, 512, dtype=torch.bfloat16), w) is None
    assert linear.sms_taken(q.float(), w) is None
    assert linear.sms_taken(q, torch.zeros(8, 16, 64, dtype=torch.bfloat16)) == (3, 16, 64, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,keys", [(1, 2048), (1, 300), (4, 130)])
def test_the_launch_behind_gives_the_same_rows_let_in_or_not(rows, keys):
    from test_kernels_gpu import DEV, rnd
    from freetoken_b200.parts.base import Workspace
    H, G, D, page = 32, 4, 128, 64
    pages = -(-keys // page)
    kv = rnd(2, rows * pages + 1, G, page, D, dtype=torch.bfloat16, seed=1)
    table = torch.arange(1, rows * pages + 1, dtype=torch.int32, device=DEV).view(rows, pages)
    q, w = rnd(rows, H * D, dtype=torch.bfloat16, seed=2), rnd(2048, H * D, dtype=torch.bfloat16, seed=3, scale=0.02)
    pos = torch.full((rows,), keys - 1, dtype=torch.int32, device=DEV)
    seg = torch.arange(rows, dtype=torch.int32, device=DEV)
    ws = Workspace(DEV)
    got = []
    for behind in (None, 0):                 # closed, and open whatever comes
        for _ in range(10):
            o, y = torch.zeros_like(q), torch.zeros(rows, 2048, dtype=torch.bfloat16, device=DEV)
            ops.attn_decode(q, o, kv, None, rows, pos, seg, table, H, G, D, D ** -0.5, None, keys, ws, sms_behind=behind)
            ops.skinny_gemm(o, w, y)
            got.append(y)
    assert ops.decode_lets_in(1, 0, ops.sm_count(DEV))
    for y in got[1:]:
        assert torch.equal(y, got[0])


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
