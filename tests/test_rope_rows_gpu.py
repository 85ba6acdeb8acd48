"""The rotation and store of many tokens (rows kept in registers) beside the kernel of up to 64 tokens."""

import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


# head sizes of 4, 8, 16 and 32 pieces; rows that end inside a block's round and inside a warp; no rotation, a part of
# a head, all of it; no norm, one a row, one a head; pairs; blended values; a stop that stores nothing
@pytest.mark.parametrize("nq,nkv,d,R,mode,pairs,blend,store", [
    (6, 2, 32, 16, 2, False, False, True), (3, 1, 64, 64, 1, False, False, True), (5, 5, 128, 0, 1, False, False, True),
    (16, 4, 128, 64, 0, False, True, True), (7, 1, 128, 128, 2, False, False, True), (4, 4, 256, 128, 1, False, False, True),
    (9, 3, 64, 24, 0, True, False, True), (48, 8, 128, 64, 1, False, False, True), (24, 8, 256, 32, 0, False, False, False),
    (12, 3, 64, 48, 1, False, False, True)])             # a rotary half of three pieces: the general kernel either way
def test_many_tokens_like_few(nq, nkv, d, R, mode, pairs, blend, store):
    T, P = 70, 16
    bf = torch.bfloat16
    qkv = rnd(T, (nq + 2 * nkv) * d + 8, dtype=bf, seed=1)[:, :(nq + 2 * nkv) * d]
    qw = kw = None
    if mode:
        qw, kw = (rnd(n * d if mode == 1 else d, seed=2 + i) for i, n in enumerate((nq, nkv)))
    turn = rnd(T, R, seed=4) if R else None
    more = dict(value_first=rnd(T, nkv * d, dtype=bf, seed=5), value_lambda=torch.tensor([0.4], device=DEV)) if blend else {}
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seg = torch.zeros(T, dtype=torch.int32, device=DEV)
    table = torch.tensor([[3, 1, 5, 2, 4]], dtype=torch.int32, device=DEV)
    results = []
    for rows in (T, 10):
        q = torch.full((T, nq * d), float("nan"), dtype=bf, device=DEV)
        pages = torch.zeros(2, 6, nkv, P, d, dtype=bf, device=DEV)
        for a in range(0, T, rows):
            b = min(T, a + rows)
            part = {k: v[a:b] if k == "value_first" else v for k, v in more.items()}
            ops().qk_rope_store(qkv[a:b], q[a:b], pages if store else None, qw, kw, turn, pos[a:b], seg[a:b], table, nq, nkv, d,
                                R, mode, mode == 2, pairs, 1e-6, **part)
        results.append((q.float(), pages.float()))
    for many, few in zip(*results):
        # Both round a rotation's two products and their sum in float32, one of the three inside a fused multiply-add;
        # which one, and the order of a norm's sum, is not the same: values of up to 16 then differ by some 2^-23 * 16
        # (2e-6) before they are stored, and by one bfloat16 step (2^-7 of the value) where that crosses a rounding
        # boundary, which is 2^-8 * 16 wide: in about one value of 10,000.
        assert torch.allclose(many, few, rtol=2 ** -7, atol=1e-5)
        assert (many != few).float().mean() < 1e-3
