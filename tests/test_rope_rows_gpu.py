"""The rotation and store of many tokens (rows kept in registers) beside the kernel of up to 64 tokens, bit for bit,
and beside PyTorch in float32."""

import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


def plain(qkv, qw, kw, turn, pos, nq, nkv, d, R, mode, pairs, eps):
    """Queries, keys and values of rows [q | k | v] in float32."""
    T = qkv.shape[0]
    x = qkv.float().view(T, nq + 2 * nkv, d)
    parts = [x[:, :nq], x[:, nq:nq + nkv]]
    for i, w in enumerate((qw, kw)):
        if mode:
            dims = (-2, -1) if mode == 1 else -1
            scale = torch.rsqrt(parts[i].pow(2).mean(dims, keepdim=True) + eps)
            parts[i] = parts[i] * scale * (w.view(-1, d) + (mode == 2))
        if R:
            z, h = parts[i].clone(), R // 2
            c, s = turn[pos.long(), None, :h], turn[pos.long(), None, h:]
            a, b = (slice(0, R, 2), slice(1, R, 2)) if pairs else (slice(0, h), slice(h, R))
            z[..., a] = parts[i][..., a] * c - parts[i][..., b] * s
            z[..., b] = parts[i][..., b] * c + parts[i][..., a] * s
            parts[i] = z
    return parts[0].reshape(T, nq * d), parts[1], x[:, nq + nkv:]


# head sizes of 4, 8, 16 and 32 pieces; one to eight pieces a thread; rows that end inside a block's round and inside
# a warp; keys that begin with a block's first thread and elsewhere; no rotation, a part of a head, all of it; no norm,
# one a row, one a head; pairs; blended values; a stop that stores nothing
@pytest.mark.parametrize("nq,nkv,d,R,mode,pairs,blend,store", [
    (6, 2, 32, 16, 2, False, False, True), (3, 1, 64, 64, 1, False, False, True), (5, 5, 128, 0, 1, False, False, True),
    (16, 4, 128, 64, 0, False, True, True), (7, 1, 128, 128, 2, False, False, True), (4, 4, 256, 128, 1, False, False, True),
    (9, 3, 64, 24, 0, True, False, True), (48, 8, 128, 64, 1, False, False, True), (24, 8, 256, 32, 0, False, False, False),
    (32, 8, 128, 64, 2, False, False, True), (32, 8, 128, 128, 1, False, True, True), (40, 8, 256, 64, 1, False, False, True),
    (24, 12, 256, 256, 2, True, False, True), (21, 11, 128, 64, 1, False, False, True),
    (12, 3, 64, 48, 1, False, False, True)])             # a rotary half of three pieces: the general kernel either way
def test_many_tokens_like_few(nq, nkv, d, R, mode, pairs, blend, store):
    T, first, P, eps = 150, 83, 16, 1e-6                 # two requests: 83 tokens from place 0, 67 from place 9
    bf = torch.bfloat16
    qkv = rnd(T, (nq + 2 * nkv) * d + 8, dtype=bf, seed=1)[:, :(nq + 2 * nkv) * d]
    qw = kw = None
    if mode:
        qw, kw = (rnd(n * d if mode == 1 else d, seed=2 + i) for i, n in enumerate((nq, nkv)))
    turn = rnd(T, R, seed=4) if R else None
    value_first, lam = rnd(T, nkv * d, dtype=bf, seed=5), 0.4
    pos = torch.cat([torch.arange(first), torch.arange(9, 9 + T - first)]).to(torch.int32).to(DEV)
    seg = (torch.arange(T) >= first).to(torch.int32).to(DEV)
    table = torch.tensor([[3, 1, 5, 2, 4, 11], [7, 10, 6, 9, 8, 0]], dtype=torch.int32, device=DEV)
    results = []
    for rows in (T, 64, 10):
        q = torch.full((T, nq * d), float("nan"), dtype=bf, device=DEV)
        pages = torch.zeros(2, 12, nkv, P, d, dtype=bf, device=DEV)
        for a in range(0, T, rows):
            b = min(T, a + rows)
            more = dict(value_first=value_first[a:b], value_lambda=torch.tensor([lam], device=DEV)) if blend else {}
            ops().qk_rope_store(qkv[a:b], q[a:b], pages if store else None, qw, kw, turn, pos[a:b], seg[a:b], table, nq, nkv, d,
                                R, mode, mode == 2, pairs, eps, **more)
        results.append((q, pages))
    for few in results[1:]:
        assert torch.equal(results[0][0], few[0]) and torch.equal(results[0][1], few[1])
    q, k, v = plain(qkv, qw, kw, turn, pos, nq, nkv, d, R, mode, pairs, eps)
    if blend:
        v = (1 - lam) * v + lam * value_first.float().view(T, nkv, d)
    # float32 inside, of values up to about 20 (1e-5), then one rounding to bfloat16 (2^-9 of the value)
    close = dict(rtol=2 ** -8, atol=1e-5)
    assert torch.allclose(results[0][0].float(), q, **close)
    if not store:
        return
    page, place = table[seg.long(), pos.long() // P].long(), pos.long() % P
    assert torch.allclose(results[0][1][0, page, :, place].float(), k, **close)
    assert torch.allclose(results[0][1][1, page, :, place].float(), v, **close)
