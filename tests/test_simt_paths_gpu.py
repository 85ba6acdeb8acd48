"""The CUDA-core kernels' variants against each other: which of them a launch takes depends on its rows, columns
and alignment, a row's result on none of these."""

import pytest
import torch

from test_kernels_gpu import DEV, DT, GEMM_TYPES, _grouped_case, ops, rnd

pytestmark = pytest.mark.gpu


def _misaligned(x):
    """The same rows one element into wider ones: no 16-byte pieces, so the plain kernel runs."""
    wide = torch.zeros(x.shape[0], x.shape[1] + 3, dtype=x.dtype, device=DEV)
    wide[:, 1:1 + x.shape[1]] = x
    return wide[:, 1:1 + x.shape[1]]


@pytest.mark.parametrize("at,wt,ct", GEMM_TYPES)
@pytest.mark.parametrize("M,N,K", [
    (1, 31, 8), (2, 33, 136), (3, 32, 128), (5, 100, 512), (9, 70, 392), (17, 40, 1040),   # streamed, 1 .. 16 rows a block
    (64, 8192, 16), (65, 8200, 48), (130, 4100, 144),                                      # register tiles and their edges
    (400, 8, 264),                                                                         # many rows, few columns: streamed
    (1, 65535 * 32, 8), (2, 65535 * 32 + 33, 8)])                                          # as many blocks as a grid holds; more
def test_dense_products_agree_bitwise(at, wt, ct, M, N, K):
    a, w = rnd(M, K, dtype=DT[at], seed=1), rnd(N, K, dtype=DT[wt], seed=2, scale=0.1)
    got, want = (torch.full((M, N), float("nan"), dtype=DT[ct], device=DEV) for _ in range(2))
    ops().gemm_rows(a, w, got)
    ops().gemm_rows(_misaligned(a), w, want)
    assert torch.equal(got, want)


@pytest.mark.parametrize("E,k,T,H,I", [(8, 2, 1, 64, 40), (8, 3, 19, 96, 48), (70, 2, 9, 136, 24),
                                       (4, 2, 300, 64, 520),                               # 150 rows a group: tiles
                                       (40, 1, 33, 40, 24)])
def test_grouped_products_agree_bitwise(E, k, T, H, I):
    _, order, token, offsets = _grouped_case(E, k, T)
    R = T * k
    x = rnd(T, H, seed=1)
    w1, w2 = rnd(E, 2 * I, H, dtype=torch.bfloat16, seed=2, scale=0.1), rnd(E, H, I, dtype=torch.bfloat16, seed=3, scale=0.1)
    rw = torch.rand(R, generator=torch.Generator().manual_seed(4)).to(DEV)
    out = []
    for view in (lambda t: t, _misaligned):
        mid, parts = torch.zeros(R, I, device=DEV), torch.zeros(R, H, device=DEV)
        ops().gemm_rows(view(x), w1, mid, group_offsets=offsets, a_rows=token, rows=R, glu=True)
        ops().gemm_rows(view(mid), w2, parts, group_offsets=offsets, c_rows=order, row_scale=rw, rows=R)
        out.append((mid, parts))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nq,nkv,d,window", [(8, 4, 16, None), (6, 2, 64, 33), (24, 2, 40, None)])
def test_attention_rows_do_not_depend_on_their_block(dtype, nq, nkv, d, window):
    """Enough tokens that neighbours share a block, requests ending inside one; every row again by itself."""
    from test_kernels_gpu import _paged_case
    lens = [(0, 75), (40, 41), (7, 50)]
    q, kv, pos, seg, table = _paged_case(dtype, nq, nkv, d, 16, lens, window)
    out = torch.empty_like(q)
    args = (kv, pos, seg, table, nq, nkv, d, d ** -0.5, window)
    ops().attn_paged_simt(q, out, *args)
    for t in range(0, q.shape[0], 5):
        one = torch.zeros_like(q)
        ops().attn_paged_simt(q, one, *args, rows=torch.tensor([t], dtype=torch.int32, device=DEV))
        assert torch.equal(one[t], out[t]), t


STREAM, TILE, DENSE, ROWS = range(4)


# each kernel at its edges: tiles of 64 x 64 that end inside rows and columns, one and several of K's tiles; fewer
# columns than a block's, of every number of them that repeats differently; K in pieces of 8 with many tiles
@pytest.mark.parametrize("at,wt,ct", GEMM_TYPES)
@pytest.mark.parametrize("M,N,K,route", [
    (64, 3000, 32, DENSE), (65, 3009, 64, DENSE), (2000, 200, 96, DENSE), (2048, 256, 512, DENSE),
    (40, 1, 64, STREAM), (33, 3, 136, STREAM), (50, 20, 64, STREAM), (9, 31, 264, STREAM), (70, 33, 64, STREAM),
    (1000, 2000, 104, ROWS), (515, 4100, 1000, ROWS), (2048, 1024, 48, TILE)])
def test_dense_products_by_kernel_agree_bitwise(at, wt, ct, M, N, K, route):
    from freetoken_b200.csrc import build
    assert build.load("gemm_simt").ft_gemm_route(M, N, K, 1, 1, 0, 0, 1, int(at == "bfloat16"), int(wt == "float32")) == route
    a, w = rnd(M, K, dtype=DT[at], seed=1), rnd(N, K, dtype=DT[wt], seed=2, scale=0.1)
    got, want = (torch.full((M, N), float("nan"), dtype=DT[ct], device=DEV) for _ in range(2))
    ops().gemm_rows(a, w, got)
    ops().gemm_rows(_misaligned(a), w, want)
    assert torch.equal(got, want)
