"""Products of few tokens whose warps read eight chunks of 32 k a round, beside the launch that reads two."""

import pytest
import torch

from test_kernels_gpu import DEV, DT, TOL, ops, rnd

pytestmark = pytest.mark.gpu


# 4, 8 and 16 warps a block; a warp's chunks: 5 (the first that takes eight a round), 8, 9 (a round of one), a last
# warp with fewer or none; K that ends inside a chunk; weight rows that end inside a tile
@pytest.mark.parametrize("ct", ["bfloat16", "float32"])
@pytest.mark.parametrize("M,N,K", [(1, 40, 544), (3, 33, 552), (8, 16, 1024), (9, 50, 1160), (5, 100, 2056),
                                   (8, 1000, 2048), (7, 24, 4104), (2, 64, 4616), (1, 6200, 1504)])
def test_eight_chunks_a_round(ct, M, N, K):
    o = ops()
    a, w = (rnd(n, K, dtype=torch.bfloat16, seed=s, scale=x) for n, s, x in ((M, 1, 1.0), (N, 2, 0.1)))
    c, two = (torch.empty(M, N, dtype=DT[ct], device=DEV) for _ in range(2))
    o.skinny_gemm(a, w, c, rows_per_pass=8)
    o.skinny_gemm(a, w, two, rows_per_pass=16)
    assert torch.equal(c, two)                   # the same products in the same order
    want = a.float() @ w.float().t()
    assert torch.allclose(c.float(), want, atol=TOL[ct]["atol"] * 3, rtol=TOL[ct]["rtol"])


# experts of rows longer than 2,048 values: groups without a row, of one, of more than a pass
@pytest.mark.parametrize("ct", ["bfloat16", "float32"])
@pytest.mark.parametrize("rows,N,K", [([1, 0, 2], 40, 2056), ([9, 1, 0, 3], 33, 2688), ([0, 8], 100, 4736), ([3] * 6, 1600, 2312)])
def test_eight_chunks_a_round_of_experts(ct, rows, N, K):
    o, E, M = ops(), len(rows), sum(rows)
    a = rnd(M, K, dtype=torch.bfloat16, seed=1)
    w = rnd(E, N, K, dtype=torch.bfloat16, seed=2, scale=0.1)
    offsets = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device=DEV)
    c, two = (torch.empty(M, N, dtype=DT[ct], device=DEV) for _ in range(2))
    o.skinny_gemm(a, w, c, group_offsets=offsets, rows_per_pass=8)
    o.skinny_gemm(a, w, two, group_offsets=offsets, rows_per_pass=16)
    assert torch.equal(c, two)
    want = torch.cat([a[offsets[e]:offsets[e + 1]].float() @ w[e].float().t() for e in range(E)])
    assert torch.allclose(c.float(), want, atol=TOL[ct]["atol"] * 3, rtol=TOL[ct]["rtol"])
