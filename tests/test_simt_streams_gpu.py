"""The weight-streaming CUDA-core product whose warps beyond the rows' only fetch: the same bits as the kernel without pieces of
16 bytes."""

import pytest
import torch

from test_kernels_gpu import DEV, DT, GEMM_TYPES, ops, rnd
from test_simt_paths_gpu import _misaligned

pytestmark = pytest.mark.gpu


# K of fewer, as many and more pieces of 128 than the four stages, ending inside one; every number of multiplying warps
@pytest.mark.parametrize("at,wt,ct", GEMM_TYPES)
@pytest.mark.parametrize("M,N,K", [(1, 70, 8), (2, 65, 384), (3, 33, 520), (4, 100, 512), (7, 31, 648), (16, 64, 1288), (31, 40, 1024)])
def test_streams_of_few_rows_agree_bitwise(at, wt, ct, M, N, K):
    a, w = rnd(M, K, dtype=DT[at], seed=1), rnd(N, K, dtype=DT[wt], seed=2, scale=0.1)
    got, want = (torch.full((M, N), float("nan"), dtype=DT[ct], device=DEV) for _ in range(2))
    ops().gemm_rows(a, w, got)
    ops().gemm_rows(_misaligned(a), w, want)
    assert torch.equal(got, want)
