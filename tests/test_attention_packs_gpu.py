"""The CUDA-core attention over several requests: a block's tokens are one request's, wherever the requests begin."""

import pytest
import torch

from test_kernels_gpu import DEV, _paged_case, ops

pytestmark = pytest.mark.gpu


def plain(q, kv, pos, seg, table, nq, nkv, d, window):
    out = torch.empty(q.shape[0], nq, d, device=DEV)
    for s in range(table.shape[0]):
        rows = (seg == s).nonzero().flatten()
        k, v = (kv[i, table[s].long()].float().transpose(1, 2).reshape(-1, nkv, d).repeat_interleave(nq // nkv, 1) for i in (0, 1))
        scores = torch.einsum("thd,jhd->htj", q[rows].float().view(-1, nq, d), k) * d ** -0.5
        far = pos[rows, None] - torch.arange(k.shape[0], device=DEV)
        hidden = (far < 0) | (far >= (window or 1 << 30))
        out[rows] = torch.einsum("htj,jhd->thd", torch.softmax(scores.masked_fill(hidden, float("-inf")), -1), v)
    return out.view(q.shape)


# requests that begin inside a block's tokens, at its first one and at the last; single tokens between portions; eight,
# four, two tokens a block, three heads that leave warps without a row; one request; windows
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nq,nkv,d,window", [(16, 16, 16, None), (8, 4, 40, None), (16, 4, 64, 21), (12, 4, 32, None), (40, 40, 8, 5)])
@pytest.mark.parametrize("lens", [[(0, 75), (40, 1), (7, 1), (3, 50)], [(5, 8), (0, 7), (30, 1), (9, 16), (2, 33)],
                                  [(70, 1)] * 40, [(0, 130)], [(20, 3)] * 21])
def test_blocks_of_one_request(dtype, nq, nkv, d, window, lens):
    q, kv, pos, seg, table = _paged_case(dtype, nq, nkv, d, 16, lens, window)
    starts = [0]
    for _, n in lens:
        starts.append(starts[-1] + n)
    starts = torch.tensor(starts, dtype=torch.int32, device=DEV)
    args = (kv, pos, seg, table, nq, nkv, d, d ** -0.5, window)
    out, apart, alone = (torch.full_like(q, float("nan")) for _ in range(3))
    ops().attn_paged_simt(q, out, *args, seg_q_start=starts)
    ops().attn_paged_simt(q, apart, *args)
    assert torch.equal(out, apart)
    for t in range(0, q.shape[0], 7):
        ops().attn_paged_simt(q, alone, *args, rows=torch.tensor([t], dtype=torch.int32, device=DEV))
        assert torch.equal(alone[t], out[t]), t
    want = plain(q, kv, pos, seg, table, nq, nkv, d, window)
    tol = 2e-5 if dtype == "float32" else 2e-2            # as the other attention tests: float32 sums, bfloat16 results
    assert torch.allclose(out.float(), want, atol=tol, rtol=tol)
