"""A product per head of few tokens in one launch, heads and tokens any distance apart."""

import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


# one pass and several, heads that end inside a tile, K that ends inside a chunk, the smallest of all
@pytest.mark.parametrize("T,H,K,N,gap", [(1, 1, 8, 1, 0), (1, 32, 128, 512, 64), (8, 4, 96, 40, 8), (9, 3, 136, 33, 0), (32, 16, 512, 128, 16),
                                         (17, 5, 64, 576, 24)])
def test_heads(T, H, K, N, gap):
    o = ops()
    wide = rnd(T, H * (K + gap) + 8, dtype=torch.bfloat16, seed=1)
    x = wide[:, 8:].unflatten(1, (H, K + gap))[:, :, :K]
    w = rnd(H, N, K, dtype=torch.bfloat16, seed=2, scale=K ** -0.5)
    room = torch.full((T, H, N + gap), 7.0, dtype=torch.bfloat16, device=DEV)
    out = room[:, :, gap:]
    assert o.skinny_heads_takes(x, w, out)
    o.skinny_heads(x, w, out)
    want = torch.einsum("thk,hnk->thn", x.float(), w.float())
    # one rounding of a value of size one
    assert torch.allclose(out.float(), want, atol=1e-3, rtol=5e-3)
    assert (room[:, :, :gap] == 7).all()


def test_what_is_not_taken():
    o = ops()
    w = rnd(2, 16, 24, dtype=torch.bfloat16)
    out = torch.empty(3, 2, 16, dtype=torch.bfloat16, device=DEV)
    for x in (rnd(3, 2, 25, dtype=torch.bfloat16)[:, :, 1:], rnd(3, 2, 24), rnd(3, 24, 2, dtype=torch.bfloat16).transpose(1, 2),
              rnd(3, 2, 28, dtype=torch.bfloat16)[:, :, :24]):
        assert not o.skinny_heads_takes(x, w, out)
        with pytest.raises(o.KernelError):
            o.skinny_heads(x, w, out)
