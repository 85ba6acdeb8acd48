"""Products in bfloat16 of rows that lie in more than two dimensions go to the library as before."""

import torch

from freetoken_b200.parts.linear import linear


def test_rows_in_three_dimensions():
    g = torch.Generator().manual_seed(1)
    x, w = (torch.randn(*s, generator=g).bfloat16() for s in ((5, 40, 24), (16, 24)))
    out = torch.empty(5, 40, 16, dtype=torch.bfloat16)
    assert linear(x, w, out) is out
    # one rounding to bfloat16 (2^-9 of the value) of a float32 sum of 24 products
    assert torch.allclose(out.double(), x.double() @ w.double().t(), rtol=2 ** -8, atol=1e-5)
