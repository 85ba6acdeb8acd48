"""Which kernel a launch takes, where two of equal results were measured against each other: lines of the rules on
the host, without a GPU."""

import pytest

from freetoken_b200.csrc import build


# T rows of S requests, blocks a token, tokens that fit a block, starts known
@pytest.mark.parametrize("T,S,rest,fit,known,tokens", [
    (64, 64, 8, 8, 1, 1), (64, 64, 16, 8, 0, 1),      # single tokens: nothing to share
    (512, 1, 16, 8, 0, 8), (512, 1, 16, 8, 1, 8),     # one prompt
    (287, 32, 16, 8, 1, 8), (287, 32, 16, 8, 0, 1),   # a prompt beside single tokens
    (18, 1, 16, 8, 1, 1), (19, 1, 16, 8, 1, 8)])      # SMs without a block
def test_tokens_that_share_an_attention_block(T, S, rest, fit, known, tokens):
    assert build.load("attention_simt").ft_attn_tokens_per_block(T, S, rest, fit, known) == tokens
