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


# channels, tokens, segments, taps, two channels a thread: runs of eight tokens a thread (0: a thread a token)
@pytest.mark.parametrize("C,T,S,taps,pairs,groups", [
    (512, 1023, 1, 4, 1, 0), (512, 1024, 1, 4, 1, 1), (2304, 1500, 1, 4, 1, 1), (2304, 2048, 1, 4, 1, 2),
    (6144, 1024, 1, 4, 1, 2), (6144, 1024, 17, 4, 1, 1),                       # many segments: a window anew at each
    (6144, 4096, 1, 3, 1, 1), (1024, 4096, 1, 4, 0, 1), (2304, 2048, 1, 3, 0, 4), (2304, 2048, 64, 3, 0, 1)])
def test_runs_of_a_long_convolution(C, T, S, taps, pairs, groups):
    assert build.load("recurrent").ft_conv_groups(C, T, S, taps, pairs) == groups
