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


DELTA, CHANNEL, RETENTION, SSD = range(4)


# kind, float32, heads, value size, key size, segments, tokens, longest (0: not known): sixteen lanes a column or not
@pytest.mark.parametrize("kind,f32,H,P,D,S,T,longest,several", [
    (DELTA, 0, 16, 128, 128, 32, 32, 1, 0), (DELTA, 0, 16, 128, 128, 32, 33, 2, 0),    # single tokens, one of two
    (DELTA, 0, 16, 128, 128, 1, 2048, 2048, 1), (DELTA, 0, 16, 128, 128, 4, 12, 3, 1), (CHANNEL, 0, 4, 64, 64, 1, 2, 2, 0),
    (DELTA, 0, 16, 128, 128, 32, 64, 2, 0), (DELTA, 0, 16, 128, 128, 32, 512, 16, 1),  # a full chip, even segments
    (DELTA, 0, 16, 128, 128, 64, 263, 200, 1), (DELTA, 0, 16, 128, 128, 64, 263, 0, 0),       # a long one beside single tokens
    (DELTA, 1, 16, 128, 128, 32, 512, 16, 0), (DELTA, 1, 16, 128, 128, 32, 1024, 32, 1),      # two columns a lane
    (SSD, 1, 32, 64, 128, 32, 1024, 32, 0), (RETENTION, 1, 16, 128, 128, 32, 1024, 32, 1),
    (DELTA, 0, 8, 256, 256, 1, 16, 16, 0), (DELTA, 0, 8, 256, 256, 1, 512, 512, 1),    # one column a lane
    (DELTA, 0, 8, 256, 256, 32, 512, 16, 0), (CHANNEL, 0, 8, 256, 256, 4, 4096, 1335, 0), (RETENTION, 0, 8, 256, 256, 8, 307, 300, 1),
    (SSD, 0, 8, 256, 256, 8, 135, 128, 1), (SSD, 0, 8, 256, 256, 32, 159, 128, 0)])
def test_lanes_of_a_scan(kind, f32, H, P, D, S, T, longest, several):
    assert build.load("recurrent").ft_scan_several(kind, f32, H, P, D, S, T, longest) == several


STREAM, TILE, DENSE, ROWS = range(4)


# rows, columns, K, groups, batch, grouped, gated, plain, bfloat16 rows, float32 weights
@pytest.mark.parametrize("M,N,K,G,batch,grouped,glu,plain,b16,w32,route", [
    (1, 4096, 2048, 1, 1, 0, 0, 1, 0, 0, STREAM), (64, 2048, 2048, 1, 1, 0, 0, 1, 0, 0, STREAM),
    (4096, 32, 512, 1, 1, 0, 0, 1, 0, 0, STREAM), (342, 8, 2048, 1, 1, 0, 0, 1, 0, 0, STREAM),
    (1024, 4096, 2048, 1, 1, 0, 0, 1, 0, 0, TILE), (342, 3072, 2048, 1, 1, 0, 0, 1, 0, 0, TILE),
    (2048, 256, 512, 1, 1, 0, 0, 1, 0, 0, DENSE), (64, 512, 128, 1, 16, 0, 0, 1, 0, 0, DENSE),
    (700, 512, 1024, 1, 1, 0, 0, 1, 0, 1, DENSE), (2048, 256, 512, 1, 1, 0, 0, 0, 0, 0, TILE),
    (2048, 4096, 1000, 1, 1, 0, 0, 1, 0, 0, ROWS), (512, 2048, 2056, 1, 1, 0, 0, 1, 0, 1, ROWS),
    (64, 1024, 1000, 1, 1, 0, 0, 1, 0, 0, STREAM),
    (2000, 1024, 2048, 8, 1, 1, 1, 0, 0, 0, TILE), (2000, 1024, 1000, 8, 1, 1, 1, 0, 0, 1, ROWS),
    (8, 512, 1024, 64, 1, 1, 1, 0, 0, 0, STREAM),
    (1, 65535 * 32, 8, 1, 1, 0, 0, 1, 0, 0, STREAM), (1, 65535 * 32 + 1, 8, 1, 1, 0, 0, 1, 0, 0, ROWS),     # a grid's most blocks
    (64, 65535 * 32 + 1, 8, 1, 1, 0, 0, 1, 0, 0, ROWS), (8, 65535 * 32 + 1, 16, 8, 1, 1, 1, 0, 0, 0, ROWS)])
def test_kernel_of_a_float32_product(M, N, K, G, batch, grouped, glu, plain, b16, w32, route):
    assert build.load("gemm_simt").ft_gemm_route(M, N, K, G, batch, grouped, glu, plain, b16, w32) == route


# float32, width, partial rows
@pytest.mark.parametrize("f32,H,k,early", [(0, 2048, 4, 1), (0, 2048, 5, 0), (0, 4096, 1, 1), (0, 4096, 2, 1), (0, 4096, 3, 0),
                                           (1, 4096, 8, 1), (0, 512, 8, 0)])
def test_early_fetches_of_an_output_norm(f32, H, k, early):
    assert build.load("rowwise").ft_norm_add_fetches_early(f32, H, k) == early


@pytest.mark.parametrize("f32,S,H,k,early", [(0, 4, 4096, 4, 1), (0, 2, 3000, 8, 0), (0, 4, 512, 8, 0), (0, 4, 2048, 8, 1),
                                             (0, 2, 8192, 8, 1), (1, 4, 6144, 8, 0), (1, 4, 4096, 8, 1), (1, 2, 8192, 8, 1)])
def test_early_fetches_of_a_stream_norm(f32, S, H, k, early):
    assert build.load("rowwise").ft_hyper_fetches_early(f32, S, H, k) == early


# blocks, warps a block, K, experts
@pytest.mark.parametrize("blocks,ks,K,experts,eight", [
    (384, 4, 4096, 0, 1), (592, 4, 4096, 0, 1), (593, 4, 4096, 0, 0), (1036, 4, 4096, 0, 0), (1037, 4, 4096, 0, 1),
    (296, 8, 4096, 0, 1), (297, 8, 4096, 0, 0), (445, 8, 4096, 0, 1), (128, 4, 512, 0, 0),
    (512, 4, 2304, 1, 1), (640, 4, 2304, 1, 0), (4096, 4, 2304, 1, 0), (4096, 4, 2688, 1, 1), (1024, 4, 4736, 1, 0)])
def test_chunks_a_round_of_a_weight_streaming_product(blocks, ks, K, experts, eight):
    assert build.load("skinny_gemm").ft_skinny_eight_chunks(blocks, ks, K, experts) == eight


@pytest.mark.parametrize("T,H,one", [(1, 1024, 0), (1, 1028, 1), (8, 2048, 1), (9, 2048, 0), (64, 2048, 0), (1, 2052, 1), (64, 2052, 1),
                                     (64, 4096, 1), (65, 4096, 0), (1, 4100, 0)])
def test_rows_of_one_piece_a_thread(T, H, one):
    assert build.load("rowwise").ft_norm_add_one_piece(T, H) == one


@pytest.mark.parametrize("sms", [74, 132, 148, 160])
def test_rounds_are_those_of_the_device_that_runs_them(sms):
    """Both lines of the rule lie at a whole house of blocks, whatever number of multiprocessors that is."""
    rule = build.load("skinny_gemm").ft_skinny_eight_chunks_on
    for ks, eight, four in ((4, 4, 7), (8, 2, 3), (16, 1, 1)):
        assert rule(sms, sms * eight, ks, 4096, 0) == 1
        assert rule(sms, sms * eight + 1, ks, 4096, 0) == int(eight == four)
        assert rule(sms, sms * four + 1, ks, 4096, 0) == 1
    assert rule(sms, 2 * sms, 4, 512, 0) == 0


def test_nothing_that_a_device_is_asked_is_kept_for_all_devices():
    """The streaming product's launch rule holds no device's answer in a static of its own, and no number of multiprocessors."""
    import os
    with open(os.path.join(build.HERE, "skinny_gemm.cu")) as f:
        code = "\n".join(line.split("//")[0] for line in f)
    assert "static const int" not in code and code.count("148") == 1            # the exported rule of the tests above


@pytest.mark.parametrize("H,k,two", [(2048, 1, 1), (2048, 2, 0), (2052, 2, 1), (3072, 3, 1), (3072, 4, 0), (8192, 8, 0), (512, 1, 1)])
def test_pieces_of_a_norm_of_few_tokens(H, k, two):
    assert build.load("elementwise").ft_rmsnorm_two_pieces(H, k) == two


# both forms of few tokens and the form of many: a token's row has the same bits
@pytest.mark.gpu
@pytest.mark.parametrize("H", [128, 2048, 2052, 3072, 8192])
@pytest.mark.parametrize("k", [0, 1, 2, 3, 4, 5, 9])
def test_norms_of_few_and_many_tokens_agree(H, k):
    import torch
    from test_kernels_gpu import DEV, ops, rnd
    delta = rnd(65, max(k, 1), H, dtype=torch.bfloat16, seed=1) if k else None
    residual, weight = rnd(65, H, seed=2), rnd(H, seed=3)
    got = []
    for T in (65, 64, 1):
        r, out = residual[:T].clone(), torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
        ops().rmsnorm(delta[:T].contiguous() if k else None, r, weight, out, 1e-5, False)
        got.append((r, out))
    for r, out in got[1:]:
        assert torch.equal(r, got[0][0][:len(r)]) and torch.equal(out, got[0][1][:len(r)])
