"""The scans of the recurrent mixers, the short convolution and the latent store: a launch of several tokens takes
other kernels than a launch of one token a segment, and gives the same bits."""

import pytest
import torch

from test_kernels_gpu import DEV, DT, ops, rnd

pytestmark = pytest.mark.gpu

# heads, value size, key size, tokens a segment, groups: remainders of chunks of 8, of lanes' columns and rows;
# the last two fill the chip (four columns a lane)
SIZES = [(4, 10, 12, [9], 2), (2, 36, 40, [3, 1, 17], 1), (4, 64, 64, [16, 7], 2), (3, 28, 20, [33], 3),
         (2, 130, 200, [12, 5], 1), (1, 7, 129, [8], 1), (8, 16, 32, [1, 2, 25], 4), (2, 8, 256, [10], 2),
         (32, 64, 96, [11, 8, 3], 1), (40, 130, 33, [9], 40)]


def _segments(lens):
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    return (torch.arange(len(lens), dtype=torch.int32, device=DEV) + 1,
            torch.tensor(starts, dtype=torch.int32, device=DEV))


def _token_by_token(lens, launch):
    """``launch(token rows, slots, starts)`` for the first token of every segment, then the second ..."""
    starts = [sum(lens[:i]) for i in range(len(lens))]
    for t in range(max(lens)):
        live = [i for i, n in enumerate(lens) if t < n]
        rows = torch.tensor([starts[i] + t for i in live], device=DEV)
        launch(rows, torch.tensor([i + 1 for i in live], dtype=torch.int32, device=DEV),
               torch.arange(len(live) + 1, dtype=torch.int32, device=DEV), t)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("kind", ["delta", "channel_delta", "retention", "ssd"])
@pytest.mark.parametrize("H,P,D,lens,G", SIZES)
def test_scans_agree_bitwise(dtype, kind, H, P, D, lens, G):
    T, dt, o = sum(lens), DT[dtype], ops()
    slot, starts = _segments(lens)
    a_log, bias = rnd(H, seed=3, scale=0.5) - 1, rnd(H, seed=4, scale=0.5) - 1
    gates = rnd(T, 2 * H, dtype=dt, seed=2)
    first = rnd(len(lens) + 2, H * D * P + 5, seed=5, scale=0.1)
    if kind == "ssd":
        x, skip = rnd(T, H * P + 2 * G * D, dtype=dt, seed=1), rnd(H, seed=6)
        call = lambda state, y, rows, s, q, t: o.ssd_scan(x[rows], gates[rows][:, :H], bias, a_log, skip, state, y, s, q,
                                                          H, P, D, G)
    elif kind == "retention":
        x, decay = rnd(T, 2 * H * D + H * P, dtype=dt, seed=1), torch.linspace(0.9, 0.999, H, device=DEV)
        rot = 2 * (D // 4)
        turn = rnd(64, rot, seed=7) if rot else None
        call = lambda state, y, rows, s, q, t: o.retention_scan(x[rows], decay, turn, torch.full_like(s, t), state, y, s,
                                                                q, H, D, P, D ** -0.5)
    else:
        x = rnd(T, 2 * G * D + H * P, dtype=dt, seed=1)
        per_channel = rnd(T, H * D, seed=8), rnd(H * D, seed=9, scale=0.5) - 1
        if kind == "delta":
            call = lambda state, y, rows, s, q, t: o.delta_scan(
                x[rows], gates[rows][:, :H], gates[rows][:, H:], bias, a_log, state, y, s, q, H, G, D, P, 1e-6, D ** -0.5)
        else:
            call = lambda state, y, rows, s, q, t: o.channel_delta_scan(
                x[rows], gates[rows][:, :H], per_channel[0][rows], per_channel[1], a_log, state, y, s, q, H, G, D, P, 1e-6,
                D ** -0.5)
    whole, y = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)
    call(whole, y, torch.arange(T, device=DEV), slot, starts, 0)
    steps, want = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)

    def launch(rows, s, q, t):
        out = torch.empty(rows.numel(), H * P, device=DEV)
        call(steps, out, rows, s, q, t)
        want[rows] = out
    _token_by_token(lens, launch)
    assert torch.equal(y, want) and torch.equal(whole, steps)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("C,taps,lens,act", [(6, 4, [5, 1, 9], True), (130, 2, [3], False), (7, 8, [12, 2], True),
                                             (64, 1, [4], True), (33, 9, [3, 12], True)])
def test_convolutions_agree_bitwise(dtype, C, taps, lens, act):
    T, dt = sum(lens), DT[dtype]
    slot, starts = _segments(lens)
    seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32).to(DEV)
    x, w, b = rnd(T, C + 2, dtype=dt, seed=1)[:, :C], rnd(C, taps, seed=2), rnd(C, seed=3)
    first = rnd(len(lens) + 2, max(1, (taps - 1) * C), seed=4)
    whole, y = first.clone(), torch.empty(T, C, dtype=dt, device=DEV)
    ops().conv_silu(x, y, w, b, whole, seg, slot, starts, activation=act)
    steps, want = first.clone(), torch.empty(T, C, dtype=dt, device=DEV)

    def launch(rows, s, q, t):
        out = torch.empty(rows.numel(), C, dtype=dt, device=DEV)
        ops().conv_silu(x[rows], out, w, b, steps, torch.arange(rows.numel(), dtype=torch.int32, device=DEV), s, q,
                        activation=act)
        want[rows] = out
    _token_by_token(lens, launch)
    assert torch.equal(y, want) and torch.equal(whole, steps)


def test_convolution_of_as_many_tokens_as_segments_that_are_not_one_each():
    """Two tokens in one segment and none in the other."""
    x, w = rnd(2, 10, seed=1), rnd(10, 3, seed=2)
    first = rnd(3, 20, seed=4)
    out = []
    for starts in ([0, 0, 2], [0, 2]):
        state, y = first.clone(), torch.empty(2, 10, device=DEV)
        S = len(starts) - 1
        slot = torch.tensor([2, 1][-S:], dtype=torch.int32, device=DEV)
        ops().conv_silu(x, y, w, None, state, torch.full((2,), S - 1, dtype=torch.int32, device=DEV), slot,
                        torch.tensor(starts, dtype=torch.int32, device=DEV))
        out.append((y, state))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("heads,dq,rank,rot,interleaved", [(32, 16, 40, 64, False), (3, 8, 24, 6, True), (20, 8, 16, 32, True)])
def test_latent_rows_of_few_and_many_tokens_agree_bitwise(dtype, heads, dq, rank, rot, interleaved):
    T, dt, P = 70, DT[dtype], 16
    down, q = rnd(T, rank + rot, dtype=dt, seed=1), rnd(T, heads * (dq + rot), dtype=dt, seed=2)
    weight, turn = rnd(rank, seed=3), rnd(T, rot, seed=4)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seg = torch.zeros(T, dtype=torch.int32, device=DEV)
    table = torch.arange(1, 6, dtype=torch.int32, device=DEV).view(1, 5)
    results = []
    for rows in (T, 9):
        pages = torch.zeros(6, 1, P, rank + rot, dtype=dt, device=DEV)
        q_abs = torch.zeros(T, heads, rank + rot, dtype=dt, device=DEV)
        turned = q.clone()
        for a in range(0, T, rows):
            b = min(T, a + rows)
            ops().latent_store(down[a:b], turned[a:b], q_abs[a:b], pages, weight, turn, pos[a:b], seg[a:b], table,
                               heads=heads, q_dim=dq, rank=rank, rot=rot, interleaved=interleaved, eps=1e-6, turn_q=True)
        results.append((pages, q_abs, turned))
    assert all(torch.equal(x, y) for x, y in zip(*results))


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("H,P,D,lens", [(2, 36, 40, [3, 1, 17]), (1, 64, 64, [8, 9]), (3, 30, 20, [11]),
                                        (40, 41, 41, [9] * 9), (20, 70, 100, [3, 8] * 5)])    # two columns a lane
def test_time_mixing_agrees_bitwise(dtype, H, P, D, lens):
    T, dt = sum(lens), DT[dtype]
    slot, starts = _segments(lens)
    r, k, v = rnd(T, H * D, dtype=dt, seed=1), rnd(T, H * D, dtype=dt, seed=2), rnd(T, H * P, dtype=dt, seed=3)
    decay, w0, u = rnd(T, H * D, seed=4), rnd(H * D, seed=5), rnd(H, D, seed=6)
    if P != D:                                   # one row stride
        wide = max(P, D) * H
        r, k, v = (torch.cat([x, torch.zeros(T, wide - x.shape[1], dtype=dt, device=DEV)], 1) for x in (r, k, v))
    call = lambda state, y, rows, s, q: ops().time_mixing_scan(
        r[rows][:, :H * D], k[rows][:, :H * D], v[rows][:, :H * P], decay[rows], w0, u, state, y, s, q, H, P, D)
    first = rnd(len(lens) + 2, H * D * P, seed=7, scale=0.1)
    whole, y = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)
    call(whole, y, torch.arange(T, device=DEV), slot, starts)
    steps, want = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)

    def launch(rows, s, q, t):
        out = torch.empty(rows.numel(), H * P, device=DEV)
        call(steps, out, rows, s, q)
        want[rows] = out
    _token_by_token(lens, launch)
    assert torch.equal(y, want) and torch.equal(whole, steps)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("C,taps,lens", [(258, 4, [1000, 1, 31]), (70, 3, [1024]), (33, 4, [500, 700]), (8, 8, [7] * 150)])
def test_long_convolutions_agree_bitwise(dtype, C, taps, lens):
    """1,024 tokens and more take runs of 32 a thread; here against the same segments a few at a time."""
    dt = DT[dtype]
    w, b = rnd(C, taps, seed=2), rnd(C, seed=3)
    slot, starts = _segments(lens)
    seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32).to(DEV)
    x = rnd(sum(lens), C, dtype=dt, seed=1)
    first = rnd(len(lens) + 2, max(1, (taps - 1) * C), seed=4)
    whole, y = first.clone(), torch.empty_like(x)
    ops().conv_silu(x, y, w, b, whole, seg, slot, starts)
    parts, want, at = first.clone(), torch.empty_like(x), 0
    for i, n in enumerate(lens):
        for a in range(0, n, 600):
            m = min(600, n - a)
            ops().conv_silu(x[at + a:at + a + m], want[at + a:at + a + m], w, b, parts, torch.zeros(m, dtype=torch.int32, device=DEV),
                            slot[i:i + 1], torch.tensor([0, m], dtype=torch.int32, device=DEV))
        at += n
    assert torch.equal(y, want) and torch.equal(whole, parts)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("S,H,k", [(4, 256, 1), (4, 2052, 2), (2, 4100, 5), (1, 1024, 8), (3, 64, 0), (4, 6144, 2), (4, 8192, 5)])
def test_stream_norms_of_few_and_many_tokens_agree_bitwise(dtype, S, H, k):
    T, dt, o = 70, DT[dtype], ops()
    streams, branch = rnd(T, S, H, seed=1), rnd(T, max(k, 1), H, dtype=dt, seed=2)
    mix, out, read = rnd(S, S, seed=3), rnd(S, seed=4), rnd(S, seed=5)
    weight, bias = rnd(H, seed=6), rnd(H, seed=7)
    results = []
    for rows in (T, 9):
        x, y = streams.clone(), torch.empty(T, H, dtype=dt, device=DEV)
        for a in range(0, T, rows):
            b = min(T, a + rows)
            o.hyper_norm(x[a:b], branch[a:b] if k else None, mix if k else None, out if k else None, read, weight, bias, 1e-5,
                         True, y[a:b])
        results.append((x, y))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("H,k", [(512, 1), (2048, 3), (4096, 2), (6000, 1), (30, 2)])
def test_branch_norms_of_few_and_many_tokens_agree_bitwise(dtype, H, k):
    T, dt, o = 70, DT[dtype], ops()
    residual, branch = rnd(T, H, seed=1), rnd(T, k, H, dtype=dt, seed=2)
    w, w2 = rnd(H, seed=3), rnd(H, seed=4)
    results = []
    for rows in (T, 9):
        x, y = residual.clone(), torch.empty(T, H, dtype=dt, device=DEV)
        for a in range(0, T, rows):
            b = min(T, a + rows)
            o.norm_add(branch[a:b], x[a:b], w, 1e-5, True, 0.7, next_weight=w2, next_eps=1e-4, next_out=y[a:b])
        results.append((x, y))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


# a thread keeps one, two and four pieces of the row, the last with and without a remainder; fewer and more slots than
# are fetched at a time
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("H,k,m", [(1000, 1, 1), (2048, 5, 2), (2040, 2, 3), (4096, 3, 1), (3000, 9, 2), (8192, 2, 2)])
def test_routed_branches_of_few_and_many_tokens_agree_bitwise(dtype, H, k, m):
    T, dt, o = 70, DT[dtype], ops()
    residual, extra, source = rnd(T, H, seed=1), rnd(T, H, dtype=dt, seed=2), rnd(T, H, dtype=dt, seed=3)
    rows, beside = rnd(T, k, H, dtype=dt, seed=4), rnd(T, m, H, dtype=dt, seed=5)
    ids = (torch.arange(T * k, device=DEV, dtype=torch.int32) * 5 % 7).view(T, k)      # ids of 4 and more hand back
    rows[ids >= 4] = float("nan")                                                       # and are not read
    weights, gate, scale = rnd(T, k, seed=6), rnd(T, seed=7), rnd(m, seed=8)
    w, w2 = rnd(H, seed=9), rnd(H, seed=10)
    results = []
    for step in (T, 9):
        x, y, u = residual.clone(), torch.empty(T, H, dtype=dt, device=DEV), torch.empty(T, H, dtype=dt, device=DEV)
        for a in range(0, T, step):
            c = slice(a, min(T, a + step))
            branch = o.RoutedRows(rows[c], ids[c], weights[c], 4, source[c], extra[c], None, gate[c], beside[c], scale)
            o.norm_add(branch, x[c], w, 1e-5, True, 0.7, next_weight=w2, next_eps=1e-4, next_out=y[c])
            o.join_layer_norm(branch, x[c], w, 1e-5, u[c])
        results.append((x, y, u))
    assert all(torch.isfinite(r).all() and torch.equal(r, other) for r, other in zip(*results))


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("H,P,D,lens", [(40, 130, 128, [29, 16, 8]), (4, 30, 64, [61]), (6, 70, 200, [13, 24])])
def test_delta_rule_repeats_itself(dtype, per_channel, H, P, D, lens):
    """A token's write is read out later in its chunk by other lanes than computed it: the same bits in every launch."""
    T, dt, o = sum(lens), DT[dtype], ops()
    slot, starts = _segments(lens)
    a_log, bias = rnd(H, seed=3, scale=0.5) - 1, rnd(H, seed=4, scale=0.5) - 1
    gates, first = rnd(T, 2 * H, dtype=dt, seed=2), rnd(len(lens) + 2, H * D * P, seed=5, scale=0.1)
    x, decay, channel_bias = rnd(T, 2 * H * D + H * P, dtype=dt, seed=1), rnd(T, H * D, seed=8), rnd(H * D, seed=9, scale=0.5) - 1
    results = []
    for _ in range(12):
        state, y = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)
        if per_channel:
            o.channel_delta_scan(x, gates[:, :H], decay, channel_bias, a_log, state, y, slot, starts, H, H, D, P, 1e-6, D ** -0.5)
        else:
            o.delta_scan(x, gates[:, :H], gates[:, H:], bias, a_log, state, y, slot, starts, H, H, D, P, 1e-6, D ** -0.5)
        results.append((state, y))
    assert all(torch.equal(a, b) for r in results[1:] for a, b in zip(results[0], r))


# two runs a thread (bfloat16 pairs, four taps), four (single channels), and one beside: a request's edges inside runs
@pytest.mark.parametrize("dtype,C,taps,lens", [("bfloat16", 2006, 4, [1500, 20, 541]), ("bfloat16", 2311, 4, [2050]),
                                               ("float32", 2310, 3, [1201, 850]), ("bfloat16", 2006, 3, [1500, 20, 541]),
                                               ("bfloat16", 512, 4, [7, 1022])])
def test_long_convolutions_of_several_runs(dtype, C, taps, lens):
    test_long_convolutions_agree_bitwise(dtype, C, taps, lens)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("kind", ["delta", "channel_delta", "retention", "ssd"])
@pytest.mark.parametrize("H,P,D,lens", [(2, 130, 200, [12, 5]), (1, 7, 129, [8]), (2, 8, 256, [10]), (16, 66, 256, [9, 3] * 5),
                                        (40, 64, 64, [3, 1] * 8)])
def test_scans_agree_whichever_lanes_they_take(dtype, kind, H, P, D, lens):
    """The same launch told that its longest segment has one token, and so many that it is worth a chain."""
    T, dt, o = sum(lens), DT[dtype], ops()
    slot, starts = _segments(lens)
    a_log, bias = rnd(H, seed=3, scale=0.5) - 1, rnd(H, seed=4, scale=0.5) - 1
    gates, first = rnd(T, 2 * H, dtype=dt, seed=2), rnd(len(lens) + 2, H * D * P, seed=5, scale=0.1)
    results, kinds = [], ["delta", "channel_delta", "retention", "ssd"]
    for longest in (1, 1 << 20):
        state, y = first.clone(), torch.full((T, H * P), float("nan"), device=DEV)
        if kind == "ssd":
            o.ssd_scan(rnd(T, H * P + 2 * D, dtype=dt, seed=1), gates[:, :H], bias, a_log, rnd(H, seed=6), state, y, slot, starts, H, P,
                       D, 1, longest)
        elif kind == "retention":
            o.retention_scan(rnd(T, 2 * H * D + H * P, dtype=dt, seed=1), torch.linspace(0.9, 0.999, H, device=DEV), rnd(64, 2 * (D // 4),
                             seed=7), torch.arange(len(lens), dtype=torch.int32, device=DEV), state, y, slot, starts, H, D, P, D ** -0.5,
                             longest)
        elif kind == "delta":
            o.delta_scan(rnd(T, 2 * H * D + H * P, dtype=dt, seed=1), gates[:, :H], gates[:, H:], bias, a_log, state, y, slot, starts, H,
                         H, D, P, 1e-6, D ** -0.5, longest)
        else:
            o.channel_delta_scan(rnd(T, 2 * H * D + H * P, dtype=dt, seed=1), gates[:, :H], rnd(T, H * D, seed=8), rnd(H * D, seed=9) - 1,
                                 a_log, state, y, slot, starts, H, H, D, P, 1e-6, D ** -0.5, longest)
        results.append((state, y))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    from freetoken_b200.csrc import build
    worth = D <= 128 or H * P * len(lens) > 8192 or kind in ("delta", "ssd")       # others of more than 128 rows stay
    for longest, took in ((1, False), (1 << 20, worth)):
        assert took == build.load("recurrent").ft_scan_several(kinds.index(kind), dtype == "float32", H, P, D, len(lens), T, longest)
