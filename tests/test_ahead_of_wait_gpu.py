"""What kernels fetch while the launch in front of them still runs, and the choice of experts by whole-warp reductions."""

import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


# a launch of one round, of less than one and of several rounds of blocks; experts without rows
@pytest.mark.parametrize("rows,N,K", [([1, 0, 3], 40, 264), ([8, 9, 0, 1], 96, 1536), ([1] * 64, 3072, 160)])
def test_lists_that_were_there_before(rows, N, K):
    o, G, M = ops(), len(rows), sum(rows)
    a, w = rnd(M, K, dtype=torch.bfloat16, seed=1), rnd(G * N, K, dtype=torch.bfloat16, seed=2, scale=0.1).view(G, N, K)
    offsets = i32([sum(rows[:g]) for g in range(G + 1)])
    busy = [g for g in range(G) if rows[g]]
    active = i32(busy + [0] * (G - len(busy)) + [len(busy)])
    scratch, one, two = (torch.zeros(M, N, dtype=torch.bfloat16, device=DEV) for _ in range(3))
    lists = dict(group_offsets=offsets, active=active, rows=M)
    o.skinny_gemm(a, w, one, **lists)
    for _ in range(20):                                    # right behind a launch that still runs
        o.skinny_gemm(a, w, scratch, **lists)
        o.skinny_gemm(scratch[:, :K] if N >= K else a, w, two, lists_ahead=True, **lists)
    o.skinny_gemm(scratch[:, :K] if N >= K else a, w, one, **lists)
    assert torch.equal(one, two)
    if N < K:
        want = torch.cat([a[s:s + n].float() @ w[g].float().t() for g, (s, n) in enumerate(zip(offsets.tolist(), rows))])
        assert torch.allclose(two.float(), want, atol=0.05, rtol=0.02)


# one token a segment: as many steps with the state fetched ahead of the wait as without, a projection in between
@pytest.mark.parametrize("kind", ["delta", "channel_delta", "retention", "ssd", "time_mixing", "conv"])
@pytest.mark.parametrize("S,H,P,D", [(1, 2, 64, 64), (5, 3, 40, 24), (9, 16, 128, 128)])
def test_states_fetched_ahead(kind, S, H, P, D):
    o = ops()
    inner, kd = H * P, H * D
    x = rnd(S, 4 * max(inner, kd), dtype=torch.bfloat16, seed=3)
    w = rnd(x.shape[1], x.shape[1], dtype=torch.bfloat16, seed=4, scale=x.shape[1] ** -0.5)
    made = {}                                              # nothing but the package's launches between two steps

    def f32(*shape, seed):
        if (shape, seed) not in made:
            made[shape, seed] = rnd(*shape, seed=seed, scale=0.3).sigmoid()
        return made[shape, seed]
    slots, starts, segs = i32(list(range(S))[::-1]), i32(list(range(S + 1))), i32(list(range(S)))
    results = []
    for ahead in (False, True):
        state = rnd(S, 3 * inner if kind == "conv" else inner * D, seed=5)
        row = x.clone()
        for _ in range(4):
            nxt = torch.empty_like(row)
            o.skinny_gemm(row, w, nxt)                     # what stands between two visits of a state
            row = nxt
            y = torch.empty(S, inner, dtype=torch.float32, device=DEV)
            if kind == "conv":
                out = torch.empty(S, inner, dtype=torch.bfloat16, device=DEV)
                o.conv_silu(row[:, :inner], out, f32(inner, 4, seed=6), None, state, segs, slots, starts, state_ahead=ahead)
                y = out
            elif kind == "delta":
                o.delta_scan(row[:, :2 * kd + inner], row[:, -2 * H:-H], row[:, -H:], f32(H, seed=6), f32(H, seed=7), state, y,
                             slots, starts, H, H, D, P, 1e-6, 0.1, state_ahead=ahead)
            elif kind == "channel_delta":
                o.channel_delta_scan(row[:, :2 * kd + inner], row[:, -H:], f32(S, kd, seed=8), f32(kd, seed=6), f32(H, seed=7),
                                     state, y, slots, starts, H, H, D, P, 1e-6, 0.1, state_ahead=ahead)
            elif kind == "retention":
                o.retention_scan(row[:, :2 * kd + inner], f32(H, seed=6), None, segs, state, y, slots, starts, H, D, P,
                                 0.1, state_ahead=ahead)
            elif kind == "ssd":
                o.ssd_scan(row[:, :inner + 2 * D], row[:, -H:], f32(H, seed=6), f32(H, seed=7), f32(H, seed=8), state, y, slots,
                           starts, H, P, D, 1, state_ahead=ahead)
            else:
                r, k, v = (row[:, i * max(inner, kd):][:, :n] for i, n in enumerate((kd, kd, inner)))
                o.time_mixing_scan(r, k, v, f32(S, kd, seed=8), f32(kd, seed=6), f32(kd, seed=7), state, y, slots, starts, H, P,
                                   D, state_ahead=ahead)
        results.append((state, y))
    assert torch.isfinite(results[0][1].float()).all()
    for a, b in zip(*results):
        assert torch.equal(a, b)


# equal values, zeros of both signs, minus infinities and NaN; fewer experts than lanes, odd numbers, all of them chosen
@pytest.mark.parametrize("E,k", [(3, 3), (8, 2), (33, 7), (256, 8), (300, 32), (512, 40)])
def test_choice_of_experts(E, k):
    o, T = ops(), 6
    g = torch.Generator().manual_seed(E)
    logits = torch.randn(T, E, generator=g)
    bias = torch.randn(E, generator=g)
    logits[1] = 0.0                                        # all equal: the lowest ids
    logits[2] = torch.randint(-2, 3, (E,), generator=g).float()
    bias[:] = torch.where(torch.rand(E, generator=g) < 0.3, torch.zeros(()), bias.round())
    logits[3, ::2] = float("-inf")
    logits[4, 0] = float("nan")
    score = torch.sigmoid(logits)
    choice = score + bias
    choice[4] = torch.where(choice[4].isnan(), torch.full((), -float("inf")), choice[4])
    ids = torch.empty(T, k, dtype=torch.int32, device=DEV)
    weights = torch.empty(T, k, dtype=torch.float32, device=DEV)
    o.router_select(logits.to(DEV), bias.to(DEV), ids, weights, k, False, False, 1.0)
    # the kernel's own scores decide (its exp differs from the host's in the last bit): compare values, then ties by id
    for t in range(T):
        got = ids[t].tolist()
        chosen = [choice[t, e].item() for e in got]
        if t == 4 and k == E:
            got, chosen = got[:-1], chosen[:-1]            # the NaN itself is nobody's choice
        assert len(set(got)) == len(got)
        assert all(a >= b - 1e-6 for a, b in zip(chosen, chosen[1:]))
        rest = [choice[t, e].item() for e in range(E) if e not in got]
        assert not rest or max(rest) <= chosen[-1] + 1e-6
        if t in (1, 2):                                    # equal scores are equal bits: ascending ids
            same = [(a, b) for a, b in zip(got, got[1:]) if logits[t, a] == logits[t, b] and bias[a] == bias[b]]
            assert all(a < b for a, b in same)
