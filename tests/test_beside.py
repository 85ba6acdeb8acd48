"""Two pieces of a step side by side: only in a capture, only with scratch of their own; the graph's rows are the eager rows."""

import pytest
import torch

from freetoken_b200.parts.base import StepContext


def context(device="cpu", side=()):
    t = torch.zeros(1, dtype=torch.int32, device=device)
    return StepContext(device=torch.device(device), dtype=torch.bfloat16, segments=[], num_tokens=1, token_ids=t, token_pos=t,
                       token_seg=t, seg_slot=t, seg_pos0=t, seg_q_start=t, seg_kv_len=t, block_tables=[], workspace=None, page_size=64,
                       side=list(side))


def test_outside_a_capture_one_follows_the_other():
    order = []
    ctx = context()
    assert ctx.beside(lambda: order.append(1) or "a", lambda: order.append(2) or "b", ("x",), ("y",)) == ("a", "b")
    assert order == [1, 2]


def test_parts_name_every_buffer_they_write():
    """The scratch a part states covers the workspace names in its class and in the faces it calls."""
    import inspect
    import re

    from freetoken_b200.csrc import ops
    from freetoken_b200.parts import base
    for registry in (base.MIXERS, base.FEED_FORWARDS):
        for kind in registry.kinds():
            cls = registry.get(kind)
            if not cls.__module__.startswith("freetoken_b200."):
                continue
            source = "".join(inspect.getsource(c) for c in cls.__mro__ if c.__module__ == cls.__module__)
            for face in set(re.findall(r"ops\.(\w+)\(", source)):
                source += inspect.getsource(getattr(ops, face)) if inspect.isfunction(getattr(ops, face, None)) else ""
            written = {name.split(".")[0] for name in re.findall(r'(?:ws|workspace)\.get\(\s*"([\w.]+)"', source)}
            stated = cls.scratch or {"RoutedExperts": ("moe",), "MixerSum": ("mixer_sum",)}.get(cls.__name__, ())
            assert written <= set(stated), (kind, written - set(stated))


@pytest.mark.gpu
@pytest.mark.parametrize("scratch,branches", [((("a",), ("b",)), True), ((("a", "c"), ("b", "c")), False), ((None, ("b",)), False)])
def test_branches_of_a_graph(scratch, branches):
    from test_kernels_gpu import DEV, ops, rnd
    o = ops()
    side = [torch.cuda.Stream(), torch.cuda.Stream()]
    ctx = context(DEV, side)
    x = rnd(3, 512, dtype=torch.bfloat16, seed=1)
    w = [rnd(512, 512, dtype=torch.bfloat16, seed=2 + i, scale=0.05) for i in range(6)]
    rows = [torch.empty_like(x) for _ in range(8)]
    streams = []

    def chain(first, weights, out):
        def run():
            streams.append(torch.cuda.current_stream().cuda_stream)
            o.skinny_gemm(first, weights[0], out[0])
            for a, b, m in zip(out, out[1:], weights[1:]):
                o.skinny_gemm(a, m, b)
            return out[-1]
        return run

    def step():
        o.skinny_gemm(x, w[0], rows[0])
        a, b = ctx.beside(lambda: ctx.beside(chain(rows[0], w[:2], rows[1:3]), chain(rows[0], w[1:3], rows[3:5]), *scratch)[1],
                          chain(rows[0], w[3:], rows[5:8]), *scratch)
        o.skinny_gemm(a, w[5], rows[1])
        return a, b, rows[1]

    want = [t.clone() for t in step()]
    assert len(set(streams)) == 1
    graph = torch.cuda.CUDAGraph()
    del streams[:]
    with torch.cuda.graph(graph):
        got = step()
    assert len(set(streams)) == (3 if branches else 1) and len(ctx.side) == 2
    for seed in range(20):
        x.copy_(rnd(3, 512, dtype=torch.bfloat16, seed=100 + seed))
        graph.replay()
        have = [t.clone() for t in got]
        streams_before = len(streams)
        want = [t.clone() for t in step()]
        assert len(streams) > streams_before
        for a, b in zip(have, want):
            assert torch.equal(a, b)
