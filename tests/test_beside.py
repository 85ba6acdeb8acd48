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


@pytest.mark.parametrize("failing", ["first", "second", None])
def test_a_branch_is_joined_whatever_a_piece_raises(failing, monkeypatch):
    """A capture left with an open branch would end in an error of its own, in the place of the piece's."""
    import contextlib
    calls = []

    class Stream:
        def __init__(self, name):
            self.name = name

        def wait_stream(self, other):
            calls.append((self.name, other.name))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream("main"))
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    ctx = context(side=[Stream("side")])

    def piece(name):
        def run():
            if name == failing:
                raise KeyError(name)
            return name
        return run
    with contextlib.nullcontext() if failing is None else pytest.raises(KeyError):
        assert ctx.beside(piece("first"), piece("second"), ("x",), ("y",)) == ("first", "second")
    assert calls == [("side", "main"), ("main", "side")] and [s.name for s in ctx.side] == ["side"]


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


def _written(cls, ops):
    """First words of the workspace names in a class, the package's classes it inherits from, the functions of those modules
    that it calls and the faces it calls; a name that comes by a variable counts with every literal the variable is given."""
    import inspect
    import re
    import sys
    source, taken = "", set()
    for c in cls.__mro__:
        if c.__module__.startswith("freetoken_b200.") and c.__module__ != "freetoken_b200.parts.base":
            source += inspect.getsource(c)
            taken.add(c.__module__)
    seen = set()
    while True:
        called = {(ops.__name__, n) for n in re.findall(r"ops\.(\w+)\(", source)}
        called |= {(m, n) for m in taken for n in re.findall(r"(?<![\w.])(\w+)\(", source)}
        new = [(m, n) for m, n in sorted(called - seen) if inspect.isfunction(getattr(sys.modules[m], n, None))]
        seen |= called
        if not new:
            break
        source += "".join(inspect.getsource(getattr(sys.modules[m], n)) for m, n in new)
    names = set(re.findall(r'(?:ws|workspace)\.get\(\s*"([\w.]+)"', source))
    for variable in set(re.findall(r"(?:ws|workspace)\.get\(\s*([A-Za-z_]\w*),", source)):
        given = re.findall(rf'\b{variable} = (.*"[\w.]+".*)', source)
        assert given, f"{cls.__name__}: where {variable} comes from"
        for line in given:
            names |= set(re.findall(r'"(\w+\.\w+)"', line))
    return {name.split(".")[0] for name in names}


def _package_parts():
    from freetoken_b200.parts import base
    return [registry.get(kind) for registry in (base.MIXERS, base.FEED_FORWARDS) for kind in registry.kinds()
            if registry.get(kind).__module__.startswith("freetoken_b200.")]


def test_what_a_part_inherits_and_calls_is_in_its_scratch():
    from freetoken_b200.csrc import ops
    from freetoken_b200.parts.key_attention import SharedKVAttention
    assert _written(SharedKVAttention, ops) == {"kattn", "attn"}          # the splits' partial results, by two steps
    for cls in _package_parts():
        assert "scratch" in vars(cls), cls
        assert _written(cls, ops) <= set(cls.scratch), cls


def test_a_class_states_its_own_scratch():
    """One that inherits a forward may write more buffers than that: nothing runs beside it until it says which."""
    for cls in _package_parts():
        bare = object.__new__(type("Derived", (cls,), {}))
        bare.members, bare.shared = [], None
        assert bare.scratch_names() is None, cls
        stated = object.__new__(type("Derived", (cls,), {"scratch": ("own",)}))
        stated.members, stated.shared = [], None
        assert stated.scratch_names() == ("own",), cls


MODELS = [("besuzen", which) for which in "ABC"] + [("tonapel", which) for which in "ABC"] + [("mezapel", which) for which in "ABCD"]
OTHERS = [("nirelix", which) for which in "ABC"] + [("dizatar", which) for which in "ABCD"] + [("fazinex", which) for which in "ABC"]
SETS = {"besuzen": "BZ", "tonapel": "TN", "mezapel": "MZ", "nirelix": "NX", "dizatar": "DZ", "fazinex": "FZ"}


def tiny_engine(folder, model, which, **more):
    import importlib
    from freetoken_b200.engine import Engine, EngineArgs
    tiny = importlib.import_module(f"{model}_tiny")
    tiny.write_tiny(folder, which)
    engine = Engine.from_folder(folder, EngineArgs(dtype="bfloat16", page_size=tiny.PAGE[which], max_tokens=3 * 128, **more))
    return engine, {r: tiny.tokens(90 + i, 90, getattr(tiny, SETS[model])[which]["vocab"]) for i, r in enumerate("xyz")}


@pytest.mark.gpu
@pytest.mark.parametrize("model,which", MODELS + OTHERS)
def test_branches_write_the_scratch_they_state(model, which, tmp_path, monkeypatch):
    """Every workspace name that a branch of a decode step takes, against what its parts say of themselves."""
    from freetoken_b200.engine import StepEntry
    from freetoken_b200.parts.base import Workspace
    engine, toks = tiny_engine(str(tmp_path / "m"), model, which)
    engine.step([StepEntry(r, t[:20], []) for r, t in toks.items()])
    open_branches, checked = [], []
    get, beside = Workspace.get, StepContext.beside

    def noted(self, name, shape, dtype):
        for names in open_branches:
            names.add(name.split(".")[0])
        return get(self, name, shape, dtype)

    def recorded(self, first, second, *scratch, filler=False):
        def run(piece, stated):
            def inner():
                names = set()
                open_branches.append(names)
                out = piece()
                open_branches.pop()
                checked.append(stated is None or names <= set(stated))
                assert checked[-1], (names, stated)
                return out
            return inner
        return beside(self, run(first, scratch[0]), run(second, scratch[1]), *scratch, filler=filler)
    monkeypatch.setattr(Workspace, "get", noted)
    monkeypatch.setattr(StepContext, "beside", recorded)
    engine.step([StepEntry(r, [t[20]], [0]) for r, t in toks.items()])
    assert all(checked) and (checked or (model, which) not in MODELS[:3])


@pytest.mark.gpu
@pytest.mark.parametrize("model,which", MODELS)
def test_replayed_branches_give_the_rows_of_eager_steps(model, which, tmp_path):
    """Models of parallel halves, sums of mixers and shared experts: the same tokens with and without graph replay."""
    from freetoken_b200.engine import StepEntry
    outs = []
    for most in (64, 0):
        engine, toks = tiny_engine(str(tmp_path / str(most)), model, which, cuda_graph_max_bs=most)
        engine.step([StepEntry(r, t[:30], []) for r, t in toks.items()])
        rows = [engine.step([StepEntry(r, [t[i]], [0]) for r, t in toks.items()]).clone() for i in range(30, 90)]
        engine.check_status()
        assert (engine.graph_replays > 30) == (most > 0)
        outs.append(torch.stack(rows))
    assert torch.equal(*outs)


@pytest.mark.gpu
@pytest.mark.parametrize("scratch,branches", [((("a",), ("b",)), True), ((("a",), ("a",)), False), ((("a",), None), False)])
def test_a_filler_takes_the_minor_streams(scratch, branches):
    """A long chain and a short one of lower priority beside it, nested once: the graph's rows are the eager ones."""
    from test_kernels_gpu import DEV, ops, rnd
    from freetoken_b200.csrc.ops import own_stream
    o = ops()
    ctx = context(DEV, [own_stream(DEV, -1), own_stream(DEV, -1)])
    ctx.minor = [own_stream(DEV, 0), own_stream(DEV, 0)]
    minor = {s.cuda_stream for s in ctx.minor}
    x = rnd(3, 512, dtype=torch.bfloat16, seed=1)
    w = [rnd(512, 512, dtype=torch.bfloat16, seed=2 + i, scale=0.05) for i in range(4)]
    rows = [torch.empty_like(x) for _ in range(10)]
    fillers = []

    def long(source, out):
        def run():
            o.skinny_gemm(source, w[0], out[0])
            o.skinny_gemm(out[0], w[1], out[1])
            o.skinny_gemm(out[1], w[2], out[2])
            return out[2]
        return run

    def short(source, out):
        def run():
            fillers.append(torch.cuda.current_stream().cuda_stream)
            o.skinny_gemm(source, w[3], out)
            return out
        return run

    def step():
        a, b = ctx.beside(long(x, rows[:3]), short(x, rows[3]), *scratch, filler=True)
        c, d = ctx.beside(lambda: ctx.beside(long(a, rows[4:7]), short(b, rows[7]), *scratch, filler=True)[1],
                          short(a, rows[8]), *scratch)
        o.skinny_gemm(c, w[1], rows[9])
        return a, b, c, d, rows[9]

    step()
    assert not minor & set(fillers)
    graph = torch.cuda.CUDAGraph()
    del fillers[:]
    with torch.cuda.graph(graph, stream=own_stream(DEV, -1)):
        got = step()
    assert len(minor & set(fillers)) == (1 if branches else 0) and len(ctx.minor) == len(ctx.side) == 2
    assert [s in minor for s in fillers] == ([True, False, True] if branches else [False] * 3)
    for seed in range(20):
        x.copy_(rnd(3, 512, dtype=torch.bfloat16, seed=100 + seed))
        graph.replay()
        have = [t.clone() for t in got]
        for a, b in zip(have, step()):
            assert torch.equal(a, b)
