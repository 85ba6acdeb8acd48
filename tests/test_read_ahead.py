"""What launches may read while the launch in front of them still runs is promised by whoever knows: a model whose parts all
keep to it, nobody by default."""

import ctypes
import importlib
import threading

import pytest
import torch

from freetoken_b200.csrc import ops
from freetoken_b200.models.model import Model
from freetoken_b200.parts import base
from freetoken_b200.registry import architecture_of


@pytest.fixture
def host():
    module = ops._host_module()
    module.setup(torch.Tensor, lambda: 0, lambda device: 7, ops.KernelError, ops._ERRORS)
    before = module.ahead(False)
    yield module
    module.ahead(before)
    module.setup(torch.Tensor, getattr(torch._C, "_cuda_getDevice", lambda: 0),
                 getattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 0), ops.KernelError, ops._ERRORS)


def test_the_promise_stands_behind_the_arguments_of_its_own_thread(host):
    seen = []

    def packed(words):
        seen.append(list((ctypes.c_longlong * 4).from_address(words)))
        return 0
    packed = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)(packed)
    f = host.Launcher(ctypes.cast(packed, ctypes.c_void_p).value, "i q", "ft_thing", 1)
    f(1, 2)
    assert host.ahead(True) is False
    f(1, 2)
    other = threading.Thread(target=f, args=(1, 2))
    other.start()
    other.join()
    assert ops.read_ahead(False) is True
    f(1, 2)
    assert seen == [[1, 2, 7, 0], [1, 2, 7, 1], [1, 2, 7, 0], [1, 2, 7, 0]]
    with pytest.raises(ZeroDivisionError):
        host.ahead(type("Odd", (), {"__bool__": lambda self: 1 / 0})())
    assert host.ahead(False) is False


MODELS = [("besuzen", "BZ"), ("tonapel", "TN"), ("mezapel", "MZ"), ("nirelix", "NX"), ("dizatar", "DZ"), ("fazinex", "FZ")]


def tiny_model(name, configs):
    tiny = importlib.import_module(f"{name}_tiny")
    config = next(iter(getattr(tiny, configs).values()))
    arch = architecture_of(config)
    return Model(arch.build_plan(arch.read_config(config)))


@pytest.mark.parametrize("name,configs", MODELS)
def test_a_model_promises_it_if_all_its_parts_do(name, configs, monkeypatch):
    model = tiny_model(name, configs)
    assert model.reads_ahead
    for part in {type(p): p for p in model.leaf_parts()}.values():
        derived = type("Derived", (type(part),), {})              # says nothing of its own launches
        part.__class__, was = derived, type(part)
        assert not part.keeps_ahead() and not all(p.keeps_ahead() for p in model.leaf_parts())
        part.__class__ = was


def test_the_promise_holds_for_the_length_of_a_step(host, monkeypatch):
    model = tiny_model("nirelix", "NX")
    held = []

    def step(*a):
        held.append(host.ahead(True))
        host.ahead(held[-1])
        if len(held) == 2:
            raise RuntimeError("in the middle of a step")
    monkeypatch.setattr(model, "_forward", step)
    model.forward(None, [], None, None)
    with pytest.raises(RuntimeError):
        model.forward(None, [], None, None)
    assert host.ahead(False) is False
    model.reads_ahead = False
    host.ahead(True)
    model.forward(None, [], None, None)
    assert held == [True, True, False] and host.ahead(False) is True


def test_no_part_without_its_own_statement():
    for registry in (base.MIXERS, base.FEED_FORWARDS, base.BLOCKS, base.NORMS, base.EMBEDDINGS, base.HEADS, base.STREAM_MAPS):
        for kind in registry.kinds():
            cls = registry.get(kind)
            if cls.__module__.startswith("freetoken_b200."):
                assert vars(cls).get("reads_ahead") is True, cls


# A weight, a table or a list that the package's launch right in front has written: without the promise every face waits for it.
# (gather_rows writes it: 6,000 rows, the last of them the one that is used.)
@pytest.mark.gpu
@pytest.mark.parametrize("face", ["rmsnorm", "rmsnorm_parts", "norm_add", "norm_add_parts", "join", "hyper", "rms_rows", "gated",
                                  "router_logits", "route_small", "skinny", "skinny_heads", "gemm_rows", "gemm_heads"])
def test_what_the_launch_in_front_wrote_may_be_a_weight(face):
    from test_kernels_gpu import DEV, ops as get, rnd
    o, T, H, rows = get(), 3, 2048, 6000
    bf = torch.bfloat16
    f32 = lambda *s, seed: rnd(*s, seed=seed)
    wide = face in ("skinny", "skinny_heads")
    source = [rnd(rows, H, dtype=bf if wide else torch.float32, seed=40 + i, scale=0.05) for i in range(2)]
    pick = torch.arange(rows, dtype=torch.int32, device=DEV)
    table = torch.zeros_like(source[0])
    x, parts, residual = rnd(T, H, dtype=bf, seed=1), rnd(T, 6, H, dtype=bf, seed=2), f32(T, H, seed=3)
    streams, ones = f32(T, 4, H, seed=4), torch.ones(4, device=DEV)
    last = table[-1]
    logits = f32(T, 128, seed=5)

    def used():
        if face in ("rmsnorm", "rmsnorm_parts"):
            r, out = residual.clone(), torch.empty_like(x)
            return lambda: (o.rmsnorm(x if face == "rmsnorm" else parts, r, last, out, 1e-5, False), r, out)[1:]
        if face in ("norm_add", "norm_add_parts"):
            r, out = residual.clone(), torch.empty_like(x)
            return lambda: (o.norm_add(x if face == "norm_add" else parts, r, last, 1e-5, False, 1.0, next_weight=table[-2],
                                       next_eps=1e-5, next_out=out), r, out)[1:]
        if face == "join":
            r, out = residual.clone(), torch.empty_like(x)
            return lambda: (o.join_layer_norm(x, r, last, 1e-5, out, bias=table[-2]), r, out)[1:]
        if face == "hyper":
            s, out = streams.clone(), torch.empty_like(x)
            return lambda: (o.hyper_norm(s, x, last[:16].view(4, 4), last[16:20], ones, last, None, 1e-5, False, out), s, out)[1:]
        if face == "rms_rows":
            out = torch.empty_like(x)
            return lambda: (o.rms_rows(x, last, out, 1e-5), out)[1:]
        if face == "gated":
            out = torch.empty_like(x)
            return lambda: (o.gated_norm(residual, x, last[:128], out, 16, 1e-5, False), out)[1:]
        if face == "router_logits":
            out = torch.empty(T, 64, device=DEV)
            return lambda: (o.router_logits(x, table[-64:], out), out)[1:]
        if face == "route_small":
            ids, w = torch.empty(T, 4, dtype=torch.int32, device=DEV), torch.empty(T, 4, device=DEV)
            lists = [torch.empty(n, dtype=torch.int32, device=DEV) for n in (128, 129, 12, 12, 129)]
            return lambda: (o.route_small(logits, last[:128], ids, w, *lists, 4, False, True, 1.0), ids, w)[1:]
        if face == "skinny":
            out = torch.empty(T, 512, dtype=bf, device=DEV)
            return lambda: (o.skinny_gemm(x, table[-512:], out), out)[1:]
        if face == "skinny_heads":
            out, w = torch.empty(T, 8, 64, dtype=bf, device=DEV), table[-64:].view(8, 64, 256)
            return lambda: (o.skinny_heads(x.view(T, 8, 256), w, out), out)[1:]
        if face == "gemm_rows":
            out = torch.empty(T, 512, device=DEV)
            return lambda: (o.gemm_rows(residual, table[-512:], out), out)[1:]
        out, w = torch.empty(T, 8, 64, device=DEV), table[-64:].view(8, 64, 256)
        return lambda: (o.gemm_heads(residual.view(T, 8, 256), w, out), out)[1:]

    want = []
    for s in source:
        call = used()
        table.copy_(s)
        torch.cuda.synchronize()
        want.append([t.clone() for t in call()])
    assert not torch.equal(want[0][-1], want[1][-1])
    assert o.read_ahead(False) is False
    for turn in range(12):
        call = used()
        o.gather_rows(source[1 - turn % 2], pick, table)
        o.gather_rows(source[turn % 2], pick, table)
        got = call()
        for a, b in zip(got, want[turn % 2]):
            assert torch.equal(a, b), turn


# with the promise, a weight that was there before: the same rows
@pytest.mark.gpu
def test_promised_steps_give_the_same_rows():
    from test_kernels_gpu import DEV, ops as get, rnd
    o, T, H = get(), 4, 4096
    x = rnd(T, H, dtype=torch.bfloat16, seed=1)
    w = [rnd(H, H, dtype=torch.bfloat16, seed=2 + i, scale=H ** -0.5) for i in range(4)]
    n = rnd(H, seed=9)
    results = []
    for promise in (False, True):
        before = o.read_ahead(promise)
        try:
            r, rows = rnd(T, H, seed=7), [x.clone() for _ in range(9)]
            for i in range(4):
                o.skinny_gemm(rows[2 * i], w[i], rows[2 * i + 1])
                o.rmsnorm(rows[2 * i + 1], r, n, rows[2 * i + 2], 1e-5, False)
        finally:
            o.read_ahead(before)
        results.append([r, *rows])
    for a, b in zip(*results):
        assert torch.equal(a, b)
