"""The streams decode steps are captured on are an engine's own, and go back when it is gone."""

import gc

import pytest
import torch

from freetoken_b200.engine import streams


@pytest.fixture
def made(monkeypatch):
    out = []

    def own_stream(device, priority=0):
        out.append((str(device), priority))
        return len(out)
    monkeypatch.setattr(streams.ops, "own_stream", own_stream)
    monkeypatch.setattr(torch.cuda, "Stream", lambda *a, **k: pytest.fail("a stream of the shared pool"))
    monkeypatch.setattr(streams, "_free", {})
    return out


def test_live_engines_share_no_stream_and_sets_go_round(made):
    a, b, other = streams.take("cuda:0", True), streams.take("cuda:0", True), streams.take("cuda:1", True)
    plain = streams.take("cuda:0", False)
    ids = [i for s in (a, b, other, plain) for i in (s.main, *s.side, *s.minor)]
    assert len(set(ids)) == len(ids) == len(made) == 5 + 5 + 5 + 3
    assert {p for d, p in made[:3]} == {-1} and {p for d, p in made[3:5]} == {0} and {p for d, p in made[15:]} == {0}
    streams.give_back("cuda:0", True, a)
    assert streams.take("cuda:0", False) not in (a, plain)
    assert streams.take("cuda:0", True) is a and len(made) == 21
    assert streams.take("cuda:0", True) is not a and len(made) == 26


@pytest.mark.gpu
def test_an_engine_gives_its_streams_back_and_nobody_else_has_them(tmp_path):
    import besuzen_tiny as tiny
    from freetoken_b200.engine import Engine, EngineArgs, StepEntry
    folder = str(tmp_path / "model")
    which = next(iter(tiny.BZ))
    tiny.write_tiny(folder, which)
    streams._free.clear()

    def lives():
        engine = Engine.from_folder(folder, EngineArgs(dtype="bfloat16", page_size=tiny.PAGE[which], max_tokens=512))
        for t in range(6):
            engine.step([StepEntry("a", [t], [0])])
        assert engine.graph_replays > 0
        return engine, engine._streams
    one, first = lives()
    two, second = lives()
    pool = {torch.cuda.Stream(priority=p).cuda_stream for p in (0, -1) for _ in range(64)}
    mine = [s.cuda_stream for t in (first, second) for s in (t.main, *t.side, *t.minor)]
    assert len(set(mine)) == len(mine) and not pool & set(mine)
    del one
    gc.collect()
    assert lives()[1] is first
