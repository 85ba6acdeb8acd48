"""Streams that decode steps are captured on.

Whatever runs on a capturing stream is recorded instead of run, so nobody else may be given one: PyTorch's own streams
come out of a pool of a few dozen that every thread of the process shares.  An engine takes a set at its first capture
and the set goes back when the engine is gone: there are as many sets as engines that lived at the same time, and
no two live engines share one (nor the library workspaces that PyTorch keeps a stream).
"""

from __future__ import annotations

import threading
from typing import Any, Dict, List, NamedTuple, Tuple

from ..csrc import ops


class CaptureStreams(NamedTuple):
    main: Any
    side: Tuple[Any, ...]        # for the branches of a step
    minor: Tuple[Any, ...]       # of lower priority, for fillers (none where no part has one)


_lock = threading.Lock()
_free: Dict[Tuple[str, bool], List[CaptureStreams]] = {}


def take(device, fills: bool) -> CaptureStreams:
    """A set of streams on ``device``.  ``fills``: a filler's blocks wait for those of everything else.  Only models that
    have one pay for priorities: with the same one on every launch a step of two equal branches took 2 % longer than
    with none."""
    with _lock:
        kept = _free.get((str(device), fills))
        if kept:
            return kept.pop()
    high = -1 if fills else 0
    return CaptureStreams(ops.own_stream(device, high), tuple(ops.own_stream(device, high) for _ in range(2)),
                          tuple(ops.own_stream(device) for _ in range(2 if fills else 0)))


def give_back(device, fills: bool, streams: CaptureStreams) -> None:
    with _lock:
        _free.setdefault((str(device), fills), []).append(streams)
