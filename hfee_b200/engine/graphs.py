"""CUDA graphs of engines that are gone are freed when no capture is running.

A capture does not survive a graph being freed under it, and the collector frees a dead engine's graphs whenever it runs, in
whichever thread.  A runner therefore hands its graphs to :func:`retire` (through ``weakref.finalize``, and those it evicts itself);
they are dropped at once, or, while a :func:`capturing` block of any runner is open, at the end of the last such block.
"""
from __future__ import annotations

import contextlib
import threading

_lock = threading.RLock()        # held while graphs are dropped, so that no capture starts meanwhile; a collector run inside may call retire()
_captures = 0
_retired: list = []


def retire(graphs: dict, *keys) -> None:
    """Take the graphs of ``keys`` (all, if none are given) out of ``graphs`` and drop them now, or when the last capture that is
    running has ended."""
    with _lock:
        for key in keys or list(graphs):
            _retired.append(graphs.pop(key))
        if not _captures:
            _retired.clear()


@contextlib.contextmanager
def capturing():
    """Nothing given to :func:`retire` is freed while the block runs."""
    global _captures
    with _lock:
        _captures += 1
    try:
        yield
    finally:
        with _lock:
            _captures -= 1
            if not _captures:
                _retired.clear()
