"""Graphs of engines that are gone outlive every capture that is running, whoever drops them."""
import gc
import threading
import weakref

import pytest

from hfee_b200.engine import graphs


class _Graph:
    pass


class _Runner:
    """As ModelRunner: its graphs are handed on when it goes, and it is part of a cycle."""

    def __init__(self):
        self.graphs = {1: _Graph()}
        self.me = self
        weakref.finalize(self, graphs.retire, self.graphs).atexit = False


def _dead_runner():
    return weakref.ref(_Runner().graphs[1])


def test_without_a_capture_graphs_go_at_once():
    graph = _dead_runner()
    gc.collect()
    assert graph() is None


def test_a_collector_run_inside_a_capture_frees_no_graph():
    graph = _dead_runner()
    with graphs.capturing():
        gc.collect()
        assert graph() is not None
    assert graph() is None
    with pytest.raises(RuntimeError), graphs.capturing():
        graph = _dead_runner()
        gc.collect()
        raise RuntimeError
    assert graph() is None


def test_one_capture_ending_leaves_the_others_protected():
    started, end, seen = threading.Event(), threading.Event(), []

    def second():
        with graphs.capturing():
            started.set()
            assert end.wait(30)
        seen.append(graph() is not None)
    graph = _dead_runner()
    with graphs.capturing():
        other = threading.Thread(target=second)
        other.start()
        assert started.wait(30)
        gc.collect()
        end.set()
        other.join()
        gc.collect()
        assert seen == [True] and graph() is not None and gc.isenabled()
    assert graph() is None


@pytest.mark.gpu
def test_a_capture_survives_the_collector(tiny_dirs):
    from hfee_b200 import Engine, EngineConfig, StepEntry

    def decode(engine, steps=4):
        slot = engine.runner.open()
        out = [engine.runner.step([StepEntry(slot, [7, 8, 9], want=(2,))]).clone()]
        out += [engine.runner.step([StepEntry(slot, [t], want=(0,))]).clone() for t in range(steps)]
        engine.runner.close(slot)
        return out
    config = EngineConfig(max_requests=2, max_batch_tokens=64, page_size=16, max_context=128)
    first = Engine(tiny_dirs["A"], config)
    want = decode(first)
    assert first.runner.graph_replays > 0
    first.cycle = first                                     # only the collector frees it
    del first
    second = Engine(tiny_dirs["A"], config)
    forward, collected = second.runner.model.forward, []
    second.runner.model.forward = lambda *a: (collected.append(gc.collect()), forward(*a))[1]
    got = decode(second)
    assert second.runner.graph_replays > 0 and len(collected) >= 3
    for a, b in zip(got, want):
        assert (a == b).all()
