"""Graphs of steps that die while another step is captured are destroyed after
the last capture has ended, also with several threads; Python's collector is
left as it is."""
import gc
import threading
import weakref

from ubs.render import _Graphs


class _Graph:
    pass


class _Step:
    def __init__(self, graphs):
        self.graph = _Graph()
        self.cycle = self
        weakref.finalize(self, graphs.release, self.graph).atexit = False


def _dead_in_a_cycle(graphs):
    s = _Step(graphs)
    return weakref.ref(s), weakref.ref(s.graph)


def test_destroyed_at_once_without_a_capture():
    step, graph = _dead_in_a_cycle(_Graphs())
    gc.collect()
    assert step() is None and graph() is None


def test_kept_until_the_capture_has_ended():
    g = _Graphs()
    step, graph = _dead_in_a_cycle(g)
    with g.capturing():
        assert gc.isenabled()
        gc.collect()
        assert step() is None and graph() is not None
    assert graph() is None and gc.isenabled()


def test_kept_after_a_failed_capture_only_until_its_end():
    g = _Graphs()
    step, graph = _dead_in_a_cycle(g)
    try:
        with g.capturing():
            gc.collect()
            raise ValueError
    except ValueError:
        pass
    assert graph() is None


def test_two_threads_that_capture_interleave():
    g = _Graphs()
    first_in, second_in, first_out = (threading.Event() for _ in range(3))
    seen = []

    def first():
        with g.capturing():
            first_in.set()
            second_in.wait(10)
        first_out.set()

    def second():
        first_in.wait(10)
        with g.capturing():
            second_in.set()
            first_out.wait(10)
            step, graph = _dead_in_a_cycle(g)  # the other capture is over, this one is not
            gc.collect()
            seen.append((step() is None, graph() is not None))
            seen.append(graph)

    ts = [threading.Thread(target=f) for f in (first, second)]
    [t.start() for t in ts]
    [t.join(30) for t in ts]
    assert seen[0] == (True, True)
    assert seen[1]() is None
