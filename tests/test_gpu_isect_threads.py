"""The intersection operator on threads that come and go: the end of one does
not touch another thread's graph capture, and threads in turn and at once get
their own counts."""
import threading

import pytest
import torch

from scenes import beta_params, projected_scene

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_thread_that_ends_inside_a_capture():
    from gsplat.cuda._wrapper import isect_tiles
    from ubs import scene as S
    from ubs.render import GraphedStep, Renderer, Views
    s = projected_scene(200, 64, 48, seed=2, device=DEV)
    want = isect_tiles(s["means2d"], s["radii"], s["depths"], 16, 4, 3)
    p = {k: torch.nn.Parameter(v.to(DEV))
         for k, v in beta_params(300, 6, seed=0, log_scale_mu=-2.5).items()}
    views = Views([S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)], device=DEV)
    warm, go, done, got = threading.Event(), threading.Event(), threading.Event(), []
    stream = torch.cuda.Stream()

    def call():
        with torch.cuda.stream(stream):
            got.append(isect_tiles(s["means2d"], s["radii"], s["depths"], 16, 4, 3))

    def other():
        try:
            call()
            warm.set()
            go.wait(30)
        except Exception as e:  # noqa: BLE001 (reported below)
            got.append(e)
        finally:
            warm.set()
            done.set()

    t = threading.Thread(target=other)
    t.start()
    assert warm.wait(30)
    ends = []

    def loss(c, a):
        if torch.cuda.is_current_stream_capturing() and not ends:
            go.set()
            done.wait(30)
            t.join(30)  # the thread ends inside the capture
            ends.append(not t.is_alive())
        return c.sum()

    step = GraphedStep(Renderer(dim=6), p, views, None, loss)
    assert ends == [True]
    a = float(step.replay().detach())
    torch.cuda.synchronize()
    assert a == float(step.loss.detach())
    assert len(got) == 1 and not isinstance(got[0], Exception), got
    for x, y in zip(got[0], want):
        assert torch.equal(x, y)


def test_threads_in_turn_and_at_once():
    from gsplat.cuda._wrapper import isect_tiles
    scenes = [projected_scene(50 + 37 * i, 64, 48, seed=i, device=DEV) for i in range(6)]

    def ids(s):
        return isect_tiles(s["means2d"], s["radii"], s["depths"], 16, 4, 3)[1]

    want = [ids(s) for s in scenes]
    assert len({w.numel() for w in want}) == len(want)
    wrong = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                if not torch.equal(ids(scenes[i]), want[i]):
                    wrong.append(i)

    for _ in range(5):
        ts = [threading.Thread(target=work, args=(i,)) for i in range(6)]
        [t.start() for t in ts]
        [t.join(60) for t in ts]
        for i in range(6):
            t = threading.Thread(target=work, args=(i,))
            t.start()
            t.join(60)
    torch.cuda.synchronize()
    assert not wrong
