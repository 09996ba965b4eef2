"""A call that waits for room in a full launch queue blocks its own thread
only: other Python threads go on."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _loss():
    from ubs.loss import l1_loss
    a, b = torch.rand(100, device=DEV), torch.rand(100, device=DEV)
    return lambda: l1_loss(a, b)


def _render():
    from scenes import beta_params
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(200, 6, seed=0, log_scale_mu=-2.5).items()}
    views = Views([S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)], device=DEV)
    r = Renderer(dim=6)
    r.render(p, views)
    return lambda: r.render(p, views, check="none")


@pytest.mark.parametrize("make", [_loss, _render])
def test_other_threads_run_while_a_call_blocks(make):
    call = make()
    call()
    x = torch.rand(20480, 20480, device=DEV)
    y = torch.empty_like(x)
    torch.mm(x, x, out=y)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    t = threading.Thread(target=tick)
    t.start()
    for _ in range(3):  # about half a second of work in front
        torch.mm(x, x, out=y)
    longest = start = end = 0.0
    for _ in range(1500):  # more launches than the queue holds
        a = time.perf_counter()
        call()
        b = time.perf_counter()
        if b - a > longest:
            longest, start, end = b - a, a, b
    torch.cuda.synchronize()
    stop.set()
    t.join(10)
    assert longest > 0.05  # a call did block
    inside = [start] + [s for s in ticks if start < s < end] + [end]
    assert max(b - a for a, b in zip(inside, inside[1:])) < 0.5 * longest
