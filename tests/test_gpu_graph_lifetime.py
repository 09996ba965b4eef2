"""A captured step that dies inside a later step's capture."""
import gc
import weakref

import pytest
import torch

from scenes import beta_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _step(loss):
    from ubs import scene as S
    from ubs.render import GraphedStep, Renderer, Views
    p = {k: torch.nn.Parameter(v.to(DEV))
         for k, v in beta_params(300, 6, seed=0, log_scale_mu=-2.5).items()}
    views = Views([S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)], device=DEV)
    return GraphedStep(Renderer(dim=6), p, views, None, loss)


def test_collection_inside_a_capture():
    old = _step(lambda c, a: c.sum())
    old.cycle = old
    graph = weakref.ref(old.graph)
    held, capturing = [old], []
    del old

    def loss(c, a):
        if torch.cuda.is_current_stream_capturing():
            held.clear()
            gc.collect()
            capturing.append(graph() is not None)
        return c.sum()

    new = _step(loss)
    assert capturing == [True] and graph() is None
    a = float(new.replay())
    torch.cuda.synchronize()
    assert a == float(new.replay()) > 0
    assert gc.isenabled()
