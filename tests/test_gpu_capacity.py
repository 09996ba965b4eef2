"""Unchecked frames of a scene whose intersections grow slowly: the capacity
grows before a frame overflows; a jump past it is still reported."""
import pytest
import torch

from scenes import beta_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_capacity_follows_a_growing_scene():
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(3000, 6, seed=0, log_scale_mu=-3.0).items()}
    cam = S.orbit_view(1, 3.0, 320, 240, 260.0, 260.0, device=DEV)
    views, r = Views([cam], device=DEV), Renderer(dim=6)
    with torch.no_grad():
        r.render(p, views)
        first = r.last_isects
        r.capacity = int(first * 1.2)  # room for the first steps
        for _ in range(120):
            p["scale"][:, :3] += 0.02  # a few per cent more intersections per frame
            r.render(p, views, check=False)
        r._check_pending()
        assert r.last_isects > 2 * first
        r.capacity = r.last_isects // 2
        r.render(p, views, check=False)
        with pytest.raises(RuntimeError, match="capacity is now"):
            r.render(p, views, check=False)
