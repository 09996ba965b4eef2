"""Every tensor input of a call makes its outputs differentiable, those whose
gradient is not defined (backgrounds of the fused render, the conditioning's
query, the intrinsics) included: backward passes and leaves them without one,
as the reference's autograd functions do."""
import pytest
import torch

from scenes import beta_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_render_with_only_backgrounds():
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(200, 6, seed=0, log_scale_mu=-2.5).items()}
    views = Views([S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)], device=DEV)
    bg = torch.rand(1, 3, device=DEV, requires_grad=True)
    colors, alphas = Renderer(dim=6).render(p, views, bg)
    assert colors.requires_grad and alphas.requires_grad
    (colors.sum() + alphas.sum()).backward()
    assert bg.grad is None


def test_cond_with_only_the_query():
    from gsplat.cuda._wrapper import cond_mean_convariance_opacity as cond
    n = 100
    V = torch.eye(6, device=DEV).expand(n, 6, 6).contiguous()
    q = torch.rand(n, 3, device=DEV, requires_grad=True)
    outs = cond(torch.rand(n, 6, device=DEV), V, torch.rand(n, 1, device=DEV),
                torch.rand(n, 3, device=DEV), q)
    assert all(o.requires_grad for o in outs)
    sum(o.sum() for o in outs).backward()
    assert q.grad is None


def test_projection_with_only_the_intrinsics():
    from gsplat.cuda._wrapper import fully_fused_projection
    from ubs import scene as S
    cam = S.orbit_view(3, 3.0, 70, 50, 60.0, 60.0, device=DEV)
    V = 0.01 * torch.eye(3, device=DEV).expand(100, 3, 3).contiguous()
    K = cam.K[None].clone().requires_grad_(True)
    outs = fully_fused_projection(torch.rand(100, 3, device=DEV), V, None, None,
                                  cam.viewmat[None], K, 70, 50)[1:4]
    assert all(o.requires_grad for o in outs)
    sum(o.sum() for o in outs).backward()
    assert K.grad is None
