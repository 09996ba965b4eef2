"""What saved-tensor hooks return reaches the backward's kernels only as the
forward's values: other strides give the same gradients, another device, type
or size is refused before a launch."""
import pytest
import torch

from scenes import beta_params, projected_scene, rest_indices

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _render():
    from ubs import scene as S
    from ubs.render import PARAM_ORDER, Renderer, Views
    p = beta_params(400, 6, seed=0, log_scale_mu=-2.5)
    views = Views([S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)], device=DEV)
    r = Renderer(dim=6)
    return ([p[k].to(DEV) for k in PARAM_ORDER],
            lambda *t: r.render(dict(zip(PARAM_ORDER, t)), views))


def _cond():
    from gsplat.cuda._wrapper import cond_mean_convariance_opacity as cond
    g = torch.Generator().manual_seed(1)
    L = torch.randn(300, 6, 6, generator=g) * 0.2 + torch.eye(6)
    return [t.to(DEV) for t in (torch.randn(300, 6, generator=g), L @ L.transpose(1, 2),
                                torch.rand(300, 1, generator=g), torch.rand(300, 3, generator=g) * 4,
                                torch.randn(300, 3, generator=g))], cond


def _covar():
    from gsplat.cuda._wrapper import rot_scale_l_triangle_to_covar as covar
    ri, rj = (t.to(DEV) for t in rest_indices(6))
    g = torch.Generator().manual_seed(2)
    return [t.to(DEV) for t in (torch.randn(300, 3, 3, generator=g), torch.rand(300, 6, generator=g),
                                torch.randn(300, 15, generator=g))], \
        lambda R, s, l: covar(R, s, l, ri, rj)


def _projection():
    from gsplat.cuda._wrapper import fully_fused_projection
    from ubs import scene as S
    cam = S.orbit_view(3, 3.0, 70, 50, 60.0, 60.0, device=DEV)
    g = torch.Generator().manual_seed(3)
    L = torch.randn(300, 3, 3, generator=g) * 0.1
    V = L @ L.transpose(1, 2) + 0.01 * torch.eye(3)
    return [torch.randn(300, 3, generator=g).to(DEV), V.to(DEV)], \
        lambda m, C: fully_fused_projection(m, C, None, None, cam.viewmat[None], cam.K[None], 70,
                                            50, calc_compensations=True)[1:]


def _blend():
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles, rasterize_to_pixels
    s = projected_scene(200, 64, 48, seed=2, device=DEV)
    _, ids, fl = isect_tiles(s["means2d"], s["radii"], s["depths"], 16, 4, 3)
    offs = isect_offset_encode(ids, 1, 4, 3)
    masks = torch.rand(1, 3, 4, generator=torch.Generator().manual_seed(4)).to(DEV) < 0.8
    return [s[k] for k in ("means2d", "conics", "colors", "opacities", "betas")], \
        lambda *t: rasterize_to_pixels(*t, 64, 48, 16, offs, fl, masks=masks)


CALLS = [_render, _cond, _covar, _projection, _blend]


def _grads(make, unpack):
    ins, f = make()
    x = [t.clone().requires_grad_(True) for t in ins]
    if unpack is None:
        outs = f(*x)
    else:
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            outs = f(*x)
    outs = outs if isinstance(outs, tuple) else (outs,)
    sum((o * o).sum() for o in outs).backward()
    torch.cuda.synchronize()
    return [t.grad for t in x]


def _strided(t):
    """The same values, last dimension first in memory."""
    return t if t.dim() < 2 else t.movedim(-1, 0).contiguous().movedim(0, -1)


@pytest.mark.parametrize("make", CALLS)
def test_other_strides(make):
    seen = []

    def unpack(t):
        s = _strided(t.clone())
        seen.append(s.is_contiguous())
        return s

    want, got = _grads(make, None), _grads(make, unpack)
    assert not all(seen)
    for a, b in zip(got, want):
        if b is not None:
            torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("make", CALLS)
def test_refused(make):
    for unpack, error in ((lambda t: t.cpu(), ValueError), (lambda t: t.double(), TypeError),
                          (lambda t: t[:1], ValueError)):
        with pytest.raises(error):
            _grads(make, unpack)
