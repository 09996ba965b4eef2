"""torch.jit.trace over the operators, the fused render and the losses: the
traced program renders new inputs, with gradients, as the eager calls do."""
import pytest
import torch

from scenes import beta_params, projected_scene, rest_indices

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _same(traced, eager, inputs):
    x = [t.detach().clone().requires_grad_(t.is_floating_point()) for t in inputs]
    y = [t.detach().clone().requires_grad_(t.is_floating_point()) for t in inputs]
    a, b = traced(*x), eager(*y)
    a, b = (o if isinstance(o, tuple) else (o,) for o in (a, b))
    assert len(a) == len(b)
    for s, t in zip(a, b):
        assert torch.equal(s, t)
    for o in (a, b):
        sum((t * t).sum() for t in o if t.requires_grad).backward()
    for s, t in zip(x, y):
        if t.grad is not None:
            torch.testing.assert_close(s.grad, t.grad, rtol=1e-4, atol=1e-6)


def _inputs(dim, seed, n=300):
    p = beta_params(n, dim, seed=seed, log_scale_mu=-2.5)
    return [p[k].to(DEV) for k in ("xyz", "mean", "scale", "l_triangle", "opacity", "beta", "rgb")]


@pytest.mark.parametrize("dim", [6, 7])
def test_traced_render(dim):
    from ubs import scene as S
    from ubs.render import PARAM_ORDER, Renderer, Views
    cam = S.orbit_view(3, 3.0, 70, 50, 60.0, 60.0, timestamp=0.3, device=DEV)
    r = Renderer(dim=dim)

    def f(*tensors):
        return r.render(dict(zip(PARAM_ORDER, tensors)), Views([cam], device=DEV))

    t = torch.jit.trace(f, tuple(v.requires_grad_(True) for v in _inputs(dim, 0)))
    _same(t, f, _inputs(dim, 1))


def test_traced_operators():
    from gsplat.cuda._wrapper import (cond_mean_convariance_opacity, fully_fused_projection,
                                      l_triangle_to_rotmat, rot_scale_l_triangle_to_covar)
    from ubs import scene as S
    cam = S.orbit_view(3, 3.0, 70, 50, 60.0, 60.0, device=DEV)
    ri, rj = (t.to(DEV) for t in rest_indices(6))

    def f(xyz, mean, scale, ltri, opacity, beta, query):
        R = l_triangle_to_rotmat(ltri[:, :3])
        V = rot_scale_l_triangle_to_covar(R, scale.exp(), ltri, ri, rj)
        m, C, o = cond_mean_convariance_opacity(torch.cat([xyz, mean], 1), V, opacity.sigmoid(),
                                                beta[:, 1:].exp(), query)
        radii, m2, dep, con, _ = fully_fused_projection(m, C, None, None, cam.viewmat[None],
                                                        cam.K[None], 70, 50)
        return radii, m2, dep, con, o

    a, b = _inputs(6, 0), _inputs(6, 1)
    a[6], b[6] = a[0] / a[0].norm(dim=1, keepdim=True), b[0] / b[0].norm(dim=1, keepdim=True)
    _same(torch.jit.trace(f, tuple(v.requires_grad_(True) for v in a)), f, b)


def test_traced_blend():
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles, rasterize_to_pixels

    def f(m2, conics, colors, opac, betas, radii, depths):
        _, ids, fl = isect_tiles(m2, radii, depths, 16, 4, 3)
        offs = isect_offset_encode(ids, 1, 4, 3)
        return rasterize_to_pixels(m2, conics, colors, opac, betas, 64, 48, 16, offs, fl)

    def ins(seed):
        s = projected_scene(200, 64, 48, seed=seed, device=DEV)
        return [s[k] for k in ("means2d", "conics", "colors", "opacities", "betas", "radii",
                               "depths")]

    first = [t.requires_grad_(True) if i < 5 else t for i, t in enumerate(ins(2))]
    _same(torch.jit.trace(f, tuple(first)), f, ins(5))


@pytest.mark.parametrize("grad", [False, True])
def test_traced_losses(grad):
    from ubs.loss import l1_loss, l1_ssim_loss
    g = torch.Generator().manual_seed(0)
    imgs = [torch.rand(1, 3, 40, 50, generator=g).to(DEV) for _ in range(4)]
    for f in (l1_loss, l1_ssim_loss):
        t = torch.jit.trace(lambda x, y, f=f: f(x, y) * 1.0,
                            (imgs[0].clone().requires_grad_(grad), imgs[1]))
        x, y = (imgs[2].clone().requires_grad_(grad) for _ in range(2))
        a, b = t(x, imgs[3]), f(y, imgs[3])
        assert torch.equal(a, b)
        if grad:
            a.backward()
            b.backward()
            torch.testing.assert_close(x.grad, y.grad, rtol=1e-6, atol=0)
