"""Autograd behaviour of the host path's nodes (csrc/host/native.cpp): what the
operators refuse (other types and devices, forward-mode derivatives, function
transforms, a second backward, inputs changed in between), saved-tensor hooks,
inputs that are not contiguous or need no gradient, and renders from several
threads on their own streams."""
import threading

import pytest
import torch

from scenes import beta_params, projected_scene

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _scene(n=400, seed=0, dim=6):
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(n, dim, seed=seed, log_scale_mu=-2.5).items()}
    cam = S.orbit_view(seed + 1, 3.0, 70, 50, 60.0, 60.0, timestamp=0.3, device=DEV)
    return p, Views([cam], device=DEV), Renderer(dim=dim)


def _raster_inputs(n=200, W=64, H=48):
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles
    s = projected_scene(n, W, H, seed=2, device=DEV)
    _, ids, fl = isect_tiles(s["means2d"], s["radii"], s["depths"], 16, 4, 3)
    leaves = [s[k].requires_grad_(True) for k in ("means2d", "conics", "colors", "opacities",
                                                  "betas")]
    return leaves, (W, H, 16, isect_offset_encode(ids, 1, 4, 3), fl)


def test_second_backward_is_refused():
    from gsplat.cuda._wrapper import rasterize_to_pixels
    p, views, r = _scene()
    p["rgb"].requires_grad_(True)
    leaves, rest = _raster_inputs()
    for out in (r.render(p, views)[0].sum(), rasterize_to_pixels(*leaves, *rest)[0].sum()):
        out.backward(retain_graph=True)
        with pytest.raises(RuntimeError, match="released"):
            out.backward()


def test_other_types_and_devices_are_refused():
    from gsplat.cuda._wrapper import l_triangle_to_rotmat, rasterize_to_pixels
    from ubs.loss import l1_loss
    p, views, r = _scene()
    with pytest.raises(TypeError):
        r.render(dict(p, rgb=p["rgb"].double()), views)
    with pytest.raises(ValueError):
        r.render(dict(p, rgb=p["rgb"].cpu()), views)
    with pytest.raises(TypeError):
        l_triangle_to_rotmat(p["l_triangle"][:, :3].half())
    with pytest.raises(TypeError):
        l1_loss(p["rgb"].cpu(), p["rgb"].cpu())
    leaves, rest = _raster_inputs()
    with pytest.raises(TypeError):
        rasterize_to_pixels(*leaves[:3], leaves[3].double(), leaves[4], *rest)


def test_forward_mode_and_transforms_are_refused():
    from gsplat.cuda._wrapper import l_triangle_to_rotmat
    import torch.autograd.forward_ad as fwAD
    l = torch.randn(8, 3, device=DEV)
    with fwAD.dual_level():
        with pytest.raises(NotImplementedError):
            l_triangle_to_rotmat(fwAD.make_dual(l, torch.ones_like(l)))
    with pytest.raises(RuntimeError):
        torch.func.vmap(l_triangle_to_rotmat)(l[None])
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda x: l_triangle_to_rotmat(x).sum())(l)


def test_change_between_forward_and_backward_is_detected():
    p, views, r = _scene()
    p["scale"].requires_grad_(True)
    out = r.render(p, views)[0].sum()
    with torch.no_grad():
        p["scale"].add_(0.1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward()


@pytest.mark.parametrize("dim", [6, 7])
def test_hooks_partial_gradients_and_strides(dim):
    p, views, r = _scene(dim=dim)
    ref = {k: v.clone().requires_grad_(True) for k, v in p.items()}
    w = torch.rand(views.n_pixels, 3, generator=torch.Generator().manual_seed(0)).to(DEV)
    (r.render(ref, views)[0] * w).sum().backward()
    # saved-tensor hooks see what the node keeps; only two inputs need gradients,
    # one of them is stored transposed
    packed = []
    x = dict(p)
    x["scale"] = p["scale"].t().contiguous().t().requires_grad_(True)
    x["opacity"] = p["opacity"].clone().requires_grad_(True)
    assert not x["scale"].is_contiguous()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(),
                                                  lambda t: t.to(DEV)):
        colors, alphas = r.render(x, views)
        loss = (colors * w).sum()
    assert len(packed) >= 9
    loss.backward()
    for k in ("scale", "opacity"):
        assert x[k].grad.shape == x[k].shape
        torch.testing.assert_close(x[k].grad, ref[k].grad, rtol=1e-4, atol=1e-6)
    assert x["xyz"].grad is None
    with torch.no_grad():
        assert r.render(x, views)[0].grad_fn is None


def test_alpha_only_gradient():
    p, views, r = _scene()
    x = {k: v.requires_grad_(True) for k, v in p.items()}
    r.render(x, views)[1].sum().backward()
    assert float(x["rgb"].grad.abs().max()) == 0.0
    assert float(x["opacity"].grad.abs().max()) > 0.0


def test_threads_on_their_own_streams():
    scenes = [_scene(n=300 + 100 * i, seed=i) for i in range(4)]
    want = []
    for p, views, r in scenes:
        x = {k: v.clone().requires_grad_(True) for k, v in p.items()}
        c, _ = r.render(x, views)
        c.sum().backward()
        want.append((c.detach().clone(), x["xyz"].grad.clone()))
    torch.cuda.synchronize()
    got, errors = [None] * 4, []

    def work(i):
        try:
            p, views, r = scenes[i]
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for _ in range(5):
                    x = {k: v.clone().requires_grad_(True) for k, v in p.items()}
                    c, _ = r.render(x, views)
                    c.sum().backward()
            st.synchronize()
            got[i] = (c.detach(), x["xyz"].grad)
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join(60) for t in threads]
    assert not errors, errors
    for (c, g), (wc, wg) in zip(got, want):
        assert torch.equal(c, wc)
        torch.testing.assert_close(g, wg, rtol=1e-4, atol=1e-6)
