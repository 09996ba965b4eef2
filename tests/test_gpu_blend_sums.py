"""The backward blend's tensor-core reduction of a visit's sums, against the
FP64 oracle: every packed channel count and tile edge (tiles of 24 and 32 are
cut into 8- and 16-pixel squares), ragged images, grids below and above the
small-grid bound, and inputs that take the lane-exchange reduction instead
(negative beta, infinities and NaN)."""
import numpy as np
import pytest
import torch

import oracle as orc
from scenes import projected_scene
from test_gpu_ops import grad_close, npy

pytestmark = pytest.mark.gpu
DEV = "cuda"
NAMES = ("v_means2d", "v_conics", "v_colors", "v_opac", "v_betas")


def _scene(N, W, H, ts, channels, seed):
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles
    s = projected_scene(N, W, H, seed=seed, big_frac=0.05)
    g = torch.Generator().manual_seed(seed + 1)
    ins = [s["means2d"], s["conics"], torch.rand(1, N, channels, generator=g),
           # faint and with beta >= 1.5: no cancellation in 1 - alpha and no
           # pole of (1 - sigma)^(beta - 1), so FP32 is accurate throughout
           s["opacities"] * 0.1, s["betas"].clamp(min=1.5)]
    tw, th = (W + ts - 1) // ts, (H + ts - 1) // ts
    _, ids, fl = isect_tiles(s["means2d"].to(DEV), s["radii"].to(DEV), s["depths"].to(DEV), ts,
                             tw, th)
    offs = isect_offset_encode(ids, 1, tw, th)
    wc = torch.randn(1, H, W, channels, generator=g)
    wa = torch.randn(1, H, W, 1, generator=g)
    return ins, offs, fl, wc, wa


def _grads(ins, offs, fl, wc, wa, W, H, ts):
    from gsplat.cuda._wrapper import rasterize_to_pixels
    leaves = [t.to(DEV).requires_grad_(True) for t in ins]
    rc, ra = rasterize_to_pixels(*leaves, W, H, ts, offs, fl)
    torch.autograd.backward([rc, ra], [wc.to(DEV), wa.to(DEV)])
    return [npy(t.grad) for t in leaves]


def _oracle(ins, offs, fl, wc, wa, W, H, ts):
    x = [npy(t).astype(np.float64) for t in ins]
    _, oa, li = orc.rasterize_to_pixels(*x, W, H, ts, npy(offs), npy(fl), dtype=np.float64)
    return orc.rasterize_to_pixels_bwd(*x, W, H, ts, npy(offs), npy(fl), oa, li,
                                       npy(wc).astype(np.float64), npy(wa).astype(np.float64),
                                       dtype=np.float64)


# FP32 evaluates a pair to a few 1e-6 (log2 and exp2 are good to 2^-22, times
# an exponent of up to about 20); the split keeps 2^-22 of each value.
@pytest.mark.parametrize("channels", [1, 2, 3, 4])
@pytest.mark.parametrize("ts", [8, 16, 24, 32])
def test_visit_sums(channels, ts):
    W, H = 101, 67
    ins, offs, fl, wc, wa = _scene(500, W, H, ts, channels, seed=ts + channels)
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    for a, r, nm in zip(got, _oracle(ins, offs, fl, wc, wa, W, H, ts), NAMES):
        grad_close(a, r, nm, rel_l2=5e-5)


def test_visit_sums_large_grid():
    W, H, ts = 1009, 803, 16  # 3264 tiles
    ins, offs, fl, wc, wa = _scene(20000, W, H, ts, 3, seed=4)
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    for a, r, nm in zip(got, _oracle(ins, offs, fl, wc, wa, W, H, ts), NAMES):
        grad_close(a, r, nm, rel_l2=5e-5)


def test_negative_beta():
    W, H, ts = 101, 67, 16
    ins, offs, fl, wc, wa = _scene(500, W, H, ts, 3, seed=9)
    ins[4][0, ::50] = -0.25  # opacity (1 - sigma)^beta grows towards the edge
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    for a, r, nm in zip(got, _oracle(ins, offs, fl, wc, wa, W, H, ts), NAMES):
        grad_close(a, r, nm, rel_l2=1e-3)  # (1 - sigma)^(beta - 1) has a pole at the edge


@pytest.mark.parametrize("where", ["pixel", "colour"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_non_finite_values_stay_in_their_tiles(where, value):
    W, H, ts = 128, 96, 16
    ins, offs, fl, wc, wa = _scene(300, W, H, ts, 3, seed=21)
    clean = _grads(ins, offs, fl, wc, wa, W, H, ts)
    starts = np.append(npy(offs).reshape(-1), fl.numel())
    order = npy(fl)
    if where == "pixel":
        wc = wc.clone()
        wc[0, 40, 40, 1] = value
        bad_tiles = [40 // ts * (W // ts) + 40 // ts]
    else:
        g = int(order[starts[10]])  # a primitive of tile 10
        ins[2] = ins[2].clone()
        ins[2][0, g, 0] = value
        bad_tiles = [t for t in range(len(starts) - 1) if g in order[starts[t]:starts[t + 1]]]
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    touched = np.zeros(300, bool)
    for t in bad_tiles:
        touched[order[starts[t]:starts[t + 1]]] = True
    assert touched.any() and not touched.all()
    for a, b, nm in zip(got, clean, NAMES):
        assert np.isfinite(a[0, ~touched]).all()
        np.testing.assert_allclose(a[0, ~touched], b[0, ~touched], rtol=1e-4,
                                   atol=1e-5 * np.abs(b).max(), err_msg=nm)
    assert not all(np.isfinite(a).all() for a in got)
