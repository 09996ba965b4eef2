"""Colour rows of more than four channels: CTAs over 16x16- and 8x8-pixel squares
of a tile, entry rows per warp in the backward; gradients against the FP64 oracle
over tile sizes, ragged images and lists that overflow, and the tiles that stay
refused.  Tolerances as for the narrow rows (a visit's pairs are evaluated to a
few 1e-6; the dense scene's records lie behind hundreds of others)."""
import numpy as np
import pytest
import torch

from test_gpu_blend_sums import NAMES, _grads, _oracle, _scene
from test_gpu_ops import grad_close, npy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,ts", [(5, 8), (5, 16), (5, 24), (5, 32), (8, 32), (13, 16),
                                         (16, 24), (17, 8), (32, 8), (32, 16), (33, 16)])
def test_wide_rows(channels, ts):
    W, H = 101, 67
    ins, offs, fl, wc, wa = _scene(500, W, H, ts, channels, seed=ts + channels)
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    for a, r, nm in zip(got, _oracle(ins, offs, fl, wc, wa, W, H, ts), NAMES):
        grad_close(a, r, nm, rel_l2=5e-5)


@pytest.mark.parametrize("channels", [4, 8, 32])
def test_list_overflow(channels):
    # every record covers every 8x8 box and no pixel terminates: 128 visits per
    # warp and batch against 64 entry rows
    from test_gpu_ops import _blend_inputs
    N, W, H, ts = 1200, 64, 48, 16
    s, _, offs, fl = _blend_inputs(N, W, H, 1, seed=5, ts=ts, big_frac=1.0)
    assert np.diff(np.append(npy(offs).reshape(-1), fl.numel())).min() > 4 * 128
    g = torch.Generator().manual_seed(3)
    ins = [s["means2d"], s["conics"], torch.rand(1, N, channels, generator=g),
           s["opacities"] * 0.01, s["betas"]]
    wc = torch.randn(1, H, W, channels, generator=g)
    wa = torch.randn(1, H, W, 1, generator=g)
    got = _grads(ins, offs, fl, wc, wa, W, H, ts)
    for a, r, nm in zip(got, _oracle(ins, offs, fl, wc, wa, W, H, ts), NAMES):
        grad_close(a, r, nm, rel_l2=1e-3)


@pytest.mark.parametrize("channels,ts", [(16, 32), (32, 24), (32, 32)])
def test_refused_tiles(channels, ts):
    W, H = 64, 64
    ins, offs, fl, wc, wa = _scene(50, W, H, ts, channels, seed=1)
    with pytest.raises(RuntimeError, match="shared memory"):
        _grads(ins, offs, fl, wc, wa, W, H, ts)
