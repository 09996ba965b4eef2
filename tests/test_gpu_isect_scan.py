"""The drop-in intersection count scans up to 65,536 buckets with one launch (one
CTA up to 1024, else a cluster) that also reports the total to the host, more with
separate launches: bucket counts around those edges, several cameras and threads,
against the oracle, bit for bit; and the zeroed gradient arrays of the blend."""
import threading

import numpy as np
import pytest
import torch

import oracle as orc
from test_gpu_ops import npy

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(C, N, tw, th, ts, seed):
    g = torch.Generator().manual_seed(seed)
    m2 = torch.rand(C, N, 2, generator=g) * torch.tensor([tw * ts, th * ts])
    radii = torch.randint(0, 3 * ts, (C, N), generator=g, dtype=torch.int32)
    return m2, radii, torch.rand(C, N, generator=g) * 4 + 0.5


def _check(C, N, tw, th, ts, seed):
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles
    m2, radii, depths = _inputs(C, N, tw, th, ts, seed)
    tpg, ids, fl = isect_tiles(m2.to(DEV), radii.to(DEV), depths.to(DEV), ts, tw, th)
    tpg_o, ids_o, fl_o = orc.isect_tiles(npy(m2), npy(radii), npy(depths), ts, tw, th)
    np.testing.assert_array_equal(npy(tpg), tpg_o)
    np.testing.assert_array_equal(npy(ids), ids_o)
    np.testing.assert_array_equal(npy(fl), fl_o)
    np.testing.assert_array_equal(npy(isect_offset_encode(ids, C, tw, th)),
                                  orc.isect_offset_encode(ids_o, C, tw, th))


@pytest.mark.parametrize("C,tw,th", [(1, 1, 1), (1, 2, 1), (1, 32, 32), (1, 41, 25), (3, 33, 31),
                                     (1, 256, 256), (2, 182, 181), (1, 257, 256)])
def test_bucket_counts(C, tw, th):
    _check(C, 3000, tw, th, 16, tw)


def test_counts_of_concurrent_threads():
    errors = []

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for r in range(5):
                    _check(1, 500 + 100 * k, 8 + k, 7, 16, 10 * k + r)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors


@pytest.mark.parametrize("N,channels", [(1, 1), (3, 3), (1023, 5), (5000, 32)])
def test_untouched_gradients_are_zero(N, channels):
    # nothing visible: every gradient is what the zeroing left
    from gsplat.cuda._wrapper import rasterize_to_pixels
    g = torch.Generator().manual_seed(N)
    m2, _, _ = _inputs(1, N, 4, 4, 16, N)
    m2[0, 0] = 24.0
    fl = torch.zeros(1, dtype=torch.int32, device=DEV)  # primitive 0 in tile 5
    offs = (torch.arange(16, device=DEV) > 5).int().view(1, 4, 4)
    ins = [m2, torch.tensor([0.01, 0.0, 0.01]).expand(1, N, 3),
           torch.rand(1, N, channels, generator=g), torch.rand(1, N, generator=g),
           torch.full((1, N), 2.0)]
    leaves = [t.to(DEV).contiguous().requires_grad_(True) for t in ins]
    rc, ra = rasterize_to_pixels(*leaves, 64, 64, 16, offs, fl)
    (rc.sum() + ra.sum()).backward()
    for t in leaves:
        assert (t.grad[0, 1:] == 0).all() and torch.isfinite(t.grad).all()
    assert (leaves[2].grad[0, 0] != 0).all()
