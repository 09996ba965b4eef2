"""The per-bucket sort on 32-bit composites against numpy's sort of the 64-bit
keys: bucket sizes around every size class, and depths that the composites
cannot separate (all equal, a few distinct values, neighbours in the last place
beside outliers, as they come and reversed)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = [1, 2, 31, 33, 64, 65, 127, 300, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 3000,
         4095, 4096, 4097, 9000, 20000]


def _depths(kind, n, rng):
    if kind == "random":
        return rng.uniform(2.0, 6.0, n)
    if kind == "equal":
        return np.full(n, 3.25)
    if kind == "few":
        return rng.choice([2.5, 2.75, 2.7500002, 40.0, 1e6], n)
    if kind == "two":
        return np.where(np.arange(n) % 2, 4.0, 3.0)
    # neighbours in the last place and one far outlier: all share the bits kept
    d = np.float32(3.0) + np.arange(n, dtype=np.float32) * np.float32(2.4e-7)
    d[-1] = 1e30
    return d[::-1] if kind == "reversed" else d


@pytest.mark.parametrize("kind", ["random", "equal", "few", "two", "ulps", "reversed"])
def test_sort_matches_numpy(kind):
    from gsplat.cuda._wrapper import isect_tiles
    rng = np.random.default_rng(0)
    # one 16x16 tile per size: primitives of radius 1 at the tile's middle
    means, depths = [], []
    for i, n in enumerate(SIZES):
        means.append(np.stack([np.full(n, 16 * i + 8.0), np.full(n, 8.0)], 1))
        depths.append(_depths(kind, n, rng))
    m, d = np.concatenate(means), np.concatenate(depths).astype(np.float32)
    order = rng.permutation(len(d))
    m, d = m[order], d[order]
    m2 = torch.tensor(m, dtype=torch.float32, device=DEV)[None]
    dd = torch.tensor(d, device=DEV)[None]
    radii = torch.ones(1, len(d), dtype=torch.int32, device=DEV)
    _, ids, flat = isect_tiles(m2, radii, dd, 16, len(SIZES), 1)
    tile = (m[:, 0] // 16).astype(np.int64)
    want = np.lexsort((np.arange(len(d)), d.view(np.int32), tile))
    np.testing.assert_array_equal(flat.cpu().numpy(), want)
    keys = (tile[want] << 32) | d.view(np.int32)[want].astype(np.int64)
    np.testing.assert_array_equal(ids.cpu().numpy(), keys)
