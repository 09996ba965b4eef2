"""Position noise from draws that round to 1 in single precision: finite."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
M64 = (1 << 64) - 1


def _bits(seed, i):
    """The top 53 bits of draw i of the library's counter-based generator."""
    z = (seed + (i + 1) * 0x9e3779b97f4a7c15) & M64
    z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
    z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
    return (z ^ (z >> 31)) >> 11


# (seed, primitive, pair of draws): found by running the generator over 200 seeds
@pytest.mark.parametrize("seed, prim, pair", [(85, 190153, 1), (38, 354185, 1), (135, 675486, 0)])
def test_noise_is_finite(monkeypatch, seed, prim, pair):
    from ubs import mcmc
    assert _bits(seed, 4 * prim + 2 * pair) >= (1 << 53) - (1 << 28)  # rounds to 1.0
    n = prim + 1
    m = types.SimpleNamespace(
        _xyz=torch.zeros(n, 3, device=DEV), _opacity=torch.full((n, 1), -30.0, device=DEV),
        _scale=torch.zeros(n, 6, device=DEV), _l_triangle=torch.zeros(n, 15, device=DEV))
    monkeypatch.setattr(mcmc, "_seed", lambda generator: seed)
    mcmc.perturb_xyz(m, 1.0)
    assert bool(torch.isfinite(m._xyz).all())
    # the largest radius of Box-Muller from 24 bits: sqrt(2 ln 2^24) sigma^2
    assert float(m._xyz.abs().max()) <= 5.77 * 0.6931472 ** 2 * 1.001
