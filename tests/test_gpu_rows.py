"""The per-primitive operators pass a block's rows (128 primitives) through shared
memory, and place the lower triangle's rest entries at compile time when the index
lists are the full row-major order.  Sizes around the block, every width, lists in
that order, permuted and partial, against the oracle.  The covariance is a sum of
at most D products in float32 on both sides and its gradient one of 2 D, so 1e-5
relative with 1e-6 of the largest value covers the rounding."""
import numpy as np
import pytest
import torch

import oracle as orc
from scenes import beta_params, rest_indices

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def npy(t):
    return t.detach().cpu().numpy()


def close(a, b, what):
    a, b = npy(a).astype(np.float64), np.asarray(b, np.float64)
    assert a.shape == b.shape
    scale = np.abs(b).max() if b.size else 0.0
    np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6 * scale, err_msg=what)


@pytest.mark.parametrize("spatial", [False, True])
@pytest.mark.parametrize("order", ["rows", "permuted", "partial"])
@pytest.mark.parametrize("D,n", [(4, 129), (6, 1), (6, 128), (6, 300), (7, 127), (8, 130)])
def test_covariance_rows(D, n, order, spatial):
    from gsplat.cuda._wrapper import rot_scale_l_triangle_to_covar
    p = beta_params(n, D, seed=D + n)
    ri, rj = rest_indices(D)
    if order == "permuted":
        k = torch.randperm(len(ri), generator=torch.Generator().manual_seed(1))
        ri, rj = ri[k], rj[k]
    elif order == "partial":
        ri, rj = ri[1:], rj[1:]
    lt = p["l_triangle"].to(DEV).requires_grad_(True)
    sc = torch.nn.functional.softplus(p["scale"]).to(DEV).requires_grad_(True)
    R = torch.tensor(orc.l_triangle_to_rotmat(npy(lt))).to(DEV).requires_grad_(True)
    cov = rot_scale_l_triangle_to_covar(R, sc, lt, ri.to(DEV), rj.to(DEV), spatial)
    args = [npy(t) for t in (R, sc, lt, ri, rj)]
    close(cov, orc.rot_scale_l_triangle_to_covar(*args, spatial), "covar")
    g = torch.randn(cov.shape, generator=torch.Generator().manual_seed(2))
    (cov * g.to(DEV)).sum().backward()
    want = orc.rot_scale_l_triangle_to_covar_bwd(*args, npy(g), spatial)
    for t, w, what in zip((R, sc, lt), want, ("v_rot", "v_scale", "v_l_triangle")):
        close(t.grad, w, what)


@pytest.mark.parametrize("n", [1, 127, 129])
@pytest.mark.parametrize("stride", [3, 15])
def test_rotation_rows(n, stride):
    from gsplat.cuda._wrapper import l_triangle_to_rotmat
    l = torch.randn(n, stride, generator=torch.Generator().manual_seed(n)).to(DEV)
    l.requires_grad_(True)
    R = l_triangle_to_rotmat(l[:, :3])
    np.testing.assert_array_equal(npy(R), orc.l_triangle_to_rotmat(npy(l)))
    g = torch.randn(R.shape, generator=torch.Generator().manual_seed(3)).to(DEV)
    R.backward(g)
    np.testing.assert_array_equal(npy(l.grad)[:, :3], orc.l_triangle_to_rotmat_bwd(npy(g)))
