"""Backward of the losses: the stored gradient times the incoming scalar, as one
kernel over dense tensors (whole quads, remainders, one value, unaligned views)
and as a general product where the gradient is differentiated, batched or taken
from a saved-tensor hook.  One product per value: bit-equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _sign_grad(x, y):
    return torch.sign(x - y) * torch.tensor(1.0 / x.numel(), dtype=torch.float32)


@pytest.mark.parametrize("shape", [(1,), (3,), (4,), (5, 3), (2, 33, 65, 3), (1, 300, 401, 3)])
@pytest.mark.parametrize("factor", [1.0, -0.37, float("inf")])
def test_scaled_gradient(shape, factor):
    from ubs.loss import l1_loss
    g = torch.Generator().manual_seed(len(shape))
    x, y = (torch.rand(shape, generator=g).to(DEV) for _ in range(2))
    x.requires_grad_(True)
    loss = l1_loss(x, y)
    loss.backward(torch.tensor(factor, device=DEV))
    torch.testing.assert_close(x.grad, _sign_grad(x.detach(), y) * factor, rtol=0, atol=0,
                               equal_nan=True)


def test_kernel_on_unaligned_values():
    from ubs import _lib as L
    x = torch.rand(1031, device=DEV)
    by = torch.tensor(3.25, device=DEV)
    for a, b in ((0, 0), (1, 0), (0, 1), (3, 3)):
        n = 1024 if a or b else 1031
        out = torch.full((1031,), -1.0, device=DEV)
        L.call("ubs_scale", L.ptr(x[a:]), L.ptr(by), L.ptr(out[b:]), n,
               torch.cuda.current_stream().cuda_stream)
        assert torch.equal(out[b:b + n], x[a:a + n] * by)
        assert (out[b + n:] == -1).all() and (out[:b] == -1).all()


def test_general_products():
    from ubs.loss import l1_loss
    x, y = torch.rand(7, 9, device=DEV), torch.rand(7, 9, device=DEV)
    x.requires_grad_(True)
    want = _sign_grad(x.detach(), y)
    go = torch.tensor(2.0, device=DEV, requires_grad=True)
    gx, = torch.autograd.grad(l1_loss(x, y), x, go, create_graph=True)
    ggo, = torch.autograd.grad(gx.sum(), go)
    torch.testing.assert_close(ggo, want.sum())
    many = torch.arange(3.0, device=DEV)
    gx, = torch.autograd.grad(l1_loss(x, y), x, many, is_grads_batched=True)
    torch.testing.assert_close(gx, want * many[:, None, None])
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.double(), lambda t: t.float()):
        loss = l1_loss(x, y)
    gx, = torch.autograd.grad(loss, x)
    torch.testing.assert_close(gx, want)
