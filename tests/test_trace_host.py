"""torch.jit.trace over calls whose work does not pass through the dispatcher:
each is recorded as a node that makes the call again (ubs._lib.op)."""
import types

import pytest
import torch

from ubs import _lib as L


class _Square(torch.autograd.Function):
    """x * x, computed where the dispatcher does not see it."""

    @staticmethod
    def forward(ctx, x):
        ctx.save_for_backward(x)
        out = torch.empty_like(x)
        out.numpy()[:] = x.numpy() ** 2
        return out

    @staticmethod
    def backward(ctx, g):
        return 2 * ctx.saved_tensors[0] * g


@pytest.fixture
def standin(monkeypatch):
    def pair(x, scale, y, flag):
        s = _Square.apply(x)
        return s * scale + y, (s > 1).to(torch.int32), None if flag else s.sum()

    mod = types.SimpleNamespace(square=_Square.apply, pair=pair,
                                table=lambda n: torch.full((n,), 2.0))
    monkeypatch.setattr(L, "_native", mod)
    return mod


@pytest.mark.parametrize("grad", [False, True])
def test_traced_operator_runs_on_new_inputs(standin, grad):
    f = torch.jit.trace(lambda x: L.op("square", x) + 1, (torch.rand(5, requires_grad=grad),))
    for seed in range(3):
        x = torch.rand(5, generator=torch.Generator().manual_seed(seed)).requires_grad_(grad)
        y = f(x)
        torch.testing.assert_close(y, x * x + 1, rtol=0, atol=1e-6)
        if grad:
            y.sum().backward()
            torch.testing.assert_close(x.grad, 2 * x.detach())
            with pytest.raises(RuntimeError):
                y.sum().backward()


@pytest.mark.parametrize("flag", [False, True])
def test_traced_operator_of_several_results(standin, flag):
    def f(x, y):
        a, b, c = L.op("pair", x, 3.0, y, flag)
        assert (c is None) == flag
        return (a, b) if flag else (a, b, c)

    x, y = torch.rand(4, requires_grad=True), torch.rand(4, requires_grad=True)
    t = torch.jit.trace(f, (x, y))
    x2, y2 = (torch.rand(4) * 2).requires_grad_(True), torch.rand(4, requires_grad=True)
    got, want = t(x2, y2), f(x2, y2)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and torch.equal(a, b)
    assert got[0].requires_grad and not got[1].requires_grad
    ga, gb = (torch.autograd.grad(o[0].sum() + (0 if flag else o[2]), (x2, y2)) for o in (got, want))
    for a, b in zip(ga, gb):
        torch.testing.assert_close(a, b)


def test_nothing_inside_is_recorded(standin):
    def f(x):
        return x * L.untraced("table", 3)

    t = torch.jit.trace(f, (torch.ones(3),))
    assert not L.tracing()
    assert "full" not in str(t.graph)
    assert torch.equal(t(torch.arange(3.0)), torch.tensor([0.0, 2.0, 4.0]))
