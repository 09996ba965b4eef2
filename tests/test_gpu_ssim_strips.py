"""SSIM strips: a warp takes 64 columns and a number of rows that depends on the
image.  Widths around the strip, heights of less than the window, of one strip
and of several, both layouts, against conv2d in float64.  The windowed sums are
float32 over 121 taps (relative error about 1e-6); the variance's cancellation
against C2 = 9e-4 raises it by at most 1 / C2 ~ 1e3 times the squared mean, so 2e-4 of
the largest gradient and 1e-5 of the loss bound it for images in [0, 1]."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ssim64(x, y, valid):
    C = x.shape[1]
    g = torch.exp(-(torch.arange(11, device=x.device).double() - 5) ** 2 / 4.5)
    k = (g[:, None] * g[None] / g.sum() ** 2).expand(C, 1, 11, 11)

    def f(t):
        return F.conv2d(t, k, padding=5, groups=C)
    mx, my = f(x), f(y)
    vx, vy, cxy = f(x * x) - mx * mx, f(y * y) - my * my, f(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    m = ((2 * mx * my + c1) * (2 * cxy + c2)) / ((mx * mx + my * my + c1) * (vx + vy + c2))
    return (m[..., 5:-5, 5:-5] if valid else m).mean()


@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("n,c,h,w", [(1, 1, 1, 1), (1, 3, 4, 63), (1, 3, 11, 64), (2, 3, 29, 65),
                                     (1, 3, 300, 129), (1, 1, 700, 3), (3, 4, 121, 203)])
def test_strips(n, c, h, w, channels_last):
    from fused_ssim import fused_ssim
    gen = torch.Generator().manual_seed(h * w)
    x, y = (torch.rand(n, c, h, w, generator=gen).to(DEV) for _ in range(2))
    if channels_last:
        x, y = (t.permute(0, 2, 3, 1).contiguous().permute(0, 3, 1, 2) for t in (x, y))
    for padding in ["same"] + (["valid"] if h > 10 and w > 10 else []):
        a = x.clone().requires_grad_(True)
        v = fused_ssim(a, y, padding=padding)
        v.backward()
        b = x.double().requires_grad_(True)
        r = ssim64(b, y.double(), padding == "valid")
        r.backward()
        assert abs(v.item() - r.item()) <= 1e-5
        assert (a.grad - b.grad).abs().max() <= 2e-4 * b.grad.abs().max()
