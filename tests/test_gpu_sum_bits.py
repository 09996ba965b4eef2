"""The backward blend sums a record's per-pixel values with all their 24 bits:
one pixel carries a colour gradient whose last bits would be lost in a shorter
format, every other one carries none, so the sum is that value."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("channels", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ts", [8, 16, 32])
def test_one_value_survives_its_sum(channels, ts):
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles, rasterize_to_pixels
    W = H = 32
    t = (W + ts - 1) // ts
    m2 = torch.tensor([[[16.0, 16.0]]], device=DEV)
    conics = torch.tensor([[[1e-3, 0.0, 1e-3]]], device=DEV)
    opac, betas = torch.full((1, 1), 0.5, device=DEV), torch.zeros(1, 1, device=DEV)
    colors = torch.ones(1, 1, channels, device=DEV, requires_grad=True)
    _, ids, fl = isect_tiles(m2, torch.full((1, 1), 32, dtype=torch.int32, device=DEV),
                             torch.ones(1, 1, device=DEV), ts, t, t)
    img, _ = rasterize_to_pixels(m2, conics, colors, opac, betas, W, H, ts,
                                 isect_offset_encode(ids, 1, t, t), fl)
    # (1 - sigma)^0 = 1: alpha is 0.5 and the colour gradient 0.5 v; 13 bits of v
    # lie below its leading 11
    v = torch.zeros_like(img)
    want = torch.zeros(channels)
    for k in range(channels):
        v[0, 5 + 6 * (k % 4), 9 + 3 * k, k] = 1 + 2.0 ** -11 + (3 - k % 2 * 2) * 2.0 ** -23
        want[k] = 0.5 * v[0, ..., k].max().item()
    img.backward(v)
    # one unit in the last place of 0.5 v, for the reciprocal of 1 - alpha
    assert (colors.grad.cpu()[0, 0] - want).abs().max() <= 2.0 ** -24
