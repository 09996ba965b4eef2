"""Frames whose image the blend stores to pinned host memory (tiles of 16 pixels and
more; smaller ones are copied): bit-equal to the image in device memory over tile
sizes, ragged and odd images, several views, and the frame that is re-run because
its first capacity was too small."""
import pytest
import torch

import scenes as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _views(sizes, tile):
    from ubs.render import Views
    from ubs.scene import Camera
    g = torch.Generator().manual_seed(3)
    cams = [Camera(S.orbit_camera(g, 4.0), S.intrinsics(w * 0.8, w * 0.8, w / 2, h / 2), w, h)
            for w, h in sizes]
    return Views(cams, tile_size=tile, device=DEV)


@pytest.mark.parametrize("tile", [8, 16, 24, 32])
@pytest.mark.parametrize("sizes", [[(1, 1)], [(16, 16)], [(101, 67)], [(640, 479)],
                                   [(33, 50), (128, 31)]])
def test_host_image(tile, sizes):
    from ubs.render import Renderer
    p = {k: v.to(DEV) for k, v in S.beta_params(3000, 6, seed=tile).items()}
    views = _views(sizes, tile)
    bg = torch.rand(len(sizes), 3, generator=torch.Generator().manual_seed(1)).to(DEV)
    n = sum(w * h for w, h in sizes)
    want, want_a, want_l, _, _ = Renderer(dim=6, tile_size=tile).forward_raw(p, views, bg)
    r = Renderer(dim=6, tile_size=tile)
    for cap in (None, 64):  # the second frame overflows and is run again
        if cap:
            r.capacity = cap
        host = torch.full((3 * n,), -7.0).pin_memory()
        got, a, last, _, _ = r.forward_raw(p, views, bg, image=host)
        torch.cuda.synchronize()
        assert got.data_ptr() == host.data_ptr() and got.shape == (n, 3)
        assert torch.equal(got, want.cpu())
        assert torch.equal(a, want_a) and torch.equal(last, want_l)


def test_host_image_is_checked():
    from ubs.render import Renderer
    p = {k: v.to(DEV) for k, v in S.beta_params(100, 6, seed=1).items()}
    views = _views([(32, 32)], 16)
    bg = torch.zeros(1, 3, device=DEV)
    for bad in (torch.zeros(3 * 32 * 32), torch.zeros(10).pin_memory(),
                torch.zeros(3 * 32 * 32, device=DEV)):
        with pytest.raises(ValueError):
            Renderer(dim=6).forward_raw(p, views, bg, image=bad)
