"""As many views in one call as a call takes: more than a grid has rows."""
import pytest
import torch

from scenes import beta_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("count", [65_535, 65_536])
def test_one_primitive_in_many_views(count):
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(1, 6, seed=3, log_scale_mu=-1.5).items()}
    p["xyz"].zero_()
    cams = [S.orbit_view(1, 3.0, 8, 8, 8.0, 8.0), S.orbit_view(2, 3.0, 8, 8, 8.0, 8.0)]
    small = Views(cams, tile_size=8, device=DEV)
    # the second camera is the last view alone
    many = Views([cams[0]] * (count - 1) + [cams[1]], tile_size=8, device=DEV)
    w = torch.rand(8, 8, 3, generator=torch.Generator().manual_seed(0)).to(DEV)

    def run(views, counts):
        x = {k: v.clone().requires_grad_(True) for k, v in p.items()}
        colors, _ = Renderer(dim=6, tile_size=8).render(x, views)
        images = colors.view(-1, 8, 8, 3)
        first = (images[:-1] * w).sum() / counts
        (first + (images[-1] * w).sum()).backward()
        return images.detach(), {k: v.grad for k, v in x.items()}

    a, ga = run(small, 1)
    b, gb = run(many, count - 1)
    assert float(a.abs().max()) > 0
    assert torch.equal(b[:-1], a[:1].expand(count - 1, 8, 8, 3)) and torch.equal(b[-1], a[1])
    for k in ga:  # sums of 65,535 equal terms, each weighted by their inverse count
        torch.testing.assert_close(gb[k], ga[k], rtol=2e-3, atol=1e-6)
