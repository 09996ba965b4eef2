"""The per-primitive kernels loop over views inside a thread; with few
primitives the views are split into groups that add their gradients.  Batched
renders against the same views one at a time, at one view, one group, several
groups and primitive counts around a warp's and a block's edge."""
import pytest
import torch

from scenes import beta_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 59,000 primitives fill the backward's CTAs (one group), fewer are split
@pytest.mark.parametrize("n,dim,views", [(1, 6, 2), (31, 7, 3), (129, 6, 1), (1000, 7, 5),
                                         (30_000, 6, 3), (59_000, 7, 2)])
def test_batched_views_match_single_views(n, dim, views):
    from ubs import scene as S
    from ubs.render import Renderer, Views
    p = {k: v.to(DEV) for k, v in beta_params(n, dim, seed=n, log_scale_mu=-3.0).items()}
    cams = [S.orbit_view(i, 3.0, 60 + 7 * i, 44 + i, 50.0, 50.0, timestamp=0.2 * i, device=DEV)
            for i in range(views)]
    g = torch.Generator().manual_seed(n)
    w = [torch.rand(c.width * c.height, 3, generator=g).to(DEV) for c in cams]

    def grads(groups):
        x = {k: v.clone().requires_grad_(True) for k, v in p.items()}
        images = []
        for ids in groups:
            colors, _ = Renderer(dim=dim).render(x, Views([cams[i] for i in ids], device=DEV))
            (colors * torch.cat([w[i] for i in ids])).sum().backward()
            images.append(colors.detach())
        return torch.cat(images), {k: v.grad for k, v in x.items()}

    one, g1 = grads([[i] for i in range(views)])
    all_, ga = grads([list(range(views))])
    assert torch.equal(one, all_)  # the forward does not depend on the batch
    for k in g1:
        # sums over views and of atomics in another order
        scale = float(g1[k].abs().max())
        torch.testing.assert_close(ga[k], g1[k], rtol=1e-3, atol=2e-5 * scale + 1e-12)
