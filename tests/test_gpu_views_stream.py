"""Camera tables built for a side stream: the cameras' tensors are read in the
order of the stream they were made on, the upload runs on the given one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("center", [False, True])
def test_cameras_made_on_the_current_stream(center):
    from ubs import scene as S
    from ubs.render import Views
    cam = S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0, device=DEV)
    want = Views([cam], device=DEV)
    vm, K = torch.zeros(4, 4, device=DEV), torch.zeros(3, 3, device=DEV)
    pos = torch.zeros(3, device=DEV)
    late = S.Camera(vm, K, 70, 50, cam.timestamp, position=pos if center else None)
    side, x = torch.cuda.Stream(), torch.rand(4096, 4096, device=DEV)
    torch.cuda.synchronize()
    for _ in range(20):  # some milliseconds of work in front of the values
        x = x @ x * 1e-4
    vm.copy_(cam.viewmat)
    K.copy_(cam.K)
    pos.copy_(want.centers[0])
    views = Views([late], device=DEV, stream=side)
    side.synchronize()
    for name in ("viewmats", "intr", "centers", "times", "dims", "tile_base", "pix_base"):
        assert torch.equal(getattr(views, name), getattr(want, name)), name


def test_upload_is_on_the_given_stream():
    from ubs import scene as S
    from ubs.render import Views
    cam = S.orbit_view(1, 3.0, 70, 50, 60.0, 60.0)  # on the host
    want = Views([cam], device=DEV)
    side, x = torch.cuda.Stream(), torch.rand(4096, 4096, device=DEV)
    torch.cuda.synchronize()
    for _ in range(200):
        x = x @ x * 1e-4
    views = Views([cam], device=DEV, stream=side)
    with torch.cuda.stream(side):
        got = views.viewmats.cpu()
    assert not torch.cuda.current_stream().query()  # the current stream was not waited for
    torch.cuda.synchronize()
    assert torch.equal(got, want.viewmats.cpu())
