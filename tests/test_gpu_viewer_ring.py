"""Two frames under way on one renderer (two threads) do not share a host
buffer, and a frame that fails leaves the last image alone."""
import numpy as np
import pytest
import torch

from scenes import beta_params
from ubs import scene as S

pytestmark = pytest.mark.gpu
DEV = "cuda"
W, H = 97, 63


def _setup(seed, mode="RGB"):
    from ubs.viewer import FrameRenderer, ViewState
    p = {k: v.to(DEV) for k, v in beta_params(800, 6, seed=0, log_scale_mu=-2.5).items()}
    cam = S.orbit_view(seed, 3.0, W, H, 90.0, 90.0)
    args = (p, torch.inverse(cam.viewmat.cpu()).numpy(), cam.K.cpu().numpy(), W, H)
    return FrameRenderer(dim=6), args, ViewState(render_mode=mode, backgrounds=(0, 0, 255))


@pytest.mark.parametrize("mode", ["RGB", "Depth"])
def test_interleaved_frames(monkeypatch, mode):
    frames, a, state = _setup(1, mode)
    _, b, _ = _setup(2, mode)
    want_a, want_b = (frames.render(*x, state, copy=True) for x in (a, b))
    assert not np.array_equal(want_a, want_b)
    inner, got = frames._frame, []

    def frame(*args, **kw):
        # the other frame starts and ends while this one is being prepared
        monkeypatch.setattr(frames, "_frame", inner)
        got.append(frames.render(*b, state))
        return inner(*args, **kw)

    monkeypatch.setattr(frames, "_frame", frame)
    got_a = frames.render(*a, state)
    assert np.array_equal(got_a, want_a)
    assert np.array_equal(got[0], want_b)


def test_failed_frame_leaves_the_last_image():
    frames, a, state = _setup(1)
    _, b, bad = _setup(2)
    want = frames.render(*a, state, copy=True)
    last = frames.render(*a, state)
    bad.render_mode = "none"
    for _ in range(3):
        with pytest.raises(ValueError):
            frames.render(*b, bad)
    frames.render(*b, state)
    assert np.array_equal(last, want)
