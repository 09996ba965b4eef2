"""The reference's training loss in two kernel launches (csrc/ssim.cu).

train.py:117-121 trains on  (1 - l) L1(image, gt) + l (1 - SSIM(image, gt))
(l = lambda_dssim, 0.2) with SSIM from the fused_ssim package, which
evaluates utils/loss_utils.py:26-80's definition.  `l1_ssim_loss` computes
that loss and writes d loss / d image in the same launches (the backward
pass only scales it by the incoming gradient); `ssim` is the SSIM term
alone and `l1_loss` the L1 term alone (utils/loss_utils.py:18-19), one
launch with its gradient.

Images may be laid out as [..., C, H, W] or, with channels_last=True, as
[..., H, W, C] (the renderer's layout) with any strides: nothing is copied.
"""
import torch

from . import _lib as L

_W_SSIM_ONLY = (0.0, 1.0, 0.0)


def _check(img, gt, channels_last):
    if not (img.is_cuda and gt.is_cuda):
        raise TypeError("the loss kernel needs CUDA tensors")
    if img.dtype != torch.float32 or gt.dtype != torch.float32:
        raise TypeError("the loss kernel handles float32 images")
    if img.shape != gt.shape:
        raise ValueError("image and target shapes differ: %s vs %s"
                         % (tuple(img.shape), tuple(gt.shape)))
    if img.dim() not in (3, 4):
        raise ValueError("expected [C, H, W] / [N, C, H, W] images (or the channels-last "
                         "forms), got %s" % (tuple(img.shape),))


def _apply(img, gt, channels_last, valid, weights, index):
    _check(img, gt, channels_last)
    return L.op("ssim_loss", img, gt.detach(), channels_last, valid, *weights, index)


def l1_ssim_loss(img, gt, lambda_dssim=0.2, channels_last=False, padding="same"):
    """(1 - lambda_dssim) mean|img - gt| + lambda_dssim (1 - SSIM(img, gt)),
    train.py:117-121's loss, as a 0-dim tensor differentiable w.r.t. img."""
    if padding not in ("same", "valid"):
        raise ValueError("padding must be 'same' or 'valid'")
    lam = float(lambda_dssim)
    return _apply(img, gt, channels_last, padding == "valid", (1.0 - lam, -lam, lam), 2)


def ssim(img, gt, channels_last=False, padding="same"):
    """Mean SSIM of img against gt (utils/loss_utils.py:45-80 with size_average),
    differentiable w.r.t. img."""
    if padding not in ("same", "valid"):
        raise ValueError("padding must be 'same' or 'valid'")
    return _apply(img, gt, channels_last, padding == "valid", _W_SSIM_ONLY, 0)


def l1_loss(img, gt):
    """mean |img - gt| (utils/loss_utils.py:18-19) of two contiguous float32
    CUDA tensors of one shape, differentiable w.r.t. img; one launch writes
    the value and the gradient."""
    if not (img.is_cuda and gt.is_cuda) or img.dtype != torch.float32 or \
            gt.dtype != torch.float32:
        raise TypeError("l1_loss needs float32 CUDA tensors")
    if img.shape != gt.shape:
        raise ValueError("shapes differ: %s vs %s" % (tuple(img.shape), tuple(gt.shape)))
    if not (img.is_contiguous() and gt.is_contiguous()):
        raise ValueError("l1_loss needs contiguous tensors")
    return L.op("l1_loss", img, gt.detach())
