"""Drop-in replacement of the reference's gsplat.cuda._wrapper for the Universal
Beta Splatting rasteriser path, running the GB300 kernels of libubs_gb300.so.

Function names, argument meaning, shapes and autograd behaviour follow
submodules/gsplat/cuda/_wrapper.py of the reference.  Every compute call goes
through the C ABI (include/ubs.h); there is no CPU or PyTorch fallback.  The
argument checks are here, allocation, calls and autograd nodes in
csrc/host/native.cpp.

Operators the reference defines but the UBS path never calls
(quat_scale_to_covar_preci, proj, world_to_cam, rasterize_to_indices_in_range)
raise NotImplementedError.
"""
import os
from typing import Optional, Tuple

import torch
from torch import Tensor

from ubs import _lib as L

# Conditioning backward: "reference" reproduces the reference CUDA backward
# (cond_mean_convariance_opacity_bwd.cu), including its transposed Cholesky
# factor; "exact" returns the true gradient of the forward.  The mode in effect
# when the forward runs is the one its backward uses.
_COND_GRAD_MODE = os.environ.get("UBS_COND_GRAD", "reference")

# channel counts with a dedicated kernel; others are padded (as the reference
# does, _wrapper.py:419-464) or split into 32-channel chunks above 33
_NATIVE_CHANNELS = (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33)


def set_cond_grad_mode(mode: str) -> None:
    global _COND_GRAD_MODE
    if mode not in ("reference", "exact"):
        raise ValueError("cond grad mode must be 'reference' or 'exact'")
    _COND_GRAD_MODE = mode


def get_cond_grad_mode() -> str:
    return _COND_GRAD_MODE


# --------------------------------------------------------------------- a4
def cond_mean_convariance_opacity(
    means: Tensor,  # [N, D]
    covars: Tensor,  # [N, D, D]
    opacities: Tensor,  # [N, 1]
    betas: Tensor,  # [N, D-3]
    query: Tensor,  # [N, D-3]
) -> Tuple[Tensor, Tensor, Tensor]:
    """Condition mean, covariance and opacity on a query (_wrapper.py:18-31)."""
    N, D = means.shape
    assert covars.shape == (N, D, D), covars.shape
    assert opacities.numel() == N and betas.shape == (N, D - 3) and query.shape == (N, D - 3)
    # the mode at forward time applies
    return L.op("cond", means, covars, opacities, betas, query, _COND_GRAD_MODE == "exact")


# --------------------------------------------------------------------- a2
def l_triangle_to_rotmat(l_triangle: Tensor) -> Tensor:
    """R = I + A from the 3 skew entries (_wrapper.py:34-36)."""
    assert l_triangle.shape[1] == 3, l_triangle.shape
    return L.op("rotmat", l_triangle)


# --------------------------------------------------------------------- a3
def rot_scale_l_triangle_to_covar(
    rot: Tensor,  # [N, 3, 3]
    scale: Tensor,  # [N, D]
    l_triangle: Tensor,  # [N, D*(D-1)//2]
    rest_i: Tensor,
    rest_j: Tensor,
    spatial_block: bool = False,
) -> Tensor:
    """Sigma = L L^T (_wrapper.py:39-55)."""
    return L.op("covar", rot, scale, l_triangle, rest_i, rest_j, bool(spatial_block))


# --------------------------------------------------------------------- a6
def fully_fused_projection(
    means: Tensor,  # [N, 3]
    covars: Optional[Tensor],  # [N, 6] or None
    quats: Optional[Tensor],  # [N, 4] or None
    scales: Optional[Tensor],  # [N, 3] or None
    viewmats: Tensor,  # [C, 4, 4]
    Ks: Tensor,  # [C, 3, 3]
    width: int,
    height: int,
    eps2d: float = 0.3,
    near_plane: float = 0.01,
    far_plane: float = 1e10,
    radius_clip: float = 0.0,
    sparse_grad: bool = False,
    calc_compensations: bool = False,
    ortho: bool = False,
) -> Tuple[Tensor, Tensor, Tensor, Tensor, Tensor]:
    """Projects primitives to 2D (_wrapper.py:185-282).

    Returns radii [C,N] int32, means2d [C,N,2], depths [C,N], conics [C,N,3],
    compensations [C,N] or None.  Culled entries have radius 0 and zeros.
    """
    C = viewmats.size(0)
    N = means.size(0)
    assert means.size() == (N, 3), means.size()
    assert viewmats.size() == (C, 4, 4), viewmats.size()
    assert Ks.size() == (C, 3, 3), Ks.size()
    if ortho:
        raise NotImplementedError("orthographic projection is not on the UBS path")
    if covars is not None:
        assert covars.size() in ((N, 6), (N, 3, 3)), covars.size()
    else:
        assert quats is not None and scales is not None, "covars or quats+scales is required"
        assert quats.size() == (N, 4) and scales.size() == (N, 3)
    return L.op("projection", means, covars, quats, scales, viewmats, Ks, int(width), int(height),
                float(eps2d), float(near_plane), float(far_plane), float(radius_clip),
                bool(calc_compensations))


# --------------------------------------------------------------- a7 / a8
def _isect(means2d, radii, depths, tile_size, tile_width, tile_height, sort=True):
    """Intersections plus the (camera, tile) offsets the count step yields."""
    return L.op("isect", means2d, radii, depths, int(tile_size), int(tile_width), int(tile_height),
                bool(sort))


@torch.no_grad()
def isect_tiles(
    means2d: Tensor,  # [C, N, 2]
    radii: Tensor,  # [C, N]
    depths: Tensor,  # [C, N]
    tile_size: int,
    tile_width: int,
    tile_height: int,
    sort: bool = True,
    n_cameras: Optional[int] = None,
    camera_ids: Optional[Tensor] = None,
    primitive_ids: Optional[Tensor] = None,
) -> Tuple[Tensor, Tensor, Tensor]:
    """Maps projected primitives to intersecting tiles (_wrapper.py:286-343).

    Returns tiles_per_gauss [C,N] int32, isect_ids [n_isects] int64
    (camera | tile | depth bits) and flatten_ids [n_isects] int32.
    """
    if camera_ids is not None or primitive_ids is not None:
        raise NotImplementedError("packed intersection input is not on the UBS path")
    C, N, _ = means2d.shape
    assert means2d.shape == (C, N, 2), means2d.size()
    assert radii.shape == (C, N), radii.size()
    assert depths.shape == (C, N), depths.size()
    tpg, ids, fl, _ = _isect(means2d, radii, depths, tile_size, tile_width, tile_height, sort)
    return tpg, ids, fl


@torch.no_grad()
def isect_offset_encode(isect_ids: Tensor, n_cameras: int, tile_width: int,
                        tile_height: int) -> Tensor:
    """First sorted intersection of every (camera, tile) (_wrapper.py:347-363)."""
    return L.op("offset_encode", isect_ids, int(n_cameras), int(tile_width), int(tile_height))


# ------------------------------------------------------------ a9 / a10
def rasterize_to_pixels(
    means2d: Tensor,  # [C, N, 2]
    conics: Tensor,  # [C, N, 3]
    colors: Tensor,  # [C, N, channels]
    opacities: Tensor,  # [C, N]
    betas: Tensor,  # [C, N]
    image_width: int,
    image_height: int,
    tile_size: int,
    isect_offsets: Tensor,  # [C, tile_height, tile_width]
    flatten_ids: Tensor,  # [n_isects]
    backgrounds: Optional[Tensor] = None,  # [C, channels]
    masks: Optional[Tensor] = None,  # [C, tile_height, tile_width]
) -> Tuple[Tensor, Tensor]:
    """Front-to-back Beta-kernel blend (_wrapper.py:366-491).

    Returns render_colors [C,H,W,channels] and render_alphas [C,H,W,1].
    """
    C = isect_offsets.size(0)
    device = means2d.device
    N = means2d.size(1)
    assert means2d.shape == (C, N, 2), means2d.shape
    assert conics.shape == (C, N, 3), conics.shape
    assert colors.shape[:2] == (C, N), colors.shape
    assert opacities.shape == (C, N), opacities.shape
    assert betas.shape == (C, N), betas.shape
    if backgrounds is not None:
        assert backgrounds.shape == (C, colors.shape[-1]), backgrounds.shape
    if masks is not None:
        assert masks.shape == isect_offsets.shape, masks.shape
    channels = colors.shape[-1]
    if channels > 513 or channels == 0:
        raise ValueError(f"Unsupported number of color channels: {channels}")
    tile_height, tile_width = isect_offsets.shape[1:3]
    assert tile_height * tile_size >= image_height, \
        f"Assert Failed: {tile_height} * {tile_size} >= {image_height}"
    assert tile_width * tile_size >= image_width, \
        f"Assert Failed: {tile_width} * {tile_size} >= {image_width}"

    if channels > 33:
        # 32-channel chunks; alphas are identical across chunks and only the
        # first chunk's alphas are returned, so the gradient is unchanged
        outs, alphas = [], None
        for s in range(0, channels, 32):
            cc = colors[..., s:s + 32]
            bb = backgrounds[..., s:s + 32] if backgrounds is not None else None
            o, a = rasterize_to_pixels(means2d, conics, cc, opacities, betas, image_width,
                                       image_height, tile_size, isect_offsets, flatten_ids, bb,
                                       masks)
            outs.append(o)
            alphas = a if alphas is None else alphas
        return torch.cat(outs, dim=-1), alphas

    padded = 0
    if channels not in _NATIVE_CHANNELS:
        padded = (1 << (channels - 1).bit_length()) - channels
        colors = torch.cat([colors, torch.zeros(*colors.shape[:-1], padded, device=device)], -1)
        if backgrounds is not None:
            backgrounds = torch.cat(
                [backgrounds, torch.zeros(*backgrounds.shape[:-1], padded, device=device)], -1)
    render_colors, render_alphas = L.op(
        "raster", means2d, conics, colors, opacities, betas, backgrounds, masks, int(image_width),
        int(image_height), int(tile_size), isect_offsets, flatten_ids)
    if padded > 0:
        render_colors = render_colors[..., :-padded]
    return render_colors, render_alphas


# ------------------------------------------- operators outside the UBS path
def _not_on_path(name):
    def f(*args, **kwargs):
        raise NotImplementedError(
            "%s is part of the reference's generic gsplat operator set but is never called on "
            "the Universal Beta Splatting rasteriser path" % name)
    f.__name__ = name
    return f


quat_scale_to_covar_preci = _not_on_path("quat_scale_to_covar_preci")
persp_proj = _not_on_path("persp_proj")
proj = _not_on_path("proj")
world_to_cam = _not_on_path("world_to_cam")
rasterize_to_indices_in_range = _not_on_path("rasterize_to_indices_in_range")
