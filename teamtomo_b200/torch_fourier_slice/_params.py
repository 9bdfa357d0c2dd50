"""Host-side argument normalisation shared by the slice operators."""

from __future__ import annotations

from functools import lru_cache

import numpy as np
import torch

from .. import _lib


def rotation_arg(rotation_matrices: torch.Tensor, device: torch.device):
    """(..., 3, 3) -> contiguous (n, 3, 3) float32/float64 on ``device``.

    float64 matrices are passed as they are: the kernels round them to float32
    exactly as ``Tensor.to(torch.float32)`` does.  Other dtypes are cast to
    float32 first."""
    R = torch.as_tensor(rotation_matrices)
    if R.shape[-2:] != (3, 3):
        raise ValueError(f"rotation matrices must have shape (..., 3, 3), got {tuple(R.shape)}")
    stack = tuple(R.shape[:-2])
    if R.dtype not in (torch.float32, torch.float64):
        R = R.to(torch.float32)
    if R.device != device:
        R = R.to(device)
    if R.ndim != 3:
        R = R.reshape(-1, 3, 3)
    return R.contiguous(), stack


@lru_cache(maxsize=256)
def _rounded(x: float) -> float:
    return float(np.float32(x))


def _f32(x) -> float:
    return _rounded(float(x))


def slice_params(n, image_shape, volume, rotation, fftfreq_max=None, zyx_matrices=False,
                 x_tolerance=1e-8, rot_tolerance=None, volume_unshifted=False,
                 slices_unshifted=False, vol_dims=None, deterministic=False) -> _lib.SliceParams:
    d, h, w = (int(s) for s in image_shape)
    vd, vh, vw = vol_dims if vol_dims is not None else (int(s) for s in volume.shape[-3:])
    return _lib.SliceParams(
        int(n), d, h, w, vd, vh, vw,
        int(fftfreq_max is not None), _f32(fftfreq_max) if fftfreq_max is not None else 0.0,
        int(bool(zyx_matrices)), _f32(x_tolerance), _f32(x_tolerance * 10),
        int(rot_tolerance is not None), _f32(rot_tolerance) if rot_tolerance is not None else 0.0,
        int(rotation.dtype == torch.float64), int(bool(volume_unshifted)), int(bool(slices_unshifted)),
        int(bool(deterministic)), 0)


def resolve_deterministic(flag: bool | None) -> bool:
    """``None`` follows ``torch.use_deterministic_algorithms``."""
    return torch.are_deterministic_algorithms_enabled() if flag is None else bool(flag)


def rfft_shape(shape):
    """Output shape of an rfft over ``shape`` (torch_grid_utils.rfft_shape)."""
    s = list(int(x) for x in shape)
    s[-1] = s[-1] // 2 + 1
    return tuple(s)
