"""Real-space reconstruction (drop-in for torch_fourier_slice.backproject_2d_to_3d).

Same steps as torch_fourier_slice/backproject.py:11-92 — pad, 2D rfft,
central-slice insertion, division by max(weights, 1), 3D irfft, division by
sinc^2, crop — with the fftshifts folded into kernel addressing.  Untracked
float32 images of supported boxes run on the library's own transforms
(_reconstruct), which skip the zeros of the padding and the rows that the crop
drops, and apply the completion and the normalisation while they load the
accumulator.  The others: one kernel
pads and shifts the images, the insertion reads the unshifted 2D rfft, one
kernel applies the Friedel completion, the normalisation and the inverse
shift, and one kernel recentres, divides by sinc^2 and crops.

When the images require grad, the same steps run as differentiable pieces
(each fused pass has its exact adjoint; the insertion's backward is the
gather adjoint of the splat; the normalisation divides by the weights, which
do not depend on the images), so a reconstruction can be differentiated
w.r.t. its projections, as with the reference's torch code.
"""

from __future__ import annotations

import torch

from .. import _lib
from . import _wrappers
from ._params import rotation_arg, slice_params
from .slice_insertion import (
    _InsertCentralSlices,
    insert_accumulate,
    insert_accumulate_multichannel,
    new_accumulator,
)


def _pad_amount(n: int, pad_factor: float) -> int:
    return int((n * (pad_factor - 1.0)) // 2)


def _reconstruct(flat, R, c, pad, fftfreq_max, zyx_matrices):
    """(n * c, d, d) float32 images -> (c, d, d, d') maps with the library's
    own transforms (csrc/fft.cu) around the insertion."""
    dev = flat.device
    d = flat.shape[-1]
    e = d + 2 * pad
    wr = e // 2 + 1
    L = _lib.load()
    st = _lib.stream_of(dev)
    params = slice_params(n=R.shape[0], image_shape=(e, e, e), volume=None, rotation=R, fftfreq_max=fftfreq_max,
                          zyx_matrices=zyx_matrices, vol_dims=(e, e, wr))
    row = int(L.tt_transform_row(d, pad))
    slices = torch.empty((flat.shape[0], e, row), dtype=torch.complex64, device=dev)
    nbytes = max(int(L.tt_transform_workspace_bytes(0, flat.shape[0], d, pad)),
                 int(L.tt_transform_workspace_bytes(1, c, d, pad)))
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    _lib.check(L.tt_backproject_spectra(_lib.ptr(flat), flat.shape[0], d, pad, _lib.ptr(slices), _lib.ptr(ws), nbytes,
                                        st), "backproject_2d_to_3d")
    bricked = bool(L.tt_insert_prefers_bricks(params))
    if bricked:
        acc = torch.zeros(c * (int(L.tt_insert_bricked_accumulator_bytes(e, e, wr)) // 4), dtype=torch.float32,
                          device=dev)
    else:
        acc = new_accumulator((e, e, e), False, dev, channels=c)
    _lib.check(L.tt_insert_accumulate_rows(_lib.ptr(slices), c, row, _lib.ptr(R), _lib.ptr(acc), int(bricked), params,
                                           st), "backproject_2d_to_3d")
    out = torch.empty((c, d, d, 2 * (wr - 1) - 2 * pad), dtype=torch.float32, device=dev)
    _lib.check(L.tt_backproject_volume(_lib.ptr(acc), int(bricked), c, d, pad, _lib.ptr(out), _lib.ptr(ws), nbytes,
                                       st), "backproject_2d_to_3d")
    return out


def _backproject(images, rotation_matrices, pad_factor, fftfreq_max, zyx_matrices, channels):
    h, w = images.shape[-2:]
    if h != w:
        raise ValueError("images must be square.")
    if pad_factor < 1.0:
        raise ValueError("pad_factor must be >= 1.0")
    _lib.require_cuda(images)
    if images.dtype not in (torch.float32, torch.float64):
        images = images.to(torch.float32)
    dev = images.device
    p = _pad_amount(images.shape[-1], pad_factor) if pad_factor > 1.0 else 0
    d = images.shape[-1]
    n = d + 2 * p
    shape = (n, n, n)
    R, _ = rotation_arg(rotation_matrices, dev)
    nrot = R.shape[0]
    lead = images.shape[:-3] if channels else images.shape[:-2]
    c = images.shape[-3] if channels else 1
    flat = _lib.dense(images.reshape(-1, d, d))
    track = torch.is_grad_enabled() and images.requires_grad
    # images that any derivative can be asked of (forward mode and functorch
    # too) go through the autograd Functions; the rotations are constants here
    if (_lib.untracked(images) and images.dtype == torch.float32 and nrot * c == flat.shape[0] > 0
            and _lib.load().tt_transform_supported(d, p)):
        out = _reconstruct(flat, R, c, p, fftfreq_max, zyx_matrices)
        return out if channels else out[0]
    fft_in = _wrappers.pad_fftshift_2d(flat, p)
    spec = torch.fft.rfftn(fft_in, dim=(-2, -1)).reshape(*lead, c, n, n // 2 + 1)
    spec = spec.reshape(nrot, c, n, n // 2 + 1)
    if track:
        vols, weights = _InsertCentralSlices.apply(spec, R, shape, fftfreq_max, zyx_matrices, False, True)
        dft = torch.fft.ifftshift(vols / torch.clamp(weights, min=1.0), dim=(-3, -2))
        real = _wrappers.irfftn_last(dft, 3)
        out = _wrappers.backproject_finish(real, p)
        return out if channels else out[0]
    c128 = spec.dtype == torch.complex128
    acc = new_accumulator(shape, c128, dev, channels=c)
    if c > 1 and not c128:
        insert_accumulate_multichannel(spec.contiguous(), R, shape, acc, fftfreq_max, zyx_matrices,
                                       images_unshifted=True)
    else:
        for ch in range(c):
            insert_accumulate(spec[:, ch].contiguous(), R, shape, acc[ch], fftfreq_max, zyx_matrices,
                              images_unshifted=True)
    dft = _wrappers.backproject_normalize(acc)
    # irfftn without an output size, as the reference (odd boxes lose one x column)
    real = _wrappers.irfftn_last(dft, 3)
    out = _wrappers.backproject_finish(real, p)
    return out if channels else out[0]


def backproject_2d_to_3d(
    images: torch.Tensor,  # (b, d, d)
    rotation_matrices: torch.Tensor,  # (b, 3, 3)
    pad_factor: float = 2.0,
    fftfreq_max: float | None = None,
    zyx_matrices: bool = False,
) -> torch.Tensor:
    """Reconstruct a (d, d, d) volume from (..., d, d) projection images."""
    return _backproject(images, rotation_matrices, pad_factor, fftfreq_max, zyx_matrices, False)


def backproject_2d_to_3d_multichannel(
    images: torch.Tensor,  # (..., c, d, d)
    rotation_matrices: torch.Tensor,  # (..., 3, 3)
    pad_factor: float = 2.0,
    fftfreq_max: float | None = None,
    zyx_matrices: bool = False,
) -> torch.Tensor:
    """Reconstruct (c, d, d, d) volumes from (..., c, d, d) images."""
    return _backproject(images, rotation_matrices, pad_factor, fftfreq_max, zyx_matrices, True)
