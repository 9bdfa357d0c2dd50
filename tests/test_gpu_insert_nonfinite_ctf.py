"""CTF-weighted insertion of images whose CTF is not a number.

An amplitude contrast above one has no CTF (the square root of a negative
number).  Its image spoils the voxels that its pixels are interpolated to, and
no others: a corner of zero interpolation weight, which past the last index of
an axis has no voxel at all, stays out of the reductions."""

import math

import numpy as np
import pytest
import torch

from teamtomo_b200 import _lib
from teamtomo_b200.batched import ctf_params
from teamtomo_b200.torch_fourier_slice._params import rfft_shape, slice_params

pytestmark = pytest.mark.gpu

BRICKS = 2


def _axis_rotations():
    """Identity and quarter turns: their pixels sit on voxels, the outermost at exactly the last index."""
    R = [np.eye(3), np.diag([-1.0, -1.0, 1.0])]
    for perm in ((1, 2, 0), (2, 0, 1), (1, 0, 2)):
        P = np.zeros((3, 3))
        P[range(3), perm] = 1.0
        R += [P * np.round(np.linalg.det(P)), P]
    return torch.tensor(np.stack(R), dtype=torch.float32, device="cuda")


def _accumulate(images, R, ctf, d, layout, tile_shape):
    """Accumulator (and the slack behind it) of one batched insertion."""
    L = _lib.load()
    shape = rfft_shape((d, d, d))
    p = slice_params(n=R.shape[0], image_shape=(d, d, d), volume=None, rotation=R, vol_dims=shape)
    p.volume_layout = layout
    size = int(L.tt_insert_bricked_accumulator_bytes(*shape)) // 4 if layout else math.prod(shape) * 4
    slack = 2 * (d + 2) * (d // 2 + 3) * 4 * 2  # more than a plane of bricks
    acc = torch.zeros(size + slack, dtype=torch.float32, device="cuda")
    ws = torch.empty(int(L.tt_batch_workspace_bytes()), dtype=torch.uint8, device="cuda")
    entry = _lib.BatchVolume(p, None, images.data_ptr(), acc.data_ptr(), R.data_ptr(), ctf.data_ptr())
    _lib.check(L.tt_insert_central_slices_rfft_3d_batched((_lib.BatchVolume * 1)(entry), 1, tile_shape, _lib.ptr(ws),
                                                          ws.numel(), _lib.stream_of(acc.device)), "batched insertion")
    return acc[:size], acc[size:]


def _unbricked(acc, d):
    """(z, y, x, 4) of a bricked accumulator, and whether its padding is zero."""
    e, w = (d + 1) // 2, (d // 2 + 2) // 2
    a = acc.reshape(e, e, w, 2, 2, 2, 4).permute(0, 3, 1, 4, 2, 5, 6).reshape(2 * e, 2 * e, 2 * w, 4)
    inside = torch.zeros(a.shape[:3], dtype=torch.bool, device=a.device)
    inside[:d, :d, :d // 2 + 1] = True
    return a[:d, :d, :d // 2 + 1], bool((a[~inside] == 0).all())


@pytest.mark.parametrize("tile_shape", [0, 1, 2])
@pytest.mark.parametrize("d", [23, 24, 26])  # an odd box, and both parities of the rfft axis
def test_nan_ctf_reaches_the_same_voxels_in_both_layouts(d, tile_shape):
    R = _axis_rotations()
    n = R.shape[0]
    g = torch.Generator(device="cuda").manual_seed(d)
    images = torch.randn(n, d, d // 2 + 1, dtype=torch.complex64, device="cuda", generator=g)
    ctf = ctf_params(1.5, n=n, device="cuda").clone()
    ctf[::2, 5] = 7.0  # amplitude contrast: 0.07 was meant
    plain, slack = _accumulate(images, R, ctf, d, 0, tile_shape)
    assert (slack == 0).all()
    plain = plain.reshape(d, d, d // 2 + 1, 4)
    assert plain.isnan().any() and plain.isfinite().any()
    bricks, slack = _accumulate(images, R, ctf, d, BRICKS, tile_shape)
    assert (slack == 0).all()
    bricks, padding = _unbricked(bricks, d)
    assert padding
    assert torch.equal(bricks.isnan(), plain.isnan())
    ok = plain.isfinite()
    # sums of at most eight slices' corners in another order: a few units in the last place of the largest term
    assert torch.allclose(bricks[ok], plain[ok], rtol=1e-5, atol=1e-5)
