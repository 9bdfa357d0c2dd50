"""Coordinates and flags of the slice geometry at many box sizes, bit for bit
against the oracle's float32 arithmetic (IEEE divisions): the kernels divide by
reciprocals with two FMA corrections."""

import numpy as np
import pytest
import torch

from helpers import rotations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 5, 8, 24, 45, 63, 64, 67, 96, 100, 127, 162, 200, 251, 256, 320, 400])
@pytest.mark.parametrize("mode", ["extract", "insert"])
def test_coordinates_bitwise(n, mode):
    from teamtomo_b200.torch_fourier_slice.slice_extraction import central_slice_geometry

    R = rotations(3, seed=n).astype(np.float32)
    flags, coords = central_slice_geometry(torch.tensor(R, device="cuda"), (n, n, n), (n, n, n // 2 + 1), mode=mode)
    flags, coords = flags.cpu().numpy(), coords.cpu().numpy()
    f = np.float32
    k = np.arange(n)
    qy = np.fft.fftshift((np.where(k < (n + 1) // 2, k, k - n).astype(f) * f(1.0 / n)).astype(f))
    qx = (np.arange(n // 2 + 1).astype(f) * f(1.0 / n)).astype(f)
    m = R[:, ::-1, ::-1]
    p = [(m[:, i, 1, None, None] * qy[:, None]).astype(f) + (m[:, i, 2, None, None] * qx).astype(f) for i in range(3)]
    kept, conj = (flags & 1) > 0, (flags & 2) > 0
    p = [np.where(conj, -x, x) for x in p]
    iw = f(1) - f(1) / f(n)
    with np.errstate(all="ignore"):
        ref = np.stack([((p[0] + f(0.5)) / iw) * f(n - 1), ((p[1] + f(0.5)) / iw) * f(n - 1),
                        (p[2] * f(2)) * f(n // 2)], axis=-1)
    assert ref.dtype == np.float32 and kept.any()
    assert np.array_equal(coords[kept], ref[kept])
