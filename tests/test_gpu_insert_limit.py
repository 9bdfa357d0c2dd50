"""The bricked splat up to a resolution limit skips whole patches of pixels that
lie beyond it: the same pixels as the plain splat, which tests each, in the
one-shot and in the batched kernel's tile shapes.

Limits on a pixel's frequency exactly, just below and above it, none kept but
the origin, and beyond the corner; odd and even boxes, more than 32 tiles to a
row, rows stored from the origin on.  The sums are those of the same terms in
another order: at most eight corners of n slices, 1e-5 of the largest."""

import numpy as np
import pytest
import torch

from helpers import rotations
from teamtomo_b200 import _lib
from teamtomo_b200.torch_fourier_slice._params import rfft_shape, slice_params

pytestmark = pytest.mark.gpu


def _limits(d):
    q = [float(np.float32(k) * np.float32(1.0 / d)) for k in (1, d // 5, d // 4, d // 2 - 1)]
    return [0.0, *q, float(np.nextafter(np.float32(q[2]), np.float32(0))), 0.301, 0.6, 0.8]


def _unbricked(acc, d):
    e, w = (d + 1) // 2, (d // 2 + 2) // 2
    a = acc.reshape(e, e, w, 2, 2, 2, 4).permute(0, 3, 1, 4, 2, 5, 6).reshape(2 * e, 2 * e, 2 * w, 4)
    return a[:d, :d, :d // 2 + 1]


def _same(bricks, plain, what):
    assert torch.equal(bricks[..., 2] != 0, plain[..., 2] != 0), what
    assert (bricks - plain).abs().max() <= 1e-5 * plain.abs().max().clamp(min=1e-30), what


@pytest.mark.parametrize("unshifted", [False, True])
@pytest.mark.parametrize("d,n", [(24, 40), (33, 40), (64, 30), (100, 10), (530, 1)])
def test_one_shot_kernel(d, n, unshifted):
    L = _lib.load()
    shape = rfft_shape((d, d, d))
    R = torch.as_tensor(rotations(n, seed=d)).reshape(n, 3, 3).float().cuda()
    img = torch.randn(n, d, d // 2 + 1, dtype=torch.complex64, device="cuda",
                      generator=torch.Generator(device="cuda").manual_seed(d))
    for fmax in _limits(d):
        p = slice_params(n=n, image_shape=(d, d, d), volume=None, rotation=R, fftfreq_max=fmax, vol_dims=shape,
                         slices_unshifted=unshifted)
        plain = torch.zeros(*shape, 4, device="cuda")
        bricks = torch.zeros(int(L.tt_insert_bricked_accumulator_bytes(*shape)) // 4, device="cuda")
        for acc, bricked in ((plain, 0), (bricks, 1)):
            _lib.check(L.tt_insert_accumulate_rows(_lib.ptr(img), 1, d // 2 + 1, _lib.ptr(R), _lib.ptr(acc), bricked, p,
                                                   _lib.stream_of(img.device)), "insertion")
        assert (plain[..., 2] != 0).any()  # the origin at least
        _same(_unbricked(bricks, d), plain, fmax)


@pytest.mark.parametrize("tile_shape", [0, 1, 2])
@pytest.mark.parametrize("d,n", [(24, 40), (33, 40), (100, 10), (530, 1)])
def test_batched_kernel(d, n, tile_shape):
    L = _lib.load()
    shape = rfft_shape((d, d, d))
    R = torch.as_tensor(rotations(n, seed=d)).reshape(n, 3, 3).float().cuda()
    img = torch.randn(n, d, d // 2 + 1, dtype=torch.complex64, device="cuda",
                      generator=torch.Generator(device="cuda").manual_seed(d))
    ws = torch.empty(int(L.tt_batch_workspace_bytes()), dtype=torch.uint8, device="cuda")
    for fmax in _limits(d):
        accs = []
        for layout in (0, 2):
            p = slice_params(n=n, image_shape=(d, d, d), volume=None, rotation=R, fftfreq_max=fmax, vol_dims=shape)
            p.volume_layout = layout
            acc = torch.zeros(int(L.tt_insert_bricked_accumulator_bytes(*shape)) // 4 if layout else
                              shape[0] * shape[1] * shape[2] * 4, device="cuda")
            entry = _lib.BatchVolume(p, None, img.data_ptr(), acc.data_ptr(), R.data_ptr(), None)
            _lib.check(L.tt_insert_central_slices_rfft_3d_batched((_lib.BatchVolume * 1)(entry), 1, tile_shape,
                                                                  _lib.ptr(ws), ws.numel(), _lib.stream_of(img.device)),
                       "batched insertion")
            accs.append(acc)
        # the plain one-shot splat tests every pixel by itself
        p = slice_params(n=n, image_shape=(d, d, d), volume=None, rotation=R, fftfreq_max=fmax, vol_dims=shape)
        want = torch.zeros(*shape, 4, device="cuda")
        _lib.check(L.tt_insert_accumulate(_lib.ptr(img), 0, _lib.ptr(R), _lib.ptr(want), p,
                                          _lib.stream_of(img.device)), "insertion")
        _same(accs[0].reshape(want.shape), want, fmax)
        _same(_unbricked(accs[1], d), want, fmax)
