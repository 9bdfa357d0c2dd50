"""The bricked splat (lane octets; corners that two neighbouring pixels of a row
share are added up before the reduction) against the plain one, which adds
every corner by itself: the same corner terms in another order, so the sums
agree within float32 rounding of at most a few hundred terms (1e-6 relative L2)
and the weights' non-zero pattern is the same.

Boxes below one tile, at its edges and past them, odd ones; identity,
axis-aligned, 45-degree and half-turn rotations (every offset between
neighbouring cells, whole rows of zero fractions, the x' < 0 redirect inside a
row) beside random ones; padded rows, interleaved channels, a CTF, infinities
and NaN."""

import ctypes

import numpy as np
import pytest
import torch

from helpers import rel_l2, rotations

pytestmark = pytest.mark.gpu


def _rots(n):
    ax = [np.eye(3)]
    for p in ((0, 2, 1), (2, 1, 0), (1, 2, 0)):
        m = np.eye(3)[list(p)]
        ax.append(m * np.sign(np.linalg.det(m)))
    c = np.sqrt(0.5)
    ax += [np.array([[c, -c, 0], [c, c, 0], [0, 0, 1]]), np.array([[c, 0, c], [0, 1, 0], [-c, 0, c]]),
           np.diag([-1.0, 1.0, -1.0]), np.diag([1.0, -1.0, -1.0])]
    return torch.tensor(np.concatenate([np.stack(ax), rotations(n, seed=n)]), dtype=torch.float32, device="cuda")


def _insert(img, n, R, bricked, pitch, channels=1, fmax=None):
    """(volumes, weights) of channel-interleaved (m, c, n, pitch) images."""
    from teamtomo_b200 import _lib
    from teamtomo_b200.torch_fourier_slice._params import rfft_shape, slice_params

    L = _lib.load()
    d, h, w = rfft_shape((n, n, n))
    p = slice_params(n=R.shape[0], image_shape=(n, n, n), volume=None, rotation=R, fftfreq_max=fmax,
                     vol_dims=(d, h, w))
    st = _lib.stream_of(R.device)
    slots = int(L.tt_insert_bricked_accumulator_bytes(d, h, w)) // 16 if bricked else d * h * w
    acc = torch.zeros((channels, slots, 4), device="cuda")
    assert L.tt_insert_accumulate_rows(_lib.ptr(img), channels, pitch, _lib.ptr(R), _lib.ptr(acc), int(bricked),
                                       ctypes.byref(p), st) == 0
    vol, wts = [], []
    for ch in range(channels):
        v = torch.empty((1, d, h, w), dtype=torch.complex64, device="cuda")
        wt = torch.empty((d, h, w), device="cuda")
        if bricked:
            assert L.tt_insert_finalize_bricked(_lib.ptr(acc[ch]), d, h, w, _lib.ptr(v), _lib.ptr(wt), st) == 0
        else:
            assert L.tt_insert_finalize(_lib.ptr(acc[ch]), 0, 1, d, h, w, _lib.ptr(v), _lib.ptr(wt), st) == 0
        vol.append(v[0])
        wts.append(wt)
    return torch.stack(vol), torch.stack(wts)


@pytest.mark.parametrize("n,channels,pad,fmax", [(4, 1, 0, None), (7, 1, 3, None), (8, 2, 0, None), (15, 1, 0, 0.4),
                                                 (16, 1, 7, None), (31, 2, 0, None), (33, 1, 0, 0.3), (64, 1, 0, None),
                                                 (90, 1, 2, None)])
def test_bricked_matches_plain(n, channels, pad, fmax):
    R = _rots(20)
    pitch = n // 2 + 1 + pad
    g = torch.Generator(device="cuda").manual_seed(n)
    img = torch.view_as_complex(torch.randn((R.shape[0], channels, n, pitch, 2), generator=g, device="cuda"))
    a, wa = _insert(img, n, R, True, pitch, channels, fmax)
    b, wb = _insert(img, n, R, False, pitch, channels, fmax)
    assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-6 and rel_l2(wa.cpu().numpy(), wb.cpu().numpy()) < 1e-6
    assert torch.equal(wa != 0, wb != 0)


def test_non_finite_data_reach_the_same_voxels():
    n, R = 24, _rots(6)
    g = torch.Generator(device="cuda").manual_seed(1)
    img = torch.view_as_complex(torch.randn((R.shape[0], 1, n, n // 2 + 1, 2), generator=g, device="cuda"))
    img[0, 0, 5, 3] = complex(float("nan"), 1.0)
    img[9, 0, 7, 4] = complex(float("inf"), 0.0)
    img[4, 0, 20, 2] = complex(0.0, float("-inf"))
    a, _ = _insert(img, n, R, True, n // 2 + 1)
    b, _ = _insert(img, n, R, False, n // 2 + 1)
    for x, y in ((a.real, b.real), (a.imag, b.imag)):
        assert torch.equal(torch.isfinite(x), torch.isfinite(y))


def test_batched_ctf_small_and_large_choose_their_layout():
    """A batch whose volumes take both layouts equals the volumes one by one."""
    from teamtomo_b200 import batched as B

    boxes, counts = [40, 40, 65], [3, 300, 120]
    g = torch.Generator(device="cuda").manual_seed(2)
    imgs = [torch.view_as_complex(torch.randn((k, b, b // 2 + 1, 2), generator=g, device="cuda"))
            for b, k in zip(boxes, counts)]
    rots = [torch.tensor(rotations(k, seed=k), dtype=torch.float32, device="cuda") for k in counts]
    ctfs = [B.ctf_params(np.linspace(0.8, 2.5, k), astigmatism_um=0.03, astigmatism_angle_deg=20.0, n=k,
                         device="cuda") for k in counts]
    for i, (v, w) in enumerate(B.insert_central_slices_rfft_3d_batched(imgs, rots, ctf=ctfs)):
        # a few slices at a time go to plain accumulators
        parts = [B.insert_central_slices_rfft_3d_batched([imgs[i][k:k + 40]], [rots[i][k:k + 40]],
                                                         ctf=[ctfs[i][k:k + 40]])[0] for k in range(0, counts[i], 40)]
        assert rel_l2(v.cpu().numpy(), sum(p[0] for p in parts).cpu().numpy()) < 1e-6
        assert rel_l2(w.cpu().numpy(), sum(p[1] for p in parts).cpu().numpy()) < 1e-6
