"""The library's own transforms around projection and reconstruction
(csrc/fft.cu) against the same call in float64 torch (projection) and against
the general path (gradients, reconstruction).

Sizes: factors 2 to 20 in lengths of two and three factors, odd padded boxes
(whose inverse real transform is one sample shorter), no padding, one and more
than one block of eight transforms, boxes beyond 48 KB of shared memory, one
rotation, several channels.

Tolerances: a float32 transform of n samples has a relative L2 error of about
eps * log2(n) with eps = 6e-8, three of them in a row below 2e-6 at these
sizes; the geometry and the sampled values are the general path's bit for bit.
The projection is compared at 1e-5 (its float32 slice coordinates, which both
paths share, are off the float64 ones by up to 1e-5 of a voxel)."""

import numpy as np
import pytest
import torch

from helpers import blob_volume, rel_l2, rotations

pytestmark = pytest.mark.gpu

# (d, pad factor): padded 8, 25 -> 24, 26, 22, 27 -> 26, 45 -> 44, 65 -> 64, 98, 104, 128, 180, 256, 320, 49 -> 48
BOXES = [(4, 2.0), (25, 1.0), (26, 1.0), (22, 1.0), (27, 1.0), (45, 1.0), (33, 2.0), (98, 1.0), (70, 1.5), (64, 2.0),
         (90, 2.0), (128, 2.0), (160, 2.0), (33, 1.5)]


def tt():
    import teamtomo_b200

    return teamtomo_b200


def _own(d, pad_factor):
    from teamtomo_b200 import _lib

    p = int((d * (pad_factor - 1.0)) // 2)
    return bool(_lib.load().tt_transform_supported(d, p))


def _both(monkeypatch, fn):
    out = []
    for mode in ("auto", "bricks"):  # a forced layout takes the general path
        monkeypatch.setenv("TT_VOLUME_LAYOUT", mode)
        out.append(fn())
    return out


@pytest.mark.parametrize("d,pad", BOXES)
@pytest.mark.parametrize("channels,fmax", [(0, None), (2, 0.37)])
def test_projection_and_gradients(monkeypatch, d, pad, channels, fmax):
    n = 1 if d == 128 else 9
    vol = np.stack([blob_volume(d, seed=700 + d + i) for i in range(max(channels, 1))])
    vol = torch.as_tensor(vol if channels else vol[0]).float().cuda()
    R = torch.as_tensor(rotations(n, seed=701 + d)).float().cuda()
    fn = tt().project_3d_to_2d_multichannel if channels else tt().project_3d_to_2d

    def run():
        v, r = vol.clone().requires_grad_(True), R.clone().requires_grad_(True)
        out = fn(v, r, pad_factor=pad, fftfreq_max=fmax)
        G = torch.randn(out.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(d))
        return (out.detach(), *torch.autograd.grad(out, [v, r], grad_outputs=G))

    assert _own(d, pad)
    own, general = _both(monkeypatch, run)
    for a, b, tol in zip(own, general, (2e-6, 4e-6, 2e-5)):  # d/drotation differences cancel: the looser bound
        assert a.shape == b.shape and a.dtype == b.dtype
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < tol
    # no gradient asked for, and each gradient alone, are the same calls
    with torch.no_grad():
        monkeypatch.setenv("TT_VOLUME_LAYOUT", "auto")
        monkeypatch.setenv("TT_PROJECT_GRAPHS", "0")
        assert torch.equal(fn(vol, R, pad_factor=pad, fftfreq_max=fmax), own[0])


@pytest.mark.parametrize("want", ["volume", "rotation"])
def test_single_gradients(monkeypatch, want):
    vol = torch.as_tensor(blob_volume(24, seed=3)).float().cuda().requires_grad_(want == "volume")
    R = torch.as_tensor(rotations(5, seed=4)).double().cuda().requires_grad_(want == "rotation")

    def run():
        out = tt().project_3d_to_2d(vol, R)
        (g,) = torch.autograd.grad(out.square().sum(), [vol if want == "volume" else R])
        return g

    a, b = _both(monkeypatch, run)
    assert a.dtype == b.dtype and rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-5


@pytest.mark.parametrize("d,pad", BOXES)
def test_projection_against_oracle(oracle, d, pad):
    vol = blob_volume(d, seed=720 + d)
    R = rotations(4, seed=721 + d).astype(np.float32)
    out = tt().project_3d_to_2d(torch.as_tensor(vol).float().cuda(), torch.as_tensor(R).cuda(), pad_factor=pad)
    assert rel_l2(out.cpu().numpy(), oracle.project_3d_to_2d(vol, R, pad_factor=pad)) < 1e-5


@pytest.mark.parametrize("d,pad", BOXES)
@pytest.mark.parametrize("channels", [0, 2])
def test_reconstruction(d, pad, channels):
    """Images with a gradient take the general path: the same reconstruction."""
    n = 7 if d >= 128 else 40
    g = torch.Generator(device="cuda").manual_seed(d)
    images = torch.randn((n, channels, d, d) if channels else (n, d, d), device="cuda", generator=g)
    R = torch.as_tensor(rotations(n, seed=730 + d)).float().cuda()
    fn = tt().backproject_2d_to_3d_multichannel if channels else tt().backproject_2d_to_3d
    a = fn(images, R, pad_factor=pad)
    b = fn(images.clone().requires_grad_(True), R, pad_factor=pad).detach()
    assert a.shape == b.shape and rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 4e-6


@pytest.mark.parametrize("d,n,channels", [(33, 5, 2), (32, 5, 3), (16, 6000, 3), (27, 1, 5)])
def test_channels_match_single_maps(d, n, channels):
    """Channels are sampled in pairs: a pair, a pair and a rest, launches with whole
    and with split rows of tiles.  Up to the transforms' rounding (rows of an odd
    box pair up differently)."""
    vol = torch.stack([torch.as_tensor(blob_volume(d, seed=i)).float() for i in range(channels)]).cuda()
    R = torch.as_tensor(rotations(n, seed=4)).float().cuda()
    got = tt().project_3d_to_2d_multichannel(vol, R)
    for c in range(channels):
        ref = tt().project_3d_to_2d(vol[c], R)
        assert rel_l2(got[:, c].cpu().numpy(), ref.cpu().numpy()) < 4e-6


def test_unsupported_boxes_keep_the_general_path(monkeypatch):
    """A prime factor above 13 (68 = 4 * 17) and float64 maps."""
    assert not _own(34, 2.0) and not _own(600, 2.0)
    R = torch.as_tensor(rotations(3, seed=9)).float().cuda()
    for d, dtype in ((34, torch.float32), (16, torch.float64)):
        vol = torch.as_tensor(blob_volume(d, seed=5)).to(dtype).cuda()
        a, b = _both(monkeypatch, lambda: tt().project_3d_to_2d(vol, R))
        assert a.dtype == dtype and torch.equal(a, b)
