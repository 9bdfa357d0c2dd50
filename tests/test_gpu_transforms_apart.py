"""Images that are transformed in one launch stay apart: a channel, map or
orientation comes out as it would alone, beside one of a million times its
amplitude, one of zeros or one that is not a number.

Real rows are transformed in pairs; with an odd number of rows a pair must not
take the last row of one image and the first of the next.

Tolerances as in test_gpu_transforms.py: each result against the same call on
its own, a transform's float32 rounding (4e-6; 2e-5 for the gradient of the
rotations, whose terms cancel)."""

import pytest
import torch

from helpers import blob_volume, rel_l2, rotations

pytestmark = pytest.mark.gpu

# odd boxes, with fewer and more than eight pairs of rows to an image, and an even one
BOXES = [(5, 2.0), (9, 1.0), (11, 2.0), (33, 2.0), (41, 2.0), (85, 2.0), (45, 1.0), (32, 2.0)]


def tt():
    import teamtomo_b200

    return teamtomo_b200


def _supported(d, pad):
    from teamtomo_b200 import _lib

    return bool(_lib.load().tt_transform_supported(d, int((d * (pad - 1.0)) // 2)))


def _rel(a, b):
    return rel_l2(a.cpu().numpy(), b.cpu().numpy())


def _beside(x):
    """Channels: x, its mirror image at 1e6, zeros, NaN, x again."""
    return [x, 1e6 * x.flip(-1), torch.zeros_like(x), torch.full_like(x, float("nan")), x]


@pytest.mark.parametrize("d,pad", BOXES)
def test_maps(d, pad):
    assert _supported(d, pad)
    one = torch.as_tensor(blob_volume(d, seed=d)).float().cuda()
    R = torch.as_tensor(rotations(6, seed=2)).float().cuda()
    vols = torch.stack(_beside(one)).requires_grad_(True)
    out = tt().project_3d_to_2d_multichannel(vols, R, pad_factor=pad)
    ref_in = one.clone().requires_grad_(True)
    ref = tt().project_3d_to_2d(ref_in, R, pad_factor=pad)
    G = torch.randn(ref.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(d))
    (gv,) = torch.autograd.grad(out, vols, grad_outputs=torch.stack(_beside(G), dim=1))
    (gref,) = torch.autograd.grad(ref, ref_in, grad_outputs=G)
    out, ref = out.detach(), ref.detach()
    for c in (0, 4):
        assert _rel(out[:, c], ref) < 4e-6
        assert _rel(gv[c], gref) < 4e-6
    assert (out[:, 2] == 0).all() and (gv[2] == 0).all()
    assert out[:, 3].isnan().all() and gv[3].isnan().all()


@pytest.mark.parametrize("d,pad", BOXES)
def test_images(d, pad):
    n = 30
    g = torch.Generator(device="cuda").manual_seed(d)
    one = torch.randn(n, d, d, device="cuda", generator=g)
    R = torch.as_tensor(rotations(n, seed=3)).float().cuda()
    vols = tt().backproject_2d_to_3d_multichannel(torch.stack(_beside(one), dim=1), R, pad_factor=pad)
    ref = tt().backproject_2d_to_3d(one, R, pad_factor=pad)
    assert _rel(vols[0], ref) < 4e-6 and _rel(vols[4], ref) < 4e-6
    assert (vols[2] == 0).all()


@pytest.mark.parametrize("bad", [1e6, float("nan")])
@pytest.mark.parametrize("d,pad", BOXES)
def test_orientations(d, pad, bad):
    """The gradient of one rotation beside an orientation whose image gradient is huge or not a number."""
    vol = torch.as_tensor(blob_volume(d, seed=d)).float().cuda()
    R = torch.as_tensor(rotations(5, seed=4)).float().cuda()
    r = R.clone().requires_grad_(True)
    out = tt().project_3d_to_2d(vol, r, pad_factor=pad)
    G = torch.randn(out.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(d))
    G[[1, 3]] *= bad
    (gr,) = torch.autograd.grad(out, r, grad_outputs=G)
    for i in (0, 2, 4):
        ri = R[i:i + 1].clone().requires_grad_(True)
        (ref,) = torch.autograd.grad(tt().project_3d_to_2d(vol, ri, pad_factor=pad), ri, grad_outputs=G[i:i + 1])
        assert _rel(gr[i], ref[0]) < 2e-5
