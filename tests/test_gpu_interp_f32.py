"""The single-precision trilinear sampling / insertion kernels (one index and
three strides per cell, lane pairs in the reductions) against the general
kernels, which run in double precision on the same numbers.

Points: random ones, voxel centres (zero fractions), the last index of each
axis (no high corner), just outside; counts below, at and above a warp and a
block; images one voxel thin.  A float32 sum of eight products is within
8 eps = 5e-7 of the double one relative to its terms; sums of many points per
voxel (about 20 here) within sqrt(20) times that: 3e-6 covers both."""

import pytest
import torch

from helpers import rel_l2

pytestmark = pytest.mark.gpu

WIDE = {torch.float32: torch.float64, torch.complex64: torch.complex128}


def tt():
    import teamtomo_b200

    return teamtomo_b200


def _points(n, shape, g):
    size = torch.tensor(shape, device="cuda", dtype=torch.float32)
    c = torch.rand((n, 3), generator=g, device="cuda") * (size + 1) - 1  # some outside
    c[::5] = torch.round(c[::5])
    c[::7, 0] = size[0] - 1
    c[1::7, 1] = size[1] - 1
    c[2::7, 2] = size[2] - 1
    return c


def _randn(shape, dtype, g):
    x = torch.randn(shape, generator=g, device="cuda")
    return torch.complex(x, torch.randn(shape, generator=g, device="cuda")) if dtype.is_complex else x


CASES = [((9, 10, 11), 1, 1), ((9, 10, 11), 1, 31), ((8, 16, 5), 2, 33), ((1, 7, 9), 1, 300), ((6, 1, 9), 3, 257),
         ((7, 9, 1), 1, 256), ((20, 24, 28), 2, 20000)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
@pytest.mark.parametrize("shape,c,n", CASES)
def test_sample_and_gradients(shape, c, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    img, co = _randn((c, *shape), dtype, g), _points(n, shape, g)
    G = _randn((n, c), dtype, g)
    res = []
    for d in (dtype, WIDE[dtype]):
        i, x = img.to(d).requires_grad_(True), co.to(i_real(d)).requires_grad_(True)
        out = tt().sample_image_3d(i, x)
        res.append((out.detach(), *torch.autograd.grad(out, [i, x], grad_outputs=G.to(d))))
    for a, b in zip(*res):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 3e-6
    # each gradient alone
    i, x = img.clone().requires_grad_(True), co.clone().requires_grad_(True)
    (gi,) = torch.autograd.grad(tt().sample_image_3d(i, co), [i], grad_outputs=G)
    (gx,) = torch.autograd.grad(tt().sample_image_3d(img, x), [x], grad_outputs=G)
    assert rel_l2(gi.cpu().numpy(), res[1][1].cpu().numpy()) < 3e-6
    assert torch.equal(gx, res[0][2])


def i_real(d):
    return torch.float64 if d in (torch.float64, torch.complex128) else torch.float32


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape,c,n", CASES)
def test_insert(shape, c, n, dtype, wdtype):
    """Into images that already hold values; voxels no point touches stay as they were."""
    g = torch.Generator(device="cuda").manual_seed(n + 1)
    vals, co = _randn((n, c), dtype, g), _points(n, shape, g)
    start, wstart = _randn((c, *shape), dtype, g), torch.rand(shape, generator=g, device="cuda")
    img, wts = tt().insert_into_image_3d(vals, co, start.clone(), wstart.clone().to(wdtype))
    d = WIDE[dtype]
    ref, rw = tt().insert_into_image_3d(vals.to(d), co, start.to(d), wstart.to(torch.float64))
    assert img.dtype == dtype and wts.dtype == wdtype
    assert rel_l2(img.cpu().numpy(), ref.cpu().numpy()) < 3e-6
    assert rel_l2(wts.cpu().numpy(), rw.cpu().numpy()) < 3e-6
    same = rw == wstart.to(torch.float64)
    assert torch.equal(wts[same], wstart.to(wdtype)[same]) and torch.equal(img[:, same], start[:, same])


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64])
@pytest.mark.parametrize("shape,n", [((24, 31, 17), 200003), ((1, 300, 5), 200000), ((58, 58, 59), 200000),
                                     ((60, 60, 60), 210000)])
def test_insert_many_points(shape, n, dtype):
    """From one point per voxel (and 200,000 points) the splat goes through a
    bricked accumulator; the third shape has 198,476 voxels, just enough, the
    last 216,000, too many.  Neighbouring points in neighbouring, equal and far
    cells."""
    g = torch.Generator(device="cuda").manual_seed(n)
    co = _points(n, shape, g)
    step = torch.tensor([0.3, 0.5, 0.8], device="cuda")
    k = torch.arange(n // 2, device="cuda") % 32
    co[: n // 2] = co[: n // 2 : 32].repeat_interleave(32, 0)[: n // 2] + k[:, None] * step  # runs of points
    vals = _randn((n,), dtype, g)
    start, wstart = _randn(shape, dtype, g), torch.rand(shape, generator=g, device="cuda")
    img, wts = tt().insert_into_image_3d(vals, co, start.clone(), wstart.clone())
    ref, rw = tt().insert_into_image_3d(vals.to(WIDE[dtype]), co, start.to(WIDE[dtype]), wstart.double())
    assert rel_l2(img.cpu().numpy(), ref.cpu().numpy()) < 3e-6 and rel_l2(wts.cpu().numpy(), rw.cpu().numpy()) < 3e-6
    same = rw == wstart.double()
    assert torch.equal(wts[same], wstart[same]) and torch.equal(img[same], start[same])


def test_non_finite_values():
    """Infinities and NaN in the image reach the same samples, and those in the upstream
    gradient the same voxels, as in double precision."""
    g = torch.Generator(device="cuda").manual_seed(5)
    img, co = torch.randn((6, 7, 8), generator=g, device="cuda"), _points(500, (6, 7, 8), g)
    img[2, 3, 4], img[5, 6, 7] = float("inf"), float("nan")
    G = torch.randn(500, generator=g, device="cuda")
    G[3], G[20], G[35] = float("nan"), float("inf"), float("nan")
    res = []
    for d in (torch.float32, torch.float64):
        i = img.to(d).requires_grad_(True)
        out = tt().sample_image_3d(i, co.to(d))
        res.append((out.detach(), *torch.autograd.grad(out, [i], grad_outputs=G.to(d))))
    for a, b in zip(*res):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
