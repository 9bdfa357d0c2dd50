"""The lengths that the library's transforms take (csrc/fft.cuh), by a
restatement of the rule that splits them, and the transforms at lengths that
between them run every factor in every place of a plan, two to four passes,
and tiles on both sides of 48 KB of shared memory.

Tolerances as in test_gpu_transforms.py: a float32 transform of n samples has a
relative L2 error of about eps * log2(n), up to three of them in a row stay
below 2e-6; 4e-6 where the insertion's sums come in another order, 2e-5 for the
gradient of the rotations."""

import numpy as np
import pytest
import torch

from helpers import blob_volume, rel_l2, rotations

FACTORS = (20, 16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2)


def _split(n, passes, cap):
    if passes == 0:
        return [] if n == 1 else None
    for r in FACTORS:
        if r <= cap and n % r == 0:
            rest = _split(n // r, passes - 1, r)
            if rest is not None:
                return [r] + rest
    return None


def plan(n):
    """Fewest factors, then the smallest largest one; None when there is no such split."""
    if 4 <= n <= 1024:
        for passes in (2, 3, 4):
            for cap in range(2, 21):
                f = _split(n, passes, cap)
                if f:
                    return f
    return None


def _supported(e):
    return plan(e) is not None and plan(2 * (e // 2)) is not None


def _features(e):
    """What a padded box of e runs: in its transforms and in the inverse real ones, of 2 (e // 2)."""
    out = set()
    for what, n in (("box", e), ("inverse", 2 * (e // 2))):
        f = plan(n)
        for i, r in enumerate(f):
            out.add((what, r, "first" if i == 0 else "last" if i == len(f) - 1 else "middle"))
        out.add((what, "passes", len(f), n % 2))
        tile = n // f[0] * (f[0] | 1) * 8
        out.add((what, "two tiles above 48 KB", (2 * tile + n) * 8 > 48 * 1024, len(f)))
    return out


# transforms of images: all of the features above
IMAGES = [4, 6, 12, 21, 28, 56, 72, 100, 108, 110, 154, 156, 162, 208, 210, 216, 240, 242, 243, 250, 256, 264, 312, 330,
          338, 350, 400, 625, 784, 1024]
# of volumes: three and four passes, odd and even, on both sides of 48 KB
VOLUMES = [100, 108, 162, 210, 242, 243, 250, 264, 338, 350, 400, 625]


def test_supported_lengths_follow_the_rule():
    from teamtomo_b200 import _lib

    L = _lib.load()
    for e in range(1, 1100):
        assert bool(L.tt_transform_supported(e, 0)) == _supported(e), e


def test_the_lengths_below_cover_the_plans():
    every = set().union(*(_features(e) for e in range(4, 1025) if _supported(e)))
    assert set().union(*(_features(e) for e in IMAGES)) == every
    for e in IMAGES + VOLUMES:
        assert _supported(e), e
    volumes = set().union(*(_features(e) for e in VOLUMES))
    for what in ("box", "inverse"):
        assert {f[2] for f in volumes if f[:2] == (what, "passes")} >= {2, 3}
        assert {(what, "two tiles above 48 KB", big, 3) for big in (False, True)} <= volumes
    assert ("box", "passes", 4, 1) in volumes and ("box", "passes", 3, 1) in volumes


def test_index_arithmetic_of_the_plans():
    """The quotients that the kernels form by a product and a shift are exact over the ranges they are used on."""
    for n in range(4, 1025):
        ns = 1
        for r in plan(n) or ():
            nb = n // r
            # a row pass's butterfly -> its transform; a butterfly, or a sample, -> its place in the earlier factors
            for divisor, count in ((nb, 8 * nb), (ns, n)):
                i = np.arange(count, dtype=np.uint64)
                inverse = (1 << 20) // divisor + 1
                assert i.max() * inverse < 1 << 32
                assert np.array_equal((i * inverse) >> 20, i // divisor), (n, divisor)
            ns *= r


@pytest.mark.gpu
@pytest.mark.parametrize("e", IMAGES)
def test_image_spectra(e):
    from teamtomo_b200 import _lib

    L = _lib.load()
    count = 3
    x = torch.randn(count, e, e, device="cuda", generator=torch.Generator(device="cuda").manual_seed(e))
    row, nbytes = int(L.tt_transform_row(e, 0)), int(L.tt_transform_workspace_bytes(0, count, e, 0))
    out = torch.zeros((count, e, row), dtype=torch.complex64, device="cuda")
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    st = _lib.stream_of(x.device)
    _lib.check(L.tt_backproject_spectra(_lib.ptr(x), count, e, 0, _lib.ptr(out), _lib.ptr(ws), nbytes, st), "spectra")
    want = torch.fft.fftshift(torch.fft.rfft2(torch.fft.fftshift(x.double(), dim=(-2, -1))), dim=-2)
    for got, ref in zip(out[..., :e // 2 + 1].cpu().numpy(), want.cpu().numpy()):
        assert rel_l2(got, ref) < 2e-6
    # the adjoint of the projections' inverse transforms: real transforms of 2 (e // 2)
    length = 2 * (e // 2)
    g = x[..., :length].contiguous()
    grad = torch.zeros((count, e, e // 2 + 1), dtype=torch.complex64, device="cuda")
    _lib.check(L.tt_project_slices_backward(_lib.ptr(g), count, e, 0, _lib.ptr(grad), _lib.ptr(ws), nbytes, st), "adjoint")
    rows = torch.fft.rfft(torch.fft.fftshift(g.double(), dim=-1)) / (e * length)  # sample x at (x + length / 2)
    rows[..., 1:-1] *= 2
    want = torch.fft.fftshift(torch.fft.fft(torch.fft.fftshift(rows, dim=-2), dim=-2), dim=-2)
    for got, ref in zip(grad.cpu().numpy(), want.cpu().numpy()):
        assert rel_l2(got, ref) < 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("e", VOLUMES)
def test_volumes_against_the_general_path(monkeypatch, e):
    """Projection with both gradients, and the reconstruction, of a small map padded to e."""
    import teamtomo_b200 as tt

    d = 24 + e % 2
    pad = (e + 0.5) / d  # (e - d) / 2 on each side
    n = 5
    vol = torch.as_tensor(blob_volume(d, seed=e)).float().cuda()
    R = torch.as_tensor(rotations(n, seed=e + 1)).float().cuda()
    images = torch.randn(n, d, d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(e))

    def project():
        v, r = vol.clone().requires_grad_(True), R.clone().requires_grad_(True)
        out = tt.project_3d_to_2d(v, r, pad_factor=pad)
        G = torch.randn(out.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(e + 2))
        return (out.detach(), *torch.autograd.grad(out, [v, r], grad_outputs=G))

    own = project()
    monkeypatch.setenv("TT_VOLUME_LAYOUT", "bricks")  # a forced layout takes the general path
    for a, b, tol in zip(own, project(), (2e-6, 4e-6, 2e-5)):
        assert a.shape == b.shape and rel_l2(a.cpu().numpy(), b.cpu().numpy()) < tol
    monkeypatch.delenv("TT_VOLUME_LAYOUT")
    a = tt.backproject_2d_to_3d(images, R, pad_factor=pad)
    b = tt.backproject_2d_to_3d(images.clone().requires_grad_(True), R, pad_factor=pad).detach()
    assert a.shape == b.shape and rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 4e-6
