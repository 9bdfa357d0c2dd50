"""Functions that run their kernels without autograd where no derivative can be
asked for do so only there: none of them has a forward-mode derivative or a
vmap rule, and a call that asks for one is refused, not answered without it."""

import pytest
import torch
from torch.autograd import forward_ad

from helpers import rotations

pytestmark = pytest.mark.gpu


def _calls():
    """Name -> (function of one differentiable tensor, that tensor)."""
    import teamtomo_b200 as tt
    from teamtomo_b200.torch_image_interpolation import insert_into_image_3d, sample_image_3d

    d, n = 16, 4
    g = torch.Generator(device="cuda").manual_seed(0)
    rand = lambda *s, dtype=torch.float32: torch.randn(s, dtype=dtype, device="cuda", generator=g)  # noqa: E731
    R = torch.as_tensor(rotations(n, seed=1)).float().cuda()
    spec, c64 = (d, d, d // 2 + 1), torch.complex64
    coords = torch.rand(50, 3, device="cuda", generator=g) * (d - 1)
    image, values = rand(d, d, d), rand(50)
    return {
        "backproject": (lambda x: tt.backproject_2d_to_3d(x, R), rand(n, d, d)),
        "backproject, no padding": (lambda x: tt.backproject_2d_to_3d(x, R, pad_factor=1.0), rand(n, d, d)),
        "backproject multichannel": (lambda x: tt.backproject_2d_to_3d_multichannel(x, R), rand(n, 2, d, d)),
        "project": (lambda x: tt.project_3d_to_2d(x, R), rand(d, d, d)),
        "project multichannel": (lambda x: tt.project_3d_to_2d_multichannel(x, R), rand(2, d, d, d)),
        "project, rotations": (lambda x: tt.project_3d_to_2d(image, x), R),
        "extract": (lambda x: tt.extract_central_slices_rfft_3d(x, (d, d, d), R), rand(*spec, dtype=c64)),
        "insert": (lambda x: tt.insert_central_slices_rfft_3d(x, (d, d, d), R)[0], rand(n, *spec[1:], dtype=c64)),
        "insert multichannel": (lambda x: tt.insert_central_slices_rfft_3d_multichannel(x, (d, d, d), R)[0],
                                rand(n, 2, *spec[1:], dtype=c64)),
        "sample": (lambda x: sample_image_3d(x, coords), image),
        "sample, coordinates": (lambda x: sample_image_3d(image, x), coords),
        "splat": (lambda x: insert_into_image_3d(x, coords, torch.zeros(d, d, d, device="cuda"))[0], values),
    }


NAMES = ["backproject", "backproject, no padding", "backproject multichannel", "project", "project multichannel",
         "project, rotations", "extract", "insert", "insert multichannel", "sample", "sample, coordinates", "splat"]


@pytest.mark.parametrize("name", NAMES)
def test_derivatives_that_do_not_exist_are_refused(monkeypatch, name):
    monkeypatch.setenv("TT_PROJECT_GRAPHS", "0")
    fn, x = _calls()[name]
    ref = fn(x)
    with forward_ad.dual_level():
        with pytest.raises((NotImplementedError, RuntimeError)):
            fn(forward_ad.make_dual(x, torch.ones_like(x)))
    with pytest.raises((NotImplementedError, RuntimeError)):
        torch.func.jvp(fn, (x,), (torch.ones_like(x),))
    # a plain call inside a level, and the same call after it, are answered
    with forward_ad.dual_level():
        again = fn(x)
    for y in (again, fn(x)):
        # at most 2 x 8 x 4 terms a sum, in another order or from the other path
        assert y.shape == ref.shape and (y - ref).abs().max() <= 1e-5 * ref.abs().max()
