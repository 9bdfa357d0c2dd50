"""When a call may skip autograd's Function (``_lib.untracked``), and the
parameter rounding (CPU)."""

import numpy as np
import torch


def test_untracked_follows_every_way_to_differentiate():
    from teamtomo_b200 import _lib

    a, b = torch.zeros(3), torch.zeros(3, requires_grad=True)
    assert _lib.untracked(a) and not _lib.untracked(a, b)
    with torch.no_grad():
        assert _lib.untracked(a, b)
    with torch.inference_mode():
        assert _lib.untracked(a)
    with torch.autograd.forward_ad.dual_level():
        assert not _lib.untracked(a)
    seen = []

    def f(x):
        seen.append(_lib.untracked(x))
        return x * 2

    torch.func.vmap(f)(torch.zeros(2, 3))
    torch.func.jvp(f, (a,), (a,))
    torch.func.grad(lambda x: f(x).sum())(a)
    assert seen == [False, False, False] and _lib.untracked(a)


def test_scalar_parameters_are_rounded_by_value():
    from teamtomo_b200.torch_fourier_slice._params import slice_params

    R = torch.zeros((1, 3, 3))
    t = torch.tensor(0.1, dtype=torch.float64)
    make = lambda f: slice_params(1, (8, 8, 8), None, R, fftfreq_max=f, vol_dims=(8, 8, 5)).fftfreq_max  # noqa: E731
    assert make(t) == make(0.1) == float(np.float32(0.1))
    t.fill_(0.2)  # a tensor is read at each call
    assert make(t) == float(np.float32(0.2))
    assert make(np.float64(0.3)) == float(np.float32(0.3)) and make(None) == 0.0
