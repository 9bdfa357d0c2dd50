"""Transforms of different lengths from several threads at once, each on its own
stream: lengths whose tiles take more than 48 KB of shared memory need the
kernels' limit raised, which is the kernel's and not the call's."""

import threading

import pytest
import torch

from teamtomo_b200 import _lib

pytestmark = pytest.mark.gpu


def _spectra(images):
    L = _lib.load()
    d = images.shape[-1]
    row, nbytes = int(L.tt_transform_row(d, 0)), int(L.tt_transform_workspace_bytes(0, images.shape[0], d, 0))
    out = torch.zeros((images.shape[0], d, row), dtype=torch.complex64, device="cuda")
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _lib.check(L.tt_backproject_spectra(_lib.ptr(images), images.shape[0], d, 0, _lib.ptr(out), _lib.ptr(ws), nbytes,
                                        _lib.stream_of(images.device)), "spectra")
    return out


def test_lengths_from_several_threads():
    sizes = [360, 500, 720, 1000, 352, 1024]  # 48 to 145 KB
    images = [torch.randn(2, d, d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(d))
              for d in sizes]
    want = [_spectra(x) for x in images]
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    got = _spectra(images[i])
                    assert torch.equal(got, want[i]), sizes[i]
        except BaseException as e:  # noqa: BLE001 - handed to the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
