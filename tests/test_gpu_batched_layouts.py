"""Batched insertions whose volumes go to plain and to bricked accumulators in
one launch, by the rule that the insertion asks (tt_insert_prefers_bricks):
each volume against the one-shot insertion, and with a CTF against the oracle's
insertions of ctf * image and ctf^2, as in test_gpu_batched.py."""

import numpy as np
import pytest
import torch

from helpers import blob_volume, rel_l2, rfft_volume_np, rotations

pytestmark = pytest.mark.gpu

BOXES, COUNTS = [216, 48, 230, 64], [40, 30, 25, 400]


def test_both_layouts_in_one_launch(oracle):
    import teamtomo_b200 as tt
    from teamtomo_b200 import _lib, batched
    from teamtomo_b200.torch_fourier_slice._params import rfft_shape, slice_params

    L = _lib.load()
    rots = [torch.as_tensor(rotations(k, seed=b + k)).float().cuda() for b, k in zip(BOXES, COUNTS)]
    bricked = [L.tt_insert_prefers_bricks(slice_params(n=k, image_shape=(b, b, b), volume=None, rotation=R,
                                                       vol_dims=rfft_shape((b, b, b))))
               for b, k, R in zip(BOXES, COUNTS, rots)]
    # 200,000 pixels and an eighth of a pixel per voxel: 941,760 of 5.1 M, 36,000, 667,000 of 6.1 M, 844,800 of 135,168
    assert bricked == [1, 0, 0, 1]
    vols = [torch.as_tensor(rfft_volume_np(blob_volume(b, seed=b, n_blobs=8))).cuda() for b in BOXES]
    imgs = [tt.extract_central_slices_rfft_3d(v, (b, b, b), R) for b, v, R in zip(BOXES, vols, rots)]
    for b, im, R, (vol, w) in zip(BOXES, imgs, rots, batched.insert_central_slices_rfft_3d_batched(imgs, rots)):
        v1, w1 = tt.insert_central_slices_rfft_3d(im, (b, b, b), R)
        assert rel_l2(vol.cpu().numpy(), v1.cpu().numpy()) < 1e-6, b
        assert rel_l2(w.cpu().numpy(), w1.cpu().numpy()) < 1e-6, b
        assert torch.equal(w != 0, w1 != 0), b
    ctfs = [batched.ctf_params(np.linspace(0.8, 2.5, k), n=k, device="cuda") for k in COUNTS]
    outs = batched.insert_central_slices_rfft_3d_batched(imgs, rots, ctf=ctfs)
    for b, im, R, c, (vol, w) in zip(BOXES, imgs, rots, ctfs, outs):
        cc = c.cpu().numpy()
        ctf = np.stack([oracle.ctf_2d(*cc[j], image_shape=(b, b)) for j in range(len(cc))])
        rv, _ = oracle.insert((im.cpu().numpy() * ctf).astype(np.complex64), (b, b, b), R.cpu().numpy(), nthreads=8)
        rw, _ = oracle.insert((ctf * ctf).astype(np.complex64), (b, b, b), R.cpu().numpy(), nthreads=8)
        assert rel_l2(vol.cpu().numpy(), rv) < 1e-4, b
        assert rel_l2(w.cpu().numpy(), rw.real) < 1e-4, b
