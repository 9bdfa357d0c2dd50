"""Argument checks of tt_insert_accumulate_rows (no GPU, no kernel launches)."""

import pytest

FAKE = 16  # the C side must refuse the call before touching it


def _status(bricked, **kw):
    from teamtomo_b200 import _lib

    p = _lib.SliceParams()
    p.n, p.img_d, p.img_h, p.img_w = 4, 16, 16, 16
    p.vol_d, p.vol_h, p.vol_w = 16, 16, 9
    for k, v in kw.items():
        setattr(p, k, v)
    L = _lib.load()
    return L.tt_insert_accumulate_rows(FAKE, 1, p.vol_w, FAKE, FAKE, bricked, p, None), L.tt_last_error().decode()


@pytest.mark.fake_pointers
def test_bricked_accumulator_slots_fit_32_bits():
    """A brick's slots are addressed in 32 bits, and odd dims are rounded up: 9 * 2^27 voxels take 2^31 slots."""
    wide = dict(img_d=3, img_h=3, img_w=2**28 - 2, vol_d=3, vol_h=3, vol_w=2**27)
    status, text = _status(1, **wide)
    assert status == 1 and "2^31" in text
