"""Geometry of the LayerNorm backward (csrc/ln_geometry.h, compiled for the host)."""
import ctypes

import pytest


def _geometry(H, rows, sms=148):
    from terapipe_b200.ops.lib import host_lib
    out = (ctypes.c_int * 3)()
    return None if host_lib().tp_ln_bwd_geometry(H, rows, sms, out) else tuple(out)


def test_every_row_fits_its_geometry():
    for H in list(range(8, 2048, 8)) + list(range(2048, 16385, 56)) + [16384]:
        for rows in (1, 77, 148, 444, 600, 888, 1184, 1777, 2048, 4096, 100000):
            nv, wpr, per_cta = _geometry(H, rows)
            assert wpr in (1, 2, 4, 8, 16) and 1 <= nv <= 4
            assert nv * wpr * 256 >= H and per_cta * wpr in (16, 24)
            assert per_cta * 2 * H * 4 <= 192 * 1024       # shared memory of the partial sums
            assert wpr == 1 or per_cta <= 15               # a named barrier each


def test_refused_widths():
    assert all(_geometry(H, 10) is None for H in (0, -8, 4, 100, 16392))


@pytest.mark.parametrize("H,rows,nv,wpr", [
    # one round of CTAs with as few vectors per lane as possible
    (768, 77, 1, 4), (768, 1024, 2, 2), (768, 2048, 3, 1), (2304, 256, 2, 8), (2304, 600, 3, 4),
    (2048, 256, 1, 8), (2048, 600, 2, 4), (2048, 1024, 4, 2), (4096, 512, 4, 4), (5120, 77, 2, 16),
    # several rounds: four vectors on 16 warps where these are fewer rounds
    (2048, 16384, 4, 2), (1024, 2048, 4, 1), (4096, 600, 2, 8), (4096, 1024, 4, 4), (2560, 6144, 3, 4),
    (2048, 4096, 2, 4), (1600, 6144, 2, 4),
    (6144, 2048, 3, 8), (12288, 4096, 3, 16),
    (8192, 256, 2, 16), (8192, 1024, 2, 16), (8192, 2048, 4, 8), (16384, 100, 4, 16)])
def test_geometry(H, rows, nv, wpr):
    assert _geometry(H, rows)[:2] == (nv, wpr)
