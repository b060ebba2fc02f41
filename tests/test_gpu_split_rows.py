"""GPU test of the split's row modes (forward-only rows, piece-product rows; ffg_rows.cu)
at every row length they are instantiated for, forced by ffg_set_geometry whatever the
tuning file holds: squares with an even and an odd number of pieces, and a product of
unlike lengths, modulo three 64-bit primes and 2^128."""
import pytest

from test_gpu_passes import _check

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [9, 10, 11, 12, 13])
def test_split_rows(ff, c):
    ff.init(1 << 21)
    lg, cap0, max0 = c + 6, ff.g_ntt_max_L(), ff.ntt_max_L()
    try:
        ff.set_max_lg(lg)
        ff.set_geometry(lg, 0, c, 16)
        piece = (1 << lg) // 2 * 32 // 64  # limbs of a piece at width 32
        for na, nb in ((4 * piece, None), (5 * piece - 7, None), (6 * piece + 3, 2 * piece + 1)):
            pl = ff.plan(64 * na, 64 * (nb or na), nb is None)
            assert pl["split"] and pl["L"] == 1 << lg and pl["row_lg"] == c, pl
            _check(ff, na, nb or na, nb is None)
    finally:
        ff.set_geometry(lg, 0, 0, 0)
        ff.load_tuning()
        ff.set_max_lg(25)
        ff.lib().ffg_set_ntt_max_L(max0)
        ff.set_g_ntt_max_L(cap0)
