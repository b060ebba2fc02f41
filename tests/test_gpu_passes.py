"""GPU test of the fixed-shape four-step passes (ffg_rows.cu, ffg_cols.cu) at
every column length and row length they instantiate, forced by
ffg_set_geometry: squares and products, one of them with a short operand (most
rows of its columns are zero), against the product modulo three 64-bit primes
and modulo 2^128 (a wrong residue changes the product everywhere)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

PRIMES = (18446744073709551557, 18446744073709551533, 9223372036854775783)

# (columns of 2^rn or 3 2^rn words, rows of 2^c): every rn with rows of 512, every c with columns of 64 or 192
SHAPES = [(rn, 9) for rn in range(6, 13)] + [(6, c) for c in range(10, 14)] + [(10, 12), (11, 11)]


def _check(ff, na, nb, square):
    rng = np.random.default_rng(na * 7 + nb)
    a = rng.integers(0, 2**64, na, dtype=np.uint64)
    b = a if square else rng.integers(0, 2**64, nb, dtype=np.uint64)
    da = torch.from_numpy(a.view(np.int64)).cuda()
    db = da if square else torch.from_numpy(b.view(np.int64)).cuda()
    out = torch.full((na + nb + 1,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ff.mul_device(out.data_ptr(), da.data_ptr(), na, 64 * na, db.data_ptr(), nb, 64 * nb, square)
    torch.cuda.synchronize()
    x, y = ff.limbs_to_int(a), ff.limbs_to_int(b)
    z = ff.limbs_to_int(out.cpu().numpy().view(np.uint64))
    assert z.bit_length() <= 64 * (na + nb)
    for m in PRIMES + (1 << 128,):
        assert z % m == (x % m) * (y % m) % m, (na, nb, square, m)


@pytest.mark.parametrize("r3", [0, 1])
@pytest.mark.parametrize("rn,c", SHAPES)
def test_pass_shapes(ff, rn, c, r3):
    if r3 and rn > 11:
        pytest.skip("columns of 3 2^12 words do not fit a tile")
    ff.init(1 << 23)
    lg = rn + c
    L = (3 if r3 else 1) << lg
    hit = 0
    for wc in (8, 32):
        try:
            ff.set_geometry(lg, r3, c, wc)
        except ff.FfgError:
            continue  # 32 long columns do not fit shared memory
        try:
            # (limbs of a, of b): 32-bit digits, digits of over 32 bits, a short operand
            for na, nb in ((L // 4 - 3, None), (L // 4 + L // 256, L // 4 - 4), (L // 2 - L // 32, L // 40)):
                if ff.plan(64 * na, 64 * (nb or na), nb is None)["L"] == L:
                    _check(ff, na, nb or na, nb is None)
                    hit += 1
        finally:
            ff.set_geometry(lg, r3, 0, 0)
            ff.load_tuning()
    assert hit


@pytest.mark.parametrize("lg", [13, 16, 17, 18, 19, 20])
def test_split_row_shapes(ff, lg):
    """The split's row modes at every row length (rows of 2^9 .. 2^13 for
    pieces of 2^16 .. 2^20 words, and one piece length below): squares with an
    even and an odd number of pieces, a product of unlike lengths."""
    ff.init(1 << 20)
    cap0, max0 = ff.g_ntt_max_L(), ff.ntt_max_L()
    try:
        ff.set_max_lg(lg)
        piece = (1 << lg) // 2 * 32 // 64  # limbs of a piece at width 32
        for na, nb in ((4 * piece, None), (5 * piece - 7, None), (6 * piece + 3, 2 * piece + 1)):
            pl = ff.plan(64 * na, 64 * (nb or na), nb is None)
            assert pl["split"]
            _check(ff, na, nb or na, nb is None)
    finally:
        ff.set_max_lg(25)
        ff.lib().ffg_set_ntt_max_L(max0)
        ff.set_g_ntt_max_L(cap0)


def test_one_cta_lengths(ff):
    """The one-CTA convolution at every length 2^4 .. 2^14 and 3 2^4 .. 3 2^12:
    batches of 64 products (which run it past 4096 words too) with operands
    around half of the length, a short one, nearly full ones, for products and
    squares, against Python integers."""
    ff.init(1 << 20)
    rng = np.random.default_rng(3)
    lengths = set()
    for r3, top in ((0, 14), (1, 12)):
        for lg in range(4, top + 1):
            L = (3 if r3 else 1) << lg
            for na, nb in ((L // 4, None), (max(1, L // 4 - 1), L // 4), (max(1, L // 2 - L // 16 - 1), max(1, L // 32)),
                           (L // 4 + max(1, L // 128), None)):
                pl = ff.plan(64 * na, 64 * (nb or na), nb is None)
                if pl["L"] != L or pl["split"]:
                    continue
                pairs = []
                for _ in range(64):
                    a = rng.integers(0, 2**64, na, dtype=np.uint64)
                    a[-1] |= np.uint64(1 << 63)
                    b = None
                    if nb:
                        b = rng.integers(0, 2**64, nb, dtype=np.uint64)
                        b[-1] |= np.uint64(1 << 63)
                    pairs.append((a, b))
                lengths.add(L)
                for (a, b), out in zip(pairs[:6], ff.mul_batch(pairs, method="ntt")[:6]):
                    x = ff.limbs_to_int(a)
                    y = x if b is None else ff.limbs_to_int(b)
                    assert ff.limbs_to_int(out) == x * y, (L, na, nb)
    assert len(lengths) >= 18
