"""GPU test of the host entry point's copies through the pinned slots (ffg_host.cu):
operands and products around one slot (16384 limbs) and around all four, with the
product's top limb zero and not, exact modulo three 64-bit primes, and nothing
written past the product's limbs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRIMES = (18446744073709551557, 18446744073709551533, 9223372036854775783)
SLOT = 16384


@pytest.mark.parametrize("top", [1, 2**64 - 1])
@pytest.mark.parametrize("na,nb", [(SLOT - 1, 2000), (SLOT, 2048), (SLOT + 1, SLOT - 1), (2 * SLOT, 2 * SLOT),
                                   (2 * SLOT + 1, 2 * SLOT), (4 * SLOT + 1, 3), (5 * SLOT - 1, 4 * SLOT + 1)])
def test_host_product(ff, na, nb, top):
    rng = np.random.default_rng(na + nb)
    a = rng.integers(0, 2**64, na, dtype=np.uint64)
    b = rng.integers(0, 2**64, nb, dtype=np.uint64)
    a[-1] = b[-1] = top
    x, y = ff.limbs_to_int(a), ff.limbs_to_int(b)
    want = ((x * y if nb < 100 else 0).bit_length() + 63) // 64 or na + nb - (top == 1)
    out = np.full(na + nb, 0x5A5A5A5A5A5A5A5A, dtype=np.uint64)
    n = ctypes.c_size_t()
    u64p = ctypes.POINTER(ctypes.c_uint64)
    rc = ff.lib().ffg_mul_host(out.ctypes.data_as(u64p), ctypes.byref(n), a.ctypes.data_as(u64p), na,
                               b.ctypes.data_as(u64p), nb, 0)
    assert rc == 0 and n.value == want
    z = ff.limbs_to_int(out[:n.value])
    for m in PRIMES + (1 << 128,):
        assert z % m == (x % m) * (y % m) % m, m
    assert (out[n.value:] == 0x5A5A5A5A5A5A5A5A).all()
