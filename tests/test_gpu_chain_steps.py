"""GPU test of the doubling steps that run in one launch (k_chain_steps, ffg_crt.cu):
chains from pairs of 1, 2, 3 limbs and around its longest operand (160 limbs), of
every parity of k and of each bit, against fast doubling on Python integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(n):
    """(F(n), F(n + 1))"""
    if n == 0:
        return 0, 1
    a, b = _pair(n >> 1)
    c, d = a * (2 * b - a), a * a + b * b
    return (d, c + d) if n & 1 else (c, d)


def _limbs(x):
    n = max(1, (x.bit_length() + 63) // 64)
    return np.frombuffer(x.to_bytes(8 * n, "little"), dtype=np.uint64)


# 92.2 indices a limb
@pytest.mark.parametrize("k", [1, 2, 3, 90, 93, 94, 186, 190, 278, 1569, 3137, 7300, 14700, 14751, 14752, 14753, 20001])
@pytest.mark.parametrize("tail,bits", [(0b00, 2), (0b01, 2), (0b1010, 4), (0b0111, 4), (0b110100101, 9), (0b0011011010, 10)])
def test_steps(ff, k, tail, bits):
    n = k << bits | tail
    if n > 3_000_000:
        n, bits = k << 4 | (tail & 15), 4
    f0, f1 = _pair(k - 1)
    ff.init(n // 92 + 8)
    got = ff.fib_chain(n, bits, _limbs(f0), _limbs(f1))
    assert ff.limbs_to_int(got) == _pair(n)[0], (k, n)
