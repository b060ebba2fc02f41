"""GPU test of ffg_last_chain_io: the bytes the chain's copies move.  The starting pair
goes up as one block, each number padded to 32 limbs (with its zeros, so that nothing on
the device has to be cleared); F(n) comes back with its leading zeros."""
import pytest

pytestmark = pytest.mark.gpu


def _pair(n):
    if n == 0:
        return 0, 1
    a, b = _pair(n >> 1)
    c, d = a * (2 * b - a), a * a + b * b
    return (d, c + d) if n & 1 else (c, d)


@pytest.mark.parametrize("k", [90, 2000, 2950, 2960, 20000])
def test_bytes_copied(ff, k):
    f0, f1 = (ff.int_to_limbs(v) for v in _pair(k - 1))
    ff.init(16 * k // 92 + 64)
    got = ff.fib_chain(k << 3, 3, f0, f1)
    up, down = ff.last_chain_io()
    assert up == 2 * 8 * ((max(f0.size, f1.size) + 31) // 32 * 32)
    assert down >= 8 * got.size
