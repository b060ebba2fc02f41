"""GPU tests of every form of the CRT on numbers that stress its carries: the largest
coefficients, and long runs of ones with a carry (or a borrow) that starts at the
bottom or in the middle and has to cross threads, warps, CTAs and the rounds of 2048
CTAs in which the last CTA settles them.  Expected values are sums of few powers of
two, so that lengths of tens of millions of coefficients stay quick.

The forms: k_crt<CF_BATCH> (297..1024 CTAs of 2048 coefficients) and k_crt<CF_LONG>
(more) at every width; k_crt_flat (batches); k_crt_lin (a doubling step, one output a
CTA and both); k_crt_narrow (widths below 32)."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P = (2113929217, 2013265921, 1811939329)
M = P[0] * P[1] * P[2]


def _ones(n, b):
    """sum of 2^(i b) over i < n"""
    s, m = 0, 0
    for bit in bin(n)[2:]:
        s, m = s | (s << m * b), 2 * m
        if bit == "1":
            s, m = s | (1 << m * b), m + 1
    return s


def _int(t):
    return int.from_bytes(t.cpu().numpy().tobytes(), "little")


def _shape(ff, w, L):
    """Bit lengths of a product whose plan has width w and just under L coefficients."""
    for conv in (L - 5, L - 6):
        ca = min(conv // 2 + 1, 5_900_000 if w == 35 else conv)  # a short side below the bound of the width
        bits = ca * w, (conv + 1 - ca) * w
        pl = ff.plan(*bits)
        if (pl["width"], pl["L"], pl["split"], pl["kernel"]) == (w, L, 0, 1):
            return bits, pl
    raise AssertionError((w, L, pl))


# lengths of 384 and 512 CTAs of 2048 coefficients; 384 and 3072 CTAs of 8192
@pytest.mark.parametrize("L", [3 << 18, 1 << 20, 3 << 20, 3 << 23])
@pytest.mark.parametrize("w", [32, 33, 34, 35])
def test_crt_of_constant_coefficients(ff, w, L):
    ff.init(1 << 24)
    (bits_a, bits_b), pl = _shape(ff, w, L)
    conv, na, nb = pl["conv"], (bits_a + 63) // 64, (bits_b + 63) // 64
    s = _ones(conv, w)
    y = torch.full((3, L), -559038737, dtype=torch.int32, device="cuda")  # words past conv are not residues
    side = torch.cuda.Stream()
    for x, at in ((M - 1, None), (2**w - 1, 0), (2**w - 1, conv // 2)):
        for k, p in enumerate(P):
            y[k, :conv] = x % p
            if at is not None:
                y[k, at] = (x + 1) % p
        out = torch.full((na + nb + 1,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ff.crt_residues(out.data_ptr(), y.data_ptr(), na, bits_a, nb, bits_b, False, side.cuda_stream)
        side.synchronize()
        want = x * s + (0 if at is None else 1 << at * w)
        assert _int(out) == want % (1 << 64 * (na + nb + 1)), (x == M - 1, at)
    assert ff.tickets_in_use() == 0


def _thirds(na, h):
    """(2^n - 1) / 3 + 2^(64 h), n = 64 na: times 3 it is 2^n - 1 and a carry from limb h to the top."""
    a = torch.full((na,), 0x5555555555555555, dtype=torch.int64, device="cuda")
    a[h] += 1
    return a


def _times3(na, h):
    """The na + 2 limbs of 3 ((2^n - 1) / 3 + 2^(64 h))."""
    out = torch.zeros(na + 2, dtype=torch.int64, device="cuda")
    out[:h] = -1
    out[h] = 2
    out[na] += 1
    return out


# limbs: under a CTA, about one (1024 to 1120 limbs), a few, past 2048 CTAs (a second round of maps)
BATCH = [5, 1119, 1120, 1121, 9000, 2_400_000]


def test_batch_crt_carries(ff):
    ff.init(1 << 24)
    three = torch.tensor([3], dtype=torch.int64, device="cuda")
    jobs, outs, wants, keep = [], [], [], []
    for na in BATCH:
        for h in (0, na // 2):
            a = _thirds(na, h)
            out = torch.full((na + 2,), -1, dtype=torch.int64, device="cuda")
            jobs.append({"a": a.data_ptr(), "b": three.data_ptr(), "na": na, "nb": 1, "bits_a": 64 * na, "bits_b": 2,
                         "out": out.data_ptr(), "method": "ntt"})
            outs.append(out)
            wants.append(_times3(na, h))
            keep.append(a)
        ones = torch.full((na,), -1, dtype=torch.int64, device="cuda")  # (2^n - 1)^2 = 2^2n - 2^(n + 1) + 1
        out = torch.full((2 * na + 1,), -2, dtype=torch.int64, device="cuda")
        jobs.append({"a": ones.data_ptr(), "na": na, "bits_a": 64 * na, "out": out.data_ptr(), "square": True,
                     "method": "ntt"})
        want = torch.zeros(2 * na + 1, dtype=torch.int64, device="cuda")
        want[0] = 1
        want[na] = -2
        want[na + 1: 2 * na] = -1
        outs.append(out)
        wants.append(want)
        keep.append(ones)
    torch.cuda.synchronize()
    ff.mul_batch_device(jobs)
    torch.cuda.synchronize()
    for j, out, want in zip(jobs, outs, wants):
        assert torch.equal(out, want), (j["na"], j.get("square", False))


# 40, 350 and more than 1024 CTAs of 2048 coefficients: each form of the plain product
@pytest.mark.parametrize("na", [45_000, 390_000, 1_500_000, 12_000_000])
def test_plain_product_carries(ff, na):
    ff.init(1 << 24)
    three = torch.tensor([3], dtype=torch.int64, device="cuda")
    for h in (0, na // 2):
        a = _thirds(na, h)
        out = torch.full((na + 2,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ff.mul_device(out.data_ptr(), a.data_ptr(), na, 64 * na, three.data_ptr(), 1, 2, False)
        torch.cuda.synchronize()
        assert torch.equal(out, _times3(na, h)), h


def _mul(x, y):
    z = {}
    for e, c in x.items():
        for f, d in y.items():
            z[e + f] = z.get(e + f, 0) + c * d
    return z


def _lin(*terms):
    z = {}
    for c, x in terms:
        for e, d in x.items():
            z[e] = z.get(e, 0) + c * d
    return z


def _value(x):
    return sum(c << e for e, c in x.items())


# one doubling step on operands as long as F(k), widths 32..35 in each form: 3 to 64 CTAs (one
# output a CTA), 141 to 188 (both outputs) and 2289 (a second round of maps)
STEPS = [150_000, 150_902, 155_030, 188_957, 3_000_001, 6_621_122, 9_068_445, 9_372_237, 9_657_236, 108_000_001]


@pytest.mark.parametrize("k,tail", [(k, t) for k in STEPS for t in range(4) if k < 10**8 or t in (1, 2)])
def test_doubling_step_carries(ff, k, tail):
    """The step's linear combinations of the squares of sparse numbers (F(k) and F(k - 1)
    in place, never longer than they are), through the last product: long runs of zeros,
    where the biased coefficients carry, and of ones, where a borrow runs."""
    ff.init((k << 2) // 92 + 64)
    bits = int(k * 0.6942419136306174 - 1.1609640474436812) - 2
    for y, x in (({bits: 1}, {bits - 1: 1}),
                 ({bits: 1, bits // 3: 1}, {bits - 1: 1, bits // 5: 1}),
                 ({bits: 1, 0: -1}, {bits - 1: 1, 0: -1})):
        vy, vx = _value(y), _value(x)
        py, px = ff.plan(vy.bit_length(), vy.bit_length(), True), ff.plan(vx.bit_length(), vx.bit_length(), True)
        assert all(py[f] == px[f] for f in ("width", "L", "kernel", "row_lg", "split")) and not py["split"]
        s1, s2, pm2 = _mul(y, y), _mul(x, x), {0: -2 if k & 1 else 2}
        if tail & 2:
            lo, hi = _lin((3, s1), (-2, s2), (1, pm2)), _lin((4, s1), (-1, s2), (1, pm2))
        else:
            lo, hi = _lin((1, s1), (1, s2)), _lin((3, s1), (-2, s2), (1, pm2))
        if tail & 1:
            want = _lin((1, _mul(_lin((2, hi), (1, lo)), _lin((2, hi), (-1, lo)))), (-2 if tail & 2 else 2, {0: 1}))
        else:
            want = _mul(hi, _lin((1, hi), (2, lo)))
        got = ff.fib_chain(k << 2 | tail, 2, ff.int_to_limbs(vx), ff.int_to_limbs(vy))
        assert ff.limbs_to_int(got) == _value(want), (y, x)


_NARROW = textwrap.dedent("""
    import sys
    import torch
    sys.path.insert(0, sys.argv[1])
    import fastfib_b200 as ff
    ff.init(1 << 24)
    BITS = 13_400_000_000  # past the bound of width 32

    def product(a, na, bits_a, b, nb, bits_b, square, width):
        pl = ff.plan(bits_a, bits_b, square)
        assert pl["split"] and pl["width"] == width, pl
        out = torch.full((na + nb + 1,), -3, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ff.mul_device(out.data_ptr(), a.data_ptr(), na, bits_a, b.data_ptr(), nb, bits_b, square)
        torch.cuda.synchronize()
        return out

    # short numbers whose bit lengths are given as upper bounds: a carry from limb h to the top
    three = torch.tensor([3], dtype=torch.int64, device="cuda")
    for na, h in ((100, 0), (991, 0), (992, 0), (993, 500), (70_000, 0), (70_000, 35_001), (2_500_000, 0)):
        a = torch.full((na,), 0x5555555555555555, dtype=torch.int64, device="cuda")
        a[h] += 1
        out = product(a, na, BITS, three, 1, BITS, False, 31)
        want = torch.zeros(na + 2, dtype=torch.int64, device="cuda")
        want[:h] = -1
        want[h] = 2
        want[na] += 1
        assert torch.equal(out, want), (na, h)
    # random numbers, against the product the other widths give
    gen = torch.Generator(device="cuda").manual_seed(5)
    for na, nb in ((3000, 2900), (400_000, 70_001)):
        a = torch.randint(-(2**63), 2**63 - 1, (na,), dtype=torch.int64, device="cuda", generator=gen)
        b = torch.randint(-(2**63), 2**63 - 1, (nb,), dtype=torch.int64, device="cuda", generator=gen)
        want = torch.empty(na + nb + 1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ff.mul_device(want.data_ptr(), a.data_ptr(), na, 64 * na, b.data_ptr(), nb, 64 * nb, False)
        assert torch.equal(product(a, na, BITS, b, nb, BITS, False, 31), want), (na, nb)
    # (2^N - 1)^2 at that length: the largest coefficients it can have
    na = BITS // 64
    a = torch.full((na,), -1, dtype=torch.int64, device="cuda")
    out = product(a, na, 64 * na, a, na, 64 * na, True, 31)
    assert int(out[0]) == 1 and int(out[na]) == -2 and int(out[2 * na]) == 0
    assert not out[1:na].any() and bool((out[na + 1:2 * na] == -1).all())
    print("ok", ff.tickets_in_use())
""")


def test_narrow_crt():
    """Widths below 32: operands past 1.3e10 bits (a process of its own, for the
    80 GB of residues it holds)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _NARROW, root], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and r.stdout.split() == ["ok", "0"], r.stdout[-500:] + r.stderr[-3000:]
