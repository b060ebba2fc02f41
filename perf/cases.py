"""Timed cases of the framework's public entry points.

Each case is one call (or one batch call) as a program makes it: F(n) through
the reference's surface, single products on device limbs, a product of host
numbers, batches of independent products, decimal conversion.  ``prepare``
makes the operands from the seed alone (uniform random limbs: the digits of
the large numbers this library multiplies look random), ``run`` is the call,
``exact`` the same value from Python integers and a double-precision FFT.

Operands already lie on the GPU for the device entry points; ``run`` passes no
stream, so the work goes to the library's own stream, in the order of the
calls.
"""
import ctypes
import math
import weakref

import numpy as np
import torch

import fastfib_b200 as ff
from fastfib_b200.workload import uneven_sizes

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # F(n) as fibonacci() serves it: the prefix on the host, the doubling chain
        # on the device, the limbs back on the host.  Short numbers, where launches
        # and latency count ...
        {"name": "fib_1e5", "kind": "fib", "n": 100_000},
        # ... the headline size ...
        {"name": "fib_1e8", "kind": "fib", "n": 100_000_000},
        # ... and one of the largest in use, a chain of long transforms.
        {"name": "fib_1e9", "kind": "fib", "n": 1_000_000_000},
        # One short product of device numbers: the one-CTA transform and its CRT.
        {"name": "mul_300x257", "kind": "mul", "na": 300, "nb": 257, "square": False},
        # Two host numbers of middle size through the reference's surface (big_mul):
        # copies in, product, copy out.
        {"name": "big_50001x48000", "kind": "big", "na": 50_001, "nb": 48_000},
        # A middle product of device numbers, odd sizes (a launch that only just
        # fills the GPU).
        {"name": "mul_131071x120001", "kind": "mul", "na": 131_071, "nb": 120_001, "square": False},
        # A long square, the largest of the multiply microbench: transform length 2^24.
        {"name": "sqr_2e22", "kind": "mul", "na": 4_194_304, "nb": 4_194_304, "square": True},
        # A ragged long product, aspect ratio 16.
        {"name": "mul_3000001x190001", "kind": "mul", "na": 3_000_001, "nb": 190_001, "square": False},
        # A square past the longest transform: the piecewise split multiply.
        {"name": "sqr_split_12000001", "kind": "mul", "na": 12_000_001, "nb": 12_000_001, "square": True},
        # A stream of 4096 independent uneven products (2^10 .. 2^24 bits a side,
        # aspect ratio up to 16) under the plain dispatch.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 10, "hi": 24, "method": "plain", "sizes": 4},
        # A small stream of shorter products under the learned dispatch.
        {"name": "batch_300_learned", "kind": "batch", "count": 300, "lo": 10, "hi": 19, "method": "learned",
         "sizes": 11},
        # The decimal digits of a number as long as F(10^8) (20.9 million digits).
        {"name": "decimal_20900000", "kind": "decimal", "limbs": 1_084_750},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "fib", "fib", "batch", "decimal", "big"])
    if kind == "fib":
        return {"kind": "fib", "n": _log(rng, 100_000, 1_000_000_000)}
    if kind == "mul":
        na = _log(rng, 200, 12_000_001)
        square = rng.random() < 0.4
        nb = na if square else max(200, _log(rng, max(1, na // 16), na))
        return {"kind": "mul", "na": na, "nb": nb, "square": square}
    if kind == "big":
        na = _log(rng, 200, 1_000_000)
        return {"kind": "big", "na": na, "nb": max(200, _log(rng, max(1, na // 16), na))}
    if kind == "batch":
        hi = rng.choice([16, 18, 19, 20, 22, 24])
        # no more limbs than the largest listed stream
        return {"kind": "batch", "count": _log(rng, 32, 4096), "lo": 10, "hi": hi,
                "method": rng.choice(["plain", "learned", "ntt"]), "sizes": rng.randrange(1 << 20)}
    return {"kind": "decimal", "limbs": _log(rng, 600, 1_084_750)}


# ------------------------------------------------------------------ inputs


def _limbs(n, seed):
    """n uniform random limbs on the GPU, the top bit set (n limbs exactly)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randint(-(2**63), 2**63 - 1, (n,), dtype=torch.int64, device="cuda", generator=gen)
    x[n - 1] |= -(2**63)
    return x


def _fib_index(case, seed):
    """The index of this seed: one of the 90 about the case's whose F(n) have as many limbs."""
    first = int(((_fib_limbs(case["n"]) - 1) * 64 + 1.1609640474436812) / 0.6942419136306174) + 2
    return first + (seed * 7919) % 90


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fib":
        ff.ntt_init(case["n"] // 92 + 8)
        return {"kind": kind, "n": _fib_index(case, seed)}
    if kind in ("mul", "big"):
        na, nb = case["na"], case["nb"]
        a = _limbs(na, 2 * seed)
        if kind == "big":
            ff.ntt_init(na + nb)
            return {"kind": kind, "a": a.cpu().numpy().view(np.uint64),
                    "b": _limbs(nb, 2 * seed + 1).cpu().numpy().view(np.uint64)}
        ff.init(na + nb)
        b = a if case["square"] else _limbs(nb, 2 * seed + 1)
        out = torch.empty(na + nb + 1, dtype=torch.int64, device="cuda")
        return {"kind": kind, "a": a, "b": b, "out": out, "square": case["square"]}
    if kind == "batch":
        sizes = uneven_sizes(case["sizes"], case["count"], case["lo"], case["hi"])
        bits = np.array(sizes, dtype=np.int64)                    # count x 2
        limbs = (bits + 63) // 64
        end = np.cumsum(limbs.reshape(-1))
        x = _limbs(int(end[-1]), seed)
        # every operand has its bit length exactly
        top = bits.reshape(-1) - 64 * (limbs.reshape(-1) - 1)     # 1 .. 64 bits in the top limb
        keep = np.where(top == 64, -1, (np.int64(1) << np.minimum(top, 63)) - 1)
        one = np.int64(1) << (top - 1)
        at = torch.from_numpy(end - 1).cuda()
        x[at] = (x[at] & torch.from_numpy(keep).cuda()) | torch.from_numpy(one).cuda()
        nout = limbs.sum(axis=1) + 1
        out0 = np.concatenate([[0], np.cumsum(nout)])
        out = torch.empty(int(out0[-1]), dtype=torch.int64, device="cuda")
        first = np.concatenate([[0], end[:-1]]).reshape(-1, 2)
        ff.init(int(limbs.sum(axis=1).max()))
        jobs = ff.device_jobs([
            {"a": x.data_ptr() + 8 * int(first[i, 0]), "b": x.data_ptr() + 8 * int(first[i, 1]),
             "na": int(limbs[i, 0]), "nb": int(limbs[i, 1]), "bits_a": int(bits[i, 0]), "bits_b": int(bits[i, 1]),
             "out": out.data_ptr() + 8 * int(out0[i]), "method": case["method"]} for i in range(case["count"])])
        return {"kind": kind, "jobs": jobs, "x": x, "out": out, "limbs": limbs, "first": first}
    n = case["limbs"]
    ff.init(n + 8)
    return {"kind": kind, "x": _limbs(n, seed), "n": n}


# ------------------------------------------------------------------ the calls


def _digits(ptr, n):
    """The library's digit buffer as an array; the buffer goes back when it is collected."""
    a = np.ctypeslib.as_array(ctypes.cast(ptr, ctypes.POINTER(ctypes.c_uint8)), shape=(n,))
    weakref.finalize(a, ff.lib().ffg_free, ptr)
    return a


def run(state):
    kind = state["kind"]
    if kind == "fib":
        return ff.fibonacci(state["n"]).view(np.int64)
    if kind == "mul":
        a, b = state["a"], state["b"]
        na, nb = a.numel(), b.numel()
        ff.mul_device(state["out"].data_ptr(), a.data_ptr(), na, 64 * na, b.data_ptr(), nb, 64 * nb, state["square"])
        return state["out"]
    if kind == "big":
        return ff.big_mul(state["a"], state["b"]).view(np.int64)
    if kind == "batch":
        ff.mul_batch_device(state["jobs"])
        return state["out"]
    # the digits as a C program takes them: a buffer of the library's
    out, nout, done = ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_int()
    rc = ff.lib().ffg_to_decimal_device(state["x"].data_ptr(), state["n"], ctypes.byref(out), ctypes.byref(nout),
                                        ctypes.byref(done))
    if rc or not done.value:
        raise RuntimeError("decimal conversion: " + ff.lib().ffg_last_error().decode())
    return _digits(out, nout.value)


# ------------------------------------------------------------------ sizes


def _fib_limbs(n):
    return int((n * 0.6942419136306174 - 1.1609640474436812) / 64) + 1


def work(case):
    """Operands read once, results written once (no operations are counted:
    the transforms are integer work, for which no peak is measured)."""
    kind = case["kind"]
    if kind == "fib":
        return {"bytes": 8.0 * _fib_limbs(case["n"]), "flops": 0.0}
    if kind in ("mul", "big"):
        ops = case["na"] if case.get("square") else case["na"] + case["nb"]
        return {"bytes": 8.0 * (ops + case["na"] + case["nb"] + 1), "flops": 0.0}
    if kind == "batch":
        sizes = uneven_sizes(case["sizes"], case["count"], case["lo"], case["hi"])
        return {"bytes": 16.0 * sum((a + 63) // 64 + (b + 63) // 64 for a, b in sizes), "flops": 0.0}
    return {"bytes": 8.0 * case["limbs"] + 64 * case["limbs"] * math.log10(2), "flops": 0.0}


# ------------------------------------------------------------------ exact values


def _int(x):
    return int.from_bytes(x.contiguous().cpu().numpy().tobytes(), "little")


def _array(v, n):
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype=np.int64).copy()


def _times(x, y):
    """x y for Python integers: long ones by one double-precision FFT over
    their bytes (coefficients below 2^44, so every one rounds to itself)."""
    nx, ny = (x.bit_length() + 7) // 8, (y.bit_length() + 7) // 8
    if min(nx, ny) < 5000:
        return x * y
    n = 1 << (nx + ny - 1).bit_length()
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def spectrum(v, nv):
        raw = torch.from_numpy(np.frombuffer(v.to_bytes(nv, "little"), dtype=np.uint8).copy())
        return torch.fft.rfft(raw.to(dev).to(torch.float64) - 127.5, n=n), float(nv)

    # digits centred at 127.5 keep the rounding error small; the product of the
    # constant parts is added back by running sums
    (fx, _), (fy, _) = spectrum(x, nx), spectrum(y, ny)
    c = torch.fft.irfft(fx * fy, n=n)[: nx + ny - 1]
    del fx, fy
    bx = torch.from_numpy(np.frombuffer(x.to_bytes(nx, "little"), dtype=np.uint8).copy()).to(dev).to(torch.float64)
    by = torch.from_numpy(np.frombuffer(y.to_bytes(ny, "little"), dtype=np.uint8).copy()).to(dev).to(torch.float64)

    def windows(v, nv, other):
        # sum of v_i over i with 0 <= k - i < other, for every k
        s = torch.cumsum(torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), v]), 0)
        k = torch.arange(nx + ny - 1, device=dev)
        return s[torch.clamp(k + 1, max=nv)] - s[torch.clamp(k + 1 - other, min=0)]

    k = torch.arange(nx + ny - 1, device=dev, dtype=torch.float64)
    terms = torch.clamp(torch.minimum(k + 1, nx + ny - 1 - k), max=float(min(nx, ny)))
    c = c + 127.5 * (windows(bx, nx, ny) + windows(by, ny, nx)) - 127.5 * 127.5 * terms
    c = torch.round(c).to(torch.int64)
    pad = -c.numel() % 8
    c = torch.cat([c, torch.zeros(pad, dtype=torch.int64, device=dev)]).reshape(-1, 8).t().contiguous().cpu().numpy()
    return sum(int.from_bytes(c[j].tobytes(), "little") << (8 * j) for j in range(8))


def _fib(n):
    a, b = 0, 1  # F(k), F(k + 1)
    for bit in bin(n)[2:]:
        aa, bb = _times(a, a), _times(b, b)
        c, d = 2 * _times(a, b) - aa, aa + bb
        a, b = (d, c + d) if bit == "1" else (c, d)
    return a


def exact(case, seed):
    kind = case["kind"]
    if kind == "fib":
        if case["n"] > 120_000_000:
            return None
        v = _fib(_fib_index(case, seed))
        return _array(v, (v.bit_length() + 63) // 64)
    if kind in ("mul", "big"):
        if case["na"] + case["nb"] > 10_000_000:
            return None
        a = _int(_limbs(case["na"], 2 * seed))
        b = a if case.get("square") else _int(_limbs(case["nb"], 2 * seed + 1))
        v = _times(a, b)
        return _array(v, (v.bit_length() + 63) // 64 if kind == "big" else case["na"] + case["nb"] + 1)
    if kind == "batch":
        s = prepare(case, seed)
        if s["x"].numel() > 2_000_000:
            return None
        x = s["x"].cpu()
        got = []
        for (na, nb), (ia, ib) in zip(s["limbs"].tolist(), s["first"].tolist()):
            got.append(_array(_times(_int(x[ia: ia + na]), _int(x[ib: ib + nb])), na + nb + 1))
        return np.concatenate(got)
    if case["limbs"] > 60_000:
        return None
    return np.frombuffer(_decimal(_int(_limbs(case["limbs"], seed))).encode(), dtype=np.uint8).copy()


def _decimal(x):
    """Decimal digits by halves: str() has a digit limit and is slow for long numbers."""
    def digits(v, d):
        if d <= 4000:
            return str(v).rjust(d, "0")
        lo = d // 2
        q, r = divmod(v, 10**lo)
        return digits(q, d - lo) + digits(r, lo)

    return digits(x, int(x.bit_length() * math.log10(2)) + 2).lstrip("0")
