"""GPU test of the CRT alone (ffg_crt_residues): residues of chosen
coefficients X_i < p1 p2 p3, for every width and around the edges of its
super-limbs (32 coefficients), CTAs (2048 and 8192) and last quads, against
sum X_i 2^(i b) in Python integers.  Besides random coefficients: the largest
ones (every carry the column sums can hold), and runs of all-ones words with a
carry started at the bottom or in the middle, which has to cross threads,
warps and CTAs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P = (2113929217, 2013265921, 1811939329)
M = P[0] * P[1] * P[2]


def _total(xs, b):
    """sum xs[i] 2^(i b): every eighth value lies b bytes from the next."""
    t = 0
    for k in range(8):
        raw = bytearray(b * ((len(xs) + 7) // 8) + 16)
        for q, x in enumerate(xs[k::8]):
            raw[q * b: q * b + 12] = x.to_bytes(12, "little")
        t += int.from_bytes(raw, "little") << (k * b)
    return t


def _coefficients(kind, n, b, rng):
    if kind == "random":
        return [int(h) << 62 | int(l) for h, l in zip(rng.integers(0, 2**30, n), rng.integers(0, 2**62, n))]
    if kind == "largest":
        return [M - 1] * n
    xs = [2**b - 1] * n               # every bit of the sum is one ...
    at = 0 if kind == "ripple" else n // 2
    xs[at] += 1                       # ... and a carry runs from here to the top
    return xs


# (coefficients of a, of b): conv = ca + cb - 1 about a quad's, a super-limb's, a CTA's edge; one CTA, a few,
# and enough for the CTAs of 8192 coefficients (more than 1024 of 2048)
SHAPES = [(2081, 2017), (2081, 2048), (2082, 2048), (2081, 4063), (2081, 4064), (5000, 3193), (5000, 3194),
          (40000, 25537), (1200000, 1100003)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["random", "largest", "ripple", "middle"])
def test_crt_alone(ff, shape, kind):
    ff.init(1 << 22)
    side = torch.cuda.Stream()
    seen = set()
    # bit lengths whose plans take each width for these coefficient counts
    for b in (32, 33, 34, 35):
        ca, cb = shape
        bits_a, bits_b = ca * b, cb * b
        pl = ff.plan(bits_a, bits_b)
        if pl["kernel"] != 1 or pl["split"] or pl["width"] in seen:
            continue
        b, conv, L = pl["width"], pl["conv"], pl["L"]
        seen.add(b)
        if conv > 100000 and len(seen) > 1:
            break  # the long shape once
        na, nb = (bits_a + 63) // 64, (bits_b + 63) // 64
        xs = _coefficients(kind, conv, b, np.random.default_rng(7 * conv + b))
        y = np.full((3, L), 0xDEADBEEF, dtype=np.uint32)  # words past conv are not residues
        for k, p in enumerate(P):
            if kind == "random":
                y[k, :conv] = [x % p for x in xs]
            else:
                y[k, :conv] = xs[1] % p
                for i in (0, conv // 2):
                    y[k, i] = xs[i] % p
        with torch.cuda.stream(side):
            dy = torch.from_numpy(y.view(np.int32)).cuda()
            out = torch.full((na + nb + 1,), -1, dtype=torch.int64, device="cuda")
            ff.crt_residues(out.data_ptr(), dy.data_ptr(), na, bits_a, nb, bits_b, False, side.cuda_stream)
            got = int.from_bytes(out.cpu().numpy().tobytes(), "little")
        want = _total(xs, b) % (1 << 64 * (na + nb + 1))
        assert got == want, (b, conv, L)
    assert seen
