"""CPU tests of the shapes that the sources state themselves: the radix steps of a
column or a one-CTA line (ColShape, ffg_cols.cuh) for every length that the column
passes and the one-CTA convolution instantiate, and the threads per column of the short
squares (SQ_TPC, ffg_crt.cu).  Each step touches every word of the padded lines once."""
import random
import re
from pathlib import Path

from test_kernel_math import M64, square_column

CSRC = Path(__file__).resolve().parent.parent / "fastfib_b200" / "csrc"


def _ternary(text, env):
    """The value of nested a ? b : c over names, numbers and <=, parenthesised or not."""
    tok = re.findall(r"<=|[?:()]|\w+", text)

    def choice(i):
        v, i = term(i)
        if i < len(tok) and tok[i] == "?":
            a, i = choice(i + 1)
            assert tok[i] == ":"
            b, i = choice(i + 1)
            v = a if v else b
        return v, i

    def atom(i):
        if tok[i] == "(":
            v, i = choice(i + 1)
            assert tok[i] == ")"
            return v, i + 1
        return (int(tok[i]) if tok[i].isdigit() else env[tok[i]]), i + 1

    def term(i):
        v, i = atom(i)
        if i < len(tok) and tok[i] == "<=":
            w, i = atom(i + 1)
            v = v <= w
        return v, i

    v, i = choice(0)
    assert i == len(tok)
    return v


def _la(rn, r3):
    text = (CSRC / "ffg_cols.cuh").read_text()
    expr = re.search(r"struct ColShape \{\s*static constexpr int LA = ([^;]*);\s*"
                     r"static constexpr int LB = RN - 4 - LA;", text).group(1)
    return _ternary(expr, {"RN": rn, "R3": r3})


def test_every_line_length():
    cols = re.search(r"G\.rn >= (\d+) && G\.rn <= \(G\.r3 \? (\d+)u : (\d+)u\)", (CSRC / "ffg_cols.cu").read_text())
    conv = re.search(r"n >= (\d+) && n <= \(r3 \? (\d+)u : (\d+)u\)", (CSRC / "ffg_conv.cu").read_text())
    lo, hi = int(cols.group(1)), {True: int(cols.group(2)), False: int(cols.group(3))}
    assert int(conv.group(1)) == lo == 6
    top = {True: int(conv.group(2)), False: int(conv.group(3))}
    assert (hi, top) == ({True: 11, False: 12}, {True: 12, False: 14})
    for r3 in (False, True):
        for rn in range(lo, max(hi[r3], top[r3]) + 1):
            la = _la(rn, r3)
            lb = rn - 4 - la
            R, nblk, ra, rb = 1 << rn, 3 if r3 else 1, 1 << la, 1 << lb
            assert 2 <= lb <= 5 and 0 <= la <= 5 and (not r3 or (la or lb) <= 3), (rn, r3)
            pad = [i + i // 16 for i in range(nblk * R)]
            bp, sa = R + R // 16, R >> la
            se, sep, re_ = (sa, sa + sa // 16, ra) if la else (16, 17, rb)
            lines = 1 if rn <= hi[r3] else 2  # the one-CTA product: a line per operand, LS words apart
            ls = nblk * bp
            first = [c * ls + q * bp + j + (j // 16 if la else 0) + t * sep
                     for sl in range(se * lines) for c, j in [(sl % lines, sl // lines)]
                     for q in range(nblk) for t in range(re_)]
            inner = [c * ls + b * 17 * rb + j + 17 * t for c in range(lines) for b in range(nblk * R // (16 * rb))
                     for j in range(16) for t in range(rb)]
            last = [c * ls + 17 * b + t for c in range(lines) for b in range(nblk * R // 16) for t in range(16)]
            want = [c * ls + a for c in range(lines) for a in pad]
            for step in (first, inner, last) if la else (first, last):
                assert sorted(step) == want, (rn, r3)


def test_short_square_columns():
    """k_school_sq_pair's column split over SQ_TPC threads (one column a group of
    threads, SQ_NL + 3 columns a CTA) gives the square."""
    text = (CSRC / "ffg_crt.cu").read_text()
    tpc, nl, threads = (int(re.search(rf"constexpr uint32_t {n} = (\d+);", text).group(1))
                        for n in ("SQ_TPC", "SQ_NL", "SQ_THREADS"))
    assert tpc * (nl + 3) <= threads
    rng = random.Random(9)
    for _ in range(30):
        n = rng.randint(1, 70)
        a = [rng.getrandbits(64) if rng.random() < 0.8 else M64 for _ in range(n)]
        x = sum(v << 64 * i for i, v in enumerate(a))
        assert sum(square_column(a, j, tpc) << 64 * j for j in range(2 * n + 1)) == x * x
