"""CPU tests of the addressing of the fixed-shape four-step passes
(ffg_rows.cu, ffg_cols.cu), restated for every shape they instantiate: each
radix step touches every word of a line exactly once and stays inside the
line, and a warp's simultaneous accesses fall in distinct banks (rows of 512
words: at most two to a bank in step B)."""
import re
from collections import Counter
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "fastfib_b200" / "csrc"


def _row_shapes():
    text = (CSRC / "ffg_rows.cu").read_text()
    return {int(c): (int(a), int(b), int(k)) for c, a, b, k in
            re.findall(r"RowShape<(\d+)> \{ static constexpr int LA = (\d), LB = (\d), KB = (\d)", text)}


def _col_shape(rn, r3):
    la = (0 if rn <= 7 else 2 if rn <= 10 else 3) if r3 else (0 if rn <= 9 else 3 if rn <= 11 else 4)
    return la, rn - 4 - la


def _worst(first):
    """Most lanes of a warp on one bank, over the warps of a step's groups."""
    return max(max(Counter(a % 32 for a in first[i: i + 32]).values()) for i in range(0, len(first), 32))


def test_row_shapes():
    shapes = _row_shapes()
    assert sorted(shapes) == [9, 10, 11, 12, 13]
    for clg, (la, lb, kb) in shapes.items():
        C, ra, rb = 1 << clg, 1 << la, 1 << lb
        T, sa = 256 if clg == 13 else C // 16, C >> la
        pad = [i + i // 32 for i in range(C)]
        stride = ((C + (C - 1) // 32 + 1 + 31) & ~31) + 1
        assert pad[-1] < stride
        A, B = [], []
        for k in range(C // ra // T):
            for tau in range(T):
                j = tau + T * k
                A.append([j + j // 32 + t * (sa + sa // 32) for t in range(ra)])
        for k in range(C // rb // T):
            for tau in range(T):
                g = tau + T * k
                j, r = g & 15, g >> 5
                b = r % kb + ((g >> 4) & 1) * kb + (r // kb) * 2 * kb
                words = [b * (16 * rb + rb // 2) + j + 16 * t + t // 2 for t in range(rb)]
                assert words == [pad[b * 16 * rb + j + 16 * t] for t in range(rb)]
                assert j == tau & 15  # the twiddles' index
                B.append(words)
        Cg = [[16 * b + b // 2 + t for t in range(16)] for b in range(C // 16)]
        for step in (A, B, Cg):
            assert sorted(a for g in step for a in g) == pad
        for step, most in ((A, 1), (B, 2 if clg == 9 else 1), (Cg, 1)):
            assert all(_worst([g[t] for g in step]) <= most for t in range(len(step[0]))), clg


def test_column_shapes():
    for rn in range(6, 13):
        for r3 in (False, True):
            if r3 and rn > 11:
                continue
            la, lb = _col_shape(rn, r3)
            R, nblk, rb = 1 << rn, 3 if r3 else 1, 1 << lb
            assert 2 <= lb <= 5 and (not r3 or (la or lb) <= 3)
            sa, bp = R >> la, R + R // 16
            pad = [i + i // 16 for i in range(nblk * R)]
            # the step next to the digits or the result: stride sa, or 16 when it is step B
            se, sep, re_ = (sa, sa + sa // 16, 1 << la) if la else (16, 17, rb)
            E = [[q * bp + j + (j // 16 if la else 0) + t * sep for q in range(nblk) for t in range(re_)]
                 for j in range(se)]
            B = [[b * 17 * rb + j + 17 * t for t in range(rb)] for b in range(nblk * R // (16 * rb)) for j in range(16)]
            Cg = [[17 * b + t for t in range(16)] for b in range(nblk * R // 16)]
            for step in (E, B, Cg) if la else (E, Cg):
                assert sorted(a for g in step for a in g) == pad, (rn, r3)
            for wc in (8, 16, 32, 64):
                LS = ((nblk * R + nblk * R // 16 + 31) & ~31) + 32 // min(wc, 32)
                assert LS > pad[-1]
                for step in (E, B, Cg) if la else (E, Cg):
                    assert _worst([(s % wc) * LS + step[s // wc][0] for s in range(wc * len(step))]) == 1, (rn, r3, wc)
