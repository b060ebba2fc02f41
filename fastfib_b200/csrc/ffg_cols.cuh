// Radix steps on lines of 2^RN or 3 2^RN words in shared memory with the line
// length fixed at compile time, and their first step straight from an operand's
// digits: the column passes (ffg_cols.cu: a tile of columns, one line each) and
// the one-CTA convolution (ffg_conv.cu: a line per operand).
#pragma once
#include "ffg_internal.h"
#include "ffg_lines.cuh"

namespace ffg {

__host__ __device__ constexpr int brev4(int u) { return ((u & 1) << 3) | ((u & 2) << 1) | ((u & 4) >> 1) | ((u & 8) >> 3); }

// The radix-3 step triples the registers of the step next to it: radix 8 at most
// there.  (RN 13, 14 and 3 2^12: one-CTA convolutions only, no column is as long.)
template <int RN, bool R3> struct ColShape {
    static constexpr int LA = R3 ? (RN <= 7 ? 0 : RN <= 10 ? 2 : 3) : (RN <= 9 ? 0 : RN <= 11 ? 3 : RN <= 13 ? 4 : 5);
    static constexpr int LB = RN - 4 - LA;
};

template <int RN, bool R3> struct ColGeo {
    static constexpr int LA = ColShape<RN, R3>::LA, LB = ColShape<RN, R3>::LB;
    static constexpr uint32_t R = 1u << RN, NBLK = R3 ? 3 : 1;
    static constexpr uint32_t BP = R + R / 16; // padded block
    static constexpr uint32_t RA = 1u << LA, RB = 1u << LB;
    static constexpr uint32_t SA = R >> LA, SAP = SA + SA / 16;
    static constexpr uint32_t NBP = 17 * RB;   // padded block of step B (16 RB words)
    // the step next to the digits (forward) or the result (inverse)
    static constexpr int LE = LA ? LA : LB;
    static constexpr uint32_t RE = 1u << LE, SE = LA ? SA : 16, SEP = LA ? SAP : 17;
    static_assert(LA + LB + 4 == RN && LB >= 2 && LB <= 5 && (!R3 || LE <= 3), "three steps cover the column");
};

// Shared words per column line: the padded length, rounded so that
// consecutive lines start 32 / min(wc, 32) banks apart.
__host__ __device__ inline uint32_t col2_stride(uint32_t R, uint32_t wc) {
    const uint32_t wl = wc < 32 ? wc : 32;
    return ((R + R / 16 + 31) & ~31u) + 32 / wl;
}

// The digits of a forward column tile: w bits each, the first of them at bit
// sft of *src; digit i is zero from cs on, words are zero from nw on.  Indices
// are below 2^26 and bit positions below 2^32 (i < 3 2^23, w <= 35).
struct ColSrc {
    const uint32_t *src;
    uint32_t nw, cs, w, sft;
};
FFG_DEV_INLINE ColSrc col_src(const uint64_t *limbs, uint64_t ns, uint64_t cs, uint64_t off, uint32_t w) {
    const uint64_t bit = off * w, q = bit >> 5, nw = 2 * ns > q ? 2 * ns - q : 0;
    ColSrc S;
    S.src = (const uint32_t *)limbs + q;
    S.nw = nw < 0xffffffffull ? (uint32_t)nw : 0xffffffffu;
    S.cs = (uint32_t)cs;
    S.w = w;
    S.sft = (uint32_t)(bit & 31);
    // 32-bit digits are words: one bound for both
    if (w == 32 && S.cs > S.nw) S.cs = S.nw;
    return S;
}

// The raw words of one digit, loaded before any of a slot's is used.
template <bool W32> struct DigitRaw;
template <> struct DigitRaw<true> {
    uint32_t v;
    FFG_DEV_INLINE void fetch(const ColSrc &S, uint32_t i) { v = i < S.cs ? S.src[i] : 0u; }
    template <int PI> FFG_DEV_INLINE uint32_t residue(const ColSrc &, uint32_t, const PrimeDev &) const {
        constexpr uint32_t p = kPrimeC[PI];
        uint32_t l = v;
        l = min(l, l - p);
        return min(l, l - p);
    }
};
template <> struct DigitRaw<false> {
    uint32_t a, b, c;
    FFG_DEV_INLINE void fetch(const ColSrc &S, uint32_t i) {
        const uint32_t bit = S.sft + i * S.w, q = bit >> 5;
        const bool ok = i < S.cs;
        a = ok && q < S.nw ? S.src[q] : 0u;
        b = ok && q + 1 < S.nw ? S.src[q + 1] : 0u;
        c = ok && (bit & 31) + S.w > 64 && q + 2 < S.nw ? S.src[q + 2] : 0u;
    }
    template <int PI> FFG_DEV_INLINE uint32_t residue(const ColSrc &S, uint32_t i, const PrimeDev &P) const {
        constexpr uint32_t p = kPrimeC[PI];
        const uint32_t s = (S.sft + i * S.w) & 31;
        uint32_t l = __funnelshift_r(a, b, s), h = __funnelshift_r(b, c, s);
        if (S.w < 32) l &= (1u << S.w) - 1, h = 0;
        else h &= (1u << (S.w - 32)) - 1;
        l = min(l, l - p);
        l = min(l, l - p);
        return ad<PI>(l, sh<PI>(h, make_uint2(P.c32, P.c32s)));
    }
};

// Digits i0 + t di (t < NZ) mod p into x[t], zeros from NZ on.  Short digits are
// loaded before any is reduced, up to 16 words (4 digits of over 32 bits) at a
// time.
template <int PI, bool W32, int RE, int NZ>
FFG_DEV_INLINE void digits(uint32_t (&x)[RE], const ColSrc &S, uint32_t i0, uint32_t di, const PrimeDev &P) {
    constexpr int AT = W32 ? 16 : 4, STEP = NZ <= AT ? NZ : AT;
#pragma unroll
    for (int t0 = 0; t0 < NZ; t0 += STEP) {
        DigitRaw<W32> raw[STEP];
#pragma unroll
        for (int t = 0; t < STEP; t++) raw[t].fetch(S, i0 + (t0 + t) * di);
#pragma unroll
        for (int t = 0; t < STEP; t++) x[t0 + t] = raw[t].template residue<PI>(S, i0 + (t0 + t) * di, P);
    }
#pragma unroll
    for (int t = NZ; t < RE; t++) x[t] = 0;
}

// A tile's place: rows of C words, 2^wlg columns from c0, dc apart (1; 0 where
// every column is an operand of its own), LS words per line.
struct ColTile {
    uint32_t C, c0, wlg, wm, LS, dc; // wm = 2^wlg - 1
};

// The first step of a forward column tile of 2^RN rows, straight from the
// digits, when only rows below NZ times its stride can be nonzero (a product's
// operands fill at most the lower half of the transform, a short operand much
// less): the zero slots are neither read nor transformed (dft_dif_nz).
// src(c): where column c's digits are.
template <int PI, int RN, int NZ, bool W32, class Src>
FFG_DEV_INLINE void col_fwd2_first(const PrimeDev &P, Src src, const ColTile &T, uint32_t *smem) {
    using Q = ColGeo<RN, false>;
    const uint32_t slots = Q::SE << T.wlg;
    const uint2 *tw = P.stw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
#pragma unroll 1
    for (uint32_t sl = threadIdx.x; sl < slots; sl += blockDim.x) {
        const uint32_t c = sl & T.wm, j = sl >> T.wlg;
        uint32_t x[Q::RE];
        digits<PI, W32, Q::RE, NZ>(x, src(c), j * T.C + T.c0 + T.dc * c, Q::SE * T.C, P);
        dft_dif_nz<PI, Q::LE, NZ>(x);
        uint32_t *d = smem + c * T.LS + j + (Q::LA ? (j >> 4) : 0);
#pragma unroll
        for (uint32_t t = 1; t < Q::RE; t++) x[t] = sh<PI>(x[t], __ldg(&tw[(t - 1) * Q::SE + j]));
#pragma unroll
        for (uint32_t t = 0; t < Q::RE; t++) d[t * Q::SEP] = x[t];
    }
}

// The same for 3 2^RN rows: radix 3 at stride 2^RN on every position of the
// slot, then the radix step in each of the three blocks.  Only the first NB of
// the blocks can hold nonzero rows (NB = 1: y0 = x0, y1 = x0 w^j, y2 = x0 w^2j,
// and only below NZ times the stride; NB = 2: x2 = 0).
template <int PI, int RN, int NB, int NZ, bool W32, class Src>
FFG_DEV_INLINE void col_fwd2_first_r3(const PrimeDev &P, Src src, const ColTile &T, uint32_t *smem) {
    using Q = ColGeo<RN, true>;
    constexpr uint32_t p = kPrimeC[PI];
    static_assert(NB == 1 || NZ == (int)Q::RE, "pruned in the first block only");
    const uint32_t slots = Q::SE << T.wlg;
    const uint2 *tw = P.stw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
#pragma unroll 1
    for (uint32_t sl = threadIdx.x; sl < slots; sl += blockDim.x) {
        const uint32_t c = sl & T.wm, j = sl >> T.wlg, i0 = j * T.C + T.c0 + T.dc * c, bi = Q::R * T.C;
        const ColSrc S = src(c);
        uint32_t x[3][Q::RE];
#pragma unroll
        for (int b = 0; b < NB; b++) digits<PI, W32, Q::RE, NZ>(x[b], S, i0 + b * bi, Q::SE * T.C, P);
#pragma unroll
        for (uint32_t t = 0; t < Q::RE; t++) {
            if (t >= (uint32_t)NZ) {
                x[1][t] = x[2][t] = 0;
                continue;
            }
            const uint4 w = __ldg(&P.r3f[Q::R + j + Q::SE * t]);
            const uint32_t x0 = x[0][t], x1 = NB > 1 ? x[NB > 1 ? 1 : 0][t] : 0u, x2 = NB > 2 ? x[NB > 2 ? 2 : 0][t] : 0u;
            if (NB == 1) {
                x[1][t] = sh<PI>(x0, make_uint2(w.x, w.y));
                x[2][t] = sh<PI>(x0, make_uint2(w.z, w.w));
            } else {
                const uint32_t u = sh<PI>(x1 - x2 + p, c_lines.w3[PI]);
                x[0][t] = ad<PI>(ad<PI>(x0, x1), x2);
                x[1][t] = sh<PI>(ad<PI>(sb<PI>(x0, x2), u), make_uint2(w.x, w.y));
                x[2][t] = sh<PI>(sb<PI>(sb<PI>(x0, x1), u), make_uint2(w.z, w.w));
            }
        }
#pragma unroll
        for (int b = 0; b < 3; b++) dft_dif_nz<PI, Q::LE, NZ>(x[b]);
        uint32_t *d = smem + c * T.LS + j + (Q::LA ? (j >> 4) : 0);
#pragma unroll
        for (uint32_t t = 0; t < Q::RE; t++) {
            if (t) {
                const uint2 w = __ldg(&tw[(t - 1) * Q::SE + j]);
#pragma unroll
                for (int b = 0; b < 3; b++) x[b][t] = sh<PI>(x[b][t], w);
            }
#pragma unroll
            for (int b = 0; b < 3; b++) d[b * Q::BP + t * Q::SEP] = x[b][t];
        }
    }
}

// The first step for the least power of two NZ covering the nonzero rows (with
// the radix-3 step: in the first block, or all rows of NB blocks).
template <int PI, int RN, bool R3, bool W32, int NZ>
FFG_DEV_INLINE void col_fwd2_first_nz(const PrimeDev &P, const ColSrc &S, const ColTile &T, uint32_t *smem) {
    auto src = [&](uint32_t) -> const ColSrc & { return S; };
    if constexpr (R3) col_fwd2_first_r3<PI, RN, 1, NZ, W32>(P, src, T, smem);
    else col_fwd2_first<PI, RN, NZ, W32>(P, src, T, smem);
}
template <int PI, int RN, bool R3, bool W32>
FFG_DEV_INLINE void col_fwd2_first_any(const PrimeDev &P, const ColSrc &S, const ColTile &T, uint32_t *smem,
                                       uint32_t rows_nz) {
    using Q = ColGeo<RN, R3>;
    constexpr int M = Q::LE, RE = Q::RE;
    if constexpr (R3) {
        auto src = [&](uint32_t) -> const ColSrc & { return S; };
        if (rows_nz > 2 * Q::R) return col_fwd2_first_r3<PI, RN, 3, RE, W32>(P, src, T, smem);
        if (rows_nz > Q::R) return col_fwd2_first_r3<PI, RN, 2, RE, W32>(P, src, T, smem);
    }
    const uint32_t nzt = (rows_nz + Q::SE - 1) / Q::SE;
    if (nzt <= 1) col_fwd2_first_nz<PI, RN, R3, W32, 1>(P, S, T, smem);
    else if (nzt <= 2) col_fwd2_first_nz<PI, RN, R3, W32, 2>(P, S, T, smem);
    else if (nzt <= 4 || M < 3) col_fwd2_first_nz<PI, RN, R3, W32, 4>(P, S, T, smem);
    else if (nzt <= 8 || M < 4) col_fwd2_first_nz<PI, RN, R3, W32, (M >= 3 ? 8 : 1)>(P, S, T, smem);
    else if (nzt <= 16 || M < 5) col_fwd2_first_nz<PI, RN, R3, W32, (M >= 4 ? 16 : 1)>(P, S, T, smem);
    else col_fwd2_first_nz<PI, RN, R3, W32, (M >= 5 ? 32 : 1)>(P, S, T, smem);
}

// One radix-2^M step of a tile in shared memory: forward DFT then twiddles, or
// twiddles then inverse DFT.  Group g of a line: block g >> slg (padded length
// blk) at offset j = g mod 2^slg (+ j / 16 where the stride is over 16).
template <int PI, int M, int SLG, bool FWD>
FFG_DEV_INLINE void col_step(const ColTile &T, uint32_t groups, const uint2 *__restrict__ tw, uint32_t *smem) {
    constexpr uint32_t RM = 1u << M, S = 1u << SLG, SP = S + S / 16, BLK = SP * RM;
    const uint32_t slots = groups << T.wlg;
#pragma unroll 1
    for (uint32_t s = threadIdx.x; s < slots; s += blockDim.x) {
        const uint32_t c = s & T.wm, g = s >> T.wlg, b = g >> SLG, j = g & (S - 1);
        uint32_t *d = smem + c * T.LS + b * BLK + j + (SLG > 4 ? (j >> 4) : 0);
        uint32_t x[RM];
#pragma unroll
        for (uint32_t t = 0; t < RM; t++) x[t] = d[t * SP];
        if (FWD) dft_dif<PI, M>(x);
#pragma unroll
        for (uint32_t t = 1; t < RM; t++) x[t] = sh<PI>(x[t], __ldg(&tw[(t - 1) * S + j]));
        if (!FWD) dft_dit<PI, M>(x);
#pragma unroll
        for (uint32_t t = 0; t < RM; t++) d[t * SP] = x[t];
    }
}

// The last inverse step (and radix 3, the generic r3_dit): out(row, value) for
// every row of the lines; a thread's column is threadIdx.x mod 2^wlg in all its
// slots (blockDim.x is a multiple of 2^wlg).
template <int PI, int RN, bool R3, class Out>
FFG_DEV_INLINE void col_last(const PrimeDev &P, const ColTile &T, const uint32_t *smem, Out out) {
    using Q = ColGeo<RN, R3>;
    constexpr uint32_t p = kPrimeC[PI];
    const uint2 *tw = P.istw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
    const uint32_t *const line = smem + (threadIdx.x & T.wm) * T.LS;
    const uint32_t slots = Q::SE << T.wlg;
#pragma unroll 1
    for (uint32_t s = threadIdx.x; s < slots; s += blockDim.x) {
        const uint32_t j = s >> T.wlg;
        const uint32_t *d = line + j + (Q::LA ? (j >> 4) : 0);
        uint32_t x[Q::NBLK][Q::RE];
#pragma unroll
        for (uint32_t t = 0; t < Q::RE; t++)
#pragma unroll
            for (uint32_t b = 0; b < Q::NBLK; b++) x[b][t] = d[b * Q::BP + t * Q::SEP];
#pragma unroll
        for (uint32_t t = 1; t < Q::RE; t++) {
            const uint2 w = __ldg(&tw[(t - 1) * Q::SE + j]);
#pragma unroll
            for (uint32_t b = 0; b < Q::NBLK; b++) x[b][t] = sh<PI>(x[b][t], w);
        }
#pragma unroll
        for (uint32_t b = 0; b < Q::NBLK; b++) dft_dit<PI, Q::LE>(x[b]);
#pragma unroll
        for (uint32_t t = 0; t < Q::RE; t++) {
            const uint32_t row = j + Q::SE * t;
            if constexpr (R3) {
                const uint4 w = __ldg(&P.r3i[Q::R + row]);
                const uint32_t y0 = x[0][t], z1 = sh<PI>(x[1][t], make_uint2(w.x, w.y));
                const uint32_t z2 = sh<PI>(x[2][t], make_uint2(w.z, w.w));
                const uint32_t u = sh<PI>(z1 - z2 + p, c_lines.v3[PI]);
                out(row, ad<PI>(ad<PI>(y0, z1), z2));
                out(row + Q::R, ad<PI>(sb<PI>(y0, z2), u));
                out(row + 2 * Q::R, sb<PI>(sb<PI>(y0, z1), u));
            } else {
                out(row, x[0][t]);
            }
        }
    }
}

} // namespace ffg
