// The four-step column passes with the column length fixed at compile time,
// for columns of R = 2^RN (6 <= RN <= 12) or 3 2^RN words (RN <= 11).
//
// A CTA holds a tile of wc columns x R rows in shared memory, one padded
// line per column (pad(i) = i + i/16).  The length-2^RN transform of each column
// (of each of its three blocks of 2^RN words when R = 3 2^RN) is two or three
// radix steps (decimation in frequency forward, in time inverse):
//   A: radix 2^LA at stride 2^RN / 2^LA (absent when LA = 0),
//   B: radix 2^LB at stride 16,
//   C: radix 16 at stride 1 (no step twiddles);
// with R = 3 2^RN a radix-3 step at stride 2^RN comes first (forward) or last
// (inverse), in the registers of the first (last) radix step, as in the
// generic line transforms (r3_dif / r3_dit).
// k_col_fwd2: the first step reads the operand's digits straight from its
//   limbs (the reference's Src reader, src/ntt_kernels.c:29-74, one digit per
//   word), step C ends with the four-step twiddle ω_L^(n2 k1) and stores the
//   residues row-major, as the generic column pass (ffg_ntt.cu k_col_fwd).
// k_col_inv2: step C^-1 reads the row pass's output (scaled there) straight from
//   global memory, the last step stores it (or adds it into the split's
//   residues), as k_col_inv.
// Each step maps thread slots p = threadIdx.x + blockDim.x k to (column p mod wc,
// group p / wc), so a warp's global accesses cover min(wc, 32) consecutive
// words of each row it touches, and consecutive lines start 32 / min(wc, 32)
// banks apart: no shared access has a bank conflict.
//
// Bound by integer issue and by the latency of the strided rows.  Radix 16 at
// stride 1 where radix 32 stood halves a thread's registers and its chain of
// dependent work for the same instruction count (12.3 a word for 4 levels
// against 16.1 for 5), so twice the threads share a tile; results keep their
// pointer in registers (a job field in shared memory was read back for every
// word), digits are 32-bit index arithmetic, and the radix-3 step needs no
// pass of its own.  Square of 2^22 limbs (L = 2^24): inverse 236 -> 164 us
// (402 MB, 37 % of the copy bandwidth), forward 178 -> 178; L = 3 2^23: inverse
// 482 -> 297 us, forward 420 -> 268; F(10^9) chain 4700 -> 4050 us.
#include "ffg_internal.h"
#include "ffg_lines.cuh"

namespace ffg {

__host__ __device__ constexpr int brev4(int u) { return ((u & 1) << 3) | ((u & 2) << 1) | ((u & 4) >> 1) | ((u & 8) >> 3); }

// The radix-3 step triples the registers of the step next to it: radix 8 at most there.
template <int RN, bool R3> struct ColShape {
    static constexpr int LA = R3 ? (RN <= 7 ? 0 : RN <= 10 ? 2 : 3) : (RN <= 9 ? 0 : RN <= 11 ? 3 : 4);
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
    FFG_DEV_INLINE void fetch(const ColSrc &S, uint32_t i) { v = i < S.cs ? __ldg(S.src + i) : 0u; }
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
        a = ok && q < S.nw ? __ldg(S.src + q) : 0u;
        b = ok && q + 1 < S.nw ? __ldg(S.src + q + 1) : 0u;
        c = ok && (bit & 31) + S.w > 64 && q + 2 < S.nw ? __ldg(S.src + q + 2) : 0u;
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

// A tile's place: rows of C words, columns [c0, c0 + 2^wlg), LS words per line.
struct ColTile {
    uint32_t C, c0, wlg, wm, LS; // wm = 2^wlg - 1
};

// The first step of a forward column tile of 2^RN rows, straight from the
// digits, when only rows below NZ times its stride can be nonzero (a product's
// operands fill at most the lower half of the transform, a short operand much
// less): the zero slots are neither read nor transformed (dft_dif_nz).
template <int PI, int RN, int NZ, bool W32>
FFG_DEV_INLINE void col_fwd2_first(const PrimeDev &P, const ColSrc &S, const ColTile &T, uint32_t *smem) {
    using Q = ColGeo<RN, false>;
    const uint32_t slots = Q::SE << T.wlg;
    const uint2 *tw = P.stw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
#pragma unroll 1
    for (uint32_t sl = threadIdx.x; sl < slots; sl += blockDim.x) {
        const uint32_t c = sl & T.wm, j = sl >> T.wlg;
        uint32_t x[Q::RE];
        digits<PI, W32, Q::RE, NZ>(x, S, j * T.C + T.c0 + c, Q::SE * T.C, P);
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
template <int PI, int RN, int NB, int NZ, bool W32>
FFG_DEV_INLINE void col_fwd2_first_r3(const PrimeDev &P, const ColSrc &S, const ColTile &T, uint32_t *smem) {
    using Q = ColGeo<RN, true>;
    constexpr uint32_t p = kPrimeC[PI];
    static_assert(NB == 1 || NZ == (int)Q::RE, "pruned in the first block only");
    const uint32_t slots = Q::SE << T.wlg;
    const uint2 *tw = P.stw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
#pragma unroll 1
    for (uint32_t sl = threadIdx.x; sl < slots; sl += blockDim.x) {
        const uint32_t c = sl & T.wm, j = sl >> T.wlg, i0 = j * T.C + T.c0 + c, bi = Q::R * T.C;
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
    if constexpr (R3) col_fwd2_first_r3<PI, RN, 1, NZ, W32>(P, S, T, smem);
    else col_fwd2_first<PI, RN, NZ, W32>(P, S, T, smem);
}
template <int PI, int RN, bool R3, bool W32>
FFG_DEV_INLINE void col_fwd2_first_any(const PrimeDev &P, const ColSrc &S, const ColTile &T, uint32_t *smem,
                                       uint32_t rows_nz) {
    using Q = ColGeo<RN, R3>;
    constexpr int M = Q::LE, RE = Q::RE;
    if constexpr (R3) {
        if (rows_nz > 2 * Q::R) return col_fwd2_first_r3<PI, RN, 3, RE, W32>(P, S, T, smem);
        if (rows_nz > Q::R) return col_fwd2_first_r3<PI, RN, 2, RE, W32>(P, S, T, smem);
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

template <int PI, int RN, bool R3>
FFG_DEV_INLINE void col_fwd2_body(const PrimeDev &P, const FourStep &G, const FSJob &J, uint32_t *smem) {
    using Q = ColGeo<RN, R3>;
    const uint32_t op = G.square ? 0 : (blockIdx.z & 1);
    const uint32_t C = 1u << G.c, wc = G.wc;
    const ColTile T{C, blockIdx.x * wc, G.wc_lg, wc - 1, col2_stride(Q::NBLK * Q::R, wc)};
    const uint64_t ns = op ? J.nb : J.na, cs = op ? J.cb : J.ca, off = op ? J.off_b : J.off_a;
    const uint32_t w = J.width;
    uint32_t *const y = (op ? J.yb : J.ya) + (size_t)PI * G.L + T.c0;

    // rows at or past rows_nz are zero in every column of the tile
    const uint64_t avail = (ns * 64 + w - 1) / w; // digits that start inside the limbs
    const uint64_t lim = cs < (avail > off ? avail - off : 0) ? cs : (avail > off ? avail - off : 0);
    const uint32_t rows_nz = lim > T.c0 ? (uint32_t)((lim - T.c0 + C - 1) >> G.c) : 0;
    const ColSrc S = col_src(op ? J.b : J.a, ns, cs, off, w);
    if (w == 32) col_fwd2_first_any<PI, RN, R3, true>(P, S, T, smem, rows_nz);
    else col_fwd2_first_any<PI, RN, R3, false>(P, S, T, smem, rows_nz);
    __syncthreads();
    if (Q::LA) {
        col_step<PI, Q::LB, 4, true>(T, Q::NBLK * (Q::R / Q::RB), P.stw + c_lines.tw_off[4 * 6 + Q::LB], smem);
        __syncthreads();
    }
    // step C, then ω_L^(n2 k1): position q 2^RN + 16 b + t holds frequency
    // k1 = q + m brev_RN(16 b + t) = q + m (brev_4(t) 2^(RN - 4) + brev_(RN - 4)(b)),
    // m = 3 with the radix-3 step (q its block), else m = 1 and q = 0; n2 < C and
    // k1 < R keep the exponents below L.  A thread's column is the same in all its
    // slots (blockDim.x is a multiple of wc).
    constexpr uint32_t m3 = R3 ? 3 : 1;
    const uint32_t ms = (uint32_t)G.mstep, slots = (Q::NBLK * (Q::R / 16)) << T.wlg;
    const uint32_t c = threadIdx.x & T.wm, n2 = T.c0 + c;
    const uint32_t step = twm<PI>(P, ((n2 * m3) << (RN - 4)) * ms);
#pragma unroll 1
    for (uint32_t s = threadIdx.x; s < slots; s += blockDim.x) {
        const uint32_t b = s >> T.wlg, q = b >> (RN - 4), bl = b & ((Q::R >> 4) - 1);
        uint32_t cur = twm<PI>(P, n2 * (q + m3 * (__brev(bl) >> (32 - (RN - 4)))) * ms);
        uint32_t x[16];
        const uint32_t *d = smem + c * T.LS + 17 * b;
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = d[t];
        dft_dif<PI, 4>(x);
        uint32_t *o = y + (size_t)(16 * b) * C + c;
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int t = brev4(u); // compile-time after unrolling
            o[(size_t)t << G.c] = mo<PI>(x[t], cur);
            if (u < 15) cur = mo<PI>(cur, step);
        }
    }
}

constexpr uint32_t kColThreads = 512; // at most; 64 registers each, 32 warps an SM

template <int RN, bool R3>
__global__ void __launch_bounds__(kColThreads, 2) k_col_fwd2(Primes3 P3, FourStep G, FSJobs jobs) {
    extern __shared__ uint32_t smem[];
    __shared__ FSJob J;
    if (threadIdx.x == 0) {
        const uint32_t i = G.square ? blockIdx.z : (blockIdx.z >> 1);
        J = jobs.ext ? jobs.ext[i] : jobs.j[i < FFG_FS_JOBS ? i : 0];
    }
    __syncthreads();
    switch (blockIdx.y + G.prime0) {
    case 0: col_fwd2_body<0, RN, R3>(P3.pr[0], G, J, smem); break;
    case 1: col_fwd2_body<1, RN, R3>(P3.pr[1], G, J, smem); break;
    default: col_fwd2_body<2, RN, R3>(P3.pr[2], G, J, smem); break;
    }
}

// Where a thread's column of results goes: written, or added into the split's
// residues.
struct ColOut {
    uint32_t *out;
    bool acc;
    uint32_t clg;
};
template <int PI> FFG_DEV_INLINE void col_out(const ColOut &O, uint32_t row, uint32_t v) {
    uint32_t *p = O.out + ((size_t)row << O.clg);
    *p = O.acc ? ad<PI>(*p, v) : v;
}

template <int PI, int RN, bool R3>
FFG_DEV_INLINE void col_inv2_body(const PrimeDev &P, const FourStep &G, const FSJob &J, uint32_t *smem) {
    using Q = ColGeo<RN, R3>;
    const uint32_t C = 1u << G.c, wc = G.wc;
    const ColTile T{C, blockIdx.x * wc, G.wc_lg, wc - 1, col2_stride(Q::NBLK * Q::R, wc)};
    const uint32_t c = threadIdx.x & T.wm; // the same in all the thread's slots
    const uint32_t *const y = J.ya + (size_t)PI * G.L + T.c0 + c;
    const ColOut O{(J.yacc ? J.yacc + (size_t)PI * J.acc_stride + J.acc_off : J.ya + (size_t)PI * G.L) + T.c0 + c,
                   J.yacc != nullptr, G.c};
    uint32_t *const line = smem + c * T.LS;
    {
        const uint32_t slots = (Q::NBLK * (Q::R / 16)) << T.wlg;
#pragma unroll 1
        for (uint32_t s = threadIdx.x; s < slots; s += blockDim.x) {
            const uint32_t b = s >> T.wlg;
            const uint32_t *g = y + ((size_t)(16 * b) << G.c);
            uint32_t x[16];
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = g[(size_t)t << G.c];
            dft_dit<PI, 4>(x);
            uint32_t *d = line + 17 * b;
#pragma unroll
            for (int t = 0; t < 16; t++) d[t] = x[t];
        }
    }
    __syncthreads();
    if (Q::LA) {
        col_step<PI, Q::LB, 4, false>(T, Q::NBLK * (Q::R / Q::RB), P.istw + c_lines.tw_off[4 * 6 + Q::LB], smem);
        __syncthreads();
    }
    // the last step (and radix 3, the generic r3_dit)
    constexpr uint32_t p = kPrimeC[PI];
    const uint2 *tw = P.istw + c_lines.tw_off[(Q::LA ? RN - Q::LE : 4) * 6 + Q::LE];
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
                col_out<PI>(O, row, ad<PI>(ad<PI>(y0, z1), z2));
                col_out<PI>(O, row + Q::R, ad<PI>(sb<PI>(y0, z2), u));
                col_out<PI>(O, row + 2 * Q::R, sb<PI>(sb<PI>(y0, z1), u));
            } else {
                col_out<PI>(O, row, x[0][t]);
            }
        }
    }
}

template <int RN, bool R3>
__global__ void __launch_bounds__(kColThreads, 2) k_col_inv2(Primes3 P3, FourStep G, FSJobs jobs) {
    extern __shared__ uint32_t smem[];
    __shared__ FSJob J;
    if (threadIdx.x == 0) J = jobs.ext ? jobs.ext[blockIdx.z] : jobs.j[blockIdx.z < FFG_FS_JOBS ? blockIdx.z : 0];
    __syncthreads();
    switch (blockIdx.y + G.prime0) {
    case 0: col_inv2_body<0, RN, R3>(P3.pr[0], G, J, smem); break;
    case 1: col_inv2_body<1, RN, R3>(P3.pr[1], G, J, smem); break;
    default: col_inv2_body<2, RN, R3>(P3.pr[2], G, J, smem); break;
    }
}

cudaError_t set_line_consts_cols(const LineConsts &h) { return cudaMemcpyToSymbol(c_lines, &h, sizeof h); }

static size_t col2_smem(const FourStep &G) { return (size_t)G.wc * col2_stride(G.R, G.wc) * sizeof(uint32_t); }

constexpr size_t kColSmemMax = 216 * 1024;

// Whether the fixed-shape column passes take this geometry: columns of
// 2^6 .. 2^12 words (3 2^6 .. 3 2^11 with the radix-3 step), in tiles of 8..64
// columns that fit in shared memory (longer columns do not).
bool col2_ok(const FourStep &G) {
    return G.rn >= 6 && G.rn <= (G.r3 ? 11u : 12u) && G.wc >= 8 && G.wc <= 64 && G.wc == (1u << G.wc_lg) && G.wc <= (1u << G.c) &&
           col2_smem(G) <= kColSmemMax;
}

template <int RN, bool R3>
static cudaError_t launch_col2_t(bool fwd, const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t nz,
                                 cudaStream_t st) {
    const void *k = fwd ? (const void *)k_col_fwd2<RN, R3> : (const void *)k_col_inv2<RN, R3>;
    static bool attr[2] = {false, false};
    if (!attr[fwd]) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColSmemMax);
        if (e) return e;
        attr[fwd] = true;
    }
    const dim3 grid((1u << G.c) / G.wc, G.nprimes, nz);
    // threads per CTA: one per 16 words, at most 256 while four CTAs fit an SM's
    // shared memory, else 512 (at L = 2^24, tiles of 70 KB, the inverse pass takes
    // 164 us with 512 threads and 183 with 256; at L = 2^22, tiles of 35 KB, 45
    // and 39).  A multiple of wc, so that a thread keeps its column.
    const uint32_t groups = G.wc * (uint32_t)(G.R / 16), tmax = col2_smem(G) > 56 * 1024 ? kColThreads : kColThreads / 2;
    uint32_t threads = groups < tmax ? groups : tmax;
    threads = threads < 64 ? 64 : threads & ~31u;
    threads -= threads % G.wc;
    if (fwd) k_col_fwd2<RN, R3><<<grid, threads, col2_smem(G), st>>>(P3, G, jobs);
    else k_col_inv2<RN, R3><<<grid, threads, col2_smem(G), st>>>(P3, G, jobs);
    return cudaGetLastError();
}

template <bool R3>
static cudaError_t launch_col2_r(bool fwd, const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t nz,
                                 cudaStream_t st) {
    switch (G.rn) {
    case 6: return launch_col2_t<6, R3>(fwd, P3, G, jobs, nz, st);
    case 7: return launch_col2_t<7, R3>(fwd, P3, G, jobs, nz, st);
    case 8: return launch_col2_t<8, R3>(fwd, P3, G, jobs, nz, st);
    case 9: return launch_col2_t<9, R3>(fwd, P3, G, jobs, nz, st);
    case 10: return launch_col2_t<10, R3>(fwd, P3, G, jobs, nz, st);
    case 11: return launch_col2_t<11, R3>(fwd, P3, G, jobs, nz, st);
    default:
        if constexpr (R3) return cudaErrorInvalidValue; // col2_ok: at most 3 2^11 rows
        else return launch_col2_t<12, R3>(fwd, P3, G, jobs, nz, st);
    }
}

// nz: grid depth (jobs x operands for the forward pass, jobs for the inverse).
cudaError_t launch_col2(bool fwd, const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t nz,
                        cudaStream_t st) {
    return G.r3 ? launch_col2_r<true>(fwd, P3, G, jobs, nz, st) : launch_col2_r<false>(fwd, P3, G, jobs, nz, st);
}

} // namespace ffg
