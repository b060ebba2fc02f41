// CRT recombination and the fast-doubling linear passes, for sm_100a.
//
// k_crt, k_crt_pair, k_crt_flat (widths 32..35, every plan but the split's
// narrow ones): one CTA per 2048 coefficients, as 64 super-limbs of 32
// coefficients, which are exactly b 32-bit words of the product.
//   1. All 256 threads run Garner's method (the reference's crt_garner8,
//      src/crt.c:38-64) on quads of coefficients straight from global memory,
//        x2 = (r2 - r1) p1^-1 mod p2,  x3 = ((r3 - r1) p1^-1 - x2) p2^-1 mod p3,
//        X  = r1 + x2 p1 + x3 p1 p2  < p1 p2 p3 < 2^93,
//      and put the three words of every X into shared memory: 64 rows of 32
//      coefficients per word, 36 words apart (16-byte accesses without bank
//      conflicts).
//   2. Each of 64 threads adds the 32 values of a row, each at its shift (a
//      compile-time constant: the pattern repeats every 32 coefficients), into a
//      running 128-bit sum that gives off one 32-bit word a coefficient
//      (crt_pack64, src/crt.c:70-87, one run per thread).  What is left over
//      (below 2^64) is the next super-limb's carry-in.
//   3. With it added, a super-limb generates or propagates single carry bits:
//      ballots over the warp, maps over the warps (ffg_ripple.cuh), and the
//      CTA that finishes last settles the bits between CTAs (settle_cta).  A
//      CTA computes the carry-in at its own lower end from the 4 coefficients
//      below it: their parts above the boundary and the column sum of the 64
//      bits below it, which the true carry exceeds by at most one bit.
// Long products are bound by issue and memory together (at 2^24 coefficients
// 80 us, 268 MB: 51 % of the copy bandwidth), short ones by latency.  The form
// this replaces summed, for every limb, the shifted 128-bit slices of the 4 to 5
// coefficients over it: about 195 instructions a coefficient against 75 here,
// 147 us at 2^24 coefficients and 13.5 against 10.6 us for one of a few CTAs.
// k_crt_narrow (the split's widths 8..31): one CTA per 2048 coefficients.
//   1. Garner per coefficient for the block plus a halo below it.
//   2. Every limb j sums the slices of the coefficients X_i 2^(i b) that
//      overlap it: the column sum lo_j + 2^64 hi_j.
//   3. cta_resolve (ffg_ripple.cuh) settles the one-bit ripples; settle_cta the
//      carries between CTAs.
// A small signed constant is added to the product on the way (the final
// +-2 of fast doubling, src/fib.c:249) in two's complement over the output.
//
// k_lin: out = alpha s1 + beta s2 + gamma over len limbs, two outputs per
// launch (the reference's step_proc / last_proc, src/fib.c:37-62, 123-143);
// negative terms in two's complement (-s = ~s + 1 mod 2^(64 len)), so every
// column sum is non-negative and the same ripple settle applies.
#include <cstdlib>

#include "ffg_internal.h"
#include "ffg_ripple.cuh"

namespace ffg {

typedef unsigned __int128 u128;

constexpr uint32_t CRT_COEF = 2048;     // coefficients per CTA
constexpr uint32_t CRT_THREADS = 256;
constexpr uint32_t CRT_HALO_MAX = 24;   // ceil(156 / b) + 1 for b >= 8, rounded up to 4
constexpr uint32_t CRT_NL_MAX = 32 * 35;
constexpr uint32_t CRT_NL_PER_W = 32;   // limbs per CTA = 32 * width

FFG_DEV_INLINE int32_t floor_div32(int32_t a, int32_t b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

FFG_DEV_INLINE uint32_t crt_ctas_dev(uint64_t nlimbs, uint32_t width) {
    const uint64_t NL = (uint64_t)CRT_NL_PER_W * width;
    return (uint32_t)((nlimbs + NL - 1) / NL);
}

// Garner's recombination of one coefficient's residues: X < p1 p2 p3 < 2^93.
FFG_DEV_INLINE u128 garner(const GarnerConst &K, uint32_t r1, uint32_t r2, uint32_t r3) {
    const uint32_t p1 = K.p[0], p2 = K.p[1], p3 = K.p[2];
    const uint32_t x1m2 = min(r1, r1 - p2);
    const uint32_t x2 = shoup(r2 - x1m2 + p2, K.i12, K.i12s, p2);
    const uint32_t x1m3 = min(r1, r1 - p3);
    const uint32_t t3 = shoup(r3 - x1m3 + p3, K.i13, K.i13s, p3);
    const uint32_t x2m3 = min(x2, x2 - p3);
    const uint32_t x3 = shoup(t3 - x2m3 + p3, K.i23, K.i23s, p3);
    return (u128)((uint64_t)x2 * p1 + r1) + (u128)x3 * K.p12;
}

// Column sum lo + 2^64 hi of limb j (relative to the CTA's first limb) over
// the values X_i 2^(i b) (i relative to the CTA's first coefficient, stored
// from -halo), every X_i below 2^93.
FFG_DEV_INLINE void column_sum(const uint64_t *Xlo, const uint32_t *Xhi, int32_t j, int32_t b, int32_t halo,
                               uint64_t &s_lo, uint32_t &s_hi) {
    const int32_t ilo = floor_div32(64 * j - 92 + b - 1, b), ihi = floor_div32(64 * j + 63, b);
    s_lo = 0;
    s_hi = 0;
    for (int32_t i = ilo < -halo ? -halo : ilo; i <= ihi; i++) {
        const u128 X = ((u128)Xhi[i + halo] << 64) | Xlo[i + halo];
        const int32_t sft = i * b - 64 * j;
        const uint64_t part = sft >= 0 ? (uint64_t)(X << sft) : (uint64_t)(X >> (-sft));
        s_lo += part;
        s_hi += s_lo < part;
    }
}

__global__ void __launch_bounds__(CRT_THREADS) k_crt_narrow(GarnerConst K, CrtJob J) {
    after_previous();
    const uint32_t cta = blockIdx.x;
    extern __shared__ __align__(16) unsigned char sm[];
    uint64_t *Xlo = (uint64_t *)sm;                              // CRT_COEF + halo
    uint64_t *lo = Xlo + CRT_COEF + CRT_HALO_MAX;                // NL limbs
    uint32_t *Xhi = (uint32_t *)(lo + CRT_NL_MAX);               // CRT_COEF + halo
    uint32_t *hi = Xhi + CRT_COEF + CRT_HALO_MAX;                // NL
    uint32_t *gG = hi + CRT_NL_MAX, *gP = gG + CRT_NL_MAX / 32, *gin = gP + CRT_NL_MAX / 32;
    __shared__ uint32_t hiprev_s;

    const uint32_t b = J.width, NL = CRT_NL_PER_W * b;
    const int32_t halo = (int32_t)(((156 + b - 1) / b + 1 + 3) & ~3u);
    const int64_t ibase = (int64_t)cta * CRT_COEF;

    // residues in 16-byte vectors of 4 coefficients, every load of the thread
    // issued before any arithmetic (ibase - halo and the strides are multiples
    // of 4, and every residue array is a multiple of 16 words long)
    constexpr int VPT = (CRT_COEF + CRT_HALO_MAX) / 4 / CRT_THREADS + 1; // vectors per thread
    const int32_t nvec = ((int32_t)CRT_COEF + halo) / 4;
    uint4 rv[VPT][3];
#pragma unroll
    for (int v = 0; v < VPT; v++) {
        const int32_t t4 = (int32_t)threadIdx.x + v * (int32_t)blockDim.x;
        const int64_t gi = ibase - halo + 4 * (int64_t)t4;
        const bool in = t4 < nvec && gi >= 0 && (uint64_t)gi < J.conv;
#pragma unroll
        for (int k = 0; k < 3; k++)
            rv[v][k] = in ? *(const uint4 *)(J.y + k * J.y_stride + gi) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int v = 0; v < VPT; v++) {
        const int32_t t4 = (int32_t)threadIdx.x + v * (int32_t)blockDim.x;
        if (t4 >= nvec) break;
        const int64_t gi0 = ibase - halo + 4 * (int64_t)t4;
        const uint32_t r1s[4] = {rv[v][0].x, rv[v][0].y, rv[v][0].z, rv[v][0].w};
        const uint32_t r2s[4] = {rv[v][1].x, rv[v][1].y, rv[v][1].z, rv[v][1].w};
        const uint32_t r3s[4] = {rv[v][2].x, rv[v][2].y, rv[v][2].z, rv[v][2].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int64_t gi = gi0 + e;
            const u128 X = gi >= 0 && (uint64_t)gi < J.conv ? garner(K, r1s[e], r2s[e], r3s[e]) : (u128)0;
            Xlo[4 * t4 + e] = (uint64_t)X;
            Xhi[4 * t4 + e] = (uint32_t)(X >> 64);
        }
    }
    __syncthreads();

    // column sums; j = -1 (the limb below the CTA) only for its high part
    const uint64_t j0 = (uint64_t)cta * NL;
    const bool neg_add = J.add < 0;
    for (int32_t j = (int32_t)threadIdx.x - 1; j < (int32_t)NL; j += blockDim.x) {
        uint64_t s_lo;
        uint32_t s_hi;
        column_sum(Xlo, Xhi, j, (int32_t)b, halo, s_lo, s_hi);
        // the constant: +add at limb 0, or 2^(64 nlimbs) + add when negative
        const int64_t jabs = (int64_t)j0 + j;
        if (J.add != 0 && jabs >= 0 && (uint64_t)jabs < J.nlimbs) {
            const uint64_t c = jabs == 0 ? (uint64_t)J.add : (neg_add ? ~0ull : 0ull);
            s_lo += c;
            s_hi += s_lo < c;
        }
        if (j < 0) hiprev_s = s_hi;
        else {
            lo[j] = s_lo;
            hi[j] = s_hi;
        }
    }
    __syncthreads();
    const uint32_t map = cta_resolve(lo, hi, cta ? hiprev_s : 0, NL, gG, gP, gin);
    for (uint32_t j = threadIdx.x; j < NL && j0 + j < J.nlimbs; j += blockDim.x) J.out[j0 + j] = lo[j];
    if (threadIdx.x == 0) J.maps[cta] = map;
    const uint32_t ncta = crt_ctas_dev(J.nlimbs, b);
    if (ncta > 1 && last_cta(J.ticket, ncta)) {
        settle_cta(J.out, J.nlimbs, NL, J.maps, ncta);
        if (threadIdx.x == 0) *J.ticket = 0;
    }
}

uint32_t crt_ctas(uint64_t nlimbs, uint32_t width) {
    const uint64_t NL = (uint64_t)CRT_NL_PER_W * width;
    return (uint32_t)((nlimbs + NL - 1) / NL);
}

// ---------------------------------------------------- widths 32..35

constexpr int CS_T = CRT_COEF / 32;  // super-limbs of a CTA (64), the unit of crt_ctas()
constexpr int CS_BIG = 256;          // super-limbs of a CTA of a long product
// T super-limbs of SL coefficients of width B: W words of output each; shared
// words of a row (SL coefficients' words, later the W words of output; rows 4
// words apart from a power of two keep 16-byte accesses off each other's banks)
// and of a plane (one word of every value).
template <int T, int SL, int B> struct CrtGeo {
    static constexpr int W = SL * B / 32;
    static constexpr uint32_t ROW = SL + 4, PLANE = T * ROW;
    static_assert(SL * B % 32 == 0 && W <= (int)ROW && W >= 8 && SL >= 8 && T % 32 == 0, "whole words");
};
// The shortest super-limbs of a width (the sums' serial chain).  The doubling step's
// fused CRT gains by them (chain of F(10^8) 633 us, with super-limbs of 32 644); a plain
// short product does not (300, 1000 and 65536 limbs equal within noise) and shares them.
template <int B> struct CrtShort {
    static constexpr int SL = B == 32 ? 8 : (B == 34 ? 16 : 32);
};

// Garner's X as words x[0] + 2^32 x[1] + 2^64 x[2].
FFG_DEV_INLINE u128 garner_lean(const GarnerConst &K, uint32_t r1, uint32_t r2, uint32_t r3) {
    const uint32_t p1 = K.p[0], p2 = K.p[1], p3 = K.p[2];
    const uint32_t x2 = shoup(r2 - min(r1, r1 - p2) + p2, K.i12, K.i12s, p2);
    const uint32_t t3 = shoup(r3 - min(r1, r1 - p3) + p3, K.i13, K.i13s, p3);
    const uint32_t x3 = shoup(t3 - min(x2, x2 - p3) + p3, K.i23, K.i23s, p3);
    // below 2^62, then below 2^64: no carries between the three products
    const uint64_t lo = (uint64_t)x2 * p1 + r1;
    const uint64_t t0 = (uint64_t)x3 * (uint32_t)K.p12 + lo;
    const uint64_t t1 = (uint64_t)x3 * (uint32_t)(K.p12 >> 32) + (t0 >> 32);
    return ((u128)t1 << 32) | (uint32_t)t0;
}

FFG_DEV_INLINE uint32_t quad_word(const uint4 &v, int e) { return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w)); }

// The carry into the boundary above coefficients x[0..3] (x[3] next below it),
// short of the single bit that may ripple through the 64 bits below it: the
// parts of x[3], x[2] above the boundary plus the carries of those 64 bits'
// column sum (all: a constant limb 2^64 - 1 is part of it).
template <int B> FFG_DEV_INLINE uint64_t boundary_carry(const u128 (&x)[4], bool all) {
    u128 s = (u128)(uint64_t)(x[3] << (64 - B)) + (uint64_t)(x[2] >> (2 * B - 64)) + (uint64_t)(x[1] >> (3 * B - 64)) +
             (uint64_t)(x[0] >> (4 * B - 64));
    if (all) s += ~0ull;
    return (uint64_t)(x[3] >> B) + (uint64_t)(x[2] >> (2 * B)) + (uint64_t)(s >> 64);
}

// A thread's super-limb: words 0..3 in registers, words 4 .. b - 1 in its row.
struct Super {
    uint64_t w01, w23;
    uint32_t ones;  // the and of words 4 .. b - 1
    uint64_t left;  // carried on into the next super-limb
    uint64_t bound; // boundary_carry of its last four coefficients
};

// Sums the 32 values of a row (its three planes).  The words are stored over the
// values' own low words, always behind the chunk read ahead (chunk c + 1 is
// loaded before chunk c's words are stored; b words for 32 never overtake it).
// eval(a, b, c): the value of a coefficient from its words in the three planes
// (a value's own words, or residues not yet recombined).
template <class Q, int SL, int B, class Eval>
FFG_DEV_INLINE void super_sum(Super &S, uint32_t *row, bool all, Eval value) {
    u128 acc = 0, last[4];
    uint32_t w[4], buf[4];
    S.ones = ~0u;
    struct Raw {
        uint4 r[3];
    } cur, nxt;
    auto load = [&](int c, Raw &q) {
#pragma unroll
        for (int k = 0; k < 3; k++) q.r[k] = *(const uint4 *)(row + k * Q::PLANE + 4 * c);
    };
    auto eval = [&](const Raw &q, int e) { return value(quad_word(q.r[0], e), quad_word(q.r[1], e), quad_word(q.r[2], e)); };
    load(0, cur);
    // a chunk at compile-time position c (only width 32 shifts all chunks alike)
    auto chunk = [&](int c, const Raw &raw) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int i = 4 * c + e, wi = i * B / 32, n = (i + 1) * B / 32 - wi;
            last[e] = eval(raw, e);
            acc += last[e] << (i * B % 32);
#pragma unroll
            for (int m = 0; m < 2; m++) {
                if (m >= n) continue;
                const uint32_t word = (uint32_t)acc;
                acc >>= 32;
                const int at = wi + m;
                if (at < 4) w[at & 3] = word;
                else {
                    S.ones &= word;
                    buf[at & 3] = word;
                    if ((at & 3) == 3) *(uint4 *)(row + at - 3) = make_uint4(buf[0], buf[1], buf[2], buf[3]);
                }
            }
        }
    };
    load(1, nxt);
    chunk(0, cur);
    if (B == 32) {
#pragma unroll 1
        for (int c = 1; c < SL / 4; c++) {
            cur = nxt;
            if (c + 1 < SL / 4) load(c + 1, nxt);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                last[e] = eval(cur, e);
                acc += last[e];
                buf[e] = (uint32_t)acc;
                acc >>= 32;
                S.ones &= buf[e];
            }
            *(uint4 *)(row + 4 * c) = make_uint4(buf[0], buf[1], buf[2], buf[3]);
        }
    } else {
#pragma unroll
        for (int c = 1; c < SL / 4; c++) {
            cur = nxt;
            if (c + 1 < SL / 4) load(c + 1, nxt);
            chunk(c, cur);
        }
#pragma unroll
        for (int m = 0; m < Q::W % 4; m++) row[(Q::W & ~3) + m] = buf[m];
    }
    S.w01 = (uint64_t)w[1] << 32 | w[0];
    S.w23 = (uint64_t)w[3] << 32 | w[2];
    S.left = (uint64_t)acc;
    S.bound = boundary_carry<B>(last, all);
}

FFG_DEV_INLINE u128 words_value(uint32_t a, uint32_t b, uint32_t c) { return (u128)c << 64 | (uint64_t)b << 32 | a; }

// Adds v to words 4 .. W - 1 (v = 1 or -1, a carry or a borrow out of the words
// below): rare.  Returns the carry or borrow out of the super-limb.
template <int W> FFG_DEV_INLINE bool super_ripple(Super &S, uint32_t *row, uint32_t v) {
    bool on = true;
    uint32_t ones = ~0u;
    for (int k = 4; k < W; k++) {
        uint32_t x = row[k];
        if (on) {
            on = v == 1 ? x == ~0u : x == 0;
            x += v;
            row[k] = x;
        }
        ones &= x;
    }
    S.ones = ones;
    return on;
}

// What the threads of a CTA share while carries are resolved.
struct SuperShared {
    uint64_t left[CS_BIG];
    uint32_t gG[CS_BIG / 32], gP[CS_BIG / 32];
    uint64_t bound;
};

// Resolves the CTA's super-limbs (thread t < T its t-th) assuming no carry
// bit comes into the CTA, and stores words 0..3 to the rows; thread 0 gets the
// CTA's carry map.  All threads call it.  cin: the first super-limb's carry-in
// (the others' is their neighbour's left).  sub > 0: the constant is -sub in the
// first limb's super-limb (1 in the others), in two's complement over the whole
// number.
template <int T, int W>
FFG_DEV_INLINE uint32_t super_resolve(Super &S, uint32_t *row, SuperShared &sh, uint64_t cin, uint64_t sub) {
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr uint32_t NW = T / 32;
    const bool mine = t < T;
    if (mine) {
        if (sub) { // plus 2^(32 b) - sub
            bool br = S.w01 < sub;
            S.w01 -= sub;
            if (br) {
                br = S.w23 == 0;
                S.w23 -= 1;
                if (br) br = super_ripple<W>(S, row, ~0u);
            }
            S.left += !br;
        }
        sh.left[t] = S.left;
        if (t == T - 1) sh.bound = S.bound;
    }
    __syncthreads();
    uint32_t Gm = 0, Pm = 0;
    if (mine) {
        const uint64_t h = t ? sh.left[t - 1] : cin;
        bool G = false;
        S.w01 += h;
        if (S.w01 < h) {
            S.w23 += 1;
            if (S.w23 == 0) G = super_ripple<W>(S, row, 1);
        }
        const bool P = !G && (S.w01 & S.w23) == ~0ull && S.ones == ~0u;
        Gm = __ballot_sync(0xffffffffu, G), Pm = __ballot_sync(0xffffffffu, P);
        if (lane == 0) {
            sh.gG[warp] = Gm;
            sh.gP[warp] = Pm;
        }
    }
    __syncthreads();
    uint32_t c0 = 0, c1 = 1, cw = 0; // carries out of the warps so far, for carry-in 0 and 1
    if (mine) {
#pragma unroll
        for (uint32_t k = 0; k < NW; k++) {
            if (k == warp) cw = c0;
            const uint32_t m = map_of_group(sh.gG[k], sh.gP[k]);
            c0 = map_apply(m, c0);
            c1 = map_apply(m, c1);
        }
        const uint64_t A = Gm | Pm, Bm = Gm;
        if ((((uint32_t)((A + Bm + cw) ^ A ^ Bm)) >> lane) & 1u) {
            if (++S.w01 == 0 && ++S.w23 == 0) super_ripple<W>(S, row, 1);
        }
        *(uint4 *)row = make_uint4((uint32_t)S.w01, (uint32_t)(S.w01 >> 32), (uint32_t)S.w23, (uint32_t)(S.w23 >> 32));
    }
    // the carry out of the CTA, less what the next CTA finds by itself: 0 or 1
    const uint32_t d = (uint32_t)(sh.left[T - 1] - sh.bound);
    __syncthreads();
    return (d + c0) | ((d + c1) << 1);
}

// The CTA's words (rows of W) to its T W / 2 limbs from j0 of out, below nlimbs.
template <int T, int W, uint32_t ROW>
FFG_DEV_INLINE void super_store(const uint32_t *rows, uint64_t *out, uint64_t j0, uint64_t nlimbs) {
    const uint32_t nl = T * W / 2;
    const uint32_t lim = nlimbs > j0 ? (nlimbs - j0 < nl ? (uint32_t)(nlimbs - j0) : nl) : 0;
    for (uint32_t l = threadIdx.x; l < lim; l += blockDim.x) {
        const uint32_t k = 2 * l, r = k / W, c = k - r * W;
        uint64_t v;
        if (W % 2 == 0) {
            v = *(const uint64_t *)(rows + r * ROW + c);
        } else {
            const uint32_t lo = rows[r * ROW + c];
            const uint32_t hi = c + 1 < W ? rows[r * ROW + c + 1] : rows[(r + 1) * ROW];
            v = (uint64_t)hi << 32 | lo;
        }
        out[j0 + l] = v;
    }
}

// What a CTA shares besides its planes: the values of the 4 coefficients below it.
struct CrtShared {
    alignas(16) uint32_t halo[2][3][4];
    SuperShared sup;
};
FFG_DEV_INLINE void halo_value(const uint32_t (&h)[3][4], u128 (&x)[4]) {
#pragma unroll
    for (int e = 0; e < 4; e++) x[e] = (u128)h[2][e] << 64 | (uint64_t)h[1][e] << 32 | h[0][e];
}

// Residues of the CTA's coefficients (and of the 4 below it) into three planes,
// zero at or past conv (Garner of zeros is zero): cp.async, so that a CTA's loads
// are all in flight at once without a register each.
template <int NT, class Q, int T, int SL>
FFG_DEV_INLINE void super_stage(uint32_t *planes, uint32_t (&halo)[3][4], const uint32_t *y, uint64_t stride,
                                int64_t ibase, uint64_t conv) {
    auto copy = [&](uint32_t *dst, const uint32_t *src, int64_t gi) {
        const uint32_t n = gi >= 0 && (uint64_t)gi < conv ? (conv - gi < 4 ? (uint32_t)(conv - gi) * 4 : 16u) : 0u;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src + (n ? gi : 0)), "r"(n)
                     : "memory");
    };
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (uint32_t v = 0; v < T * SL / 4 / NT; v++) {
            const uint32_t q = threadIdx.x + v * NT;
            copy(planes + k * Q::PLANE + q / (SL / 4) * Q::ROW + q % (SL / 4) * 4, y + k * stride, ibase + 4 * (int64_t)q);
        }
        if (threadIdx.x == NT - 1) copy(halo[k], y + k * stride, ibase - 4);
    }
}
FFG_DEV_INLINE void super_staged() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// Values of the CTA's coefficients into the planes: ld(gi) loads the residues
// of coefficients gi .. gi + 3, eval(raw, e, z) gives the values of the e-th.
// A thread's loads are issued before any arithmetic; lanes 0..3 of the last
// warp also do one coefficient each of the 4 below the CTA.
template <int NT, class Q, int SL, int NO, class Raw, class Ld, class Eval>
FFG_DEV_INLINE void super_fill(uint32_t *planes, CrtShared &sh, int64_t ibase, Ld ld, Eval eval) {
    constexpr uint32_t PER = CRT_COEF / 4 / NT, AHEAD = NO == 1 ? 2 : 1; // quads a thread, AHEAD loaded at a time
    const uint32_t t = threadIdx.x, low = t - (NT - 32); // 0..3: a coefficient below the CTA
    Raw raw[AHEAD], hr;
    if (low < 4) ld(ibase - 4, hr);
    auto put = [&](const Raw &r, uint32_t q) {
        uint32_t x[NO][3][4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            u128 z[NO];
            eval(r, e, z);
#pragma unroll
            for (int k = 0; k < NO; k++)
#pragma unroll
                for (int m = 0; m < 3; m++) x[k][m][e] = (uint32_t)(z[k] >> (32 * m));
        }
        uint32_t *d = planes + q / (SL / 4) * Q::ROW + q % (SL / 4) * 4;
#pragma unroll
        for (int k = 0; k < NO; k++)
#pragma unroll
            for (int m = 0; m < 3; m++)
                *(uint4 *)(d + (3 * k + m) * Q::PLANE) =
                    make_uint4(x[k][m][0], x[k][m][1], x[k][m][2], x[k][m][3]);
    };
#pragma unroll 1
    for (uint32_t v0 = 0; v0 < PER; v0 += AHEAD) {
#pragma unroll
        for (uint32_t v = 0; v < AHEAD; v++) ld(ibase + 4 * (int64_t)(t + (v0 + v) * NT), raw[v]);
#pragma unroll
        for (uint32_t v = 0; v < AHEAD; v++) put(raw[v], t + (v0 + v) * NT);
    }
    if (low < 4) {
        u128 z[NO];
        eval(hr, (int)low, z);
#pragma unroll
        for (int k = 0; k < NO; k++)
#pragma unroll
            for (int m = 0; m < 3; m++) sh.halo[k][m][low] = (uint32_t)(z[k] >> (32 * m));
    }
    __syncthreads();
}

struct Raw3 {
    uint4 r[3];
};
// Residues of coefficients gi .. gi + 3 (gi a multiple of 4; the arrays are a
// multiple of 16 words long), zero at or past conv: Garner of zeros is zero.
FFG_DEV_INLINE void ld_residues(uint4 *r, const uint32_t *y, uint64_t stride, int64_t gi, uint64_t conv) {
    const bool in = gi >= 0 && (uint64_t)gi < conv;
#pragma unroll
    for (int k = 0; k < 3; k++) r[k] = in ? *(const uint4 *)(y + k * stride + gi) : make_uint4(0, 0, 0, 0);
    if (in && (uint64_t)gi + 4 > conv) {
        const uint32_t n = (uint32_t)(conv - (uint64_t)gi); // 1 .. 3 words
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (n < 2) r[k].y = 0;
            if (n < 3) r[k].z = 0;
            r[k].w = 0;
        }
    }
}

// How a CTA runs a CRT.
enum CrtForm {
    // short products: 256 threads recombine two quads each from registers, the
    // sums run over short super-limbs (the time is one thread's chain)
    CF_SHORT,
    // batches of products of any size: the same with 128 threads and super-limbs
    // of 32
    CF_BATCH,
    // CTAs of 256 super-limbs: every thread recombines and adds its own 32
    // coefficients in one pass with no barrier in between, and there are a quarter
    // of the carry maps; for launches that fill the GPU twice over
    CF_LONG
};
template <CrtForm F> __host__ __device__ constexpr int crt_threads() { return F == CF_BATCH ? 128 : 256; }

template <CrtForm F, int B>
FFG_DEV_INLINE void crt_super(const GarnerConst &K, const CrtJob &J, uint32_t cta, uint32_t *planes, CrtShared &sh) {
    constexpr int NT = crt_threads<F>(), SL = F == CF_SHORT ? CrtShort<B>::SL : 32;
    constexpr int T = F == CF_LONG ? CS_BIG : CRT_COEF / SL;
    using Q = CrtGeo<T, SL, B>;
    constexpr uint32_t NL = T * Q::W / 2; // limbs
    const uint32_t t = threadIdx.x;
    const int64_t ibase = (int64_t)cta * (SL * T);
    uint32_t *const row = planes + t * Q::ROW;
    const bool neg = J.add < 0;
    Super S;
    uint64_t cin = 0;
    u128 below[4];
    auto garner = [&](uint32_t a, uint32_t b, uint32_t c) { return garner_lean(K, a, b, c); };
    if (F != CF_LONG) {
        super_fill<NT, Q, SL, 1, Raw3>(
            planes, sh, ibase, [&](int64_t gi, Raw3 &q) { ld_residues(q.r, J.y, J.y_stride, gi, J.conv); },
            [&](const Raw3 &q, int e, u128(&x)[1]) {
                x[0] = garner(quad_word(q.r[0], e), quad_word(q.r[1], e), quad_word(q.r[2], e));
            });
    } else {
        super_stage<NT, Q, T, SL>(planes, sh.halo[0], J.y, J.y_stride, ibase, J.conv);
        super_staged();
    }
    if (F == CF_LONG) {
        super_sum<Q, SL, B>(S, row, neg, garner);
        if (t == 0) {
#pragma unroll
            for (int e = 0; e < 4; e++) below[e] = garner(sh.halo[0][0][e], sh.halo[0][1][e], sh.halo[0][2][e]);
        }
    } else {
        if (t < T) super_sum<Q, SL, B>(S, row, neg, words_value);
        if (t == 0) halo_value(sh.halo[0], below);
    }
    if (t == 0) cin = cta ? boundary_carry<B>(below, neg) : (neg ? 0 : (uint64_t)J.add);
    const uint64_t sub = neg ? (t == 0 && cta == 0 ? (uint64_t)-J.add : 1) : 0;
    const uint32_t map = super_resolve<T, Q::W>(S, row, sh.sup, cin, sub);
    super_store<T, Q::W, Q::ROW>(planes, J.out, (uint64_t)cta * NL, J.nlimbs);
    const uint32_t ncta = (uint32_t)((J.nlimbs + NL - 1) / NL);
    if (ncta > 1) {
        if (t == 0) J.maps[cta] = map;
        if (last_cta(J.ticket, ncta)) {
            settle_cta(J.out, J.nlimbs, NL, J.maps, ncta);
            if (t == 0) *J.ticket = 0;
        }
    }
}

template <CrtForm F> FFG_DEV_INLINE void crt_any(const GarnerConst &K, const CrtJob &J, uint32_t cta) {
    extern __shared__ __align__(16) uint32_t cs_rows[];
    __shared__ CrtShared sh;
    switch (J.width) {
    case 32: crt_super<F, 32>(K, J, cta, cs_rows, sh); return;
    case 33: crt_super<F, 33>(K, J, cta, cs_rows, sh); return;
    case 34: crt_super<F, 34>(K, J, cta, cs_rows, sh); return;
    default: crt_super<F, 35>(K, J, cta, cs_rows, sh); return;
    }
}

template <CrtForm F>
__global__ void __launch_bounds__(crt_threads<F>(), F == CF_BATCH ? 6 : (F == CF_SHORT ? 3 : 2)) k_crt(GarnerConst K, CrtJob J) {
    after_previous();
    crt_any<F>(K, J, blockIdx.x);
}

// Two CRTs by value, product blockIdx.y, its CTA blockIdx.x: the doubling step's two
// squarings when its linear pass is a launch of its own (FFG_NO_CRT_LIN=1, the
// comparison with k_crt_lin).
struct CrtPair {
    CrtJob j[2];
};
__global__ void __launch_bounds__(256, 3) k_crt_pair(GarnerConst K, CrtPair P) {
    after_previous();
    const CrtJob J = blockIdx.y ? P.j[1] : P.j[0];
    if (blockIdx.x >= crt_ctas_dev(J.nlimbs, J.width)) return;
    crt_any<CF_SHORT>(K, J, blockIdx.x);
}

// CRTs of any sizes in one launch: CTA b runs CTA b - first[j] of job j,
// first[j] <= b < first[j + 1] (first: count + 1 prefix sums of the jobs'
// CTA counts), found by binary search.
__global__ void __launch_bounds__(128, 6) k_crt_flat(GarnerConst K, const CrtJob *__restrict__ jobs,
                                                            const uint32_t *__restrict__ first, uint32_t count) {
    after_previous();
    const uint32_t b = blockIdx.x;
    uint32_t lo = 0, hi = count; // invariant: first[lo] <= b < first[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (__ldg(&first[mid]) <= b) lo = mid;
        else hi = mid;
    }
    const CrtJob J = jobs[lo];
    crt_any<CF_BATCH>(K, J, b - __ldg(&first[lo]));
}

// Shared bytes of T super-limbs' planes (the widest rows: SL + 4 words for 8
// coefficients and more) of n values.
template <int T, int SL> constexpr size_t super_smem(uint32_t n) {
    return (size_t)3 * n * T * (SL + 4) * sizeof(uint32_t);
}
constexpr size_t kShortSmem = super_smem<CRT_COEF / 8, 8>(1), kBatchSmem = super_smem<CS_T, 32>(1),
                 kLongSmem = super_smem<CS_BIG, 32>(1);

static size_t crt_smem() {
    return (CRT_COEF + CRT_HALO_MAX) * (8 + 4) + CRT_NL_MAX * (8 + 4) + 3 * (CRT_NL_MAX / 32) * 4;
}

static bool g_crt_configured = false;

cudaError_t crt_kernel_load() {
    if (g_crt_configured) return cudaSuccess;
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k_crt<CF_SHORT>);
    if (!e) e = cudaFuncGetAttributes(&fa, k_crt<CF_LONG>);
    if (!e) e = cudaFuncSetAttribute(k_crt<CF_SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShortSmem);
    if (!e) e = cudaFuncSetAttribute(k_crt<CF_LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLongSmem);
    if (!e) e = cudaFuncSetAttribute(k_crt_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShortSmem);
    if (!e) e = cudaFuncSetAttribute(k_crt_narrow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)crt_smem());
    if (e) return e;
    g_crt_configured = true;
    return cudaSuccess;
}

// From this many CTAs of 64 super-limbs a product takes CTAs of 256 instead
// (at 2^22 coefficients, 2049 against 513 CTAs, 32.0 against 25.1 us; below,
// CTAs of 256 leave SMs idle).
constexpr uint32_t kCrtBigCtas = 1024;
// Up to this many CTAs (two an SM) a product runs the short form.
constexpr uint32_t kCrtShortCtas = 296;

cudaError_t launch_crt(const Primes3 &P3, const CrtJob &J, cudaStream_t st) {
    (void)P3;
    cudaError_t e0 = crt_kernel_load();
    if (e0) return e0;
    const uint32_t ncta = crt_ctas(J.nlimbs, J.width);
    prof_begin(PK_CRT, st);
    if (J.width < 32) launch_after(k_crt_narrow, ncta, CRT_THREADS, crt_smem(), st, garner_const(), J);
    else if (ncta <= kCrtShortCtas) launch_after(k_crt<CF_SHORT>, ncta, 256, kShortSmem, st, garner_const(), J);
    else if (ncta <= kCrtBigCtas) launch_after(k_crt<CF_BATCH>, ncta, 128, kBatchSmem, st, garner_const(), J);
    else launch_after(k_crt<CF_LONG>, (ncta + 3) / 4, 256, kLongSmem, st, garner_const(), J);
    prof_end(PK_CRT, st, 12.0 * (double)J.conv + 8.0 * (double)J.nlimbs);
    return cudaGetLastError();
}

cudaError_t launch_crt_pair(const CrtJob *jobs, uint32_t count, cudaStream_t st) {
    if (count == 1 || jobs[0].width < 32 || jobs[1].width < 32) {
        cudaError_t e = cudaSuccess;
        for (uint32_t i = 0; i < count && !e; i++) e = launch_crt(Primes3{}, jobs[i], st);
        return e;
    }
    cudaError_t e0 = crt_kernel_load();
    if (e0) return e0;
    CrtPair P;
    P.j[0] = jobs[0];
    P.j[1] = jobs[1];
    const uint32_t n0 = crt_ctas(jobs[0].nlimbs, jobs[0].width), n1 = crt_ctas(jobs[1].nlimbs, jobs[1].width);
    double bytes = 0;
    for (int i = 0; i < 2; i++) bytes += 12.0 * (double)jobs[i].conv + 8.0 * (double)jobs[i].nlimbs;
    prof_begin(PK_CRT, st);
    launch_after(k_crt_pair, dim3(n0 > n1 ? n0 : n1, 2), 256, kShortSmem, st, garner_const(), P);
    prof_end(PK_CRT, st, bytes);
    return cudaGetLastError();
}

cudaError_t launch_crt_flat(const CrtJob *d_jobs, const uint32_t *d_first, uint32_t count, uint32_t total_ctas,
                            cudaStream_t st, double bytes) {
    if (!count || !total_ctas) return cudaSuccess;
    prof_begin(PK_CRT, st);
    launch_after(k_crt_flat, total_ctas, 128, kBatchSmem, st, garner_const(), d_jobs, d_first, count);
    prof_end(PK_CRT, st, bytes);
    return cudaGetLastError();
}

// ------------------------------------------------------ CRT + linear pass
//
// k_crt_lin: the CRT of a doubling step's two squarings and the step's
// linear pass in one launch.  With X1_i, X2_i the coefficients of s1 and s2,
// output k is sum_i (alpha_k X1_i + beta_k X2_i) 2^(i b) + gamma_k.  beta_k
// may be negative; every coefficient gets the bias B = K (2^b - 1), K =
// 2^(94 - b), so that Z_i = alpha_k X1_i + beta_k X2_i + B >= 0 (|beta_k| X2_i
// <= 2 p1 p2 p3 < 2^94 - K) and Z_i < 4 2^93 + 2^94 < 2^96.  Over the N
// coefficients the CTAs cover, sum_i B 2^(i b) = K 2^(N b) - K: adding the
// constant gamma_k + K leaves the output plus K 2^(N b), a multiple of
// 2^(64 len) that falls off the top (N b >= 64 len).  The rest is crt_super
// with values of up to 96 bits.  kOuts 1: output blockIdx.y alone (short
// products, where twice the CTAs hide more than recombining twice costs); 2:
// both outputs from one recombination (as CF_BATCH).  kOuts 1: 512 threads stage the
// residues, recombine a coefficient at a time in a rolled loop (straight-line code
// for 16 of them would take longer to fetch than to run) and add short super-limbs:
// 12.5 -> 10.7 us a step of the F(10^8) chain against CF_SHORT's form.
struct Raw6 {
    uint4 r[6];
};

// Values in place of the staged residues, a coefficient at a time in a rolled loop:
// value(d, p, h, hp) from the words at d, d + p, d + 2 p and h, h + hp, h + 2 hp of
// its two squarings.
template <int NT, class Q, int SL, class Value>
FFG_DEV_INLINE void short_values(uint32_t *planes, uint32_t (*halo)[3][4], Value value) {
    auto put = [&](uint32_t *d, uint32_t pitch, uint32_t *h, uint32_t hp) {
        const u128 z = value(d, pitch, h, hp);
        d[0] = (uint32_t)z;
        d[pitch] = (uint32_t)(z >> 32);
        d[2 * pitch] = (uint32_t)(z >> 64);
    };
#pragma unroll 2
    for (uint32_t v = threadIdx.x; v < CRT_COEF; v += NT) {
        uint32_t *d = planes + v / SL * Q::ROW + v % SL;
        put(d, Q::PLANE, d + 3 * Q::PLANE, Q::PLANE);
    }
    const uint32_t low = threadIdx.x - (NT - 32); // 0..3: a coefficient below the CTA
    if (low < 4) put(&halo[0][0][low], 4, &halo[1][0][low], 4);
    __syncthreads();
}

template <int kOuts> __host__ __device__ constexpr int crt_lin_threads() { return kOuts == 1 ? 512 : 128; }

template <int B, int kOuts>
FFG_DEV_INLINE void crt_lin_super(const GarnerConst &K, const CrtLinJob &J, uint32_t *planes, CrtShared &sh) {
    constexpr int NT = crt_lin_threads<kOuts>(), SL = kOuts == 1 ? CrtShort<B>::SL : 32, T = CRT_COEF / SL;
    using Q = CrtGeo<T, SL, B>;
    const uint32_t t = threadIdx.x, cta = blockIdx.x, ncta = gridDim.x;
    const int64_t ibase = (int64_t)cta * CRT_COEF;
    const int k0 = kOuts == 1 ? (int)blockIdx.y : 0;
    const u128 bias = ((u128)1 << (94 - B)) * (((u128)1 << B) - 1);
    const uint64_t conv0 = J.conv[0], conv1 = J.conv[1];
    uint32_t al[kOuts];
    int32_t be[kOuts];
#pragma unroll
    for (int k = 0; k < kOuts; k++) {
        al[k] = (uint32_t)(k0 + k ? J.alpha[1] : J.alpha[0]);
        be[k] = k0 + k ? J.beta[1] : J.beta[0];
    }
    auto combine = [&](u128 x1, u128 x2, int k) { // exact mod 2^128, 0 <= z < 2^96
        const u128 v = x1 * al[k] + bias;
        return be[k] >= 0 ? v + x2 * (uint32_t)be[k] : v - x2 * (uint32_t)(-be[k]);
    };
    if (kOuts == 1) {
        super_stage<NT, Q, T, SL>(planes, sh.halo[0], J.y[0], J.y_stride, ibase, conv0);
        super_stage<NT, Q, T, SL>(planes + 3 * Q::PLANE, sh.halo[1], J.y[1], J.y_stride, ibase, conv1);
        super_staged();
        short_values<NT, Q, SL>(planes, sh.halo,
                                [&](const uint32_t *d, uint32_t p, const uint32_t *h, uint32_t hp) {
                                    return combine(garner_lean(K, d[0], d[p], d[2 * p]),
                                                   garner_lean(K, h[0], h[hp], h[2 * hp]), 0);
                                });
    } else {
        super_fill<NT, Q, SL, kOuts, Raw6>(
            planes, sh, ibase,
            [&](int64_t gi, Raw6 &q) {
                ld_residues(q.r, J.y[0], J.y_stride, gi, conv0);
                ld_residues(q.r + 3, J.y[1], J.y_stride, gi, conv1);
            },
            [&](const Raw6 &q, int e, u128(&z)[kOuts]) {
                const u128 x1 = garner_lean(K, quad_word(q.r[0], e), quad_word(q.r[1], e), quad_word(q.r[2], e));
                const u128 x2 = garner_lean(K, quad_word(q.r[3], e), quad_word(q.r[4], e), quad_word(q.r[5], e));
#pragma unroll
                for (int k = 0; k < kOuts; k++) z[k] = combine(x1, x2, k);
            });
    }
#pragma unroll
    for (int k = 0; k < kOuts; k++) {
        uint32_t *const row = planes + 3 * k * Q::PLANE + t * Q::ROW;
        Super S;
        uint64_t cin = 0;
        if (t < T) super_sum<Q, SL, B>(S, row, false, words_value);
        if (t == 0) {
            if (cta) {
                u128 x[4];
                halo_value(sh.halo[k], x);
                cin = boundary_carry<B>(x, false);
            } else {
                cin = (uint64_t)(k0 + k ? J.gamma[1] : J.gamma[0]) + ((uint64_t)1 << (94 - B)); // gamma + K > 0
            }
        }
        const uint32_t map = super_resolve<T, Q::W>(S, row, sh.sup, cin, 0);
        super_store<T, Q::W, Q::ROW>(planes + 3 * k * Q::PLANE, k0 + k ? J.out[1] : J.out[0],
                                     (uint64_t)cta * CRT_NL_PER_W * B, J.len);
        if (t == 0) J.maps[(size_t)(k0 + k) * ncta + cta] = map;
    }
    if (ncta > 1 && last_cta(J.ticket, ncta * gridDim.y)) {
        for (int q = 0; q < 2; q++)
            settle_cta(q ? J.out[1] : J.out[0], J.len, CRT_NL_PER_W * B, J.maps + (size_t)q * ncta, ncta);
        if (t == 0) *J.ticket = 0;
    }
}

template <int kOuts>
__global__ void __launch_bounds__(crt_lin_threads<kOuts>(), kOuts == 1 ? 2 : 4) k_crt_lin(GarnerConst K, CrtLinJob J) {
    after_previous();
    extern __shared__ __align__(16) uint32_t cs_rows[];
    __shared__ CrtShared sh;
    switch (J.width) {
    case 32: crt_lin_super<32, kOuts>(K, J, cs_rows, sh); return;
    case 33: crt_lin_super<33, kOuts>(K, J, cs_rows, sh); return;
    case 34: crt_lin_super<34, kOuts>(K, J, cs_rows, sh); return;
    default: crt_lin_super<35, kOuts>(K, J, cs_rows, sh); return;
    }
}

// Up to this many CTAs an output, the two outputs go to CTAs of their own
// (F(10^8): 200 us of CRT in the chain; with every step so 222; F(10^9) 585
// against 727).
static uint32_t crt_lin_split_max() {
    static long v = -1;
    if (v < 0) {
        const char *e = getenv("FFG_CRT_LIN_SPLIT");
        v = e && *e ? strtol(e, nullptr, 10) : 128;
        if (v < 0) v = 0;
    }
    return (uint32_t)v;
}

cudaError_t launch_crt_lin(const CrtLinJob &J, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(k_crt_lin<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * kShortSmem));
        if (!e) e = cudaFuncSetAttribute(k_crt_lin<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * kBatchSmem));
        if (e) return e;
        configured = true;
    }
    if (J.width < 32 || J.width > 35 || J.alpha[0] <= 0 || J.alpha[1] <= 0) return cudaErrorInvalidValue;
    const uint32_t ncta = crt_ctas(J.len, J.width);
    prof_begin(PK_CRT, st);
    if (ncta <= crt_lin_split_max()) launch_after(k_crt_lin<1>, dim3(ncta, 2), 512, 2 * kShortSmem, st, garner_const(), J);
    else launch_after(k_crt_lin<2>, dim3(ncta, 1), 128, 2 * kBatchSmem, st, garner_const(), J);
    prof_end(PK_CRT, st, 12.0 * (double)(J.conv[0] + J.conv[1]) + 16.0 * (double)J.len);
    return cudaGetLastError();
}

// ----------------------------------------------------------- schoolbook

// k_school: a batch of schoolbook products (blockIdx.y the product), 256
// threads per CTA and SCHOOL_NL output limbs (columns) per CTA.  Column j
// sums a_i b_(j-i) over the shorter operand into 192 bits (t0, t1, t2); then
// v_j = t0_j + t1_(j-1) + t2_(j-2) < 3 2^64 leaves single-bit ripples for
// cta_resolve, and the last CTA settles the carries between CTAs.
constexpr uint32_t SCHOOL_NL = 1024;
constexpr uint32_t SCHOOL_THREADS = 256;

__host__ __device__ uint32_t school_ctas(uint64_t nlimbs) { return (uint32_t)((nlimbs + SCHOOL_NL - 1) / SCHOOL_NL); }

FFG_DEV_INLINE void school_col(const SchoolJob &J, int64_t j, uint64_t &t0, uint64_t &t1, uint64_t &t2) {
    t0 = t1 = t2 = 0;
    if (j < 0 || (uint64_t)j >= J.na + J.nb - 1) return;
    // iterate over the shorter operand
    const bool a_short = J.na <= J.nb;
    const uint64_t *S = a_short ? J.a : J.b, *Lg = a_short ? J.b : J.a;
    const int64_t ns = (int64_t)(a_short ? J.na : J.nb), nl = (int64_t)(a_short ? J.nb : J.na);
    const int64_t i0 = j - nl + 1 > 0 ? j - nl + 1 : 0, i1 = j < ns - 1 ? j : ns - 1;
    for (int64_t i = i0; i <= i1; i++) {
        const u128 pr = (u128)S[i] * Lg[j - i];
        const uint64_t lo = (uint64_t)pr, hi = (uint64_t)(pr >> 64);
        t0 += lo;
        const uint64_t c0 = t0 < lo;
        const uint64_t h = hi + c0; // hi < 2^64 - 1, so no wrap
        t1 += h;
        t2 += t1 < h;
    }
}

FFG_DEV_INLINE void school_block(const SchoolJob &J);

__global__ void __launch_bounds__(SCHOOL_THREADS) k_school(const SchoolJob *__restrict__ jobs) {
    after_previous();
    const SchoolJob J = jobs[blockIdx.y];
    if (blockIdx.x >= school_ctas(J.nlimbs)) return;
    school_block(J);
}

// Up to two schoolbook products by value (the doubling step's two squarings
// while the operands are short).
struct SchoolPair {
    SchoolJob j[2];
};
FFG_DEV_INLINE void school_block(const SchoolJob &J) {
    constexpr uint32_t NC = SCHOOL_NL + 3; // columns j0 - 3 .. j0 + NL - 1
    __shared__ uint64_t t0s[NC], t1s[NC];
    __shared__ uint32_t t2s[NC];
    __shared__ uint64_t lo[SCHOOL_NL];
    __shared__ uint32_t hi[SCHOOL_NL];
    __shared__ uint32_t gG[SCHOOL_NL / 32], gP[SCHOOL_NL / 32], gin[SCHOOL_NL / 32];
    __shared__ uint32_t hiprev_s;
    const int64_t j0 = (int64_t)blockIdx.x * SCHOOL_NL;
    for (uint32_t c = threadIdx.x; c < NC; c += blockDim.x) {
        uint64_t a, b, d;
        school_col(J, j0 - 3 + (int64_t)c, a, b, d);
        t0s[c] = a;
        t1s[c] = b;
        t2s[c] = (uint32_t)d;
    }
    __syncthreads();
    // v_j = t0_j + t1_(j-1) + t2_(j-2), for j = j0 - 1 .. j0 + NL - 1
    for (int32_t jl = (int32_t)threadIdx.x - 1; jl < (int32_t)SCHOOL_NL; jl += blockDim.x) {
        const uint32_t c = (uint32_t)(jl + 3);
        const u128 v = (u128)t0s[c] + t1s[c - 1] + t2s[c - 2];
        if (jl < 0) hiprev_s = (uint32_t)(v >> 64);
        else {
            lo[jl] = (uint64_t)v;
            hi[jl] = (uint32_t)(v >> 64);
        }
    }
    __syncthreads();
    const uint32_t map = cta_resolve(lo, hi, blockIdx.x ? hiprev_s : 0, SCHOOL_NL, gG, gP, gin);
    for (uint32_t j = threadIdx.x; j < SCHOOL_NL && (uint64_t)j0 + j < J.nlimbs; j += blockDim.x) J.out[j0 + j] = lo[j];
    if (threadIdx.x == 0) J.maps[blockIdx.x] = map;
    const uint32_t ncta = school_ctas(J.nlimbs);
    if (ncta > 1 && last_cta(J.ticket, ncta)) {
        settle_cta(J.out, J.nlimbs, SCHOOL_NL, J.maps, ncta);
        if (threadIdx.x == 0) *J.ticket = 0;
    }
}

// k_school_sq_pair: the doubling step's two short squarings (operands of up
// to 1536 limbs) spread over more CTAs than k_school gives them: SQ_NL = 32 output
// limbs per CTA, 14 threads per column (35 columns with the three below), and the
// symmetry of a square: column j = 2 sum_{i < j - i} a_i a_(j-i) + a_(j/2)^2 (j even).  The same 192-bit column sums, ripple settle and
// last-CTA carry settle as k_school.  The time is one thread's chain of products: with
// 64 limbs and 4 threads a column the chain of F(200 000) takes 74.4 us, with 64 and 7
// 67.3, with 32 and 7 67.6, with 32 and 14 65.7 (F(10^6) 143 -> 131).
constexpr uint32_t SQ_NL = 32;
constexpr uint32_t SQ_TPC = 14; // threads per column
constexpr uint32_t SQ_THREADS = 512;

__host__ __device__ uint32_t school_sq_ctas(uint64_t nlimbs) { return (uint32_t)((nlimbs + SQ_NL - 1) / SQ_NL); }

__global__ void __launch_bounds__(SQ_THREADS) k_school_sq_pair(SchoolPair Pr) {
    after_previous();
    const SchoolJob &J = blockIdx.y ? Pr.j[1] : Pr.j[0];
    const uint32_t ncta = school_sq_ctas(J.nlimbs);
    if (blockIdx.x >= ncta) return;
    constexpr uint32_t NC = SQ_NL + 3; // columns j0 - 3 .. j0 + SQ_NL - 1
    __shared__ uint64_t p0[NC][SQ_TPC], p1[NC][SQ_TPC];
    __shared__ uint32_t p2[NC][SQ_TPC];
    __shared__ uint64_t t0s[NC], t1s[NC];
    __shared__ uint32_t t2s[NC];
    __shared__ uint64_t lo[SQ_NL];
    __shared__ uint32_t hi[SQ_NL];
    __shared__ uint32_t gG[SQ_NL / 32], gP[SQ_NL / 32], gin[SQ_NL / 32];
    __shared__ uint32_t hiprev_s;
    const int64_t j0 = (int64_t)blockIdx.x * SQ_NL, n = (int64_t)J.na;
    const uint64_t *a = J.a;
    // partial sums of a_i a_(j-i) over i < j - i, i = part (mod SQ_TPC)
    for (uint32_t slot = threadIdx.x; slot < NC * SQ_TPC; slot += blockDim.x) {
        const uint32_t c = slot / SQ_TPC, part = slot % SQ_TPC;
        const int64_t j = j0 - 3 + (int64_t)c;
        uint64_t t0 = 0, t1 = 0, t2 = 0;
        if (j >= 1 && j <= 2 * n - 3) {
            const int64_t ilo = j - n + 1 > 0 ? j - n + 1 : 0, ihi = (j - 1) / 2; // i < j - i
            for (int64_t i = ilo + part; i <= ihi; i += SQ_TPC) {
                const u128 pr = (u128)a[i] * a[j - i];
                const uint64_t l = (uint64_t)pr, h = (uint64_t)(pr >> 64);
                t0 += l;
                const uint64_t hh = h + (t0 < l);
                t1 += hh;
                t2 += t1 < hh;
            }
        }
        p0[c][part] = t0;
        p1[c][part] = t1;
        p2[c][part] = (uint32_t)t2;
    }
    __syncthreads();
    // column j: 2 S_j + a_(j/2)^2, in 192 bits
    for (uint32_t c = threadIdx.x; c < NC; c += blockDim.x) {
        const int64_t j = j0 - 3 + (int64_t)c;
        uint64_t t0 = 0, t1 = 0, t2 = 0;
        for (uint32_t q = 0; q < SQ_TPC; q++) {
            t0 += p0[c][q];
            const uint64_t c0 = t0 < p0[c][q];
            const uint64_t x1 = p1[c][q] + c0; // p1 < 2^64 - 1 is not assured: carry both ways
            const uint64_t c1 = x1 < c0;
            t1 += x1;
            t2 += p2[c][q] + c1 + (t1 < x1);
        }
        // doubled
        t2 = (t2 << 1) | (t1 >> 63);
        t1 = (t1 << 1) | (t0 >> 63);
        t0 <<= 1;
        if (j >= 0 && j <= 2 * n - 2 && (j & 1) == 0) {
            const uint64_t x = a[j / 2];
            const u128 sq = (u128)x * x;
            const uint64_t l = (uint64_t)sq, h = (uint64_t)(sq >> 64);
            t0 += l;
            const uint64_t c0 = t0 < l;
            const uint64_t x1 = h + c0;
            const uint64_t c1 = x1 < c0;
            t1 += x1;
            t2 += c1 + (t1 < x1);
        }
        t0s[c] = t0;
        t1s[c] = t1;
        t2s[c] = (uint32_t)t2;
    }
    __syncthreads();
    // v_j = t0_j + t1_(j-1) + t2_(j-2), for j = j0 - 1 .. j0 + SQ_NL - 1
    for (int32_t jl = (int32_t)threadIdx.x - 1; jl < (int32_t)SQ_NL; jl += blockDim.x) {
        const uint32_t c = (uint32_t)(jl + 3);
        const u128 v = (u128)t0s[c] + t1s[c - 1] + t2s[c - 2];
        if (jl < 0) hiprev_s = (uint32_t)(v >> 64);
        else {
            lo[jl] = (uint64_t)v;
            hi[jl] = (uint32_t)(v >> 64);
        }
    }
    __syncthreads();
    const uint32_t map = cta_resolve(lo, hi, blockIdx.x ? hiprev_s : 0, SQ_NL, gG, gP, gin);
    for (uint32_t j = threadIdx.x; j < SQ_NL && (uint64_t)j0 + j < J.nlimbs; j += blockDim.x) J.out[j0 + j] = lo[j];
    if (threadIdx.x == 0) J.maps[blockIdx.x] = map;
    if (ncta > 1 && last_cta(J.ticket, ncta)) {
        settle_cta(J.out, J.nlimbs, SQ_NL, J.maps, ncta);
        if (threadIdx.x == 0) *J.ticket = 0;
    }
}

cudaError_t launch_school_sq_pair(const SchoolJob *jobs, uint32_t count, cudaStream_t st) {
    SchoolPair P{};
    uint32_t mx = 0;
    double bytes = 0;
    for (uint32_t i = 0; i < count && i < 2; i++) {
        if (jobs[i].a != jobs[i].b || jobs[i].na != jobs[i].nb) return cudaErrorInvalidValue;
        P.j[i] = jobs[i];
        mx = max(mx, school_sq_ctas(jobs[i].nlimbs));
        bytes += 8.0 * (double)(jobs[i].na + jobs[i].nlimbs);
    }
    prof_begin(PK_SCHOOL, st);
    launch_after(k_school_sq_pair, dim3(mx, count), SQ_THREADS, 0, st, P);
    prof_end(PK_SCHOOL, st, bytes);
    return cudaGetLastError();
}

cudaError_t launch_school_batch(const SchoolJob *d_jobs, uint32_t count, uint32_t max_ctas, cudaStream_t st,
                                double bytes) {
    if (!count) return cudaSuccess;
    prof_begin(PK_SCHOOL, st);
    launch_after(k_school, dim3(max_ctas, count), SCHOOL_THREADS, 0, st, d_jobs);
    prof_end(PK_SCHOOL, st, bytes);
    return cudaGetLastError();
}

// k_chain_steps: the doubling chain's first steps, up to STEP_IN limbs of operand, in
// one launch of one CTA: both squarings, the linear combinations and the carries of
// every step in shared memory.  As k_school_sq_pair and k_lin a step this short is two
// launches' latency (chain of F(20 000) 28.0 -> 25.4 us, of F(10^5) 55.4 -> 49.2, of
// F(10^7) 234 -> 227).  Longer steps are bound by the one SM's multiplier and keep
// their CTAs: with steps of up to 288 limbs F(10^5) takes 56.7 us.
//
// A step on n limbs: columns j and j + n of a square have n / 2 products together, so
// a thread takes every P-th product of such a pair (neighbours in j: one operand is a
// broadcast, the other consecutive).  P is what the threads allow, at most 8 (the parts
// are added by one thread a column).  A column's 192-bit sum
// t0 + 2^64 t1 + 2^128 t2 gives v_j = t0_j + t1_(j-1) + t2_(j-2) < 3 2^64, and output
// limb j is alpha v1_j + beta v2_j + 8 (2^64 - 1) >= 0 (beta >= -2): the bias adds
// 8 (2^(64 N) - 1) over the N limbs, so 8 more at limb 0 takes it out modulo 2^(64 N).
// Both outputs are resolved as one row with a zero limb behind each, which takes what
// runs out of the top.
constexpr uint32_t STEP_THREADS = 1024;
constexpr uint32_t STEP_ROW = 2 * STEP_IN + 32; // limbs of an output, with at least one of padding
static_assert(STEP_ROW % 32 == 0 && STEP_ROW >= 2 * STEP_IN + 2 && 2 * STEP_IN <= STEP_THREADS, "outputs and their padding, slots");

struct StepShared {
    uint64_t lo[2 * STEP_ROW];         // the pair: F(k-1), then F(k)
    uint64_t p0[2 * STEP_THREADS], p1[2 * STEP_THREADS]; // parts of the columns' sums
    uint64_t t0[4 * STEP_IN], t1[4 * STEP_IN];       // the columns' sums
    uint32_t p2[2 * STEP_THREADS], t2[4 * STEP_IN];
    uint32_t hi[2 * STEP_ROW];
    uint32_t gG[2 * STEP_ROW / 32], gP[2 * STEP_ROW / 32], gin[2 * STEP_ROW / 32];
};

__global__ void __launch_bounds__(STEP_THREADS) k_chain_steps(ChainSteps J) {
    after_previous();
    extern __shared__ __align__(16) unsigned char step_smem[];
    StepShared &S = *(StepShared *)step_smem;
    for (uint32_t j = threadIdx.x; j < 2 * STEP_IN; j += STEP_THREADS) {
        const bool up = j >= STEP_IN;
        const uint32_t i = up ? j - STEP_IN : j;
        S.lo[up ? STEP_ROW + i : i] = i < (up ? J.nk : J.nkm1) ? (up ? J.fk : J.fkm1)[i] : 0;
    }
    __syncthreads();
    uint32_t n = J.nk, odd = J.odd, row = STEP_ROW;
    for (uint32_t step = 0; step < J.steps; step++) {
        const uint32_t N = J.n_out[step], bit = J.bits >> step & 1u;
        // parts: slot (q, p, j) of columns j and j + n of square q (0: F(k), 1: F(k-1))
        const uint32_t fit = STEP_THREADS / (2 * n), P = fit < 8 ? fit : 8;
        for (uint32_t s = threadIdx.x; s < 2 * n * P; s += STEP_THREADS) {
            const uint32_t j = s % n, r = s / n, q = r >= P, p = q ? r - P : r;
            const uint64_t *a = S.lo + (q ? 0 : row);
#pragma unroll
            for (uint32_t half = 0; half < 2; half++) {
                const uint32_t c = j + half * n, ilo = half ? j + 1 : 0, iend = (c + 1) / 2; // i < c - i
                uint64_t t0 = 0, t1 = 0, t2 = 0;
#pragma unroll 2
                for (uint32_t i = ilo + p; i < iend; i += P) {
                    const u128 pr = (u128)a[i] * a[c - i];
                    const u128 sum = (u128)t1 << 64 | t0, acc = sum + pr;
                    t2 += acc < pr;
                    t0 = (uint64_t)acc;
                    t1 = (uint64_t)(acc >> 64);
                }
                const uint32_t at = (q * P + p) * 2 * n + c;
                S.p0[at] = t0;
                S.p1[at] = t1;
                S.p2[at] = (uint32_t)t2;
            }
        }
        __syncthreads();
        // column c of square q: twice its parts, and the middle square
        for (uint32_t s = threadIdx.x; s < 4 * n; s += STEP_THREADS) {
            const uint32_t q = s >= 2 * n, c = q ? s - 2 * n : s;
            u128 acc = 0;
            uint64_t top = 0;
            for (uint32_t p = 0; p < P; p++) {
                const uint32_t at = (q * P + p) * 2 * n + c;
                const u128 v = (u128)S.p1[at] << 64 | S.p0[at];
                acc += v;
                top += S.p2[at] + (acc < v);
            }
            top = top << 1 | (uint64_t)(acc >> 127);
            acc <<= 1;
            if (!(c & 1)) {
                const uint64_t x = S.lo[(q ? 0 : row) + c / 2];
                const u128 sq = (u128)x * x;
                acc += sq;
                top += acc < sq;
            }
            S.t0[s] = (uint64_t)acc;
            S.t1[s] = (uint64_t)(acc >> 64);
            S.t2[s] = (uint32_t)top;
        }
        __syncthreads();
        const int64_t pm2 = odd ? -2 : 2;
        row = (N + 32) & ~31u; // the outputs' rows: N limbs and at least one of padding
        for (uint32_t s = threadIdx.x; s < 2 * row; s += STEP_THREADS) {
            const uint32_t k = s >= row, j = k ? s - row : s;
            u128 w = 0;
            if (j < N) {
                auto column = [&](uint32_t q) { // v_j of square q
                    const uint32_t b = q * 2 * n;
                    u128 v = j < 2 * n ? S.t0[b + j] : 0;
                    if (j >= 1 && j - 1 < 2 * n) v += S.t1[b + j - 1];
                    if (j >= 2 && j - 2 < 2 * n) v += S.t2[b + j - 2];
                    return v;
                };
                const u128 v1 = column(0), v2 = column(1);
                // bit: 3 s1 - 2 s2 +- 2 and 4 s1 - s2 +- 2, else s1 + s2 and 3 s1 - 2 s2 +- 2
                const bool plain = !bit && !k;
                w = plain ? v1 + v2 : (bit && k ? v1 * 4 - v2 : v1 * 3 - v2 * 2);
                if (!plain) {
                    w += (u128)~0ull * 8;
                    if (j == 0) w += (u128)(uint64_t)(8 + pm2);
                }
            }
            S.lo[s] = (uint64_t)w;
            S.hi[s] = (uint32_t)(w >> 64);
        }
        __syncthreads();
        cta_resolve(S.lo, S.hi, 0, 2 * row, S.gG, S.gP, S.gin);
        n = N;
        odd = bit;
    }
    for (uint32_t j = threadIdx.x; j < 2 * n; j += STEP_THREADS) {
        const bool up = j >= n;
        const uint32_t i = up ? j - n : j;
        (up ? J.ok : J.okm1)[i] = S.lo[up ? row + i : i];
    }
}

cudaError_t launch_chain_steps(const ChainSteps &J, cudaStream_t st) {
    if (J.nk < 1 || J.nk > STEP_IN || J.nkm1 > J.nk || J.steps < 1 || J.steps > FFG_CHAIN_STEPS)
        return cudaErrorInvalidValue;
    for (uint32_t k = 0, n = J.nk; k < J.steps; n = J.n_out[k++])
        if (n > STEP_IN || J.n_out[k] < 1 || J.n_out[k] > 2 * n + 1) return cudaErrorInvalidValue;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(k_chain_steps, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(StepShared));
        if (e) return e;
        configured = true;
    }
    prof_begin(PK_SCHOOL, st);
    launch_after(k_chain_steps, 1, STEP_THREADS, sizeof(StepShared), st, J);
    prof_end(PK_SCHOOL, st, 8.0 * (double)(J.nk + J.nkm1 + 2 * J.n_out[J.steps - 1]));
    return cudaGetLastError();
}

// ------------------------------------------------------------ linear passes

// Two limbs a thread: the chain's short passes are one thread's latency (with 2048 limbs
// and 256 threads a CTA the F(10^5) chain takes 47.5 us, with 1024 and 512 44.9, with 512
// and 512, one limb a thread and twice the carries between CTAs, 49.2).
constexpr uint32_t LIN_NL = 1024; // limbs per CTA
constexpr uint32_t LIN_THREADS = 512;

uint32_t lin_ctas(uint64_t len) { return (uint32_t)((len + LIN_NL - 1) / LIN_NL); }

// Column sum of output k at limb j (0 past the output), from the limbs x, y
// of s1, s2 at j.
FFG_DEV_INLINE void lin_colsum(const LinJob &J, uint32_t k, uint64_t j, uint64_t x, uint64_t y, uint64_t &s_lo,
                               uint32_t &s_hi) {
    s_lo = 0;
    s_hi = 0;
    if (j >= J.len) return;
    const int64_t al = k ? J.alpha[1] : J.alpha[0], be = k ? J.beta[1] : J.beta[0];
    const int64_t ga = k ? J.gamma[1] : J.gamma[0];
    const u128 t = (u128)(al >= 0 ? x : ~x) * (uint64_t)(al >= 0 ? al : -al) +
                   (u128)(be >= 0 ? y : ~y) * (uint64_t)(be >= 0 ? be : -be);
    // constant: gamma plus one per negative term (-s = ~s + 1), two's complement
    const int64_t c = ga + (al < 0 ? -al : 0) + (be < 0 ? -be : 0);
    const uint64_t cj = j == 0 ? (uint64_t)c : (c < 0 ? ~0ull : 0ull);
    const u128 sum = t + cj;
    s_lo = (uint64_t)sum;
    s_hi = (uint32_t)(sum >> 64);
}

__global__ void __launch_bounds__(LIN_THREADS) k_lin(LinJob J) {
    after_previous();
    __shared__ uint64_t lo[LIN_NL];
    __shared__ uint32_t hi[LIN_NL];
    __shared__ uint32_t gG[LIN_NL / 32], gP[LIN_NL / 32], gin[LIN_NL / 32];
    __shared__ uint32_t hiprev_s;
    constexpr int PER = LIN_NL / LIN_THREADS;
    const uint64_t j0 = (uint64_t)blockIdx.x * LIN_NL;
    // every limb this thread needs, loaded once for both outputs
    uint64_t xs[PER], ys[PER];
#pragma unroll
    for (int r = 0; r < PER; r++) {
        const uint64_t j = j0 + threadIdx.x + r * LIN_THREADS;
        xs[r] = j < J.n1 ? J.s1[j] : 0;
        ys[r] = j < J.n2 ? J.s2[j] : 0;
    }
    uint64_t xp = 0, yp = 0; // limb j0 - 1, for the carry into the CTA's first limb
    if (threadIdx.x == 0 && j0 > 0) {
        xp = j0 - 1 < J.n1 ? J.s1[j0 - 1] : 0;
        yp = j0 - 1 < J.n2 ? J.s2[j0 - 1] : 0;
    }
    for (uint32_t k = 0; k < J.nout; k++) {
#pragma unroll
        for (int r = 0; r < PER; r++) {
            const uint32_t jl = threadIdx.x + r * LIN_THREADS;
            uint64_t s_lo;
            uint32_t s_hi;
            lin_colsum(J, k, j0 + jl, xs[r], ys[r], s_lo, s_hi);
            lo[jl] = s_lo;
            hi[jl] = s_hi;
        }
        if (threadIdx.x == 0) {
            uint64_t s_lo = 0;
            uint32_t s_hi = 0;
            if (j0 > 0) lin_colsum(J, k, j0 - 1, xp, yp, s_lo, s_hi);
            hiprev_s = s_hi;
        }
        __syncthreads();
        const uint32_t map = cta_resolve(lo, hi, hiprev_s, LIN_NL, gG, gP, gin);
        uint64_t *o = k ? J.out[1] : J.out[0];
        for (uint32_t j = threadIdx.x; j < LIN_NL && j0 + j < J.len; j += blockDim.x) o[j0 + j] = lo[j];
        if (threadIdx.x == 0) J.maps[(size_t)k * gridDim.x + blockIdx.x] = map;
        __syncthreads();
    }
    if (gridDim.x > 1 && last_cta(J.ticket, gridDim.x)) {
        for (uint32_t k = 0; k < J.nout; k++) settle_cta(k ? J.out[1] : J.out[0], J.len, LIN_NL, J.maps + (size_t)k * gridDim.x, gridDim.x);
        if (threadIdx.x == 0) *J.ticket = 0;
    }
}

cudaError_t launch_lin(const LinJob &J, cudaStream_t st) {
    const uint32_t ncta = lin_ctas(J.len);
    prof_begin(PK_LIN, st);
    launch_after(k_lin, ncta, LIN_THREADS, 0, st, J);
    prof_end(PK_LIN, st, 8.0 * (double)(J.n1 + J.n2) + 8.0 * (double)J.len * J.nout);
    return cudaGetLastError();
}

} // namespace ffg
