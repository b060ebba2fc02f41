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
#include <utility>

#include "ffg_cols.cuh"

namespace ffg {

template <int PI, int RN, bool R3>
FFG_DEV_INLINE void col_fwd2_body(const PrimeDev &P, const FourStep &G, const FSJob &J, uint32_t *smem) {
    using Q = ColGeo<RN, R3>;
    const uint32_t op = G.square ? 0 : (blockIdx.z & 1);
    const uint32_t C = 1u << G.c, wc = G.wc;
    const ColTile T{C, blockIdx.x * wc, G.wc_lg, wc - 1, col2_stride(Q::NBLK * Q::R, wc), 1};
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
    after_previous();
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
    const ColTile T{C, blockIdx.x * wc, G.wc_lg, wc - 1, col2_stride(Q::NBLK * Q::R, wc), 1};
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
    col_last<PI, RN, R3>(P, T, smem, [&](uint32_t row, uint32_t v) { col_out<PI>(O, row, v); });
}

template <int RN, bool R3>
__global__ void __launch_bounds__(kColThreads, 2) k_col_inv2(Primes3 P3, FourStep G, FSJobs jobs) {
    after_previous();
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

// Loads a pass's kernel and opts it into its shared memory, once.
template <int RN, bool R3> static cudaError_t load_col2_t(bool fwd) {
    const void *k = fwd ? (const void *)k_col_fwd2<RN, R3> : (const void *)k_col_inv2<RN, R3>;
    static bool attr[2] = {false, false};
    if (attr[fwd]) return cudaSuccess;
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k);
    if (!e) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColSmemMax);
    if (!e) attr[fwd] = true;
    return e;
}

template <int RN, bool R3>
static cudaError_t launch_col2_t(bool fwd, const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t nz,
                                 cudaStream_t st) {
    cudaError_t e = load_col2_t<RN, R3>(fwd);
    if (e) return e;
    const dim3 grid((1u << G.c) / G.wc, G.nprimes, nz);
    // threads per CTA: one per 16 words, at most 256 while four CTAs fit an SM's
    // shared memory, else 512 (at L = 2^24, tiles of 70 KB, the inverse pass takes
    // 164 us with 512 threads and 183 with 256; at L = 2^22, tiles of 35 KB, 45
    // and 39).  A multiple of wc, so that a thread keeps its column.
    const uint32_t groups = G.wc * (uint32_t)(G.R / 16), tmax = col2_smem(G) > 56 * 1024 ? kColThreads : kColThreads / 2;
    uint32_t threads = groups < tmax ? groups : tmax;
    threads = threads < 64 ? 64 : threads & ~31u;
    threads -= threads % G.wc;
    if (fwd) launch_after(k_col_fwd2<RN, R3>, grid, threads, col2_smem(G), st, P3, G, jobs);
    else launch_after(k_col_inv2<RN, R3>, grid, threads, col2_smem(G), st, P3, G, jobs);
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

template <bool R3, int... RN>
static cudaError_t load_col2_n(uint32_t rn, std::integer_sequence<int, RN...>) {
    cudaError_t e = cudaSuccess;
    for (bool fwd : {true, false})
        ((rn == RN + 6 && !e ? (void)(e = load_col2_t<RN + 6, R3>(fwd)) : (void)0), ...);
    return e;
}
cudaError_t load_col2(const FourStep &G) {
    return G.r3 ? load_col2_n<true>(G.rn, std::make_integer_sequence<int, 6>{})   // 3 2^6 .. 3 2^11
                : load_col2_n<false>(G.rn, std::make_integer_sequence<int, 7>{}); // 2^6 .. 2^12
}

// nz: grid depth (jobs x operands for the forward pass, jobs for the inverse).
cudaError_t launch_col2(bool fwd, const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t nz,
                        cudaStream_t st) {
    return G.r3 ? launch_col2_r<true>(fwd, P3, G, jobs, nz, st) : launch_col2_r<false>(fwd, P3, G, jobs, nz, st);
}

} // namespace ffg
