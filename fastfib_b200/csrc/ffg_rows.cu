// The four-step row pass with its shape fixed at compile time, for rows of
// C = 2^CLG words (9 <= CLG <= 13).
//
// The forward transform of a row is three radix steps of decimation in
// frequency:
//   A: radix 2^LA at stride SA = C / 2^LA, straight from global memory;
//   B: radix 2^LB at stride 16, blocks of 16 2^LB words;
//   C: radix 16 at stride 1 (no step twiddles).
// Step C, the pointwise product and the first inverse step (radix 16 at
// stride 1, decimation in time) run on the same 16 registers of a thread
// with no shared-memory round trip in between; then B^-1, and A^-1 ends with
// the four-step twiddle ω_L^-(n2 k1), the scale of the convolution and the
// store of the row.  Every shared address is a compile-time offset from one
// base per group, on padded lines (pad(i) = i + i/32).  No access has a bank
// conflict (step B: the two half-warps take blocks KB apart, half the banks
// away; rows of 512 have too few blocks for that).
//
// A thread carries 16 words of a row (32 of a row of 8192); a CTA holds up to
// 256 / T rows of T threads, fewer when that would leave SMs idle (the launch
// picks the rows per CTA).
// Radix 16 at the bottom (radix 32 before) costs the same instructions and
// exchanges but halves a thread's registers and its chain of dependent work: a
// launch of few rows lasts one thread's chain (one square of 4000 limbs, L =
// 2^14: 16.8 -> 10.7 us; the row passes of the F(10^8) chain 283 -> 228 us).  Long
// rows are bound by the integer pipes (L = 2^24: 275 -> 269 us, 4 CTAs an SM).
//
// It computes the same residues as the generic row pass of ffg_ntt.cu
// (k_row_conv, mode ROW_CONV): the order of the frequencies between the
// forward and the inverse differs, but the pointwise product does not care.
#include "ffg_internal.h"
#include "ffg_lines.cuh"

namespace ffg {

template <int CLG> struct RowShape;
template <> struct RowShape<9> { static constexpr int LA = 2, LB = 3, KB = 1; };
template <> struct RowShape<10> { static constexpr int LA = 3, LB = 3, KB = 4; };
template <> struct RowShape<11> { static constexpr int LA = 3, LB = 4, KB = 2; };
template <> struct RowShape<12> { static constexpr int LA = 4, LB = 4, KB = 2; };
template <> struct RowShape<13> { static constexpr int LA = 4, LB = 5, KB = 1; };

constexpr uint32_t cx_line_stride(uint32_t N) {
    return (((N + (N - 1) / 32 + 1) + 31) & ~31u) + 1;
}

template <int CLG> struct RowGeo {
    static constexpr int LA = RowShape<CLG>::LA, LB = RowShape<CLG>::LB;
    static constexpr uint32_t C = 1u << CLG;
    static constexpr uint32_t T = CLG == 13 ? 256 : C / 16; // threads per row
    static constexpr uint32_t ROWS = 256 / T;      // most rows per CTA
    static constexpr uint32_t RA = 1u << LA, RB = 1u << LB;
    static constexpr uint32_t SA = C >> LA;        // stride of step A
    static constexpr uint32_t SAP = SA + SA / 32;  // its padded distance
    static constexpr uint32_t GA = C / RA / T, GB = C / RB / T, GC = C / 16 / T; // groups per thread
    static constexpr uint32_t NBP = 16 * RB + RB / 2; // padded block of step B
    static constexpr uint32_t KB = RowShape<CLG>::KB;
    static constexpr uint32_t LS = cx_line_stride(C); // shared words per line
    static_assert(LA + LB + 4 == CLG && GA && GB && GC && SA % 32 == 0, "three steps cover the row");
    static_assert((C / (16 * RB)) % (2 * KB) == 0, "blocks in pairs KB apart");
};

// Step B's group g: word j of block b, shared offset of its first word; word t
// of the group is 16 t + t / 2 further.
template <int CLG> FFG_DEV_INLINE uint32_t row_b_base(uint32_t g) {
    using Q = RowGeo<CLG>;
    const uint32_t j = g & 15, r = g >> 5;
    const uint32_t b = (r % Q::KB) + ((g >> 4) & 1) * Q::KB + (r / Q::KB) * (2 * Q::KB);
    return b * Q::NBP + j;
}
__host__ __device__ constexpr uint32_t row_b_off(uint32_t t) { return 16 * t + t / 2; }

// Forward steps A and B of one operand: global row g into the padded shared
// line s (a barrier in between, none after).
template <int PI, int CLG>
FFG_DEV_INLINE void row_fwd_a(const uint32_t *__restrict__ g, uint32_t *__restrict__ s, uint32_t tau,
                              const uint2 *__restrict__ tw) {
    using Q = RowGeo<CLG>;
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GA; k++) {
        const uint32_t j = tau + Q::T * k;
        uint32_t x[Q::RA];
#pragma unroll
        for (uint32_t t = 0; t < Q::RA; t++) x[t] = g[j + Q::SA * t];
        dft_dif<PI, Q::LA>(x);
#pragma unroll
        for (uint32_t t = 1; t < Q::RA; t++) x[t] = sh<PI>(x[t], __ldg(&tw[(t - 1) * Q::SA + j]));
        uint32_t *d = s + j + (j >> 5);
#pragma unroll
        for (uint32_t t = 0; t < Q::RA; t++) d[t * Q::SAP] = x[t];
    }
}
template <int PI, int CLG>
FFG_DEV_INLINE void row_fwd_b(uint32_t *__restrict__ s, uint32_t tau, const uint2 *__restrict__ tw) {
    using Q = RowGeo<CLG>;
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GB; k++) {
        uint32_t *d = s + row_b_base<CLG>(tau + Q::T * k);
        uint32_t x[Q::RB];
#pragma unroll
        for (uint32_t t = 0; t < Q::RB; t++) x[t] = d[row_b_off(t)];
        dft_dif<PI, Q::LB>(x);
#pragma unroll
        for (uint32_t t = 1; t < Q::RB; t++) x[t] = sh<PI>(x[t], __ldg(&tw[(t - 1) * 16 + (tau & 15)]));
#pragma unroll
        for (uint32_t t = 0; t < Q::RB; t++) d[row_b_off(t)] = x[t];
    }
}

template <int PI, int CLG, bool SQ>
FFG_DEV_INLINE void row2_body(const PrimeDev &P, const FourStep &G, uint32_t *ja, const uint32_t *jb, uint32_t *smem) {
    using Q = RowGeo<CLG>;
    const uint32_t r = threadIdx.x / Q::T, tau = threadIdx.x % Q::T;
    const uint32_t pos = blockIdx.x * (blockDim.x / Q::T) + r;
    const size_t rowoff = (size_t)PI * G.L + (size_t)pos * Q::C;
    uint32_t *ya = ja + rowoff;
    uint32_t *sa = smem + r * (SQ ? 1 : 2) * Q::LS;
    uint32_t *sb = sa + Q::LS;
    const uint2 *twA = P.stw + c_lines.tw_off[(4 + Q::LB) * 6 + Q::LA];
    const uint2 *twB = P.stw + c_lines.tw_off[4 * 6 + Q::LB];

    row_fwd_a<PI, CLG>(ya, sa, tau, twA);
    if (!SQ) row_fwd_a<PI, CLG>(jb + rowoff, sb, tau, twA);
    __syncthreads();
    row_fwd_b<PI, CLG>(sa, tau, twB);
    if (!SQ) row_fwd_b<PI, CLG>(sb, tau, twB);
    __syncthreads();

    // step C, the pointwise product and C^-1 on registers
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GC; k++) {
        const uint32_t b = tau + Q::T * k;
        uint32_t x[16];
        uint32_t *d = sa + 16 * b + (b >> 1);
        if (!SQ) {
            uint32_t *e = sb + 16 * b + (b >> 1);
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = e[t];
            dft_dif<PI, 4>(x);
#pragma unroll
            for (int t = 0; t < 16; t++) e[t] = x[t]; // read back below by this thread only
        }
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = d[t];
        dft_dif<PI, 4>(x);
        if (SQ) {
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = mo<PI>(x[t], x[t]);
        } else {
            const uint32_t *e = sb + 16 * b + (b >> 1);
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = mo<PI>(x[t], e[t]);
        }
        dft_dit<PI, 4>(x);
#pragma unroll
        for (int t = 0; t < 16; t++) d[t] = x[t];
    }
    __syncthreads();

    // B^-1
    const uint2 *itwB = P.istw + c_lines.tw_off[4 * 6 + Q::LB];
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GB; k++) {
        uint32_t *d = sa + row_b_base<CLG>(tau + Q::T * k);
        uint32_t x[Q::RB];
#pragma unroll
        for (uint32_t t = 0; t < Q::RB; t++) x[t] = d[row_b_off(t)];
#pragma unroll
        for (uint32_t t = 1; t < Q::RB; t++) x[t] = sh<PI>(x[t], __ldg(&itwB[(t - 1) * 16 + (tau & 15)]));
        dft_dit<PI, Q::LB>(x);
#pragma unroll
        for (uint32_t t = 0; t < Q::RB; t++) d[row_b_off(t)] = x[t];
    }
    __syncthreads();

    // A^-1, then ω_L^-(n2 k1) times the scale for n2 = j + SA t (a running product
    // over t), and the store.  n2 < C and k1 < R: the exponents are below L, their
    // multiples of M / L below M.  The scale costs one product a group here, one a
    // residue in the column pass.
    const uint32_t kms = freq_of(pos, G.rn, G.r3) * (uint32_t)G.mstep;
    auto back = [&](uint32_t n2) {
        const uint32_t e = n2 * kms;
        return twm<PI>(P, e ? (uint32_t)FFG_M - e : 0);
    };
    const uint32_t step = back(Q::SA);
    const uint2 sc = make_uint2(G.scl[PI], G.scls[PI]);
    const uint2 *itwA = P.istw + c_lines.tw_off[(4 + Q::LB) * 6 + Q::LA];
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GA; k++) {
        const uint32_t j = tau + Q::T * k;
        uint32_t cur = sh<PI>(back(j), sc);
        const uint32_t *d = sa + j + (j >> 5);
        uint32_t x[Q::RA];
#pragma unroll
        for (uint32_t t = 0; t < Q::RA; t++) x[t] = d[t * Q::SAP];
#pragma unroll
        for (uint32_t t = 1; t < Q::RA; t++) x[t] = sh<PI>(x[t], __ldg(&itwA[(t - 1) * Q::SA + j]));
        dft_dit<PI, Q::LA>(x);
#pragma unroll
        for (uint32_t t = 0; t < Q::RA; t++) {
            ya[j + Q::SA * t] = mo<PI>(x[t], cur);
            if (t + 1 < Q::RA) cur = mo<PI>(cur, step);
        }
    }
}

template <int CLG, bool SQ>
__global__ void __launch_bounds__(256, CLG == 13 && !SQ ? 3 : 4) k_row2(Primes3 P3, FourStep G, FSJobs jobs) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t *jy[2];
    if (threadIdx.x == 0) {
        const FSJob &J = jobs.ext ? jobs.ext[blockIdx.z] : jobs.j[blockIdx.z < FFG_FS_JOBS ? blockIdx.z : 0];
        jy[0] = J.ya;
        jy[1] = J.yb;
    }
    __syncthreads();
    switch (blockIdx.y + G.prime0) {
    case 0: row2_body<0, CLG, SQ>(P3.pr[0], G, jy[0], jy[1], smem); break;
    case 1: row2_body<1, CLG, SQ>(P3.pr[1], G, jy[0], jy[1], smem); break;
    default: row2_body<2, CLG, SQ>(P3.pr[2], G, jy[0], jy[1], smem); break;
    }
}

template <int CLG, bool SQ>
static cudaError_t launch_row2_t(const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t njobs,
                                 cudaStream_t st) {
    using Q = RowGeo<CLG>;
    const size_t smax = (size_t)Q::ROWS * (SQ ? 1 : 2) * Q::LS * sizeof(uint32_t);
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(k_row2<CLG, SQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax);
        if (e) return e;
        attr = true;
    }
    // rows per CTA: as many as fit 256 threads, halved while the launch would
    // have fewer than three CTAs per SM (short rows of a mid-size product)
    uint32_t rows = Q::ROWS;
    while (rows > 1 && (uint64_t)(G.R / rows) * G.nprimes * njobs < 3 * 148) rows >>= 1;
    while (rows > 1 && G.R % rows) rows >>= 1;
    const size_t sm = (size_t)rows * (SQ ? 1 : 2) * Q::LS * sizeof(uint32_t);
    k_row2<CLG, SQ><<<dim3(G.R / rows, G.nprimes, njobs), rows * Q::T, sm, st>>>(P3, G, jobs);
    return cudaGetLastError();
}

// This unit's copy of the line-transform constants (each CUDA unit has its
// own constant bank); set once with the others.
cudaError_t set_line_consts_rows(const LineConsts &h) { return cudaMemcpyToSymbol(c_lines, &h, sizeof h); }

// Whether the fixed-shape row pass takes this geometry (ROW_CONV rows of
// 2^9 .. 2^13 words).
bool row2_ok(const FourStep &G) { return G.mode == ROW_CONV && G.c >= 9 && G.c <= 13; }

cudaError_t launch_row2(const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t njobs, cudaStream_t st) {
    const bool sq = G.square != 0;
    switch (G.c) {
    case 9: return sq ? launch_row2_t<9, true>(P3, G, jobs, njobs, st) : launch_row2_t<9, false>(P3, G, jobs, njobs, st);
    case 10: return sq ? launch_row2_t<10, true>(P3, G, jobs, njobs, st) : launch_row2_t<10, false>(P3, G, jobs, njobs, st);
    case 11: return sq ? launch_row2_t<11, true>(P3, G, jobs, njobs, st) : launch_row2_t<11, false>(P3, G, jobs, njobs, st);
    case 12: return sq ? launch_row2_t<12, true>(P3, G, jobs, njobs, st) : launch_row2_t<12, false>(P3, G, jobs, njobs, st);
    default: return sq ? launch_row2_t<13, true>(P3, G, jobs, njobs, st) : launch_row2_t<13, false>(P3, G, jobs, njobs, st);
    }
}

} // namespace ffg
