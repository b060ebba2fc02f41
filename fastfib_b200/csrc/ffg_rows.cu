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
// The split's row modes run the same steps: ROW_FWD stops after step C and
// stores the transformed piece in step C's order, ROW_ACC_INV starts from the
// sum of its pieces' products in that order.
//
// It computes the same residues as the generic row pass of ffg_ntt.cu
// (k_row_conv): the order of the frequencies between the forward and the
// inverse differs, but the pointwise product does not care.
#include <utility>

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

// What k_row2 does with its rows (FourStep::mode and square).
enum RowKind { RK_SQUARE, RK_PRODUCT, RK_FORWARD, RK_PIECE };

// 16 consecutive words of a residue row (16-byte aligned: the split's pieces
// lie in the arena).
FFG_DEV_INLINE void ld16(uint32_t (&x)[16], const uint32_t *p) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint4 v = ((const uint4 *)p)[k];
        x[4 * k] = v.x, x[4 * k + 1] = v.y, x[4 * k + 2] = v.z, x[4 * k + 3] = v.w;
    }
}

// The split's output piece m on 16 words of its row: the sum over i + j = m of
// the transformed pieces' products (src/mul_split.c:62-78); of a square's equal
// pairs one is computed and doubled.  at: the words' place in a piece.
template <int PI> FFG_DEV_INLINE void piece_sum(const FSJob &J, size_t at, uint32_t (&acc)[16]) {
    const uint32_t m = J.m, i0 = m + 1 > J.kb ? m + 1 - J.kb : 0;
    uint32_t i1 = m < J.ka - 1 ? m : J.ka - 1;
    if (J.psq) i1 = m ? min(i1, (m - 1) / 2) : 0; // i < j
    const uint32_t *pa = J.pa + at, *pb = J.pb + at;
    uint32_t x[16], y[16];
#pragma unroll
    for (int t = 0; t < 16; t++) acc[t] = 0;
    if (!J.psq || m) {
#pragma unroll 1
        for (uint32_t i = i0; i <= i1; i++) {
            ld16(x, pa + i * J.piece_stride);
            ld16(y, pb + (m - i) * J.piece_stride);
#pragma unroll
            for (int t = 0; t < 16; t++) acc[t] = ad<PI>(acc[t], mo<PI>(x[t], y[t]));
        }
    }
    if (!J.psq) return;
#pragma unroll
    for (int t = 0; t < 16; t++) acc[t] = ad<PI>(acc[t], acc[t]);
    if (m % 2 == 0 && m / 2 < J.ka) {
        ld16(x, pa + (m / 2) * J.piece_stride);
#pragma unroll
        for (int t = 0; t < 16; t++) acc[t] = ad<PI>(acc[t], mo<PI>(x[t], x[t]));
    }
}

template <int PI, int CLG, int KIND>
FFG_DEV_INLINE void row2_body(const PrimeDev &P, const FourStep &G, const FSJob &J, uint32_t *smem) {
    using Q = RowGeo<CLG>;
    constexpr bool TWO = KIND == RK_PRODUCT;
    const uint32_t r = threadIdx.x / Q::T, tau = threadIdx.x % Q::T;
    const uint32_t pos = blockIdx.x * (blockDim.x / Q::T) + r;
    const size_t rowoff = (size_t)PI * G.L + (size_t)pos * Q::C;
    uint32_t *ya = J.ya + rowoff;
    uint32_t *sa = smem + r * (TWO ? 2 : 1) * Q::LS;
    uint32_t *sb = sa + Q::LS;

    if (KIND != RK_PIECE) {
        const uint2 *twA = P.stw + c_lines.tw_off[(4 + Q::LB) * 6 + Q::LA];
        const uint2 *twB = P.stw + c_lines.tw_off[4 * 6 + Q::LB];
        row_fwd_a<PI, CLG>(ya, sa, tau, twA);
        if (TWO) row_fwd_a<PI, CLG>(J.yb + rowoff, sb, tau, twA);
        __syncthreads();
        row_fwd_b<PI, CLG>(sa, tau, twB);
        if (TWO) row_fwd_b<PI, CLG>(sb, tau, twB);
        __syncthreads();
    }

    // step C, the pointwise product and C^-1 on registers
#pragma unroll 1
    for (uint32_t k = 0; k < Q::GC; k++) {
        const uint32_t b = tau + Q::T * k;
        uint32_t x[16];
        uint32_t *d = sa + 16 * b + (b >> 1);
        if (KIND == RK_PIECE) {
            piece_sum<PI>(J, rowoff + 16 * b, x);
        } else {
            if (TWO) {
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
            if (KIND == RK_FORWARD) { // the transformed piece, in the order RK_PIECE reads
#pragma unroll
                for (int t = 0; t < 4; t++)
                    ((uint4 *)(ya + 16 * b))[t] = make_uint4(x[4 * t], x[4 * t + 1], x[4 * t + 2], x[4 * t + 3]);
                continue;
            }
            if (TWO) {
                const uint32_t *e = sb + 16 * b + (b >> 1);
#pragma unroll
                for (int t = 0; t < 16; t++) x[t] = mo<PI>(x[t], e[t]);
            } else {
#pragma unroll
                for (int t = 0; t < 16; t++) x[t] = mo<PI>(x[t], x[t]);
            }
        }
        dft_dit<PI, 4>(x);
#pragma unroll
        for (int t = 0; t < 16; t++) d[t] = x[t];
    }
    if (KIND == RK_FORWARD) return;
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

template <int CLG, int KIND>
__global__ void __launch_bounds__(256, CLG == 13 && KIND == RK_PRODUCT ? 3 : 4) k_row2(Primes3 P3, FourStep G, FSJobs jobs) {
    after_previous();
    extern __shared__ uint32_t smem[];
    __shared__ FSJob J;
    if (threadIdx.x == 0) J = jobs.ext ? jobs.ext[blockIdx.z] : jobs.j[blockIdx.z < FFG_FS_JOBS ? blockIdx.z : 0];
    __syncthreads();
    switch (blockIdx.y + G.prime0) {
    case 0: row2_body<0, CLG, KIND>(P3.pr[0], G, J, smem); break;
    case 1: row2_body<1, CLG, KIND>(P3.pr[1], G, J, smem); break;
    default: row2_body<2, CLG, KIND>(P3.pr[2], G, J, smem); break;
    }
}

// Loads a kernel and opts it into its shared memory, once.
template <int CLG, int KIND> static cudaError_t load_row2_t() {
    using Q = RowGeo<CLG>;
    static bool attr = false;
    if (attr) return cudaSuccess;
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k_row2<CLG, KIND>);
    const size_t smax = (size_t)Q::ROWS * (KIND == RK_PRODUCT ? 2 : 1) * Q::LS * sizeof(uint32_t);
    if (!e) e = cudaFuncSetAttribute(k_row2<CLG, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax);
    if (!e) attr = true;
    return e;
}

template <int CLG, int KIND>
static cudaError_t launch_row2_t(const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t njobs,
                                 cudaStream_t st) {
    using Q = RowGeo<CLG>;
    constexpr uint32_t lines = KIND == RK_PRODUCT ? 2 : 1;
    cudaError_t e = load_row2_t<CLG, KIND>();
    if (e) return e;
    // rows per CTA: as many as fit 256 threads, halved while the launch would
    // have fewer than three CTAs per SM (short rows of a mid-size product)
    uint32_t rows = Q::ROWS;
    while (rows > 1 && (uint64_t)(G.R / rows) * G.nprimes * njobs < 3 * 148) rows >>= 1;
    while (rows > 1 && G.R % rows) rows >>= 1;
    const size_t sm = (size_t)rows * lines * Q::LS * sizeof(uint32_t);
    launch_after(k_row2<CLG, KIND>, dim3(G.R / rows, G.nprimes, njobs), rows * Q::T, sm, st, P3, G, jobs);
    return cudaGetLastError();
}

// This unit's copy of the line-transform constants (each CUDA unit has its
// own constant bank); set once with the others.
cudaError_t set_line_consts_rows(const LineConsts &h) { return cudaMemcpyToSymbol(c_lines, &h, sizeof h); }

template <int... CLG> static cudaError_t load_row2_c(uint32_t c, bool square, std::integer_sequence<int, CLG...>) {
    cudaError_t e = cudaSuccess;
    ((c == CLG + 9 ? (void)(e = square ? load_row2_t<CLG + 9, RK_SQUARE>() : load_row2_t<CLG + 9, RK_PRODUCT>())
                   : (void)0),
     ...);
    return e;
}
cudaError_t load_row2(const FourStep &G) {
    return load_row2_c(G.c, G.square != 0, std::make_integer_sequence<int, 5>{}); // 2^9 .. 2^13
}

// Whether the fixed-shape row pass takes this geometry (rows of 2^9 .. 2^13
// words).
bool row2_ok(const FourStep &G) { return G.c >= 9 && G.c <= 13; }

template <int CLG>
static cudaError_t launch_row2_k(const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t njobs,
                                 cudaStream_t st) {
    switch (G.mode) {
    case ROW_FWD: return launch_row2_t<CLG, RK_FORWARD>(P3, G, jobs, njobs, st);
    case ROW_ACC_INV: return launch_row2_t<CLG, RK_PIECE>(P3, G, jobs, njobs, st);
    default:
        return G.square ? launch_row2_t<CLG, RK_SQUARE>(P3, G, jobs, njobs, st)
                        : launch_row2_t<CLG, RK_PRODUCT>(P3, G, jobs, njobs, st);
    }
}

cudaError_t launch_row2(const Primes3 &P3, const FourStep &G, const FSJobs &jobs, uint32_t njobs, cudaStream_t st) {
    switch (G.c) {
    case 9: return launch_row2_k<9>(P3, G, jobs, njobs, st);
    case 10: return launch_row2_k<10>(P3, G, jobs, njobs, st);
    case 11: return launch_row2_k<11>(P3, G, jobs, njobs, st);
    case 12: return launch_row2_k<12>(P3, G, jobs, njobs, st);
    default: return launch_row2_k<13>(P3, G, jobs, njobs, st);
    }
}

} // namespace ffg
