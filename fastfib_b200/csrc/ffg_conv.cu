// The one-CTA convolution with its length fixed at compile time: lengths 2^RN
// (6 <= RN <= 14) and 3 2^RN (RN <= 12), one CTA per (product, prime) with the
// whole transform in shared memory (ffg_cols.cuh's steps on one line per
// operand).  The first step reads the digits of both operands, the last forward
// step, the pointwise product and the first inverse step share a thread's 16
// registers, the last inverse step scales by 2^32 / L and stores the
// coefficients.  This is the reference's in-cache convolution
// (src/ntt_conv.c:205-226, src/ntt_kernels.c:274-295) as one kernel; shorter
// lengths run the generic one (k_conv_small, ffg_ntt.cu).
//
// Bound by latency: a single product is three CTAs, whose time is one thread's
// chain.  A thread per 16 words of each operand (the two operands' lines side by
// side), compile-time shapes and three barriers fewer take a product of 300 x 257
// limbs from 21.6 to 12.3 us (CRT included) and the one-CTA launches of a
// 20.9-million-digit decimal conversion from 2.66 to 1.19 ms against the generic
// kernel (256 threads, runtime shapes).
#include "ffg_cols.cuh"

namespace ffg {

constexpr uint32_t kConvThreads = 512;

template <int PI, int RN, bool R3, bool SQ, bool W32>
FFG_DEV_INLINE void conv2_first(const PrimeDev &P, const ConvJob &J, const ColTile &T, uint32_t *smem) {
    using Q = ColGeo<RN, R3>;
    const ColSrc A = col_src(J.a, J.na, J.ca, 0, J.width), B = col_src(J.b, J.nb, J.cb, 0, J.width);
    auto src = [&](uint32_t c) { return SQ || c == 0 ? A : B; };
    // a balanced product's operands fill at most half of the line
    const uint64_t most = SQ || J.ca > J.cb ? J.ca : J.cb;
    if constexpr (R3) {
        if (most <= 2 * Q::R) col_fwd2_first_r3<PI, RN, 2, Q::RE, W32>(P, src, T, smem);
        else col_fwd2_first_r3<PI, RN, 3, Q::RE, W32>(P, src, T, smem);
    } else {
        if (most <= Q::R / 2) col_fwd2_first<PI, RN, Q::RE / 2, W32>(P, src, T, smem);
        else col_fwd2_first<PI, RN, Q::RE, W32>(P, src, T, smem);
    }
}

template <int PI, int RN, bool R3, bool SQ>
FFG_DEV_INLINE void conv2_body(const PrimeDev &P, const ConvJob &J, uint32_t *smem) {
    using Q = ColGeo<RN, R3>;
    constexpr uint32_t LS = Q::NBLK * Q::BP, LINES = SQ ? 1 : 2;
    const ColTile both{1, 0, LINES - 1, LINES - 1, LS, 0}, one{1, 0, 0, 0, LS, 0};
    if (J.width == 32) conv2_first<PI, RN, R3, SQ, true>(P, J, both, smem);
    else conv2_first<PI, RN, R3, SQ, false>(P, J, both, smem);
    __syncthreads();
    if (Q::LA) {
        col_step<PI, Q::LB, 4, true>(both, Q::NBLK * (Q::R / Q::RB), P.stw + c_lines.tw_off[4 * 6 + Q::LB], smem);
        __syncthreads();
    }
    // step C, the pointwise product and C^-1
#pragma unroll 1
    for (uint32_t b = threadIdx.x; b < Q::NBLK * Q::R / 16; b += blockDim.x) {
        uint32_t x[16];
        uint32_t *d = smem + 17 * b;
        if (!SQ) {
            uint32_t *e = d + LS;
#pragma unroll
            for (int t = 0; t < 16; t++) x[t] = e[t];
            dft_dif<PI, 4>(x);
#pragma unroll
            for (int t = 0; t < 16; t++) e[t] = x[t]; // read back below by this thread only
        }
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = d[t];
        dft_dif<PI, 4>(x);
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = mo<PI>(x[t], SQ ? x[t] : d[LS + t]);
        dft_dit<PI, 4>(x);
#pragma unroll
        for (int t = 0; t < 16; t++) d[t] = x[t];
    }
    __syncthreads();
    if (Q::LA) {
        col_step<PI, Q::LB, 4, false>(one, Q::NBLK * (Q::R / Q::RB), P.istw + c_lines.tw_off[4 * 6 + Q::LB], smem);
        __syncthreads();
    }
    uint32_t *const y = J.y + (size_t)PI * J.y_stride;
    const uint32_t conv = J.conv;
    const uint2 sc = make_uint2(J.scl[PI], J.scls[PI]);
    col_last<PI, RN, R3>(P, one, smem, [&](uint32_t row, uint32_t v) {
        if (row < conv) y[row] = sh<PI>(v, sc);
    });
}

template <int RN, bool R3, bool SQ>
__global__ void __launch_bounds__(kConvThreads, 2) k_conv2(Primes3 P3, ConvJobs jobs) {
    after_previous();
    extern __shared__ uint32_t smem[];
    __shared__ ConvJob J;
    if (threadIdx.x == 0) J = jobs.ext ? jobs.ext[blockIdx.x] : jobs.j[blockIdx.x < FFG_CONV_JOBS ? blockIdx.x : 0];
    __syncthreads();
    switch (blockIdx.y) {
    case 0: conv2_body<0, RN, R3, SQ>(P3.pr[0], J, smem); break;
    case 1: conv2_body<1, RN, R3, SQ>(P3.pr[1], J, smem); break;
    default: conv2_body<2, RN, R3, SQ>(P3.pr[2], J, smem); break;
    }
}

cudaError_t set_line_consts_conv(const LineConsts &h) { return cudaMemcpyToSymbol(c_lines, &h, sizeof h); }

bool conv2_ok(uint32_t n, uint32_t r3) { return n >= 6 && n <= (r3 ? 12u : 14u); }

// attr_only: configure (and load) the kernel without launching it.
template <int RN, bool R3, bool SQ>
static cudaError_t launch_conv2_t(const Primes3 &P3, const ConvJobs &jobs, uint32_t njobs, bool attr_only,
                                  cudaStream_t st) {
    using Q = ColGeo<RN, R3>;
    constexpr size_t sm = (size_t)(SQ ? 1 : 2) * Q::NBLK * Q::BP * sizeof(uint32_t);
    static bool attr = false;
    if (!attr) {
        cudaFuncAttributes fa;
        cudaError_t e = cudaFuncGetAttributes(&fa, k_conv2<RN, R3, SQ>);
        if (!e) e = cudaFuncSetAttribute(k_conv2<RN, R3, SQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e) return e;
        attr = true;
    }
    if (attr_only) return cudaSuccess;
    // a thread per 16 words of every operand
    constexpr uint32_t want = (SQ ? 1 : 2) * Q::NBLK * (Q::R / 16);
    constexpr uint32_t threads = want < 32 ? 32 : want > kConvThreads ? kConvThreads : (want + 31) & ~31u;
    launch_after(k_conv2<RN, R3, SQ>, dim3(njobs, 3), threads, sm, st, P3, jobs);
    return cudaGetLastError();
}

template <bool R3, bool SQ>
static cudaError_t launch_conv2_n(const Primes3 &P3, const ConvJobs &jobs, uint32_t njobs, uint32_t n, bool attr_only,
                                  cudaStream_t st) {
    switch (n) {
    case 6: return launch_conv2_t<6, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 7: return launch_conv2_t<7, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 8: return launch_conv2_t<8, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 9: return launch_conv2_t<9, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 10: return launch_conv2_t<10, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 11: return launch_conv2_t<11, R3, SQ>(P3, jobs, njobs, attr_only, st);
    case 12: return launch_conv2_t<12, R3, SQ>(P3, jobs, njobs, attr_only, st);
    default: break;
    }
    if constexpr (!R3) {
        if (n == 13) return launch_conv2_t<13, R3, SQ>(P3, jobs, njobs, attr_only, st);
        if (n == 14) return launch_conv2_t<14, R3, SQ>(P3, jobs, njobs, attr_only, st);
    }
    return cudaErrorInvalidValue;
}

// njobs convolutions of one length 2^n or 3 2^n, all squares or all products.
cudaError_t launch_conv2(const Primes3 &P3, const ConvJobs &jobs, uint32_t njobs, uint32_t n, uint32_t r3, bool square,
                         cudaStream_t st) {
    if (r3)
        return square ? launch_conv2_n<true, true>(P3, jobs, njobs, n, false, st)
                      : launch_conv2_n<true, false>(P3, jobs, njobs, n, false, st);
    return square ? launch_conv2_n<false, true>(P3, jobs, njobs, n, false, st)
                  : launch_conv2_n<false, false>(P3, jobs, njobs, n, false, st);
}

cudaError_t load_conv2(uint32_t n, uint32_t r3, bool square) {
    const Primes3 P{};
    const ConvJobs none{};
    if (r3)
        return square ? launch_conv2_n<true, true>(P, none, 0, n, true, nullptr)
                      : launch_conv2_n<true, false>(P, none, 0, n, true, nullptr);
    return square ? launch_conv2_n<false, true>(P, none, 0, n, true, nullptr)
                  : launch_conv2_n<false, false>(P, none, 0, n, true, nullptr);
}

} // namespace ffg
