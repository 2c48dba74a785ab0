// gemm_skinny_kernel: C[M,N] = A[M,K] . W[N,K]^T for a handful of rows (M <= 64), the shape of a decode step.
// With so few rows the GEMM is a stream over the weights: every byte of W is needed once and nothing is
// reused, so the persistent tcgen05 kernel (one 128-row tile, one CTA per 256 columns) spends its time in
// set-up, and what matters is how many weight bytes are in flight.  A CTA owns 8 output columns; its 16 warps
// split K in blocks of 32 (round-robin), each warp runs mma.sync.m16n8k16 (bf16 in, fp32 accumulate) over its
// blocks with all of its loads issued up front, and the 16 partial tiles are summed through shared memory.
// The grid is N/8 CTAs, so every SM streams a slice of W and the whole kernel is about one memory round trip.
//
// Operand loads are 16 bytes per lane.  The MMA does not care in which order the k indices are presented as
// long as A and B agree, so inside a block of 32 k values lane (g, tid) loads the 8 consecutive elements
// k = 8 tid .. 8 tid + 7 of its row and uses them as the two k-halves of two MMAs:
//   MMA j (j = 0, 1): "k pair 2 tid" = elements 4 j + {0, 1}, "k pair 2 tid + 8" = elements 4 j + {2, 3}.
// A comes straight from global memory (it is M x K, a few tens of KB, shared by every CTA through L2/L1).
//
// CHAIN: launched by launch_chained under the kernel before it.  A, C and the bias then carry no __restrict__ (their loads must
// stay behind chain_wait()) and the weights of four k-blocks, inner dimensions up to 2048, are requested before waiting.  By
// itself the kernel has nothing to fetch them under and takes two blocks a trip, W and A of one before the other's: four of W
// first cost registers that more rows need and put the rows behind them (17 x 4096 x 4096 16.9 us against 10.9, 24 x 4096 x 1024
// 7.2 against 5.4, 32 x 3072 x 768 6.0 against 5.2, 1 x 4096 x 4096 7.5 against 6.6).
#include "gemm.cuh"

namespace hx {
namespace gemm {

constexpr int kSkinnyWarps = 16;

template <int MT, typename TC, int EPI, bool CHAIN>
__device__ __forceinline__ void
gemm_skinny_body(const __nv_bfloat16 *A, int64_t lda, const __nv_bfloat16 *W, int64_t ldw, const float *bias, TC *C, int64_t ldc,
                 int M, int N, int K, int epi_col0) {
    if constexpr (CHAIN) chain_trigger();
    __shared__ float partial[kSkinnyWarps * MT * 128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tid = lane & 3;
    const int n0 = blockIdx.x * 8;
    const int n = n0 + g;                                   // the W row this lane loads
    const bool n_ok = n < N;
    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
    const __nv_bfloat16 *wrow = W + (int64_t)(n_ok ? n : 0) * ldw + tid * 8;
    const __nv_bfloat16 *arow[MT][2];
    bool a_ok[MT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = mt * 16 + h * 8 + g;
            a_ok[mt][h] = r < M;
            arow[mt][h] = A + (int64_t)(a_ok[mt][h] ? r : 0) * lda + tid * 8;
        }
    float acc[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[mt][i] = 0.f;

    auto mma = [&](const uint4 (&a)[MT][2], const uint4 &b) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            // fragment registers: a0 = (row g, k pair), a1 = (row g+8, k pair), a2 = (row g, k pair + 8), a3 = (row g+8, ...)
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                         "{%0, %1, %2, %3};"
                         : "+f"(acc[mt][0]), "+f"(acc[mt][1]), "+f"(acc[mt][2]), "+f"(acc[mt][3])
                         : "r"(a[mt][0].x), "r"(a[mt][1].x), "r"(a[mt][0].y), "r"(a[mt][1].y), "r"(b.x), "r"(b.y));
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                         "{%0, %1, %2, %3};"
                         : "+f"(acc[mt][0]), "+f"(acc[mt][1]), "+f"(acc[mt][2]), "+f"(acc[mt][3])
                         : "r"(a[mt][0].z), "r"(a[mt][1].z), "r"(a[mt][0].w), "r"(a[mt][1].w), "r"(b.z), "r"(b.w));
        }
    };
    // this warp's k-blocks: warp, warp + 16, ...
    constexpr int STEP = kSkinnyWarps * 32;
    auto ld_w = [&](int k) { return (n_ok && k < K) ? *reinterpret_cast<const uint4 *>(wrow + k) : zero4; };
    auto ld_a = [&](uint4 (&a)[MT][2], int k) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) a[mt][h] = (a_ok[mt][h] && k < K) ? *reinterpret_cast<const uint4 *>(arow[mt][h] + k) : zero4;
    };
    uint4 a[2][MT][2];
    int k0 = warp * 32;
    if constexpr (CHAIN) {  // four blocks of W before the wait, then twice two of A
        uint4 b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = ld_w(k0 + u * STEP);
        chain_wait();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (k0 >= K) break;   // warp-uniform
#pragma unroll
            for (int u = 0; u < 2; ++u) ld_a(a[u], k0 + u * STEP);
#pragma unroll
            for (int u = 0; u < 2; ++u) mma(a[u], b[half * 2 + u]);
            k0 += 2 * STEP;
        }
    }
    for (; k0 < K; k0 += 2 * STEP) {  // two blocks per trip so that their loads overlap
        uint4 b[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            b[u] = ld_w(k0 + u * STEP);
            ld_a(a[u], k0 + u * STEP);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) mma(a[u], b[u]);
    }
    // partial[warp][mt][lane][i]; accumulator layout: i = 0, 1 -> (row g, columns 2 tid, 2 tid + 1); i = 2, 3 -> row g + 8
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
        *reinterpret_cast<float4 *>(&partial[((warp * MT + mt) * 32 + lane) * 4]) =
            make_float4(acc[mt][0], acc[mt][1], acc[mt][2], acc[mt][3]);
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= MT * 128) return;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kSkinnyWarps; ++w) v += partial[w * MT * 128 + t];
    const int mt = t >> 7, ln = (t & 127) >> 2, i = t & 3;
    const int r = mt * 16 + (i >> 1) * 8 + (ln >> 2);
    const int c = n0 + 2 * (ln & 3) + (i & 1);
    if (r < M && c < N) {
        if (bias) v += bias[c];
        if constexpr (EPI == kEpiAccumulate) C[(int64_t)r * ldc + c] += TC(v);  // fp32 C; this thread owns the element
        else st_f32(C + (int64_t)r * ldc + c, c >= epi_col0 ? apply_epilogue<EPI>(v) : v);
    }
}

template <int MT, typename TC, int EPI>
__global__ void __launch_bounds__(kSkinnyWarps * 32)
gemm_skinny_kernel(const __nv_bfloat16 *__restrict__ A, int64_t lda, const __nv_bfloat16 *__restrict__ W, int64_t ldw,
                   const float *__restrict__ bias, TC *__restrict__ C, int64_t ldc, int M, int N, int K, int epi_col0) {
    gemm_skinny_body<MT, TC, EPI, false>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi_col0);
}
template <int MT, typename TC, int EPI>
__global__ void __launch_bounds__(kSkinnyWarps * 32)
gemm_skinny_chain_kernel(const __nv_bfloat16 *A, int64_t lda, const __nv_bfloat16 *__restrict__ W, int64_t ldw, const float *bias,
                         TC *C, int64_t ldc, int M, int N, int K, int epi_col0) {
    gemm_skinny_body<MT, TC, EPI, true>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi_col0);
}

template <int MT, typename TC>
static hx_status launch_skinny_epi(const void *A, int64_t lda, const void *W, int64_t ldw, const float *bias, void *C, int64_t ldc,
                                   int M, int N, int K, int epi, int epi_col0, cudaStream_t st, bool chain) {
    const dim3 grid((unsigned)((N + 7) / 8)), block(kSkinnyWarps * 32);
    auto a = static_cast<const __nv_bfloat16 *>(A), w = static_cast<const __nv_bfloat16 *>(W);
    auto c = static_cast<TC *>(C);
    cudaError_t e = cudaSuccess;
#define HX_SKINNY_LAUNCH(KERNEL, EPI) e = launch_chained(chain, KERNEL<MT, TC, EPI>, grid, block, st, a, lda, w, ldw, bias, c, ldc, M, N, K, epi_col0)
    HX_REQUIRE(!chain || epi == kEpiNone || epi == kEpiAccumulate, HX_ERR_INVALID_INPUT, "a chained launch has no epilogue %d", epi);
    switch (epi) {
        case kEpiNone:
            if (chain) HX_SKINNY_LAUNCH(gemm_skinny_chain_kernel, kEpiNone);
            else HX_SKINNY_LAUNCH(gemm_skinny_kernel, kEpiNone);
            break;
        case kEpiSilu: HX_SKINNY_LAUNCH(gemm_skinny_kernel, kEpiSilu); break;
        case kEpiSoftplus: HX_SKINNY_LAUNCH(gemm_skinny_kernel, kEpiSoftplus); break;
        case kEpiSiluFast: HX_SKINNY_LAUNCH(gemm_skinny_kernel, kEpiSiluFast); break;
        case kEpiAccumulate:
            if constexpr (sizeof(TC) == 4) {
                if (chain) HX_SKINNY_LAUNCH(gemm_skinny_chain_kernel, kEpiAccumulate);
                else HX_SKINNY_LAUNCH(gemm_skinny_kernel, kEpiAccumulate);
            } else {
                return fail(HX_ERR_DTYPE_MISMATCH, "accumulating GEMM needs an fp32 C");
            }
            break;
        default: return fail(HX_ERR_INVALID_INPUT, "unknown epilogue %d", epi);
    }
#undef HX_SKINNY_LAUNCH
    HX_CUDA(e);
    return check_launch("gemm_skinny_kernel");
}

// M <= 64, K a multiple of 32, lda / ldw multiples of 8 and 16-byte aligned bases (checked by the caller).
hx_status launch_skinny(const void *A, int64_t lda, const void *W, int64_t ldw, const float *bias, void *C, int64_t ldc,
                        int c_dtype, int M, int N, int K, int epi, int epi_col0, cudaStream_t st, bool chain) {
#define HX_SKINNY(MT)                                                                                                   \
    return c_dtype == HX_BF16 ? launch_skinny_epi<MT, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, epi_col0, st, chain)    \
                              : launch_skinny_epi<MT, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, epi_col0, st, chain)
    if (M <= 16) { HX_SKINNY(1); }
    if (M <= 32) { HX_SKINNY(2); }
    HX_SKINNY(4);
#undef HX_SKINNY
}

}  // namespace gemm
}  // namespace hx
