// fp32 CUDA-core GEMM: C[M,N] = A[M,K] . W[N,K]^T (+ bias, + activation).  Any alignment, fp32 or
// bf16 operands, fp32 accumulation.  It serves the fp32 (reference-precision) path and the shapes
// too small or too ragged for the tensor-core kernel.
#include "gemm.cuh"

namespace hx {
namespace gemm {

// A CTA of 256 threads computes a BM x BN tile; KG groups of threads each take every KG-th slice of KS inner indices and
// a thread holds TM x TN products of its group.  A slab of KG * KS inner indices is staged per step (transposed to
// [k][row] so that a thread reads its operands as 16-byte groups), the next slab's global loads are in flight under the
// current one and the slabs alternate between two buffers: one barrier per slab.  The groups' partial tiles are added in
// fixed order through shared memory, so a result does not depend on timing.
//
// Bound: the FMA pipe once a shape fills the SMs (an operand value loaded from shared memory serves TM or TN products),
// latency below that; then more and smaller tiles with the inner dimension split inside the CTA win.  Picked by how many
// tiles the shape has (launch_simt).  Against 64 x 64 tiles with 4 x 4 products a thread, one element loaded at a time and
// no overlap of load and product: block f32 [16, 2000, 1024] 17.8 -> 10.3 ms, [4, 2000, 640] 2156 -> 1476 us, [2, 500, 512]
// 405 -> 213 us; the four products of a MambaBlock [256, 512] d_state 64 together 184 -> 60 us, of one [100, 64] 27.7 -> 13.9.
//
// Staged rows are XOR-swizzled by the group of four inner indices they belong to: the transposing stores of a warp
// (consecutive 4-element groups of k for a few rows) then fall into different banks.
template <int BM_, int BN_, int TM_, int TN_, int KG_, int KS_>
struct SimtCfg {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, KG = KG_, KS = KS_;
    static constexpr int SLAB = KG * KS;
    static constexpr int GT = (BM / TM) * (BN / TN);  // threads of a group
    static constexpr int Q = SLAB / 4;                // 4-element groups of a staged row
    static constexpr int SWZ = Q >= 8 ? 4 : 32 / Q;   // rows a warp's store covers (a multiple of 4)
    static_assert(GT * KG == 256 && GT % 32 == 0, "256 threads, whole warps per group");
    static_assert(BM * Q % 256 == 0 && BN * Q % 256 == 0, "whole rounds of staging loads");
    static_assert(2 * SLAB * (BM + BN) * 4 <= 48 * 1024 && (KG == 1 || BM * BN <= 2 * SLAB * (BM + BN)), "shared memory");
};

// Four consecutive values of a row from k on; past `valid` they are zeros.
template <typename T, bool VEC> __device__ __forceinline__ float4 ld_row4(const T *p, int valid) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (VEC) {  // K is a multiple of 4: all or none
        if (valid > 0) {
            if constexpr (sizeof(T) == 4) {
                v = *reinterpret_cast<const float4 *>(p);
            } else {
                const uint2 r = *reinterpret_cast<const uint2 *>(p);
                v = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16),
                                __uint_as_float(r.y & 0xffff0000u));
            }
        }
    } else {
        if (valid > 0) v.x = ld_f32(p);
        if (valid > 1) v.y = ld_f32(p + 1);
        if (valid > 2) v.z = ld_f32(p + 2);
        if (valid > 3) v.w = ld_f32(p + 3);
    }
    return v;
}

template <typename TA, typename TC, int EPI, typename Cfg, bool VEC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA *A, int64_t lda, const TA *W, int64_t ldw, const float *bias, TC *C, int64_t ldc, int M, int N,
                 int K) {
    constexpr int BM = Cfg::BM, BN = Cfg::BN, TM = Cfg::TM, TN = Cfg::TN, SLAB = Cfg::SLAB, Q = Cfg::Q;
    constexpr int RA = BM * Q / 256, RW = BN * Q / 256;  // staging loads per thread
    __shared__ __align__(16) float smem[2 * SLAB * (BM + BN)];
    const int tid = threadIdx.x;
    const int grp = tid / Cfg::GT, gt = tid % Cfg::GT;
    const int tx = gt % (BN / TN), ty = gt / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float4 ra[RA], rw[RW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < RA; ++i) {
            const int r = (tid + i * 256) / Q, k = k0 + (tid % Q) * 4;
            ra[i] = ld_row4<TA, VEC>(A + (int64_t)(m0 + r) * lda + k, m0 + r < M ? K - k : 0);
        }
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const int r = (tid + i * 256) / Q, k = k0 + (tid % Q) * 4;
            rw[i] = ld_row4<TA, VEC>(W + (int64_t)(n0 + r) * ldw + k, n0 + r < N ? K - k : 0);
        }
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    fetch(0);
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += SLAB, buf ^= 1) {
        float *As = smem + buf * SLAB * (BM + BN), *Ws = As + SLAB * BM;  // [k][row ^ swizzle of k / 4]
        const int kq = tid % Q, sw = (kq & 7) * Cfg::SWZ;
#pragma unroll
        for (int i = 0; i < RA; ++i) {
            const int c = ((tid + i * 256) / Q) ^ sw;
            As[(kq * 4 + 0) * BM + c] = ra[i].x; As[(kq * 4 + 1) * BM + c] = ra[i].y;
            As[(kq * 4 + 2) * BM + c] = ra[i].z; As[(kq * 4 + 3) * BM + c] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const int c = ((tid + i * 256) / Q) ^ sw;
            Ws[(kq * 4 + 0) * BN + c] = rw[i].x; Ws[(kq * 4 + 1) * BN + c] = rw[i].y;
            Ws[(kq * 4 + 2) * BN + c] = rw[i].z; Ws[(kq * 4 + 3) * BN + c] = rw[i].w;
        }
        __syncthreads();
        if (k0 + SLAB < K) fetch(k0 + SLAB);
#pragma unroll
        for (int s = 0; s < Cfg::KS; ++s) {
            const int k = grp * Cfg::KS + s, swk = ((k >> 2) & 7) * Cfg::SWZ;
            float a[TM], w[TN];
            // a thread's rows (columns) are groups of four, TM / 4 (TN / 4) of them spread over the tile
#pragma unroll
            for (int v = 0; v < TM / 4; ++v) {
                const float4 f = *reinterpret_cast<const float4 *>(As + k * BM + ((v * (BM * 4 / TM) + ty * 4) ^ swk));
                a[4 * v] = f.x; a[4 * v + 1] = f.y; a[4 * v + 2] = f.z; a[4 * v + 3] = f.w;
            }
#pragma unroll
            for (int v = 0; v < TN / 4; ++v) {
                const float4 f = *reinterpret_cast<const float4 *>(Ws + k * BN + ((v * (BN * 4 / TN) + tx * 4) ^ swk));
                w[4 * v] = f.x; w[4 * v + 1] = f.y; w[4 * v + 2] = f.z; w[4 * v + 3] = f.w;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
    }
    if constexpr (Cfg::KG > 1) {  // add the groups' tiles in order: groups KG-1, ..., 1 onto group 0
        for (int g = Cfg::KG - 1; g > 0; --g) {
            __syncthreads();
            if (grp == g) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) smem[(i * TN + j) * Cfg::GT + gt] = acc[i][j];
            }
            __syncthreads();
            if (grp == g - 1) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] += smem[(i * TN + j) * Cfg::GT + gt];
            }
        }
        if (grp != 0) return;
    }
    // fp32 rows on 16-byte boundaries leave as 16-byte stores
    const bool c16 = sizeof(TC) == 4 && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + (i / 4) * (BM * 4 / TM) + ty * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int v = 0; v < TN / 4; ++v) {
            const int n = n0 + v * (BN * 4 / TN) + tx * 4;
            float o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = apply_epilogue<EPI>(acc[i][v * 4 + j] + (bias && n + j < N ? bias[n + j] : 0.f));
            TC *cp = C + (int64_t)m * ldc + n;
            if (c16 && n + 4 <= N) {
                *reinterpret_cast<float4 *>(cp) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N) st_f32(cp + j, o[j]);
            }
        }
    }
}

template <typename TA, typename TC, typename Cfg, bool VEC>
static hx_status launch_simt_cfg(const TA *a, int64_t lda, const TA *w, int64_t ldw, const float *bias, TC *c, int64_t ldc, int M,
                                 int N, int K, int epi, cudaStream_t st) {
    dim3 grid((N + Cfg::BN - 1) / Cfg::BN, (M + Cfg::BM - 1) / Cfg::BM), block(256);
    switch (epi) {
        case kEpiNone: gemm_simt_kernel<TA, TC, kEpiNone, Cfg, VEC><<<grid, block, 0, st>>>(a, lda, w, ldw, bias, c, ldc, M, N, K); break;
        case kEpiSilu: gemm_simt_kernel<TA, TC, kEpiSilu, Cfg, VEC><<<grid, block, 0, st>>>(a, lda, w, ldw, bias, c, ldc, M, N, K); break;
        case kEpiSoftplus: gemm_simt_kernel<TA, TC, kEpiSoftplus, Cfg, VEC><<<grid, block, 0, st>>>(a, lda, w, ldw, bias, c, ldc, M, N, K); break;
        default: return fail(HX_ERR_INVALID_INPUT, "unknown epilogue %d", epi);
    }
    return check_launch("gemm_simt_kernel");
}

// The largest tile that still gives three quarters of the SMs one each: a bigger tile does more products per operand
// read, but an idle SM costs more than that.  The smallest tiles split the inner dimension four ways inside the CTA.
// Up to 64 columns half or more of a big tile would be padding: 64 x 64 tiles with slabs of 16 there (100000 x 16 x 16 9.7 us
// against 17.0, 65536 x 64 x 64 17.7 against 31, 65536 x 64 x 1024 251 against 423); where the middle tile is the choice it stays
// ahead of them (8000 x 64 x 4096 209 against 273).
template <typename TA, typename TC, bool VEC>
static hx_status launch_simt_tiles(const TA *a, int64_t lda, const TA *w, int64_t ldw, const float *bias, TC *c, int64_t ldc,
                                   int M, int N, int K, int epi, cudaStream_t st) {
    using Big = SimtCfg<128, 128, 8, 8, 1, 8>;
    using Mid = SimtCfg<64, 64, 8, 8, 4, 8>;
    using Small = SimtCfg<32, 32, 4, 4, 4, 16>;
    using Narrow = SimtCfg<64, 64, 4, 4, 1, 16>;
    auto tiles = [&](int bm, int bn) { return (int64_t)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    const int64_t enough = (int64_t)sm_count() * 3 / 4;
    if (tiles(Big::BM, Big::BN) >= enough)
        return N <= 64 ? launch_simt_cfg<TA, TC, Narrow, VEC>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st)
                       : launch_simt_cfg<TA, TC, Big, VEC>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st);
    if (tiles(Mid::BM, Mid::BN) >= enough) return launch_simt_cfg<TA, TC, Mid, VEC>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st);
    return launch_simt_cfg<TA, TC, Small, VEC>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st);
}

template <typename TA, typename TC>
static hx_status launch_simt(const void *A, int64_t lda, const void *W, int64_t ldw, const float *bias, void *C,
                             int64_t ldc, int M, int N, int K, int epi, cudaStream_t st) {
    auto a = static_cast<const TA *>(A);
    auto w = static_cast<const TA *>(W);
    auto c = static_cast<TC *>(C);
    HX_REQUIRE((M + 63) / 64 <= 65535, HX_ERR_INVALID_DIMENSION, "M %d too large for the SIMT GEMM grid", M);
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) % (4 * sizeof(TA))) == 0; };
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && al(A) && al(W);
    return vec ? launch_simt_tiles<TA, TC, true>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st)
               : launch_simt_tiles<TA, TC, false>(a, lda, w, ldw, bias, c, ldc, M, N, K, epi, st);
}

hx_status validate_gemm(const void *A, int64_t lda, const void *W, int64_t ldw, void *C, int64_t ldc, int M, int N, int K) {
    HX_REQUIRE(M >= 0 && N >= 0 && K >= 0, HX_ERR_INVALID_DIMENSION, "negative GEMM dimension (%d, %d, %d)", M, N, K);
    if (M == 0 || N == 0) return HX_OK;
    HX_REQUIRE(A && W && C, HX_ERR_INVALID_INPUT, "A, W and C must not be NULL");
    HX_REQUIRE(lda >= K && ldw >= K && ldc >= N, HX_ERR_SHAPE_MISMATCH,
               "leading dimension too small (lda %lld, ldw %lld, ldc %lld for K %d, N %d)", (long long)lda,
               (long long)ldw, (long long)ldc, K, N);
    return HX_OK;
}

}  // namespace gemm
}  // namespace hx

extern "C" hx_status hx_gemm_simt(const void *A, int64_t lda, const void *W, int64_t ldw, const float *bias, void *C,
                                  int64_t ldc, int32_t ab_dtype, int32_t c_dtype, int32_t M, int32_t N, int32_t K,
                                  int32_t epilogue, void *stream) {
    using namespace hx::gemm;
    hx_status s = validate_gemm(A, lda, W, ldw, C, ldc, M, N, K);
    if (s != HX_OK) return s;
    if (M == 0 || N == 0) return HX_OK;
    HX_REQUIRE((ab_dtype == HX_F32 || ab_dtype == HX_BF16) && (c_dtype == HX_F32 || c_dtype == HX_BF16),
               HX_ERR_DTYPE_MISMATCH, "dtype unsupported (ab %d, c %d)", ab_dtype, c_dtype);
    cudaStream_t st = (cudaStream_t)stream;
    const bool ab = ab_dtype == HX_BF16, cb = c_dtype == HX_BF16;
    if (ab && cb) return launch_simt<__nv_bfloat16, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    if (ab) return launch_simt<__nv_bfloat16, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    if (cb) return launch_simt<float, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    return launch_simt<float, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
}
