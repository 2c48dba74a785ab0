// S4 recurrences for sm_100a.
//
// s4_diag_kernel: the per-channel diagonal form  h_t = abar h_{t-1} + bbar u_t,  y = C.h + D u.
//   The system is time-invariant, so the sequence is cut into 8 segments that run in parallel
//   inside one CTA (one warp per segment):
//     pass 1  every segment runs the recurrence from a zero state (no output) to get its end state,
//     combine the start state of segment g is the Horner sum of the earlier end states with
//             abar^segment_length, exchanged through shared memory,
//     pass 2  every segment reruns from its true start state and emits y.
//   With g = h / bbar the update is one FMA per state (g = abar g + u) and the output one more
//   (y += (C bbar) g).  16 states per lane, the lanes of a channel are adjacent and combine their
//   partial dot products with shuffles.
//
// s4_ref_*: the reference-literal recurrence of nn::ssm::S4Block::forward_ssm
//   (crates/nn/src/ssm.rs:138-186): one d_state-wide state driven by all d_model inputs.
//   It is computed as  V = dt * (B . U)  ->  diagonal scan over time on V (same 3-pass scheme,
//   all segments in one CTA)  ->  Y = X . C^T + D * U.
#include "hx_tma.cuh"

namespace hx {
namespace s4 {

constexpr int kSeg = 8;   // segments per sequence (= warps per CTA) in s4_diag_kernel

// kNSL = states per lane (8 or 16): fewer states per lane means more lanes per channel, i.e. more warps for a
// small problem and fewer registers per thread, at the price of one more shuffle per step.
template <typename T, int LPC, int kNSL>
__global__ void __launch_bounds__(kSeg * 32, kNSL == 8 ? 4 : 2)
s4_diag_kernel(const T *u, const float *A, const float *Bp, const float *Cp, const float *delta, const float *Dskip, T *y,
               int L, int D, int N) {
    constexpr int CW = 32 / LPC;  // channels per warp
    constexpr int TU = kNSL == 8 ? 4 : 8;  // steps loaded ahead of the arithmetic
    __shared__ float ends[kSeg][32][kNSL];  // [segment][lane][state of the lane]
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = lane / LPC, q = lane % LPC;
    const int d = blockIdx.x * CW + c;
    const int b = blockIdx.y;
    const bool chan_ok = d < D;
    const int seg_len = (L + kSeg - 1) / kSeg;
    const int t0 = min(L, g * seg_len), t1 = min(L, t0 + seg_len);

    float2 a[kNSL / 2], k[kNSL / 2], aT[kNSL / 2];
    const float dl = chan_ok ? delta[d] : 0.f;
#pragma unroll
    for (int j = 0; j < kNSL; ++j) {
        const int n = q * kNSL + j;
        float av = 0.f, kv = 0.f, atv = 0.f;
        if (chan_ok && n < N) {
            const float an = A[(int64_t)d * N + n];
            av = expf(dl * an);
            atv = expf(dl * an * (float)seg_len);
            kv = Cp[(int64_t)d * N + n] * (dl * Bp[(int64_t)d * N + n]);
        }
        if (j & 1) { a[j / 2].y = av; k[j / 2].y = kv; aT[j / 2].y = atv; }
        else { a[j / 2].x = av; k[j / 2].x = kv; aT[j / 2].x = atv; }
    }
    const T *up = u + ((int64_t)b * L) * D + (chan_ok ? d : 0);
    T *yp = y + ((int64_t)b * L) * D + (chan_ok ? d : 0);
    const float dsk = (chan_ok && Dskip) ? Dskip[d] : 0.f;

    // ---- pass 1: end state of the segment from a zero start
    float2 h[kNSL / 2];
#pragma unroll
    for (int j = 0; j < kNSL / 2; ++j) h[j] = make_float2(0.f, 0.f);
    // the loads of the next TU steps are issued before the arithmetic of the current ones: all warps of a CTA walk
    // in step, so without this every batch would wait out a full memory round trip
    auto fetch = [&](int t, float *dst) {
#pragma unroll
        for (int e = 0; e < TU; ++e) dst[e] = (t + e < t1 && chan_ok) ? ld_f32(up + (int64_t)(t + e) * D) : 0.f;
    };
    // Full batches of TU steps run without a per-step guard (a branch per step would keep the compiler from
    // overlapping the dependent chains of neighbouring steps); the ragged end of the segment runs guarded.
    float ub[TU], un[TU];
    fetch(t0, ub);
    int t = t0;
    for (; t + TU <= t1; t += TU) {
        fetch(t + TU, un);
#pragma unroll
        for (int e = 0; e < TU; ++e) {
            const float2 u2 = splat2(ub[e]);
#pragma unroll
            for (int j = 0; j < kNSL / 2; ++j) h[j] = fma2(a[j], h[j], u2);
        }
#pragma unroll
        for (int e = 0; e < TU; ++e) ub[e] = un[e];
    }
#pragma unroll
    for (int e = 0; e < TU; ++e) {
        if (t + e < t1) {  // warp-uniform
            const float2 u2 = splat2(ub[e]);
#pragma unroll
            for (int j = 0; j < kNSL / 2; ++j) h[j] = fma2(a[j], h[j], u2);
        }
    }
#pragma unroll
    for (int j = 0; j < kNSL / 2; ++j) {
        ends[g][lane][2 * j] = h[j].x;
        ends[g][lane][2 * j + 1] = h[j].y;
    }
    __syncthreads();
    // ---- combine: start state of segment g (all earlier segments are full length)
#pragma unroll
    for (int j = 0; j < kNSL / 2; ++j) h[j] = make_float2(0.f, 0.f);
    for (int gp = 0; gp < g; ++gp) {
#pragma unroll
        for (int j = 0; j < kNSL / 2; ++j)
            h[j] = fma2(aT[j], h[j], make_float2(ends[gp][lane][2 * j], ends[gp][lane][2 * j + 1]));
    }
    // ---- pass 2: the real run
    auto step_sum = [&](float uv) {
        const float2 u2 = splat2(uv);
        float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < kNSL / 2; j += 2) {
            h[j] = fma2(a[j], h[j], u2);
            h[j + 1] = fma2(a[j + 1], h[j + 1], u2);
            acc0 = fma2(k[j], h[j], acc0);
            acc1 = fma2(k[j + 1], h[j + 1], acc1);
        }
        return (acc0.x + acc0.y) + (acc1.x + acc1.y);
    };
    fetch(t0, ub);
    t = t0;
    for (; t + TU <= t1; t += TU) {
        fetch(t + TU, un);
        float sv[TU];
#pragma unroll
        for (int e = 0; e < TU; ++e) sv[e] = step_sum(ub[e]);
        // the partial sums of all TU steps cross the lanes together, then lane q of a channel stores the steps
        // e = q (mod LPC)
#pragma unroll
        for (int o = LPC / 2; o > 0; o >>= 1)
#pragma unroll
            for (int e = 0; e < TU; ++e) sv[e] += __shfl_xor_sync(0xffffffffu, sv[e], o);
#pragma unroll
        for (int e = 0; e < TU; ++e)
            if (chan_ok && q == (e % LPC)) st_f32(yp + (int64_t)(t + e) * D, sv[e] + dsk * ub[e]);
#pragma unroll
        for (int e = 0; e < TU; ++e) ub[e] = un[e];
    }
#pragma unroll
    for (int e = 0; e < TU; ++e) {
        if (t + e < t1) {  // warp-uniform
            float sv = step_sum(ub[e]);
#pragma unroll
            for (int o = LPC / 2; o > 0; o >>= 1) sv += __shfl_xor_sync(0xffffffffu, sv, o);
            if (chan_ok && q == (e % LPC)) st_f32(yp + (int64_t)(t + e) * D, sv + dsk * ub[e]);
        }
    }
}

// ---------------------------------------------------------------- reference-literal S4
// V[t][n] = sum_m (dt * B[n][m]) * u[m][t]   (m ascending, as the reference's matvec)
//
// The three kernels below are small (forward_ssm at d_model 256, 2048 steps, 64 states: 67 M FMA, 4.5 MB), so what counts
// is latency: enough CTAs, a register tile per thread so that an operand read from shared memory serves several
// products, and the next slab's global loads in flight under the current one.  Every output keeps one accumulator over
// ascending m (n), so the sums are those of a thread-per-output loop bit for bit.  At that shape, in us, as one
// thread per output with operands from global memory -> now: in 21.9 -> 10.1, scan (one CTA for all states) 31.7 -> 7.5,
// out 125.4 -> 6.0; the whole call, host array to host array, 485 -> 315.
constexpr int kRT = 32;  // tile of steps
constexpr int kRN = 32;  // tile of states (s4_ref_in), slab of the summed index
constexpr int kRM = 64;  // tile of channels (s4_ref_out)

// CTA: 32 steps x 32 states, thread: 2 steps x 4 states.
__global__ void __launch_bounds__(128)
s4_ref_in_kernel(const float *u, const float *Bm, float dt, float *V, int M, int L, int N) {
    __shared__ __align__(16) float us[kRN][kRT], bs[kRN][kRN + 4];  // [m][t], [m][n]
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int t0 = blockIdx.x * kRT, n0 = blockIdx.y * kRN;
    float ur[8], br[8];
    auto fetch = [&](int m0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = tid + k * 128, lo = i % 32, hi = i / 32;
            ur[k] = (m0 + hi < M && t0 + lo < L) ? u[(int64_t)(m0 + hi) * L + t0 + lo] : 0.f;
            br[k] = (n0 + hi < N && m0 + lo < M) ? Bm[(int64_t)(n0 + hi) * M + m0 + lo] : 0.f;
        }
    };
    float acc[2][4] = {};
    fetch(0);
    for (int m0 = 0; m0 < M; m0 += kRN) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = tid + k * 128, lo = i % 32, hi = i / 32;
            us[hi][lo] = ur[k];
            bs[lo][hi] = br[k] * dt;
        }
        __syncthreads();
        if (m0 + kRN < M) fetch(m0 + kRN);
        const int mn = min(kRN, M - m0);
#pragma unroll 8
        for (int m = 0; m < mn; ++m) {
            const float2 uv = *reinterpret_cast<const float2 *>(&us[m][tx * 2]);
            const float4 bv = *reinterpret_cast<const float4 *>(&bs[m][ty * 4]);
            const float b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[0][j] = fmaf(b4[j], uv.x, acc[0][j]);
                acc[1][j] = fmaf(b4[j], uv.y, acc[1][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int t = t0 + tx * 2 + i, n = n0 + ty * 4 + j;
            if (t < L && n < N) V[(int64_t)t * N + n] = acc[i][j];
        }
}

// In-place diagonal scan over time on V [L][N]: X_t = a X_{t-1} + V_t, a = exp(dt A_re) cos(dt A_im).
// A CTA takes the kScanN states from blockIdx.x * kScanN on (their four-byte neighbours in a row make one 32-byte
// sector); thread = (state, segment of the sequence); same 3-pass scheme through shared memory.
constexpr int kScanN = 8;
__global__ void __launch_bounds__(1024)
s4_ref_scan_kernel(float *V, const float *A_real, const float *A_imag, float dt, int L, int N, int G) {
    __shared__ float ends_s[1024];  // [G][kScanN]
    const int nl = threadIdx.x % kScanN, g = threadIdx.x / kScanN, n = blockIdx.x * kScanN + nl;
    const bool active = n < N;
    const float a = active ? expf(A_real[n] * dt) * cosf(A_imag[n] * dt) : 0.f;
    const int seg_len = (L + G - 1) / G;
    const int t0 = min(L, g * seg_len), t1 = min(L, t0 + seg_len);
    float h = 0.f;
    if (active) {
#pragma unroll 16
        for (int t = t0; t < t1; ++t) h = a * h + V[(int64_t)t * N + n];
    }
    ends_s[threadIdx.x] = h;
    __syncthreads();
    if (!active) return;
    float aT = 1.f, base = a;  // a^seg_len by binary exponentiation (a may be negative)
    for (int e = seg_len; e > 0; e >>= 1) {
        if (e & 1) aT *= base;
        base *= base;
    }
    h = 0.f;
#pragma unroll 8
    for (int gp = 0; gp < g; ++gp) h = aT * h + ends_s[gp * kScanN + nl];
    int t = t0;
    for (; t + 8 <= t1; t += 8) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = V[(int64_t)(t + e) * N + n];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            h = a * h + v[e];
            V[(int64_t)(t + e) * N + n] = h;
        }
    }
    for (; t < t1; ++t) {
        h = a * h + V[(int64_t)t * N + n];
        V[(int64_t)t * N + n] = h;
    }
}

// y[t][m] = sum_n C[m][n] X[t][n] + D[m] u[m][t]   (n ascending)
// CTA: 32 steps x 64 channels, thread: 4 steps x 4 channels.
__global__ void __launch_bounds__(128)
s4_ref_out_kernel(const float *X, const float *Cm, const float *Dv, const float *u, float *y, int M, int L, int N) {
    __shared__ __align__(16) float cs[kRN][kRM + 4], xs[kRN][kRT + 4];  // [n][m], [n][t]
    __shared__ float us[kRM][kRT + 1];                                   // [m][t]
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int t0 = blockIdx.y * kRT, m0 = blockIdx.x * kRM;
    float cr[16], xr[8];
    auto fetch = [&](int n0) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int i = tid + k * 128, lo = i % 32, hi = i / 32;
            cr[k] = (m0 + hi < M && n0 + lo < N) ? Cm[(int64_t)(m0 + hi) * N + n0 + lo] : 0.f;
            if (k < 8) xr[k] = (t0 + hi < L && n0 + lo < N) ? X[(int64_t)(t0 + hi) * N + n0 + lo] : 0.f;
        }
    };
    fetch(0);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int i = tid + k * 128, lo = i % 32, hi = i / 32;
        us[hi][lo] = (m0 + hi < M && t0 + lo < L) ? u[(int64_t)(m0 + hi) * L + t0 + lo] : 0.f;
    }
    float acc[4][4] = {};
    for (int n0 = 0; n0 < N; n0 += kRN) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int i = tid + k * 128, lo = i % 32, hi = i / 32;
            cs[lo][hi] = cr[k];
            if (k < 8) xs[lo][hi] = xr[k];
        }
        __syncthreads();
        if (n0 + kRN < N) fetch(n0 + kRN);
        const int nn = min(kRN, N - n0);
#pragma unroll 8
        for (int n = 0; n < nn; ++n) {
            const float4 cv = *reinterpret_cast<const float4 *>(&cs[n][tx * 4]);
            const float4 xv = *reinterpret_cast<const float4 *>(&xs[n][ty * 4]);
            const float c4[4] = {cv.x, cv.y, cv.z, cv.w}, x4[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(c4[j], x4[i], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int m = m0 + tx * 4 + j;
        if (m >= M) continue;
        const float dv = Dv[m];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] = fmaf(dv, us[tx * 4 + j][ty * 4 + i], acc[i][j]);
    }
    const bool row16 = m0 + tx * 4 + 4 <= M && M % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = t0 + ty * 4 + i;
        if (t >= L) continue;
        float *yp = y + (int64_t)t * M + m0 + tx * 4;
        if (row16) {
            *reinterpret_cast<float4 *>(yp) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (m0 + tx * 4 + j < M) yp[j] = acc[i][j];
        }
    }
}

template <typename T>
static hx_status launch_diag(const void *u, const float *A, const float *Bp, const float *Cp, const float *delta,
                             const float *Dskip, void *y, int B, int L, int D, int N, cudaStream_t st) {
    // 16 states per lane.  The 8-state form (twice the warps, 64 registers) was measured slower on the benchmark
    // shape (124 us against 89 us for batch 8, L 2048, d_model 256, d_state 64): the extra shuffle and the
    // per-step overhead per state outweigh the occupancy.  It remains for d_state <= 8.
    const int nsl = N <= 8 ? 8 : 16;
    int lpc = 1;
    while (lpc * nsl < N) lpc *= 2;
    auto up = static_cast<const T *>(u);
    auto yp = static_cast<T *>(y);
    dim3 block(kSeg * 32);
#define HX_S4_CASE(LPC, NSL)                                                                              \
    if (lpc == LPC && nsl == NSL) {                                                                       \
        dim3 grid((D + 32 / LPC - 1) / (32 / LPC), B);                                                    \
        s4_diag_kernel<T, LPC, NSL><<<grid, block, 0, st>>>(up, A, Bp, Cp, delta, Dskip, yp, L, D, N);    \
        return check_launch("s4_diag_kernel");                                                            \
    }
    HX_S4_CASE(1, 8) HX_S4_CASE(2, 8) HX_S4_CASE(4, 8) HX_S4_CASE(8, 8) HX_S4_CASE(16, 8) HX_S4_CASE(32, 8)
    HX_S4_CASE(1, 16) HX_S4_CASE(2, 16) HX_S4_CASE(4, 16) HX_S4_CASE(8, 16) HX_S4_CASE(16, 16)
#undef HX_S4_CASE
    return fail(HX_ERR_INVALID_DIMENSION, "d_state %d exceeds 256", N);
}

// out[i][j] *= gate[j]: the row-broadcast gate of the reference's ssm-Mamba block
__global__ void row_gate_kernel(float *out, const float *gate, int rows, int cols) {
    const int64_t n = (int64_t)rows * cols;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = __fmul_rn(out[i], gate[i % cols]);
}

}  // namespace s4
}  // namespace hx

extern "C" {

hx_status hx_s4_diag_fwd(const void *u, const float *A, const float *Bp, const float *Cp, const float *delta,
                         const float *Dskip, void *y, int32_t batch, int32_t seq_len, int32_t d_model, int32_t d_state,
                         int32_t io_dtype, void *stream) {
    HX_REQUIRE(batch >= 0 && seq_len >= 0 && d_model >= 0, HX_ERR_INVALID_DIMENSION, "negative dimension");
    HX_REQUIRE(d_state >= 1 && d_state <= 256, HX_ERR_INVALID_DIMENSION, "d_state %d outside [1, 256]", d_state);
    HX_REQUIRE(io_dtype == HX_F32 || io_dtype == HX_BF16, HX_ERR_DTYPE_MISMATCH, "io_dtype %d unsupported", io_dtype);
    if (batch == 0 || seq_len == 0 || d_model == 0) return HX_OK;
    HX_REQUIRE(u && A && Bp && Cp && delta && y, HX_ERR_INVALID_INPUT, "u, A, Bp, Cp, delta and y must not be NULL");
    HX_REQUIRE(batch <= 65535, HX_ERR_INVALID_DIMENSION, "batch %d exceeds the grid limit", batch);
    cudaStream_t st = (cudaStream_t)stream;
    if (io_dtype == HX_BF16)
        return hx::s4::launch_diag<__nv_bfloat16>(u, A, Bp, Cp, delta, Dskip, y, batch, seq_len, d_model, d_state, st);
    return hx::s4::launch_diag<float>(u, A, Bp, Cp, delta, Dskip, y, batch, seq_len, d_model, d_state, st);
}

size_t hx_s4_ref_workspace_bytes(int32_t seq_len, int32_t d_state) {
    if (seq_len <= 0 || d_state <= 0) return 0;
    return (size_t)seq_len * d_state * sizeof(float);
}

hx_status hx_s4_ref_forward_ssm(const float *u, const float *A_real, const float *A_imag, const float *Bm,
                                const float *Cm, const float *Dv, float dt, float *y, int32_t d_model, int32_t seq_len,
                                int32_t d_state, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace hx::s4;
    HX_REQUIRE(d_model >= 0 && seq_len >= 0, HX_ERR_INVALID_DIMENSION, "negative dimension");
    HX_REQUIRE(d_state >= 1 && d_state <= 256, HX_ERR_INVALID_DIMENSION, "d_state %d outside [1, 256]", d_state);
    if (d_model == 0 || seq_len == 0) return HX_OK;
    HX_REQUIRE(u && A_real && A_imag && Bm && Cm && Dv && y, HX_ERR_INVALID_INPUT, "NULL operand");
    HX_REQUIRE(seq_len <= 65535, HX_ERR_INVALID_DIMENSION, "seq_len %d exceeds the grid limit", seq_len);
    const size_t need = hx_s4_ref_workspace_bytes(seq_len, d_state);
    HX_REQUIRE(workspace && workspace_bytes >= need, HX_ERR_INVALID_INPUT,
               "hx_s4_ref_forward_ssm needs a workspace of %zu bytes (got %zu)", need, workspace_bytes);
    cudaStream_t st = (cudaStream_t)stream;
    float *V = static_cast<float *>(workspace);
    s4_ref_in_kernel<<<dim3((seq_len + kRT - 1) / kRT, (d_state + kRN - 1) / kRN), 128, 0, st>>>(u, Bm, dt, V, d_model, seq_len,
                                                                                              d_state);
    hx_status s = hx::check_launch("s4_ref_in_kernel");
    if (s != HX_OK) return s;
    // segments of at least 8 steps, up to the 1024 threads of a CTA; the segment count is a multiple of 4 so that a
    // CTA is whole warps
    int G = (seq_len + 7) / 8;
    G = (G + 3) / 4 * 4;
    if (G > 1024 / kScanN) G = 1024 / kScanN;
    s4_ref_scan_kernel<<<(d_state + kScanN - 1) / kScanN, G * kScanN, 0, st>>>(V, A_real, A_imag, dt, seq_len, d_state, G);
    if ((s = hx::check_launch("s4_ref_scan_kernel")) != HX_OK) return s;
    s4_ref_out_kernel<<<dim3((d_model + kRM - 1) / kRM, (seq_len + kRT - 1) / kRT), 128, 0, st>>>(V, Cm, Dv, u, y, d_model,
                                                                                           seq_len, d_state);
    return hx::check_launch("s4_ref_out_kernel");
}

size_t hx_mamba_ssm_ref_workspace_bytes(int32_t d_model, int32_t d_state) {
    if (d_model <= 0 || d_state <= 0) return 0;
    return ((size_t)d_model * d_model * sizeof(float) + 255) / 256 * 256 + hx_s4_ref_workspace_bytes(d_model, d_state);
}

hx_status hx_mamba_ssm_ref_forward(const float *x, const float *delta_proj, const float *gate, const float *A_real,
                                   const float *A_imag, const float *Bm, const float *Cm, const float *Dv, float *out,
                                   int32_t d_model, int32_t d_state, void *workspace, size_t workspace_bytes, void *stream) {
    HX_REQUIRE(d_model >= 0, HX_ERR_INVALID_DIMENSION, "negative dimension");
    HX_REQUIRE(d_state >= 1 && d_state <= 256, HX_ERR_INVALID_DIMENSION, "d_state %d outside [1, 256]", d_state);
    if (d_model == 0) return HX_OK;
    HX_REQUIRE(x && delta_proj && gate && A_real && A_imag && Bm && Cm && Dv && out, HX_ERR_INVALID_INPUT, "NULL operand");
    const size_t need = hx_mamba_ssm_ref_workspace_bytes(d_model, d_state);
    HX_REQUIRE(workspace && workspace_bytes >= need, HX_ERR_INVALID_INPUT,
               "hx_mamba_ssm_ref_forward needs a workspace of %zu bytes (got %zu)", need, workspace_bytes);
    const int M = d_model;
    float *delta = static_cast<float *>(workspace);
    char *s4ws = static_cast<char *>(workspace) + ((size_t)M * M * sizeof(float) + 255) / 256 * 256;
    // delta = x . delta_proj in the reference's matmul arithmetic (crates/nn/src/ssm.rs:447)
    hx_status s = hx_matmul_ref(x, delta_proj, delta, M, M, M, HX_F32, stream);
    if (s != HX_OK) return s;
    // selective_ssm ignores B and C and runs the S4 recurrence on delta with dt = 0.1 (ssm.rs:474-483, :151)
    s = hx_s4_ref_forward_ssm(delta, A_real, A_imag, Bm, Cm, Dv, 0.1f, out, M, M, d_state, s4ws, workspace_bytes - (size_t)(s4ws - static_cast<char *>(workspace)),
                              stream);
    if (s != HX_OK) return s;
    const int64_t n = (int64_t)M * M;
    const int blocks = (int)((n + 255) / 256 > 65535 ? 65535 : (n + 255) / 256);
    hx::s4::row_gate_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(out, gate, M, M);
    return hx::check_launch("row_gate_kernel");
}

}  // extern "C"
