// scan_wide_kernel: the fused selective scan for any d_state <= 256, any strides and any alignment, with the arithmetic
// of scan_simple_kernel (libm-accurate forms, one exponential per point and state).  HX_SCAN_AUTO runs it wherever no
// d_state == 16 kernel takes the call.
//
// Bound by the exponentials (one per point and state) once enough lanes work on it.  One thread per channel kept 8 of
// 148 SMs busy with a serial walk that waits out a memory round trip per step: [256, 1024 channels, 64 states] f32 took
// 1125 us, and takes 41 here.  Here the states of a channel lie on LPC adjacent lanes, NSL each (a group of four states is one 16-byte
// shared load, adjacent lanes read adjacent groups), so the same problem is 512 warps, and a CTA walks the sequence in
// chunks of 16 steps:
//   point-wise    thread = (step, channel): conv, SiLU, softplus once per point; {dt, dt u} and the chunk's B, C rows go
//                 to shared memory, the skip and the gate stay in the thread's registers;
//   recurrence    a lane runs its states over the 16 steps and keeps 16 partial sums, which the lanes of a channel
//                 reduce and scatter in 15 shuffles (16 / LPC finished steps per lane) instead of log2(LPC) per step;
//   finish        back to thread = (step, channel): skip, gate, store.
// The next chunk's global loads are issued before the recurrence of the current one.  A chunk's outputs are stored after
// every thread of the CTA has loaded the next chunk (its history rows too), so y may be x, dt or z as in the simple kernel.
#include "hx_common.cuh"

namespace hx {
namespace scan {

struct WideParams {
    int B, L, D, N, K;
    int dt_softplus;
    int z_gate;  // z already holds silu(z)
    const void *x, *dt, *z, *Bm, *Cm;
    void *y;
    int64_t xb, xr, dtb, dtr, zb, zr, Bb, Br, Cb, Cr, yb, yr;
    const float *A, *Dskip, *conv_w, *conv_b, *dt_bias;
    float *h_last;
};

template <typename T, int LPC, int NSL>
__global__ void __launch_bounds__(128) scan_wide_kernel(WideParams p) {
    constexpr int TC = 16;                 // steps per chunk
    constexpr int CH = 128 / LPC;          // channels per CTA
    constexpr int NP = LPC * NSL;          // states held (rows are zero-filled past d_state)
    constexpr int V = NSL < 4 ? NSL : 4;   // states per shared load
    constexpr int PPT = CH * TC >= 128 ? CH * TC / 128 : 1;  // points per thread
    constexpr int BPT = TC * NP / 128;     // B (and C) values per thread
    static_assert(TC * NP % 128 == 0 && NSL % V == 0, "tile shape");
    __shared__ __align__(16) float sB[TC * NP], sC[TC * NP];
    __shared__ float2 sdx[TC][CH];
    __shared__ float sacc[TC][CH + 1];
    const int tid = threadIdx.x;
    const int b = blockIdx.y, d0 = blockIdx.x * CH;
    const T *x = static_cast<const T *>(p.x) + b * p.xb;
    const T *dt = static_cast<const T *>(p.dt) + b * p.dtb;
    const T *z = p.z ? static_cast<const T *>(p.z) + b * p.zb : nullptr;
    const T *Bm = static_cast<const T *>(p.Bm) + b * p.Bb;
    const T *Cm = static_cast<const T *>(p.Cm) + b * p.Cb;
    T *y = static_cast<T *>(p.y) + b * p.yb;

    // point-wise role: points tid, tid + 128, ... of the chunk's [TC][CH]; 128 is a multiple of CH, so a thread's points
    // all belong to one channel
    const int pc = tid % CH, pt = tid / CH, pd = d0 + pc;
    const bool p_on = tid < TC * CH && pd < p.D;
    float w[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.conv_w && p_on)
        for (int j = 0; j < p.K; ++j) w[4 - p.K + j] = p.conv_w[(int64_t)pd * p.K + j];
    const float cb = p.conv_b && p_on ? p.conv_b[pd] : 0.f;
    const float bias = p.dt_bias && p_on ? p.dt_bias[pd] : 0.f;
    const float dsk = p.Dskip && p_on ? p.Dskip[pd] : 0.f;

    // recurrence role: channel rc, states (jv * LPC + q) * V + e of its lanes
    const int q = tid % LPC, rc = tid / LPC;
    float h[NSL], a_row[NSL];
    bool held[NSL];  // a state past d_state stays 0 whatever dt and u are (an infinite dt u times a zero row is a NaN)
#pragma unroll
    for (int j = 0; j < NSL; ++j) {
        const int n = ((j / V) * LPC + q) * V + j % V;
        h[j] = 0.f;
        held[j] = n < p.N;
        a_row[j] = (n < p.N && d0 + rc < p.D) ? p.A[(int64_t)(d0 + rc) * p.N + n] : 0.f;
    }

    float xr[PPT][4], dr[PPT], zr[PPT], br[BPT], cr[BPT];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int k = 0; k < PPT; ++k) {
            const int t = t0 + pt + k * (128 / CH);
            const bool on = p_on && t < p.L;
#pragma unroll
            for (int j = 0; j < 4; ++j)  // x[t-3] .. x[t]; only x[t] without a conv
                xr[k][j] = (on && t - 3 + j >= 0 && (j == 3 || p.conv_w)) ? ld_f32(x + (int64_t)(t - 3 + j) * p.xr + pd) : 0.f;
            dr[k] = on ? ld_f32(dt + (int64_t)t * p.dtr + pd) : 0.f;
            zr[k] = on && z ? ld_f32(z + (int64_t)t * p.zr + pd) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < BPT; ++k) {
            const int i = tid + k * 128, n = i % NP, t = t0 + i / NP;
            const bool on = n < p.N && t < p.L;
            br[k] = on ? ld_f32(Bm + (int64_t)t * p.Br + n) : 0.f;
            cr[k] = on ? ld_f32(Cm + (int64_t)t * p.Cr + n) : 0.f;
        }
    };
    fetch(0);
    for (int t0 = 0; t0 < p.L; t0 += TC) {
        float du[PPT], gate[PPT];
#pragma unroll
        for (int k = 0; k < PPT; ++k) {
            float u;
            if (p.conv_w) {
                // taps in ascending order, like the written definition
                float c = cb;
                c += w[0] * xr[k][0];
                c += w[1] * xr[k][1];
                c += w[2] * xr[k][2];
                c += w[3] * xr[k][3];
                u = silu_acc(c);
            } else {
                u = xr[k][3];
            }
            const float v = dr[k] + bias;
            const float dtv = p.dt_softplus ? softplus_acc(v) : v;
            if (tid < TC * CH) sdx[pt + k * (128 / CH)][pc] = make_float2(dtv, dtv * u);
            du[k] = dsk * u;
            gate[k] = !z ? 1.f : p.z_gate ? zr[k] : silu_acc(zr[k]);
        }
#pragma unroll
        for (int k = 0; k < BPT; ++k) {
            sB[tid + k * 128] = br[k];
            sC[tid + k * 128] = cr[k];
        }
        __syncthreads();
        if (t0 + TC < p.L) fetch(t0 + TC);
        float acc[TC];
#pragma unroll
        for (int t = 0; t < TC; ++t) {
            acc[t] = 0.f;
            const float2 dx = sdx[t][rc];
            const bool live = t0 + t < p.L;  // the state stays what it is after the last step
#pragma unroll
            for (int jv = 0; jv < NSL / V; ++jv) {
                float bv[V], cv[V];
                const int o = t * NP + (jv * LPC + q) * V;
                if constexpr (V == 4) {
                    const float4 b4 = *reinterpret_cast<const float4 *>(sB + o), c4 = *reinterpret_cast<const float4 *>(sC + o);
                    bv[0] = b4.x; bv[1] = b4.y; bv[2] = b4.z; bv[3] = b4.w;
                    cv[0] = c4.x; cv[1] = c4.y; cv[2] = c4.z; cv[3] = c4.w;
                } else {
#pragma unroll
                    for (int e = 0; e < V; ++e) { bv[e] = sB[o + e]; cv[e] = sC[o + e]; }
                }
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const int j = jv * V + e;
                    float hn = expf(dx.x * a_row[j]) * h[j] + dx.y * bv[e];
                    hn = held[j] ? hn : 0.f;
                    h[j] = live ? hn : h[j];
                    acc[t] += cv[e] * hn;
                }
            }
        }
        // reduce and scatter over the lanes of a channel: after the exchange at distance o a lane keeps the half of its
        // steps whose bit matches its own, so lane q ends with the steps base .. base + 16 / LPC - 1
        if constexpr (LPC == 32) {
#pragma unroll
            for (int t = 0; t < TC; ++t) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], 16);
        }
        int base = 0;
        int m = TC;
#pragma unroll
        for (int o = (LPC < 16 ? LPC : 16) / 2; o > 0; o >>= 1) {
            m >>= 1;
            const bool up = (q & o) != 0;
#pragma unroll
            for (int t = 0; t < TC / 2; ++t)
                if (t < m) {
                    const float keep = up ? acc[t + m] : acc[t], give = up ? acc[t] : acc[t + m];
                    acc[t] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            base += up ? m : 0;
        }
        constexpr int LEFT = LPC < 16 ? TC / LPC : 1;
        if (LPC < 32 || q < 16) {
#pragma unroll
            for (int t = 0; t < LEFT; ++t) sacc[base + t][rc] = acc[t];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PPT; ++k) {
            const int ts = pt + k * (128 / CH), t = t0 + ts;
            if (p_on && t < p.L) {
                float out = sacc[ts][pc] + du[k];
                if (z) out *= gate[k];
                st_f32(y + (int64_t)t * p.yr + pd, out);
            }
        }
    }
    if (p.h_last && d0 + rc < p.D) {
#pragma unroll
        for (int j = 0; j < NSL; ++j) {
            const int n = ((j / V) * LPC + q) * V + j % V;
            if (n < p.N) p.h_last[((int64_t)b * p.D + d0 + rc) * p.N + n] = h[j];
        }
    }
}

template <typename T>
static void launch_wide_t(const WideParams &p, cudaStream_t st) {
#define HX_WIDE(LPC, NSL) \
    scan_wide_kernel<T, LPC, NSL><<<dim3((p.D + 128 / LPC - 1) / (128 / LPC), p.B), 128, 0, st>>>(p)
    if (p.N <= 8) HX_WIDE(4, 2);
    else if (p.N <= 16) HX_WIDE(4, 4);
    else if (p.N <= 32) HX_WIDE(8, 4);
    else if (p.N <= 64) HX_WIDE(16, 4);
    else if (p.N <= 128) HX_WIDE(16, 8);
    else HX_WIDE(32, 8);
#undef HX_WIDE
}

hx_status launch_wide(const hx_scan_args *a, cudaStream_t st) {
    HX_REQUIRE(a->W_dt == nullptr, HX_ERR_UNSUPPORTED_OPERATION, "the general scan kernel has no fused dt projection");
    WideParams p;
    p.B = a->batch; p.L = a->seq_len; p.D = a->d_inner; p.N = a->d_state; p.K = a->conv_w ? a->d_conv : 0;
    p.dt_softplus = a->dt_softplus;
    p.z_gate = a->z_is_gate != 0;
    p.x = a->x; p.dt = a->dt; p.z = a->z; p.Bm = a->Bm; p.Cm = a->Cm; p.y = a->y;
    p.xb = a->x_batch_stride; p.xr = a->x_row_stride; p.dtb = a->dt_batch_stride; p.dtr = a->dt_row_stride;
    p.zb = a->z_batch_stride; p.zr = a->z_row_stride; p.Bb = a->B_batch_stride; p.Br = a->B_row_stride;
    p.Cb = a->C_batch_stride; p.Cr = a->C_row_stride; p.yb = a->y_batch_stride; p.yr = a->y_row_stride;
    p.A = a->A; p.Dskip = a->Dskip; p.conv_w = a->conv_w; p.conv_b = a->conv_b; p.dt_bias = a->dt_bias;
    p.h_last = a->h_last;
    if (a->io_dtype == HX_BF16) launch_wide_t<__nv_bfloat16>(p, st);
    else launch_wide_t<float>(p, st);
    return check_launch("scan_wide_kernel");
}

}  // namespace scan
}  // namespace hx
