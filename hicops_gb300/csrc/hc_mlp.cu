// Learned e-value tail: a 256 -> 128 -> 64 -> 4 MLP (FP32) that maps a
// spectrum's hyperscore histogram to the tail of its survival function, in
// place of the per-spectrum regression fit of expeRT (expeRT::ModelTailFit,
// expeRT.cpp:572-718), which stays the fallback and the yardstick.
//
// Outputs: the tail line (slope, intercept), the first bin of the regression
// window (expeRT picks it by searching the curve for its 22 % point,
// expeRT.cpp:646-661) and the RMS residual of the line over the window.
//
// Input features (fixed, not learned): bins 0..254 of the histogram and the
// sum of bins >= 255 in bin 255, turned into the log10 survival curve
// log10(1 - cumsum/cpsms) (clamped at -7); bins at and above the top hit's bin
// (excluded by expeRT, expeRT.cpp:590) repeat the last value below it.
//
// The learned e-value (k_learned_tail). A spectrum whose predicted residual
// exceeds the gate (0.1, log10 units) goes to expeRT at once. Otherwise its
// survival curve over expeRT's bins [stt1, end1] is formed in FP32 from the
// full histogram, and the network's first bin is confirmed on it: the curve
// is monotone, so the first bin is expeRT's exactly when the point after it
// is the first at or below the 22 % level, a test of two points; the kernel
// tests the predicted bin and its neighbours within the search radius (one
// lane each). The window ends at expeRT's upper cut (the 87 % rule,
// expeRT.cpp:662-676), the line is the FP32 least-squares fit over the
// window, and e = 10^(line at the top hit's bin) * cpsms
// (dslim_query.cpp:786-799). Where no bin is confirmed, or a level lies
// within FP32 rounding of a point, the spectrum is listed and the FP64
// expeRT fit (k_tailfit) runs on that list only.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "hc_device.cuh"
#include "hc_internal.h"

namespace hc {
namespace {

constexpr int kIn = 256, kH1 = 128, kH2 = 64, kOut = 4;
constexpr size_t kOffW1 = 0, kOffB1 = kOffW1 + kIn * kH1, kOffW2 = kOffB1 + kH1, kOffB2 = kOffW2 + kH1 * kH2,
                 kOffW3 = kOffB2 + kH2, kOffB3 = kOffW3 + kH2 * kOut, kParams = kOffB3 + kOut;
// target scaling: slope x 10, intercept / 4, first bin / 10, residual x 5
__host__ __device__ constexpr float tscale(int j)
{
    return j == 0 ? 10.0f : (j == 1 ? 0.25f : (j == 2 ? 0.1f : 5.0f));
}
// a 22 % or 87 % level closer than this to a curve point (log10 units) is a
// near tie the FP32 curve cannot decide the way expeRT's FP64 curve does
constexpr float kLevelMargin = 1e-4f;
constexpr int kMaxRadius = 15;  // first bins tested around the prediction: 2 * radius + 1 <= 32 lanes

}  // namespace
}  // namespace hc

struct hc_mlp
{
    hc_ctx *ctx = nullptr;
    float *d_params = nullptr;  // W1 b1 W2 b2 W3 b3
    float *d_grads = nullptr;
    float *d_m = nullptr, *d_v = nullptr;
    float *d_loss = nullptr;
    int step = 0;
    bool written = false;       // weights or moments set by copies that may not have ended (settle)
    uint64_t serial = 0;        // changes with any buffer that the learned pipeline's kernels name
    // gate of the learned tail: largest predicted RMS residual (log10 units),
    // and how far from the predicted first bin the confirmation looks
    float gate_resid = 0.1f;
    uint32_t radius = 4;
    // pipeline scratch (grown before any capture): features, outputs, fallback list
    float *d_X = nullptr, *d_net = nullptr;
    uint32_t *d_fb = nullptr;  // [0] = count, then the list
    size_t pipe_cap = 0;
};

namespace hc {
namespace {

// ---- features -------------------------------------------------------------
// One warp per spectrum. Bound by the bytes: 1 KB written a spectrum and the
// bins below the top hit read (what lies at or past it is repeated anyway, so
// the tail past bin 255 is read only for a top hit past it). 50,000 spectra:
// 24 us, against 60 us reading all 4 KB of every histogram.
// The kernels of the learned tail start under the end of the one before: features
// and targets of 50,000 histograms one after the other 73.5 -> 68.5 us.
__global__ void __launch_bounds__(256) k_features(const uint32_t *__restrict__ hist, const hc_result *__restrict__ res,
                                                  uint32_t n, float *__restrict__ X)
{
    after_predecessor();
    release_successor();
    const uint32_t s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (s >= n) return;
    const uint32_t *h = hist + (size_t)s * HC_HIST_BINS;
    const uint32_t cps = res[s].cpsms;
    const uint32_t cpi = cps > 0 ? cps : 1u;
    const float inv = 1.0f / (float)cpi;
    int hyp = hist_bin(res[s].hyperscore);
    if (hyp > kIn) hyp = kIn;
    // fold bins >= 255 into 255
    uint32_t tailsum = 0;
    if (hyp == kIn)
    {
        for (int b = 255 + lane; b < HC_HIST_BINS; b += 32) tailsum += h[b];
        tailsum = __reduce_add_sync(0xFFFFFFFFu, tailsum);
    }
    uint32_t carry = 0;
    float last = 0.0f;  // the value below the top hit: bins at/after it repeat it
    float *x = X + (size_t)s * kIn;
#pragma unroll
    for (int b0 = 0; b0 < kIn; b0 += 128)
    {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const int b = b0 + 32 * j + lane;
            v[j] = b >= hyp ? 0u : (b < 255 ? __ldg(h + b) : tailsum);
        }
        if (b0 < hyp)
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v[j], o);
                    if (lane >= o) v[j] += t;
                }
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const int b = b0 + 32 * j + lane;
            float y = last;
            if (b0 + 32 * j < hyp)  // warp-uniform
            {
                // 1 - cumsum / cpsms from the exact integer difference
                const float sv = (float)(cpi - min(cpi, carry + v[j])) * inv;
                y = log10f(fmaxf(sv, 1e-7f));
                carry += __shfl_sync(0xFFFFFFFFu, v[j], 31);
                if (b0 + 32 * j + 32 >= hyp) last = __shfl_sync(0xFFFFFFFFu, y, (hyp - 1) & 31);
                if (b >= hyp) y = last;
            }
            x[b] = y;
        }
    }
}

// ---- training: forward, backward and the weights' gradients of a minibatch ----
// One CTA takes R rows through all three layers and back without leaving
// shared memory, and writes the rows' share of every parameter's gradient;
// k_grad_reduce then adds the CTAs' shares in a fixed order (and, in training,
// applies Adam), so a step is two launches with no intermediate activations
// in global memory and its result does not vary from run to run. All sums are FP32.
// What bounds it: FMA issue and shared-memory reads while the CTAs' rows are
// worked off (about 90 k FMA a row), the shares' traffic (164 KB a CTA, L2)
// when rows are few. R is the smallest of 8, 16 and 32 that still gives at
// most one tile per SM, so small minibatches use most SMs and large ones reuse
// each weight read for 32 rows.
// A refinement is a chain of these two launches, 14 and 4 us each at 512 rows: each
// starts under the end of the one before (16 minibatches of 512: 492 -> 414 us a call).
constexpr int kGradThreads = 512;
constexpr int kW2Pitch = kH2 + 4;  // rows 16 bytes apart modulo the banks: a warp reads 32 rows' float4 without conflicts
// A CTA's share: gradients, then its loss, in 128-byte lines of its own. A CTA of several
// tiles adds to its share in place under a successor that has started (see after_predecessor).
constexpr size_t kPartStride = (kParams + 1 + 31) / 32 * 32;
static_assert(kPartStride * sizeof(float) % 128 == 0, "no line of two CTAs");

template <int R>
struct GradSmem
{
    float xs[R][kIn];
    float w2[kH1][kW2Pitch];
    float w3[kH2][kOut];
    float h1[R][kH1];
    float h2[R][kH2];
    float dout[R][kOut];
    float loss[kGradThreads / 32];
    union
    {
        float red1[4][R][kH1];  // layer 1, a quarter of the inputs each
        float red2[4][R][kH2];  // layer 2 the same
        struct
        {
            float dh2[R][kH2];
            float dh1[R][kH1];
        } d;
    } u;
};

// a += x * w, each product and sum one FP32 FMA, two to an instruction
__device__ __forceinline__ void fma4(float4 &a, float x, const float4 &w)
{
    uint64_t xx, lo, hi, wl, wh;
    asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x));
    asm("mov.b64 %0, {%1, %2};" : "=l"(lo) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(hi) : "f"(a.z), "f"(a.w));
    asm("mov.b64 %0, {%1, %2};" : "=l"(wl) : "f"(w.x), "f"(w.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(wh) : "f"(w.z), "f"(w.w));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(lo) : "l"(xx), "l"(wl));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(hi) : "l"(xx), "l"(wh));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(lo));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.z), "=f"(a.w) : "l"(hi));
}

// writes v, or adds it to what an earlier tile of this CTA left there
__device__ __forceinline__ void put4(float *p, float4 v, bool add)
{
    float4 *q = reinterpret_cast<float4 *>(p);
    if (add)
    {
        const float4 o = *q;
        v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
    }
    *q = v;
}

template <int R>
__global__ void __launch_bounds__(kGradThreads, 1) k_grad_tile(const float *__restrict__ P, const float *__restrict__ X,
                                                               const float *__restrict__ Y, int n, int ntiles,
                                                               float *__restrict__ part)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    GradSmem<R> &S = *reinterpret_cast<GradSmem<R> *>(gsm);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *mine = part + (size_t)blockIdx.x * kPartStride;
    after_predecessor();
    release_successor();
    for (int i = tid; i < kH1 * kH2 / 4; i += kGradThreads)
    {
        const int k = i / (kH2 / 4), j = i % (kH2 / 4);
        *reinterpret_cast<float4 *>(&S.w2[k][4 * j]) = __ldg(reinterpret_cast<const float4 *>(P + kOffW2) + i);
    }
    for (int i = tid; i < kH2 * kOut / 4; i += kGradThreads)
        reinterpret_cast<float4 *>(&S.w3[0][0])[i] = __ldg(reinterpret_cast<const float4 *>(P + kOffW3) + i);
    const bool aligned = ((uintptr_t)X & 15) == 0;  // a caller's buffer may start anywhere a float does
    float loss = 0.0f;
    bool add = false;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, add = true)
    {
        const int r0 = tile * R;
        // rows past the end: zero inputs and, below, zero output gradients
        for (int i = tid; i < R * kIn / 4; i += kGradThreads)
        {
            const int r = i / (kIn / 4), c = i % (kIn / 4);
            const float *x = X + (size_t)(r0 + r) * kIn + 4 * c;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r0 + r < n)
                v = aligned ? __ldg(reinterpret_cast<const float4 *>(x))
                            : make_float4(__ldg(x), __ldg(x + 1), __ldg(x + 2), __ldg(x + 3));
            reinterpret_cast<float4 *>(&S.xs[r][0])[c] = v;
        }
        __syncthreads();
        // layer 1: warps 4q .. 4q+3 take inputs [64q, 64q + 64), each R/4 rows; lane l units 4l .. 4l+3
        {
            constexpr int RT = R / 4;
            const int q = warp >> 2, rb = (warp & 3) * RT;
            float4 acc[RT];
#pragma unroll
            for (int r = 0; r < RT; r++) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 *w1 = reinterpret_cast<const float4 *>(P + kOffW1) + lane;
#pragma unroll 2
            for (int k = 64 * q; k < 64 * q + 64; k += 4)
            {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = __ldg(w1 + (k + i) * (kH1 / 4));
#pragma unroll
                for (int r = 0; r < RT; r++)
                {
                    const float4 x = *reinterpret_cast<const float4 *>(&S.xs[rb + r][k]);
                    fma4(acc[r], x.x, w[0]);
                    fma4(acc[r], x.y, w[1]);
                    fma4(acc[r], x.z, w[2]);
                    fma4(acc[r], x.w, w[3]);
                }
            }
#pragma unroll
            for (int r = 0; r < RT; r++) *reinterpret_cast<float4 *>(&S.u.red1[q][rb + r][4 * lane]) = acc[r];
        }
        __syncthreads();
        for (int i = tid; i < R * kH1; i += kGradThreads)
        {
            const int r = i / kH1, c = i % kH1;
            const float v = (S.u.red1[0][r][c] + S.u.red1[1][r][c]) + (S.u.red1[2][r][c] + S.u.red1[3][r][c]) +
                            __ldg(P + kOffB1 + c);
            S.h1[r][c] = fmaxf(v, 0.0f);
        }
        __syncthreads();
        // layer 2: the same quarters of its 128 inputs; 16 groups of 4 units x 8 groups of R/8 rows
        {
            constexpr int RT = R / 8;
            const int q = warp >> 2, t = tid & 127, cg = t & 15, rb = (t >> 4) * RT;
            float4 acc[RT];
#pragma unroll
            for (int r = 0; r < RT; r++) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int k = 32 * q; k < 32 * q + 32; k += 4)
            {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = *reinterpret_cast<const float4 *>(&S.w2[k + i][4 * cg]);
#pragma unroll
                for (int r = 0; r < RT; r++)
                {
                    const float4 x = *reinterpret_cast<const float4 *>(&S.h1[rb + r][k]);
                    fma4(acc[r], x.x, w[0]);
                    fma4(acc[r], x.y, w[1]);
                    fma4(acc[r], x.z, w[2]);
                    fma4(acc[r], x.w, w[3]);
                }
            }
#pragma unroll
            for (int r = 0; r < RT; r++) *reinterpret_cast<float4 *>(&S.u.red2[q][rb + r][4 * cg]) = acc[r];
        }
        __syncthreads();
        for (int i = tid; i < R * kH2; i += kGradThreads)
        {
            const int r = i / kH2, c = i % kH2;
            const float v = (S.u.red2[0][r][c] + S.u.red2[1][r][c]) + (S.u.red2[2][r][c] + S.u.red2[3][r][c]) +
                            __ldg(P + kOffB2 + c);
            S.h2[r][c] = fmaxf(v, 0.0f);
        }
        __syncthreads();
        // outputs (four lanes each, 16 inputs a lane), the mean squared error on
        // the scaled targets (NaN targets and rows past the end excluded) and its
        // gradient 2 (out - t) / (n * 4)
        if (tid < R * 16)
        {
            const int r = tid >> 4, c = (tid >> 2) & 3, q = tid & 3;
            float v = 0.0f;
#pragma unroll
            for (int k = 0; k < 16; k++) v = fmaf(S.h2[r][4 * k + q], S.w3[4 * k + q][c], v);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
            v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
            if (q == 0)
            {
                const float y = r0 + r < n ? Y[(size_t)(r0 + r) * kOut + c] : __int_as_float(0x7FC00000);
                const float d = isnan(y) ? 0.0f : v + __ldg(P + kOffB3 + c) - y * tscale(c);
                S.dout[r][c] = 2.0f * d / (float)(n * kOut);
                loss += d * d / (float)(n * kOut);
            }
        }
        __syncthreads();
        // back through layer 3
        for (int i = tid; i < R * kH2; i += kGradThreads)
        {
            const int r = i / kH2, j = i % kH2;
            const float4 g = *reinterpret_cast<const float4 *>(&S.dout[r][0]);
            const float4 w = *reinterpret_cast<const float4 *>(&S.w3[j][0]);
            const float v = fmaf(g.w, w.w, fmaf(g.z, w.z, fmaf(g.y, w.y, g.x * w.x)));
            S.u.d.dh2[r][j] = S.h2[r][j] > 0.0f ? v : 0.0f;
        }
        if (tid < kH2 * kOut)
        {
            const int j = tid / kOut, c = tid % kOut;
            float v = 0.0f;
#pragma unroll 8
            for (int r = 0; r < R; r++) v = fmaf(S.h2[r][j], S.dout[r][c], v);
            float *p = mine + kOffW3 + tid;
            *p = add ? *p + v : v;
        }
        else if (tid < kH2 * kOut + kOut)
        {
            float v = 0.0f;
            for (int r = 0; r < R; r++) v += S.dout[r][tid - kH2 * kOut];
            float *p = mine + kOffB3 + tid - kH2 * kOut;
            *p = add ? *p + v : v;
        }
        __syncthreads();
        // back through layer 2: a warp takes RB rows and 32 KB units, lane l units l, l + 32 ..
        {
            constexpr int RB = R == 8 ? 2 : 4, KB = R == 32 ? 2 : 1, NG = R / RB;
            const int rb = (warp % NG) * RB, kb = (warp / NG) * 32 * KB + lane;
            float acc[RB][KB];
#pragma unroll
            for (int r = 0; r < RB; r++)
#pragma unroll
                for (int i = 0; i < KB; i++) acc[r][i] = 0.0f;
#pragma unroll 4
            for (int j = 0; j < kH2; j += 4)
            {
                float4 w[KB];
#pragma unroll
                for (int i = 0; i < KB; i++) w[i] = *reinterpret_cast<const float4 *>(&S.w2[kb + 32 * i][j]);
#pragma unroll
                for (int r = 0; r < RB; r++)
                {
                    const float4 g = *reinterpret_cast<const float4 *>(&S.u.d.dh2[rb + r][j]);
#pragma unroll
                    for (int i = 0; i < KB; i++)
                        acc[r][i] = fmaf(g.w, w[i].w, fmaf(g.z, w[i].z, fmaf(g.y, w[i].y, fmaf(g.x, w[i].x, acc[r][i]))));
                }
            }
#pragma unroll
            for (int r = 0; r < RB; r++)
#pragma unroll
                for (int i = 0; i < KB; i++)
                    S.u.d.dh1[rb + r][kb + 32 * i] = S.h1[rb + r][kb + 32 * i] > 0.0f ? acc[r][i] : 0.0f;
        }
        // layer 2's weights: 4 x 4 outputs a thread
        const int kq = tid >> 4, cq = tid & 15;
        {
            float4 acc[4];
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int r = 0; r < R; r++)
            {
                const float4 h = *reinterpret_cast<const float4 *>(&S.h1[r][4 * kq]);
                const float4 g = *reinterpret_cast<const float4 *>(&S.u.d.dh2[r][4 * cq]);
                fma4(acc[0], h.x, g);
                fma4(acc[1], h.y, g);
                fma4(acc[2], h.z, g);
                fma4(acc[3], h.w, g);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) put4(mine + kOffW2 + (4 * kq + i) * kH2 + 4 * cq, acc[i], add);
        }
        __syncthreads();
        // layer 1's weights: 8 x 8 outputs a thread (inputs 4kq.., 128 + 4kq..; units 4cq.., 64 + 4cq..)
        {
            float4 acc[8][2];
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int r = 0; r < R; r++)
            {
                const float4 x0 = *reinterpret_cast<const float4 *>(&S.xs[r][4 * kq]);
                const float4 x1 = *reinterpret_cast<const float4 *>(&S.xs[r][kIn / 2 + 4 * kq]);
                const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    const float4 g = *reinterpret_cast<const float4 *>(&S.u.d.dh1[r][64 * h + 4 * cq]);
#pragma unroll
                    for (int i = 0; i < 8; i++) fma4(acc[i][h], xv[i], g);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    put4(mine + kOffW1 + ((i >> 2) * (kIn / 2) + 4 * kq + (i & 3)) * kH1 + 64 * h + 4 * cq, acc[i][h],
                         add);
        }
        // the biases' gradients: column sums
        if (tid < kH1 + kH2)
        {
            float v = 0.0f;
            if (tid < kH1)
                for (int r = 0; r < R; r++) v += S.u.d.dh1[r][tid];
            else
                for (int r = 0; r < R; r++) v += S.u.d.dh2[r][tid - kH1];
            float *p = mine + (tid < kH1 ? kOffB1 + tid : kOffB2 + tid - kH1);
            *p = add ? *p + v : v;
        }
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
    if (lane == 0) S.loss[warp] = loss;
    __syncthreads();
    if (tid == 0)
    {
        float v = 0.0f;
        for (int w = 0; w < kGradThreads / 32; w++) v += S.loss[w];
        mine[kParams] = v;
    }
}

struct AdamStep
{
    float *p, *m, *v;  // null p: gradients only
    float lr, c1, c2;  // bias corrections 1 - 0.9^t and 1 - 0.999^t
};

// The CTAs' shares added up, four parameters per thread column and eight
// threads per column (share c, c + 8, ..): the gradient, or Adam's update from
// it. Block 0 adds the minibatch's loss to *loss.
__global__ void __launch_bounds__(256) k_grad_reduce(const float *__restrict__ part, int nparts, float *__restrict__ g,
                                                     AdamStep ad, float *__restrict__ loss)
{
    __shared__ float4 s[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t i4 = (size_t)blockIdx.x * 32 + lane;  // float4 of the parameters
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    after_predecessor();
    release_successor();
    if (i4 < kParams / 4)
#pragma unroll 8
        for (int c = w; c < nparts; c += 8)
        {
            const float4 x = __ldg(reinterpret_cast<const float4 *>(part + (size_t)c * kPartStride) + i4);
            a = make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w);
        }
    s[w][lane] = a;
    __syncthreads();
    if (w == 1 && blockIdx.x == 0)
    {
        float l = 0.0f;
        for (int c = lane; c < nparts; c += 32) l += part[(size_t)c * kPartStride + kParams];
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
        if (lane == 0) *loss += l;
    }
    if (threadIdx.x >= 128 || (size_t)blockIdx.x * 128 + threadIdx.x >= kParams) return;
    const size_t i = (size_t)blockIdx.x * 128 + threadIdx.x;
    const float *c = &s[0][0].x + threadIdx.x;
    const float gi = ((c[0] + c[128]) + (c[256] + c[384])) + ((c[512] + c[640]) + (c[768] + c[896]));
    if (!ad.p)
    {
        g[i] = gi;
        return;
    }
    const float mi = 0.9f * ad.m[i] + 0.1f * gi;
    const float vi = 0.999f * ad.v[i] + 0.001f * gi * gi;
    ad.m[i] = mi;
    ad.v[i] = vi;
    ad.p[i] -= ad.lr * (mi / ad.c1) / (sqrtf(vi / ad.c2) + 1e-8f);
}

// ---- inference: the three layers fused ----
// Two kernels, both FP32 FMA throughout (41 k FMA a spectrum; the batch's FMA
// issue bounds them, not its 1 KB a spectrum of input; two FMAs to an
// instruction where a thread holds neighbouring outputs).
//
// k_infer_tile, for batches that fill the chip: a persistent CTA per SM stages
// all parameters (162 KB) in shared memory once and takes 64 spectra at a
// time, inputs arriving in chunks of 64 through cp.async. A thread of layer 1
// holds 8 x 8 outputs (one shared-memory read of 16 bytes for 16 FMAs), two
// groups of four warps take half of each layer's inputs; with two warps a
// scheduler to cover each other's reads, the loops over the inputs are unrolled
// whole (176 -> 167 us below). What is left over after whole waves of tiles goes in
// half tiles of 32 if one wave takes it (167 -> 161 us; 9,800 spectra 34.8 -> 27.9).
// 100,000 spectra: 161 us, against 344 us with two spectra per warp, where a weight
// read served 8 FMAs, and 202 us with one FMA to an instruction.
//
// k_infer_rows, for the rest: a CTA takes 8 spectra and its 16 warps 1/16 of
// each layer's inputs, so every weight is read once per CTA, straight from L2
// with no staging. 1,000 spectra: 8.2 us, against 14.3 us.
//
// The line between them: half a tile takes 12.3 us up to 32 spectra per SM, rows
// 8.2 us at 8 per SM, 12.3 us at 16, 16.4 at 20 and 20.5 us at 32.
constexpr int kTileThreads = 256, kRowsThreads = 512;
constexpr int kInferTile = 64, kInferChunk = 64, kInferRows = 8;
constexpr uint32_t kInferRowsPerSm = 16;

struct InferSmem
{
    float w1[kIn][kH1];
    float w2[kH1][kH2];
    float w3[kH2][kOut];
    float b[kH1 + kH2 + kOut];
    float xs[2][kInferTile][kInferChunk];
    float h1[kInferTile][kH1];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool in)
{
    // out of range: 16 zero bytes, nothing read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 16 : 0));
}

__device__ __forceinline__ float4 relu4(const float4 &a, const float4 &p, const float4 &b)
{
    return make_float4(fmaxf(a.x + p.x + b.x, 0.f), fmaxf(a.y + p.y + b.y, 0.f), fmaxf(a.z + p.z + b.z, 0.f),
                       fmaxf(a.w + p.w + b.w, 0.f));
}

__global__ void __launch_bounds__(kTileThreads, 1) k_infer_tile(const float *__restrict__ P, const float *__restrict__ X,
                                                                uint32_t n, uint32_t nfull, uint32_t ntiles,
                                                                float *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char ism[];
    InferSmem &S = *reinterpret_cast<InferSmem *>(ism);
    after_predecessor();
    release_successor();
    const int tid = threadIdx.x;
    // group q of 128 threads takes half of the inputs; a thread 8 rows (4 of a half tile)
    const int q = tid >> 7, cg = tid & 15;
    auto first_row = [&](uint32_t tile) {
        return tile < nfull ? tile * kInferTile : nfull * kInferTile + (tile - nfull) * (kInferTile / 2);
    };
    // chunk c of a tile's inputs, four 16-byte copies a thread (two of a half tile)
    auto load = [&](uint32_t tile, int c) {
        const uint32_t row0 = first_row(tile);
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            if (i == 2 && tile >= nfull) break;
            const int r = (tid >> 4) + 16 * i, j = 4 * (tid & 15);
            const uint32_t row = row0 + (uint32_t)r;
            cp_async16(&S.xs[c & 1][r][j], X + (size_t)min(row, n - 1) * kIn + c * kInferChunk + j, row < n);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;"); };
    auto copy = [&](float *dst, const float *src, int words) {
        for (int i = 4 * tid; i < words; i += 4 * kTileThreads) cp_async16(dst + i, src + i, true);
    };
    // the first tile's first chunk with the weights it meets, then the other weights under it
    load(blockIdx.x, 0);
    copy(&S.w1[0][0], P + kOffW1, kInferChunk * kH1);
    commit();
    copy(&S.w1[kInferChunk][0], P + kOffW1 + kInferChunk * kH1, (kIn - kInferChunk) * kH1);
    copy(&S.w2[0][0], P + kOffW2, kH1 * kH2);
    copy(&S.w3[0][0], P + kOffW3, kH2 * kOut);
    commit();
    for (int i = tid; i < kH1 + kH2 + kOut; i += kTileThreads)
        S.b[i] = __ldg(P + (i < kH1 ? kOffB1 + i : (i < kH1 + kH2 ? kOffB2 + i - kH1 : kOffB3 + i - kH1 - kH2)));
    bool first = true;
    // a tile of 8 * RT rows
    auto run = [&](auto rt, uint32_t tile) {
        constexpr int RT = decltype(rt)::value;
        const int rb = RT * ((tid >> 4) & 7);
        // layer 1: RT x 8 outputs a thread (units 4cg.., 64 + 4cg..), half of each chunk
        {
            float4 acc[RT][2];
#pragma unroll
            for (int r = 0; r < RT; r++) acc[r][0] = acc[r][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c = 0; c < kIn / kInferChunk; c++)
            {
                if (first) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                first = false;
                __syncthreads();  // chunk c is here; every thread is done with chunk c - 1
                if (c + 1 < kIn / kInferChunk)
                {
                    load(tile, c + 1);
                    commit();
                }
                const float *xc = &S.xs[c & 1][rb][0];
#pragma unroll
                for (int k = 32 * q; k < 32 * q + 32; k += 4)
                {
                    float4 x[RT];
#pragma unroll
                    for (int r = 0; r < RT; r++) x[r] = *reinterpret_cast<const float4 *>(xc + r * kInferChunk + k);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                    {
                        const float *w = &S.w1[c * kInferChunk + k + i][4 * cg];
                        const float4 wa = *reinterpret_cast<const float4 *>(w);
                        const float4 wb = *reinterpret_cast<const float4 *>(w + kH1 / 2);
#pragma unroll
                        for (int r = 0; r < RT; r++)
                        {
                            const float xv = i == 0 ? x[r].x : i == 1 ? x[r].y : i == 2 ? x[r].z : x[r].w;
                            fma4(acc[r][0], xv, wa);
                            fma4(acc[r][1], xv, wb);
                        }
                    }
                }
            }
            if (q == 1)
#pragma unroll
                for (int r = 0; r < RT; r++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        *reinterpret_cast<float4 *>(&S.h1[rb + r][64 * h + 4 * cg]) = acc[r][h];
            __syncthreads();
            // the first chunk's buffer is free: the next tile's first chunk arrives under layers 2 and 3
            if (tile + gridDim.x < ntiles)
            {
                load(tile + gridDim.x, 0);
                commit();
            }
            if (q == 0)
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    const float4 b = *reinterpret_cast<const float4 *>(&S.b[64 * h + 4 * cg]);
#pragma unroll
                    for (int r = 0; r < RT; r++)
                    {
                        float4 *p = reinterpret_cast<float4 *>(&S.h1[rb + r][64 * h + 4 * cg]);
                        *p = relu4(acc[r][h], *p, b);
                    }
                }
            __syncthreads();
        }
        // layer 2: RT x 4 outputs a thread, half of the inputs; its sums and then
        // its result take the second chunk's buffer
        float(*h2)[kH2] = S.xs[1];
        {
            float4 acc[RT];
#pragma unroll
            for (int r = 0; r < RT; r++) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 64 * q; k < 64 * q + 64; k += 4)
            {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; i++) w[i] = *reinterpret_cast<const float4 *>(&S.w2[k + i][4 * cg]);
#pragma unroll
                for (int r = 0; r < RT; r++)
                {
                    const float4 x = *reinterpret_cast<const float4 *>(&S.h1[rb + r][k]);
                    fma4(acc[r], x.x, w[0]);
                    fma4(acc[r], x.y, w[1]);
                    fma4(acc[r], x.z, w[2]);
                    fma4(acc[r], x.w, w[3]);
                }
            }
            if (q == 1)
#pragma unroll
                for (int r = 0; r < RT; r++) *reinterpret_cast<float4 *>(&h2[rb + r][4 * cg]) = acc[r];
            __syncthreads();
            if (q == 0)
            {
                const float4 b = *reinterpret_cast<const float4 *>(&S.b[kH1 + 4 * cg]);
#pragma unroll
                for (int r = 0; r < RT; r++)
                {
                    float4 *p = reinterpret_cast<float4 *>(&h2[rb + r][4 * cg]);
                    *p = relu4(acc[r], *p, b);
                }
            }
            __syncthreads();
        }
        // layer 3: four lanes a row
        if (RT == 8 || tid < 4 * 8 * RT)
        {
            const int r = tid >> 2, i = tid & 3;
            // short sums added pairwise: they round less than one long one
            float4 o4[4];
#pragma unroll
            for (int j = 0; j < kH2 / 16; j++)
            {
                o4[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 x = *reinterpret_cast<const float4 *>(&h2[r][4 * (i + 4 * j)]);
                const float4 *w = reinterpret_cast<const float4 *>(&S.w3[4 * (i + 4 * j)][0]);
                fma4(o4[j], x.x, w[0]);
                fma4(o4[j], x.y, w[1]);
                fma4(o4[j], x.z, w[2]);
                fma4(o4[j], x.w, w[3]);
            }
            float4 o = make_float4((o4[0].x + o4[1].x) + (o4[2].x + o4[3].x), (o4[0].y + o4[1].y) + (o4[2].y + o4[3].y),
                                   (o4[0].z + o4[1].z) + (o4[2].z + o4[3].z), (o4[0].w + o4[1].w) + (o4[2].w + o4[3].w));
#pragma unroll
            for (int d = 1; d < 4; d <<= 1)
            {
                o.x += __shfl_xor_sync(0xFFFFFFFFu, o.x, d);
                o.y += __shfl_xor_sync(0xFFFFFFFFu, o.y, d);
                o.z += __shfl_xor_sync(0xFFFFFFFFu, o.z, d);
                o.w += __shfl_xor_sync(0xFFFFFFFFu, o.w, d);
            }
            const uint32_t row = first_row(tile) + (uint32_t)r;
            if (row < n)
                out[(size_t)row * kOut + i] = (i == 0 ? o.x : i == 1 ? o.y : i == 2 ? o.z : o.w) + S.b[kH1 + kH2 + i];
        }
    };
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    {
        if (tile < nfull) run(std::integral_constant<int, 8>{}, tile);
        else run(std::integral_constant<int, 4>{}, tile);
    }
}

struct InferRowsSmem
{
    float xs[kInferRows][kIn];
    float red[16][kInferRows][kH1];  // a warp's sums (layer 2's in the first half)
    float h1[kInferRows][kH1];
    float h2[kInferRows][kH2];
};

__global__ void __launch_bounds__(kRowsThreads, 2) k_infer_rows(const float *__restrict__ P, const float *__restrict__ X,
                                                                 uint32_t n, float *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char ism[];
    InferRowsSmem &S = *reinterpret_cast<InferRowsSmem *>(ism);
    after_predecessor();
    release_successor();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t r0 = blockIdx.x * kInferRows;
    {
        const uint32_t row = r0 + (uint32_t)(tid >> 6);
        reinterpret_cast<float4 *>(&S.xs[0][0])[tid] =
            row < n ? __ldg(reinterpret_cast<const float4 *>(X + (size_t)row * kIn) + (tid & 63))
                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    {
        const float4 *w1 = reinterpret_cast<const float4 *>(P + kOffW1) + lane;
        float4 acc[kInferRows];
#pragma unroll
        for (int r = 0; r < kInferRows; r++) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int k = 16 * warp; k < 16 * warp + 16; k += 4)
        {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = __ldg(w1 + (k + i) * (kH1 / 4));
#pragma unroll
            for (int r = 0; r < kInferRows; r++)
            {
                const float4 x = *reinterpret_cast<const float4 *>(&S.xs[r][k]);
                fma4(acc[r], x.x, w[0]);
                fma4(acc[r], x.y, w[1]);
                fma4(acc[r], x.z, w[2]);
                fma4(acc[r], x.w, w[3]);
            }
        }
#pragma unroll
        for (int r = 0; r < kInferRows; r++) *reinterpret_cast<float4 *>(&S.red[warp][r][4 * lane]) = acc[r];
    }
    // this warp's eighth rows of layer 2's weights, loaded ahead of the sums
    float2 w2[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w2[i] = __ldg(reinterpret_cast<const float2 *>(P + kOffW2 + (8 * warp + i) * kH2) + lane);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kInferRows * kH1 / kRowsThreads; j++)
    {
        const int i = tid + j * kRowsThreads;
        const float *p = &S.red[0][0][0] + i;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 16; w++) v += p[w * kInferRows * kH1];
        (&S.h1[0][0])[i] = fmaxf(v + __ldg(P + kOffB1 + i % kH1), 0.0f);
    }
    __syncthreads();
    float *red2 = &S.red[0][0][0];  // [16][rows][kH2]
#pragma unroll
    for (int r = 0; r < kInferRows; r++)
    {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; i++)
        {
            const float x = S.h1[r][8 * warp + i];
            a.x = fmaf(x, w2[i].x, a.x);
            a.y = fmaf(x, w2[i].y, a.y);
        }
        reinterpret_cast<float2 *>(red2 + (warp * kInferRows + r) * kH2)[lane] = a;
    }
    __syncthreads();
    {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 16; w++) v += red2[w * kInferRows * kH2 + tid];
        (&S.h2[0][0])[tid] = fmaxf(v + __ldg(P + kOffB2 + tid % kH2), 0.0f);
    }
    __syncthreads();
    // layer 3: a warp's lanes per row, two inputs each
    if (warp < kInferRows)
    {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 2; j++)
            fma4(o, S.h2[warp][lane + 32 * j], __ldg(reinterpret_cast<const float4 *>(P + kOffW3) + lane + 32 * j));
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            o.x += __shfl_xor_sync(0xFFFFFFFFu, o.x, d);
            o.y += __shfl_xor_sync(0xFFFFFFFFu, o.y, d);
            o.z += __shfl_xor_sync(0xFFFFFFFFu, o.z, d);
            o.w += __shfl_xor_sync(0xFFFFFFFFu, o.w, d);
        }
        const uint32_t row = r0 + (uint32_t)warp;
        if (lane < kOut && row < n)
            out[(size_t)row * kOut + lane] =
                (lane == 0 ? o.x : lane == 1 ? o.y : lane == 2 ? o.z : o.w) + __ldg(P + kOffB3 + lane);
    }
}

// ---- the learned tail ---------------------------------------------------------
constexpr int kLtWarps = 16;
enum TailMode
{
    kApply = 0,     // gated: learned spectra written, the others listed for expeRT
    kProbe = 1,     // every spectrum's learned value, no gate, nothing written to the results
    kBaseline = 2,  // as kProbe with no network: the search starts at the curve's first bin
    kExact = 3,     // expeRT's own window by a full search: the training targets
};

struct TailGate
{
    float max_resid;  // largest predicted RMS residual of a learned spectrum
    int radius;       // first bins tested on either side of the prediction
};

// One warp per spectrum. net: the network's outputs (n x 4, scaled). lg_out
// (optional): the learned log10 e-value (NaN where there is none; in kApply
// also where the spectrum went to expeRT). aux_out (optional, kProbe and
// kBaseline): per spectrum {predicted residual, residual of the fit, offset
// of the confirmed first bin from the prediction} (NaN where none). y_out
// (kExact): the training targets {slope, intercept, first bin, residual}
// (NaN where there is no fit).
//
// The curve and its fit are FP32 and take a warp; the e-value is FP64 (two
// quotients and a power, or a logarithm), and an FP64 instruction costs the
// same for one lane as for 32, so it runs with a lane per spectrum, sixteen
// spectra at a time, and not at all for the training targets. Targets of 50,000
// spectra: 43 us, against 215 us with the FP64 part on one lane per spectrum.
struct LtJob
{
    float slope, icpt;
    uint32_t s, cps;
    int state;  // 0: nothing to write; 1: a line; 2: none found
    int stt1, end1, hyp;
};

struct LtSmem
{
    LtJob job[kLtWarps];
    alignas(16) uint32_t cum[kLtWarps][kCumRow];  // cumulative counts, then the curve in their place
};

// The e-value of a job, one lane each: e(x) from the line as the reference forms
// it from expeRT's (mu, beta) (x 1e6, truncated to int; dslim_query.cpp:786-799).
__device__ __forceinline__ void learned_value(const LtJob &j, hc_result *__restrict__ res, double expect_max, int mode,
                                              float *__restrict__ lg_out, uint32_t *__restrict__ fb)
{
    const bool have = j.state == 1;
    const int32_t mu = x86_d2i((double)j.slope * 1e6), beta = x86_d2i((double)j.icpt * 1e6);
    const double lgs = (double)mu / 1e6 * (double)j.hyp + (double)beta / 1e6;
    if (lg_out) lg_out[j.s] = have ? (float)(lgs + log10((double)j.cps)) : __int_as_float(0x7FC00000);
    if (mode != kApply) return;
    if (!have)
    {
        fb[1 + atomicAdd(fb, 1u)] = j.s;  // the expeRT fit runs on it
        return;
    }
    hc_result r = res[j.s];
    r.mu = mu;
    r.beta = beta;
    r.minhyp = j.stt1;
    r.nexthyp = j.end1;
    r.maxhyp = j.hyp;
    r.evalue = pow(10.0, lgs) * (double)j.cps;
    r.reported = r.evalue < expect_max ? 1u : 0u;
    r.flags |= HC_FLAG_LEARNED;
    res[j.s] = r;
}

__global__ void __launch_bounds__(kLtWarps * 32, 3) k_learned_tail(const uint32_t *__restrict__ hist,
                                                                const float *__restrict__ net,
                                                                hc_result *__restrict__ res, uint32_t n,
                                                                TailGate gate, uint32_t min_cpsm,
                                                                double expect_max, int mode,
                                                                float *__restrict__ lg_out,
                                                                float *__restrict__ aux_out,
                                                                float *__restrict__ y_out,
                                                                uint32_t *__restrict__ fb)
{
    extern __shared__ __align__(16) unsigned char lsm[];
    LtSmem &S = *reinterpret_cast<LtSmem *>(lsm);
    after_predecessor();  // (works on the results in place: no early successor)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float nanf_ = __int_as_float(0x7FC00000);
    // one spectrum by one warp; leaves its job
    auto fit = [&](uint32_t s, LtJob &job) {
        hc_result r = res[s];
        const float presid = (net && mode != kBaseline) ? net[(size_t)s * kOut + 3] / tscale(3) : nanf_;
        const bool early_fb = mode == kApply && !(presid <= gate.max_resid);
        if (r.cpsms < min_cpsm || r.cpsms == 0 || early_fb)
        {
            if (lane == 0)
            {
                if (mode == kApply && !early_fb)
                {
                    // no e-value (the early return of the tail fit, dslim_query.cpp:773)
                    r.mu = r.beta = r.minhyp = r.nexthyp = r.maxhyp = 0;
                    r.evalue = 0.0;
                    r.reported = 0;
                    res[s] = r;
                }
                if (early_fb) fb[1 + atomicAdd(fb, 1u)] = s;
                if (lg_out) lg_out[s] = nanf_;
                if (aux_out) aux_out[3 * s] = presid, aux_out[3 * s + 1] = aux_out[3 * s + 2] = nanf_;
                if (y_out) y_out[4 * s] = y_out[4 * s + 1] = y_out[4 * s + 2] = y_out[4 * s + 3] = nanf_;
            }
            return;
        }
        const uint32_t *yy = hist + (size_t)s * HC_HIST_BINS;
        const int hyp = hist_bin(r.hyperscore);
        const uint32_t cps = r.cpsms;
        int stt1, end1;
        const int nb = tail_curve(yy, hyp, HC_HIST_BINS, lane, S.cum[warp], stt1, end1);
        float *y = reinterpret_cast<float *>(S.cum[warp]) + stt1;
        bool have = false;
        int mark = 0, offset = 0;
        float slope = 0.0f, icpt = 0.0f, resid = nanf_;
        if (nb >= 4)
        {
            // survival curve log10((cpsms - cumsum) / cpsms) over [stt1, end1]:
            // the difference is an exact integer, positive below the top hit,
            // and the curve does not increase
            const float inv = 1.0f / (float)cps;
            for (int i = lane; i < nb; i += 32)
            {
                const uint32_t left = cps - min(cps, S.cum[warp][stt1 + i]);
                y[i] = log10f(fmaxf((float)left * inv, 1e-9f));
            }
            __syncwarp();
            const float y0 = y[0], hgt = y[nb - 1] - y0;
            // upper end (expeRT.cpp:662-676): the last point at or above the 87 % level
            const float t2 = y0 + 0.87f * hgt;
            int m2 = nb - 1;
            for (int q0 = nb - 1; q0 >= 0; q0 -= 32)
            {
                const int q = q0 - lane;
                const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && y[q] >= t2);
                if (b)
                {
                    m2 = q0 - (__ffs(b) - 1);
                    break;
                }
            }
            bool clear = fabsf(y[m2] - t2) > kLevelMargin && (m2 + 1 >= nb || fabsf(y[m2 + 1] - t2) > kLevelMargin);
            // first bin: the point before the first one at or below the 22 % level
            const float t1 = y0 + 0.22f * hgt;
            int lm = -1;  // the first point at or below t1
            if (mode == kExact)
            {
                for (int q0 = 0; q0 < nb; q0 += 32)
                {
                    const int q = q0 + lane;
                    const uint32_t b = __ballot_sync(0xFFFFFFFFu, q < nb && y[q] <= t1);
                    if (b)
                    {
                        lm = q0 + __ffs(b) - 1;
                        break;
                    }
                }
            }
            else
            {
                // lane j tests lm = center + j - radius: y[lm] <= t1 < y[lm - 1]
                const int center = mode == kBaseline ? 1 : (int)lrintf(net[(size_t)s * kOut + 2] / tscale(2)) - stt1 + 1;
                const int q = center + lane - gate.radius;
                const bool hit = lane <= 2 * gate.radius && q >= 0 && q < nb && y[q] <= t1 && (q == 0 || y[q - 1] > t1);
                const uint32_t b = __ballot_sync(0xFFFFFFFFu, hit);
                if (b)
                {
                    const int j = __ffs(b) - 1;
                    lm = center + j - gate.radius;
                    offset = j - gate.radius;
                }
            }
            if (lm >= 0)
                clear = clear && fabsf(y[lm] - t1) > kLevelMargin && (lm == 0 || fabsf(y[lm - 1] - t1) > kLevelMargin);
            mark = min(lm - 1, m2 - 1);
            // a window starting before the curve reads element -1 in the
            // reference (flagged): left to expeRT, as are near ties
            if (lm >= 0 && mark >= 0 && clear)
            {
                const int first = mark, m = m2 - first + 1;
                const float xbar = 0.5f * (float)(first + m2);  // window-relative abscissae
                float sy = 0.0f;
                for (int i = lane; i < m; i += 32) sy += y[first + i];
                for (int o = 16; o > 0; o >>= 1) sy += __shfl_xor_sync(0xFFFFFFFFu, sy, o);
                const float ybar = sy / (float)m;
                float top = 0.0f, bot = 0.0f;
                for (int i = lane; i < m; i += 32)
                {
                    const float dx = (float)(first + i) - xbar;
                    top = fmaf(dx, y[first + i] - ybar, top);
                    bot = fmaf(dx, dx, bot);
                }
                for (int o = 16; o > 0; o >>= 1)
                {
                    top += __shfl_xor_sync(0xFFFFFFFFu, top, o);
                    bot += __shfl_xor_sync(0xFFFFFFFFu, bot, o);
                }
                const float sl = top / bot;
                float se = 0.0f;
                for (int i = lane; i < m; i += 32)
                {
                    const float d = fmaf(sl, (float)(first + i) - xbar, ybar) - y[first + i];
                    se = fmaf(d, d, se);
                }
                for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xFFFFFFFFu, se, o);
                slope = sl;
                // intercept in histogram bins: the line is ybar + sl (bin - stt1 - xbar)
                icpt = ybar - sl * ((float)stt1 + xbar);
                resid = sqrtf(se / (float)m);
                have = isfinite(slope) && isfinite(icpt);
            }
            __syncwarp();
        }
        if (lane == 0)
        {
            if (aux_out)
            {
                aux_out[3 * s] = presid;
                aux_out[3 * s + 1] = have ? resid : nanf_;
                aux_out[3 * s + 2] = have ? (float)offset : nanf_;
            }
            if (y_out)
            {
                y_out[4 * s] = have ? slope : nanf_;
                y_out[4 * s + 1] = have ? icpt : nanf_;
                y_out[4 * s + 2] = have ? (float)(stt1 + mark) : nanf_;
                y_out[4 * s + 3] = have ? resid : nanf_;
            }
            job = LtJob{slope, icpt, s, cps, have ? 1 : 2, stt1, end1, hyp};
        }
        __syncwarp();
    };
    for (uint32_t w0 = blockIdx.x * kLtWarps; w0 < n; w0 += gridDim.x * kLtWarps)
    {
        LtJob &job = S.job[warp];
        if (lane == 0) job.state = 0;
        if (w0 + warp < n) fit(w0 + warp, job);
        if (mode == kExact) continue;  // targets only: no e-value
        __syncthreads();
        if (warp == 0 && lane < kLtWarps && S.job[lane].state)
            learned_value(S.job[lane], res, expect_max, mode, lg_out, fb);
        __syncthreads();
    }
}

}  // namespace

// Before work on st that reads the network: the copies that set it are blocking ones on the
// legacy stream, which may end after their call and which st need not wait for. They are
// waited for by the first work after them. (A capture only records, and forbids the wait.)
static int settle(hc_mlp *m, cudaStream_t st)
{
    if (!m->written) return HC_SUCCESS;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    HC_CUDA(m->ctx, cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return HC_SUCCESS;
    const BesideCapture beside;
    HC_CUDA(m->ctx, cudaStreamSynchronize(cudaStreamLegacy));
    m->written = false;
    return HC_SUCCESS;
}

// the fused inference kernels (no activations kept)
static int mlp_infer(hc_mlp *m, const float *X, uint32_t n, float *out, cudaStream_t st)
{
    if (n == 0) return HC_SUCCESS;
    if (const int rc = settle(m, st)) return rc;
    if (n <= kInferRowsPerSm * (uint32_t)m->ctx->sm_count)
    {
        HC_CUDA(m->ctx, cudaFuncSetAttribute(k_infer_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(InferRowsSmem)));
        HC_CUDA(m->ctx, launch_after(k_infer_rows, (n + kInferRows - 1) / kInferRows, kRowsThreads, sizeof(InferRowsSmem),
                                     st, m->d_params, X, n, out));
    }
    else
    {
        HC_CUDA(m->ctx, cudaFuncSetAttribute(k_infer_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(InferSmem)));
        // whole waves of full tiles, and what is left over in half tiles where one wave takes it
        const uint32_t sms = (uint32_t)m->ctx->sm_count;
        uint32_t nfull = n / (kInferTile * sms) * sms, rest = n - nfull * kInferTile, ntiles;
        if (rest <= kInferTile / 2 * sms) ntiles = nfull + (rest + kInferTile / 2 - 1) / (kInferTile / 2);
        else ntiles = nfull = (n - 1) / kInferTile + 1;
        HC_CUDA(m->ctx, launch_after(k_infer_tile, std::min(ntiles, sms), kTileThreads, sizeof(InferSmem), st, m->d_params,
                                     X, n, nfull, ntiles, out));
    }
    return HC_SUCCESS;
}

template <int R>
static cudaError_t grad_tile(const float *P, const float *X, const float *Y, uint32_t n, uint32_t ntiles, uint32_t grid,
                             float *part, cudaStream_t st)
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_grad_tile<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem<R>));
    if (e != cudaSuccess) return e;
    return launch_after(k_grad_tile<R>, grid, kGradThreads, sizeof(GradSmem<R>), st, P, X, Y, (int)n, (int)ntiles, part);
}

// forward + backward of one minibatch; the gradients land in d_grads, or Adam
// is applied to the parameters. d_loss grows by the minibatch's loss.
static int mlp_step(hc_mlp *m, const float *X, const float *Y, uint32_t n, const AdamStep &ad, cudaStream_t st)
{
    if (const int rc = settle(m, st)) return rc;
    const uint32_t sms = (uint32_t)m->ctx->sm_count;
    const uint32_t R = n <= 8 * sms ? 8u : (n <= 16 * sms ? 16u : 32u);
    const uint32_t ntiles = (n + R - 1) / R, grid = std::min(ntiles, sms);
    // the shares: scratch of the context (training runs on its stream only), at
    // most one per SM, 25 MB
    hc_ctx *ctx = m->ctx;
    if (ctx->grad_part_cap < grid)
    {
        cudaFree(ctx->d_grad_part);
        ctx->d_grad_part = nullptr;
        ctx->grad_part_cap = 0;
        HC_CUDA(ctx, cudaMalloc((void **)&ctx->d_grad_part, sizeof(float) * kPartStride * grid));
        ctx->grad_part_cap = grid;
    }
    const float *P = m->d_params;
    float *part = ctx->d_grad_part;
    HC_CUDA(m->ctx, R == 8    ? grad_tile<8>(P, X, Y, n, ntiles, grid, part, st)
                    : R == 16 ? grad_tile<16>(P, X, Y, n, ntiles, grid, part, st)
                              : grad_tile<32>(P, X, Y, n, ntiles, grid, part, st));
    HC_CUDA(m->ctx, launch_after(k_grad_reduce, (unsigned)((kParams + 127) / 128), 256, 0, st, part, (int)grid, m->d_grads,
                                 ad, m->d_loss));
    return HC_SUCCESS;
}

// of a network's device buffers: a new network may lie where one lay before
static uint64_t next_serial()
{
    static std::atomic<uint64_t> n{0};
    return ++n;
}

static int grow_pipe(hc_mlp *m, uint32_t n)
{
    if (m->pipe_cap >= n) return HC_SUCCESS;
    m->serial = next_serial();
    cudaFree(m->d_X);
    cudaFree(m->d_net);
    cudaFree(m->d_fb);
    m->d_X = m->d_net = nullptr;
    m->d_fb = nullptr;
    m->pipe_cap = 0;
    HC_CUDA(m->ctx, cudaMalloc((void **)&m->d_X, sizeof(float) * kIn * (size_t)n));
    HC_CUDA(m->ctx, cudaMalloc((void **)&m->d_net, sizeof(float) * kOut * (size_t)n));
    HC_CUDA(m->ctx, cudaMalloc((void **)&m->d_fb, sizeof(uint32_t) * ((size_t)n + 1)));
    m->pipe_cap = n;
    return HC_SUCCESS;
}

static int tail_kernel(hc_ctx *ctx, const TailGate &g, const uint32_t *d_hist, const float *net, hc_result *d_res,
                       uint32_t n, int mode, float *lg, float *aux, float *y, uint32_t *fb, cudaStream_t st)
{
    if (n == 0) return HC_SUCCESS;
    HC_CUDA(ctx, cudaFuncSetAttribute(k_learned_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LtSmem)));
    const uint32_t blocks = std::min<uint32_t>((n + kLtWarps - 1) / kLtWarps, (uint32_t)ctx->sm_count * 3);
    HC_CUDA(ctx, launch_after(k_learned_tail, blocks, kLtWarps * 32, sizeof(LtSmem), st, d_hist, net, d_res, n, g,
                              ctx->p.min_cpsm, ctx->p.expect_max, mode, lg, aux, y, fb));
    return HC_SUCCESS;
}

static TailGate gate_of(const hc_mlp *m) { return TailGate{m->gate_resid, (int)m->radius}; }

// what a graph with this network in it was captured with
void learned_key(const hc_mlp *m, GraphKey *key)
{
    key->gate_resid = m->gate_resid;
    key->gate_radius = m->radius;
    key->net_serial = m->serial;
    key->net_epoch = m->ctx->epoch;
}

// Allocates what the learned pipeline of n spectra needs (before any capture).
int learned_prepare(hc_mlp *m, uint32_t n)
{
    int rc = settle(m, m->ctx->stream);
    if (rc) return rc;
    if ((rc = grow_pipe(m, n))) return rc;
    QueryScratch &q = m->ctx->qs;
    if (q.fit_cap < n)
    {
        m->ctx->epoch++;
        cudaFree(q.d_fitstart);
        q.d_fitstart = nullptr;
        q.fit_cap = 0;
        HC_CUDA(m->ctx, cudaMalloc((void **)&q.d_fitstart, sizeof(int32_t) * (size_t)n));
        q.fit_cap = n;
    }
    return HC_SUCCESS;
}

// After a search without tail fit: features, network, learned e-values where
// the gates pass, and expeRT's fit on the listed rest. Enqueue only (no
// allocation after learned_prepare, no host wait). lg (optional) receives the
// learned log10 e-values.
int learned_pipeline(hc_mlp *m, const uint32_t *d_hist, hc_result *d_res, uint32_t n, float *lg, cudaStream_t st,
                     int *launches)
{
    if (n == 0) return HC_SUCCESS;
    if (m->pipe_cap < n || m->ctx->qs.fit_cap < n)
        return set_error(m->ctx, HC_ERR_INVLD_SIZE, "learned pipeline scratch not prepared");
    HC_CUDA(m->ctx, cudaMemsetAsync(m->d_fb, 0, 4, st));
    HC_CUDA(m->ctx, launch_after(k_features, (n + 7) / 8, 256, 0, st, d_hist, d_res, n, m->d_X));
    int rc = mlp_infer(m, m->d_X, n, m->d_net, st);
    if (rc) return rc;
    if ((rc = tail_kernel(m->ctx, gate_of(m), d_hist, m->d_net, d_res, n, kApply, lg, nullptr, nullptr, m->d_fb,
                          st)))
        return rc;
    if ((rc = tailfit_list(m->ctx, d_res, d_hist, m->d_fb + 1, m->d_fb, n, st))) return rc;
    if (m->ctx->profiling) HC_CUDA(m->ctx, record_stage(m->ctx, 5, st));
    if (launches) *launches += 4;
    return HC_SUCCESS;
}

}  // namespace hc

using namespace hc;

extern "C" {

int hc_mlp_create(hc_ctx *ctx, uint64_t seed, hc_mlp **out)
{
    if (!ctx || !out) return HC_ERR_INVLD_PTR;
    cudaSetDevice(ctx->device);
    hc_mlp *m = new hc_mlp();
    m->ctx = ctx;
    m->serial = next_serial();
    std::vector<float> h(kParams, 0.0f);
    // He-uniform initialisation from a splitmix64 stream
    uint64_t x = seed ? seed : 0x9E3779B97F4A7C15ull;
    auto next = [&]() {
        x += 0x9E3779B97F4A7C15ull;
        uint64_t z = x;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return (double)((z ^ (z >> 31)) >> 11) / 9007199254740992.0;
    };
    auto fill = [&](size_t off, int fan_in, size_t cnt) {
        const double lim = std::sqrt(6.0 / fan_in);
        for (size_t i = 0; i < cnt; i++) h[off + i] = (float)((2.0 * next() - 1.0) * lim);
    };
    fill(kOffW1, kIn, (size_t)kIn * kH1);
    fill(kOffW2, kH1, (size_t)kH1 * kH2);
    fill(kOffW3, kH2, (size_t)kH2 * kOut);
    if (cudaMalloc((void **)&m->d_params, 4 * kParams) != cudaSuccess ||
        cudaMalloc((void **)&m->d_grads, 4 * kParams) != cudaSuccess ||
        cudaMalloc((void **)&m->d_m, 4 * kParams) != cudaSuccess ||
        cudaMalloc((void **)&m->d_v, 4 * kParams) != cudaSuccess ||
        cudaMalloc((void **)&m->d_loss, 16) != cudaSuccess)
    {
        hc_mlp_destroy(m);
        return HC_ERR_BAD_MEM_ALLOC;
    }
    m->written = true;
    if (cudaMemcpy(m->d_params, h.data(), 4 * kParams, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(m->d_m, 0, 4 * kParams) != cudaSuccess || cudaMemset(m->d_v, 0, 4 * kParams) != cudaSuccess)
    {
        hc_mlp_destroy(m);
        return HC_ERR_CUDA;
    }
    *out = m;
    return HC_SUCCESS;
}

int hc_mlp_destroy(hc_mlp *m)
{
    if (!m) return HC_ERR_INVLD_PTR;
    cudaFree(m->d_params);
    cudaFree(m->d_grads);
    cudaFree(m->d_m);
    cudaFree(m->d_v);
    cudaFree(m->d_loss);
    cudaFree(m->d_X);
    cudaFree(m->d_net);
    cudaFree(m->d_fb);
    delete m;
    return HC_SUCCESS;
}

int hc_mlp_num_params(void) { return (int)kParams; }

int hc_mlp_get_params(hc_mlp *m, float *host)
{
    if (!m || !host) return HC_ERR_INVLD_PTR;
    HC_CUDA(m->ctx, cudaMemcpy(host, m->d_params, 4 * kParams, cudaMemcpyDeviceToHost));
    return HC_SUCCESS;
}

int hc_mlp_set_params(hc_mlp *m, const float *host)
{
    if (!m || !host) return HC_ERR_INVLD_PTR;
    m->written = true;
    HC_CUDA(m->ctx, cudaMemcpy(m->d_params, host, 4 * kParams, cudaMemcpyHostToDevice));
    return HC_SUCCESS;
}

int hc_mlp_set_gate(hc_mlp *m, float max_resid, uint32_t radius)
{
    if (!m) return HC_ERR_INVLD_PTR;
    if (radius > (uint32_t)kMaxRadius || !(max_resid >= 0.0f)) return set_error(m->ctx, HC_ERR_INVLD_PARAM, "bad gate");
    m->gate_resid = max_resid;
    m->radius = radius;
    return HC_SUCCESS;
}

int hc_mlp_get_gate(const hc_mlp *m, float *max_resid, uint32_t *radius)
{
    if (!m) return HC_ERR_INVLD_PTR;
    if (max_resid) *max_resid = m->gate_resid;
    if (radius) *radius = m->radius;
    return HC_SUCCESS;
}

int hc_mlp_features(hc_ctx *ctx, const uint32_t *d_hist, const hc_result *d_res, uint32_t n, float *d_X, void *stream)
{
    if (!ctx || (n && (!d_hist || !d_res || !d_X))) return HC_ERR_INVLD_PTR;
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    if (n) HC_CUDA(ctx, launch_after(k_features, (n + 7) / 8, 256, 0, st, d_hist, d_res, n, d_X));
    return HC_SUCCESS;
}

int hc_mlp_targets(hc_ctx *ctx, const uint32_t *d_hist, const hc_result *d_res, uint32_t n, float *d_Y, void *stream)
{
    if (!ctx || (n && (!d_hist || !d_res || !d_Y))) return HC_ERR_INVLD_PTR;
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    return tail_kernel(ctx, TailGate{0.0f, 0}, d_hist, nullptr, const_cast<hc_result *>(d_res), n, kExact, nullptr,
                       nullptr, d_Y, nullptr, st);
}

int hc_mlp_forward(hc_mlp *m, const float *d_X, uint32_t n, float *d_out, void *stream)
{
    if (!m || (n && (!d_X || !d_out))) return HC_ERR_INVLD_PTR;
    cudaStream_t st = stream ? (cudaStream_t)stream : m->ctx->stream;
    return mlp_infer(m, d_X, n, d_out, st);
}

int hc_mlp_gradients(hc_mlp *m, const float *d_X, const float *d_Y, uint32_t n, float *host_grads, float *loss)
{
    if (!m || !d_X || !d_Y) return HC_ERR_INVLD_PTR;
    cudaStream_t st = m->ctx->stream;
    HC_CUDA(m->ctx, cudaMemsetAsync(m->d_loss, 0, 4, st));
    int rc = mlp_step(m, d_X, d_Y, n, AdamStep{}, st);
    if (rc) return rc;
    if (host_grads) HC_CUDA(m->ctx, cudaMemcpyAsync(host_grads, m->d_grads, 4 * kParams, cudaMemcpyDeviceToHost, st));
    if (loss) HC_CUDA(m->ctx, cudaMemcpyAsync(loss, m->d_loss, 4, cudaMemcpyDeviceToHost, st));
    HC_CUDA(m->ctx, cudaStreamSynchronize(st));
    return HC_SUCCESS;
}

int hc_mlp_train(hc_mlp *m, const float *d_X, const float *d_Y, uint32_t n, uint32_t batch, uint32_t epochs,
                 float lr, float *final_loss)
{
    if (!m || !d_X || !d_Y || batch == 0) return HC_ERR_INVLD_PTR;
    cudaStream_t st = m->ctx->stream;
    float loss = 0.0f;
    for (uint32_t ep = 0; ep < epochs; ep++)
    {
        HC_CUDA(m->ctx, cudaMemsetAsync(m->d_loss, 0, 4, st));
        uint32_t nb = 0;
        for (uint32_t s0 = 0; s0 < n; s0 += batch)
        {
            const uint32_t b = std::min(batch, n - s0);
            const int t = m->step + 1;  // (a step that is refused is none)
            // in double: 1 - 0.999f alone is 5e-5 off 0.001
            const float c1 = (float)(1.0 - std::pow(0.9, t)), c2 = (float)(1.0 - std::pow(0.999, t));
            int rc = mlp_step(m, d_X + (size_t)s0 * kIn, d_Y + (size_t)s0 * kOut, b,
                              AdamStep{m->d_params, m->d_m, m->d_v, lr, c1, c2}, st);
            if (rc) return rc;
            m->step = t;
            nb++;
        }
        HC_CUDA(m->ctx, cudaMemcpyAsync(&loss, m->d_loss, 4, cudaMemcpyDeviceToHost, st));
        HC_CUDA(m->ctx, cudaStreamSynchronize(st));
        loss /= (float)(nb ? nb : 1);
    }
    if (final_loss) *final_loss = loss;
    return HC_SUCCESS;
}

int hc_mlp_tail_probe(hc_mlp *m, const float *d_X, const uint32_t *d_hist, const hc_result *d_res, uint32_t n,
                      int baseline, float *d_learned_log10e, float *d_aux, void *stream)
{
    if (!m || (n && (!d_hist || !d_res || !d_learned_log10e || !d_aux || (!baseline && !d_X)))) return HC_ERR_INVLD_PTR;
    cudaStream_t st = stream ? (cudaStream_t)stream : m->ctx->stream;
    if (n == 0) return HC_SUCCESS;
    int rc = grow_pipe(m, n);
    if (rc) return rc;
    const float *net = nullptr;
    if (!baseline)
    {
        if ((rc = mlp_infer(m, d_X, n, m->d_net, st))) return rc;
        net = m->d_net;
    }
    return tail_kernel(m->ctx, gate_of(m), d_hist, net, const_cast<hc_result *>(d_res), n,
                       baseline ? kBaseline : kProbe, d_learned_log10e, d_aux, nullptr, nullptr, st);
}

}  // extern "C"
