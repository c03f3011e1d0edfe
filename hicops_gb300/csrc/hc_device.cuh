// Device helpers shared by the query kernels (hc_query.cu) and the learned
// e-value tail (hc_mlp.cu). Not installed; not part of the C ABI.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "hicops_gb300.h"

namespace hc {

// Kernels that follow one another in a stream, the launch and the set-up of each under
// the end of the one before: each lets its successor's CTAs start once all of its own
// have (release_successor), and each waits for its predecessor's end, and sees
// what it wrote, before it reads any of it, writes anything or ends itself
// (after_predecessor; nothing to wait for in a launch without the attribute, or behind
// a copy). So when a kernel ends, all before it have. A kernel that waits releases
// only after its wait: its successor then starts, with an L1 emptied, when all
// kernels before the two have ended, and lines that could go stale under it are only
// those that its predecessor both reads and writes. Kernels that do work in
// place keep each CTA to 128-byte lines of its own, or have no successor launched so.
__device__ __forceinline__ void after_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;"); }

// Launches k, which calls after_predecessor, where its CTAs may start before the
// kernel in front of it has ended.
template <class... P, class... A>
cudaError_t launch_after(void (*k)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k, static_cast<P>(args)...);
}

// histogram bin of a hyperscore, (int)(h * 10 + 0.5) as the reference writes
// it (dslim_query.cpp:712, 778): a float product, then a double sum
__device__ __forceinline__ int hist_bin(float hf)
{
    const float t = __fmul_rn(hf, 10.0f);
    return (int)__dadd_rn((double)t, 0.5);
}

// cvttsd2si semantics of the reference's double -> int conversions
// (expeRT.cpp:703-704): out-of-range and NaN give INT_MIN
__device__ __forceinline__ int32_t x86_d2i(double v)
{
    if (!(v > -2147483649.0 && v < 2147483648.0)) return (int32_t)0x80000000u;
    return (int32_t)v;
}

// The tail-fit bins of a spectrum (expeRT.cpp:590-601), by one warp:
// end1 = last bin below the top hit's bin `hyp` holding a candidate, stt1 =
// the first such bin, end1 moved one up when they coincide. Bins past the
// histogram (the reference writes there only out of bounds) read as empty.
// Returns the number of points, end1 - stt1 + 1 (clamped to the histogram).
__device__ __forceinline__ int tail_bins(const uint32_t *__restrict__ yy, int hyp, int nbins, int lane, int &stt1,
                                         int &end1)
{
    end1 = hyp - 1;
    for (int q0 = min(hyp - 1, nbins - 1); q0 >= 0; q0 -= 32)
    {
        const int q = q0 - lane;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && yy[q] >= 1u);
        if (b)
        {
            end1 = q0 - (__ffs(b) - 1);
            break;
        }
    }
    stt1 = 0;
    for (int q0 = 0; q0 <= end1 && q0 < nbins; q0 += 32)
    {
        const int q = q0 + lane;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, q <= end1 && q < nbins && yy[q] >= 1u);
        if (b)
        {
            stt1 = q0 + __ffs(b) - 1;
            break;
        }
    }
    if (stt1 == end1) end1 += 1;
    int n = end1 - stt1 + 1;
    if (n < 0) n = 0;
    if (stt1 + n > nbins) n = nbins - stt1;
    return n;
}

constexpr int kCumRow = (HC_HIST_BINS + 3) / 4 * 4;  // words of a spectrum's cumulative counts, 16-byte aligned

// The same bins and, in cum[q], the cumulative counts of bins 0 .. q for every
// bin up to the last point (the bins before the first point are empty, so
// these are its cumulative counts too). One pass over the bins up to the top
// hit's, 128 at a time, four consecutive ones a lane: one scan over the lanes serves
// them all (a group of 32 each took 30 more shuffles and adds, and the targets of 50,000
// histograms, features and all, 76.5 us against 73.5). yy: a histogram's row (1002 words, so 8-byte
// aligned where the first row is); cum: kCumRow words.
__device__ __forceinline__ int tail_curve(const uint32_t *__restrict__ yy, int hyp, int nbins, int lane, uint32_t *cum,
                                          int &stt1, int &end1)
{
    const int lim = hyp < nbins ? hyp + 1 : nbins;  // the bin after a single one may be the top hit's own
    const bool pairs = ((uintptr_t)yy & 7) == 0;
    int first = -1, last = -1;
    uint32_t carry = 0;
    for (int q0 = 0; q0 < lim; q0 += 128)
    {
        const int q = q0 + 4 * lane;
        uint2 a = make_uint2(0u, 0u), b = a;
        if (pairs)  // (nbins is even: a pair that starts below lim lies in the row)
        {
            if (q < lim) a = __ldg(reinterpret_cast<const uint2 *>(yy + q));
            if (q + 2 < lim) b = __ldg(reinterpret_cast<const uint2 *>(yy + q + 2));
        }
        else
        {
            if (q < lim) a.x = __ldg(yy + q);
            if (q + 1 < lim) a.y = __ldg(yy + q + 1);
            if (q + 2 < lim) b.x = __ldg(yy + q + 2);
            if (q + 3 < lim) b.y = __ldg(yy + q + 3);
        }
        // what lies past the last bin read adds to nothing that is read, and the top
        // hit's own bin is no point
        uint32_t m = (a.x ? 1u : 0u) | (a.y ? 2u : 0u) | (b.x ? 4u : 0u) | (b.y ? 8u : 0u);
        if (hyp - q < 4) m &= hyp > q ? (1u << (hyp - q)) - 1u : 0u;
        const uint32_t any = __ballot_sync(0xFFFFFFFFu, m != 0u);
        if (any)
        {
            const int l0 = __ffs(any) - 1, l1 = 31 - __clz(any);
            if (first < 0) first = q0 + 4 * l0 + __ffs(__shfl_sync(0xFFFFFFFFu, m, l0)) - 1;
            last = q0 + 4 * l1 + 31 - __clz(__shfl_sync(0xFFFFFFFFu, m, l1));
        }
        const uint32_t t1 = a.x + a.y, t2 = t1 + b.x, t3 = t2 + b.y;
        uint32_t x = t3;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += t;
        }
        const uint32_t before = carry + x - t3;
        if (q < lim)
            *reinterpret_cast<uint4 *>(cum + q) = make_uint4(before + a.x, before + t1, before + t2, before + t3);
        carry += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    __syncwarp();
    stt1 = first < 0 ? 0 : first;
    end1 = last < 0 ? hyp - 1 : last;
    if (stt1 == end1) end1 += 1;
    int n = end1 - stt1 + 1;
    if (n < 0) n = 0;
    if (stt1 + n > nbins) n = nbins - stt1;
    return n;
}

}  // namespace hc
