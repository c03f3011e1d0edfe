// MS2 ingestion. An MS2 text file is read the way the reference's
// MSQuery::initialize / readspectrum do (source/core/msquery.cpp:88-178,
// 300-505) and its raw peaks kept: files of some size are parsed on the device
// (k_ms2_lines), small ones, and those with a peak line that is not two plain
// decimal numbers, on the host. hc_ms2_extract then hands out batches the
// way MSQuery::extractbatch does (msquery.cpp:239-297), with the peak picking
// of MSQuery::pickpeaks (msquery.cpp:509-569) on the device, a warp per
// spectrum: sort the peaks by intensity, equal ones in the order that the
// reference's quicksort leaves them in (KeyVal_Parallel_Internal,
// source/core/include/keyval.h:48-104: Hoare partition around the middle
// key), set the top peak to base_int, scale the next QALEN-1 by
// base_int / top (truncated to integers) and keep the highest ones that
// reach min_int. A second kernel prefix-sums the kept counts and a third
// copies the kept peaks into the CSR batch.
#include <fcntl.h>
#include <sys/stat.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <exception>
#include <memory>
#include <new>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "hc_internal.h"

struct hc_ms2
{
    std::vector<uint64_t> off;  // raw peaks of spectrum s: [off[s], off[s+1])
    std::vector<uint32_t> mz, intn;
    // ... or, parsed on a device, there (m/z, then intensities): one allocation of a
    // context's pool, which lives until this is freed
    int device = -1;
    uint32_t *d_mz = nullptr, *d_int = nullptr;
    std::vector<double> prec, rtime;
    std::vector<uint32_t> z;  // the reference keeps the charge unsigned (msquery.hpp _Spectrum::Z)
    uint32_t maxslen = 0;
};

namespace hc {
namespace {

constexpr int kSortStack = 128;  // the smaller side is sorted first: at most 2*32 levels

// KeyVal_Parallel_Internal (keyval.h:48-104) without recursion: its two
// recursive calls cover disjoint ranges, so the order they run in does not
// change the result. Pushing the larger side first bounds the stack.
__device__ bool key_sort(uint32_t *key, uint32_t *val, int n)
{
    if (n < 2) return true;
    int stack[kSortStack];
    int sp = 0;
    stack[sp++] = 0;
    stack[sp++] = n - 1;
    while (sp > 0)
    {
        const int right = stack[--sp], left = stack[--sp];
        int i = left, j = right;
        const uint32_t pivot = key[(left + right) / 2];
        while (i <= j)
        {
            while (key[i] < pivot) i++;
            while (key[j] > pivot) j--;
            if (i <= j)
            {
                const uint32_t k = key[i], v = val[i];
                key[i] = key[j];
                val[i] = val[j];
                key[j] = k;
                val[j] = v;
                i++;
                j--;
            }
        }
        if (sp + 4 > kSortStack) return false;
        const bool lo = left < j, hi = i < right;
        if (j - left > right - i)
        {
            if (lo) { stack[sp++] = left; stack[sp++] = j; }
            if (hi) { stack[sp++] = i; stack[sp++] = right; }
        }
        else
        {
            if (hi) { stack[sp++] = i; stack[sp++] = right; }
            if (lo) { stack[sp++] = left; stack[sp++] = j; }
        }
    }
    return true;
}

constexpr uint32_t kPickCap = 1024;  // raw peaks of a spectrum a warp sorts in shared memory
constexpr int kPickWarps = 8;

// Scales a spectrum's sorted intensities it[0, n) (ascending) as pickpeaks does
// and counts the kept ones (the last of them are kept: scaling keeps the order).
// One thread; the scaled value of sorted peak j.
struct PickScale
{
    uint32_t top, base_int;
    double factor;
    __device__ __forceinline__ PickScale(uint32_t top_, uint32_t base)
        : top(top_), base_int(base), factor((double)base / (double)top_)
    {
    }
    // an all-zero spectrum scales 0 * inf = NaN, which converts to 0
    __device__ __forceinline__ uint32_t operator()(uint32_t v) const { return top ? (uint32_t)((double)v * factor) : 0u; }
};

// A warp's part of the shared memory: a spectrum's raw peaks, the kept ones and
// those next to them in ascending order, and the work space of the tied ranges.
constexpr uint32_t kPickTop = 128;  // >= HC_QALEN + 1
static_assert(HC_QALEN < kPickTop && kPickCap <= 1u << 16, "the cut's neighbour is among the sorted; 16-bit positions");
struct PickSmem
{
    unsigned long long top[kPickTop];  // intensity above m/z
    uint32_t it[kPickCap], ms[kPickCap];
    uint16_t lp[kPickCap], rp[kPickCap];
    uint32_t stk[16];  // ranges left to split, the smaller of two first: at most 10 of 1024 peaks
};

// The reference's sort splits a range at a pivot: i walks up to the next value not
// below it, j down to the next not above it, the two are swapped, until they cross. What
// they stop at does not depend on the swaps before, so the t-th swap is of the t-th
// such value from the left and from the right, as long as the first lies left of the
// second. Splits it[l, r] that way, the warp together; i and j as the walk leaves them.
__device__ __forceinline__ void pick_split(PickSmem &S, int l, int r, int lane, int &i, int &j)
{
    const uint32_t pivot = S.it[(l + r) / 2], lt = (1u << lane) - 1u;
    int totr = 0;
    for (int b = l; b <= r; b += 32)
    {
        const int x = b + lane;
        totr += __popc(__ballot_sync(0xFFFFFFFFu, x <= r && S.it[x] <= pivot));
    }
    int totl = 0, seen = 0;
    for (int b = l; b <= r; b += 32)
    {
        const int x = b + lane;
        const uint32_t v = x <= r ? S.it[x] : 0u;
        const bool isl = x <= r && v >= pivot, isr = x <= r && v <= pivot;
        const uint32_t bl = __ballot_sync(0xFFFFFFFFu, isl), br = __ballot_sync(0xFFFFFFFFu, isr);
        if (isl) S.lp[totl + __popc(bl & lt)] = (uint16_t)x;
        if (isr) S.rp[totr - 1 - seen - __popc(br & lt)] = (uint16_t)x;
        totl += __popc(bl);
        seen += __popc(br);
    }
    __syncwarp();
    int swaps = 0;
    const int most = min(totl, totr);
    for (int b = 0; b < most; b += 32)
    {
        const int t = b + lane;
        const int x = t < most ? S.lp[t] : 1, y = t < most ? S.rp[t] : 0;
        const bool sw = x <= y;
        if (sw)
        {
            const uint32_t v = S.it[x], m = S.ms[x];
            S.it[x] = S.it[y];
            S.ms[x] = S.ms[y];
            S.it[y] = v;
            S.ms[y] = m;
        }
        const uint32_t k = __ballot_sync(0xFFFFFFFFu, sw);
        swaps += __popc(k);
        if (k != 0xFFFFFFFFu) break;
    }
    __syncwarp();
    // (the pivot stops both: at least one swap). The walks end at the next value of
    // their own or at the other's last one, which the swap left on their side; a
    // swap of one place with itself ends them at once.
    const int x = S.lp[swaps - 1], y = S.rp[swaps - 1];
    i = x == y ? x + 1 : min(swaps < totl ? (int)S.lp[swaps] : y, y);
    j = x == y ? x - 1 : max(swaps < totr ? (int)S.rp[swaps] : x, x);
    __syncwarp();
}

// One warp per spectrum of up to kPickCap raw peaks (the others are left to
// k_pick_long): its kept peaks, in the order of the reference's sort, at
// QALEN * s of omz / oint, and their count.
//
// At most HC_QALEN peaks are kept, so only the largest are sorted: a threshold that
// at least HC_QALEN + 1 and at most kPickTop peaks reach, found by halving, and a
// bitonic sort of those. The order of equal intensities is what the reference's
// quicksort leaves; it runs on the raw peaks only where a range of places holds equal
// ones among the kept, and there a warp splits the range at once. Two of five
// spectra of 100-500 log-normal intensities hold some. Bound by the latency of its short
// steps: 5,000 such spectra take 68 us, against 381 us with a sort of all peaks and the
// quicksort in one lane, and 4,210 with a thread per spectrum.
__global__ void __launch_bounds__(kPickWarps * 32) k_pick(const uint64_t *__restrict__ off,
                                                         const uint32_t *__restrict__ mz,
                                                         const uint32_t *__restrict__ intn, uint32_t nspec,
                                                         uint32_t base_int, uint32_t min_int,
                                                         uint32_t *__restrict__ count, uint32_t *__restrict__ omz,
                                                         uint32_t *__restrict__ oint)
{
    extern __shared__ __align__(16) unsigned char psm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s = blockIdx.x * kPickWarps + (uint32_t)warp, lt = (1u << lane) - 1u;
    if (s >= nspec) return;
    PickSmem &S = reinterpret_cast<PickSmem *>(psm)[warp];
    const uint64_t o = off[s] - off[0];
    const uint64_t len = off[s + 1] - off[s];
    if (len > kPickCap) return;
    const uint32_t n = (uint32_t)len;
    if (n == 0)
    {
        if (lane == 0) count[s] = 0;
        return;
    }
    uint32_t most = 0;
    for (uint32_t i = (uint32_t)lane; i < n; i += 32)
    {
        const uint32_t v = intn[o + i];
        S.it[i] = v;
        S.ms[i] = mz[o + i];
        most = max(most, v);
    }
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    __syncwarp();
    // more than kPickTop peaks reach `below`, HC_QALEN at most reach `thr`, unless one
    // is found that a number between reaches
    unsigned long long thr = 0, below = 0;
    if (n > kPickTop)
    {
        unsigned long long hi = (unsigned long long)most + 1;
        thr = hi;
        while (hi - below > 1)
        {
            const unsigned long long mid = (below + hi) / 2;
            uint32_t c = 0;
            for (uint32_t i = (uint32_t)lane; i < n; i += 32) c += S.it[i] >= mid;
            c = __reduce_add_sync(0xFFFFFFFFu, c);
            if (c > kPickTop) below = mid;
            else
            {
                thr = mid;
                if (c > HC_QALEN) break;
                hi = mid;
            }
        }
    }
    uint32_t c = 0;  // sorted peaks
    for (uint32_t b = 0; b < n; b += 32)
    {
        const uint32_t i = b + (uint32_t)lane;
        const bool in = i < n && S.it[i] >= thr;
        const uint32_t k = __ballot_sync(0xFFFFFFFFu, in);
        if (in) S.top[c + __popc(k & lt)] = ((unsigned long long)S.it[i] << 32) | S.ms[i];
        c += (uint32_t)__popc(k);
    }
    // the rest up to the cut's neighbour are some of more than 28 equal ones
    const uint32_t want = min(n, (uint32_t)HC_QALEN + 1u), take = max(c, want);
    uint32_t P = 32;
    while (P < take) P <<= 1;
    for (uint32_t i = c + (uint32_t)lane; i < P; i += 32) S.top[i] = i < take ? below << 32 : ~0ull;
    c = take;
    __syncwarp();
    for (uint32_t k = 2; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1)
        {
            for (uint32_t t = (uint32_t)lane; t < P / 2; t += 32)
            {
                const uint32_t a = 2 * t - (t & (j - 1)), b = a + j;
                const unsigned long long x = S.top[a], y = S.top[b];
                if ((x > y) == ((a & k) == 0u))
                {
                    S.top[a] = y;
                    S.top[b] = x;
                }
            }
            __syncwarp();
        }
    // (padding sorts last, as does a peak equal to it: the first c are the peaks)
    const PickScale sc((uint32_t)(S.top[c - 1] >> 32), base_int);
    const uint32_t cand = n < HC_QALEN ? n : HC_QALEN;
    uint32_t keep = 1;
    for (uint32_t b = 1; b < cand; b += 32)
    {
        const uint32_t i = b + (uint32_t)lane;
        keep += (uint32_t)__popc(
            __ballot_sync(0xFFFFFFFFu, i < cand && sc((uint32_t)(S.top[c - 1 - i] >> 32)) >= min_int));
    }
    const uint32_t first = c - keep;  // sorted peak c - keep is the first kept one
    for (uint32_t i = (uint32_t)lane; i < keep; i += 32)
    {
        const unsigned long long x = S.top[first + i];
        omz[(size_t)s * HC_QALEN + i] = (uint32_t)x;
        oint[(size_t)s * HC_QALEN + i] = i == keep - 1 ? base_int : sc((uint32_t)(x >> 32));
    }
    if (lane == 0) count[s] = keep;
    // bit e of the words of lanes 0..3: sorted peaks e and e + 1 are equally intense, and e + 1 is kept
    uint32_t tied = 0;
    bool any = false;
#pragma unroll
    for (uint32_t w = 0; w < kPickTop / 32; w++)
    {
        const uint32_t e = 32 * w + (uint32_t)lane;
        const bool t = e + 1 < c && e + 1 >= first && (S.top[e] >> 32) == (S.top[e + 1] >> 32);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, t);
        if ((uint32_t)lane == w) tied = m;
        any |= m != 0u;
    }
    if (!any) return;
    const int base = (int)n - (int)c;  // the place of sorted peak e is base + e
    auto holds_tie = [&](int l, int r) {  // two equal kept peaks at the places l .. r?
        const int lo = min(max(l - base - 32 * lane, 0), 32), hi = min(max(r - base - 32 * lane, 0), 32);
        const uint32_t m = (hi > 31 ? 0xFFFFFFFFu : (1u << hi) - 1u) & ~(lo > 31 ? 0xFFFFFFFFu : (1u << lo) - 1u);
        return __any_sync(0xFFFFFFFFu, lane < (int)(kPickTop / 32) && (tied & m) != 0u) != 0;
    };
    // the peaks of a range without such: each one that equals others elsewhere is the
    // only one here, at the first of their places that the range has
    auto settle = [&](int l, int r) {
        for (int x = l + lane; x <= r; x += 32)
        {
            const uint32_t v = S.it[x];
            uint32_t lo = 0, hi = c;  // the first sorted peak that is not below v
            while (lo < hi)
            {
                const uint32_t mid = (lo + hi) / 2;
                if ((uint32_t)(S.top[mid] >> 32) < v) lo = mid + 1;
                else hi = mid;
            }
            if (lo + 1 >= c || (uint32_t)(S.top[lo + 1] >> 32) != v) continue;
            const int e = max((int)lo, l - base);
            if ((uint32_t)(S.top[lo] >> 32) == v && e >= (int)first) omz[(size_t)s * HC_QALEN + (e - (int)first)] = S.ms[x];
        }
    };
    __syncwarp();
    int l = 0, r = (int)n - 1, sp = 0;
    for (;;)
    {
        int i, j;
        pick_split(S, l, r, lane, i, j);
        if (i - j > 1) settle(j + 1, i - 1);
        const int keep_from = base + (int)first;
        const bool ta = holds_tie(l, j), tb = holds_tie(i, r);
        if (!ta && l <= j && j >= keep_from) settle(l, j);
        if (!tb && i <= r && r >= keep_from) settle(i, r);
        if (ta && tb)
        {
            const bool lefts = j - l > r - i;  // the larger one waits
            if (lane == 0) S.stk[sp] = lefts ? (uint32_t)l << 16 | (uint32_t)j : (uint32_t)i << 16 | (uint32_t)r;
            sp++;
            __syncwarp();
            if (lefts) l = i;
            else r = j;
        }
        else if (ta) r = j;
        else if (tb) l = i;
        else
        {
            if (sp == 0) break;
            const uint32_t q = S.stk[--sp];
            __syncwarp();
            l = (int)(q >> 16);
            r = (int)(q & 0xFFFFu);
        }
    }
}

// The spectra of more than kPickCap raw peaks, a thread each, sorted in place
// (mz, intn: scratch copies).
__global__ void k_pick_long(const uint64_t *__restrict__ off, uint32_t *__restrict__ mz, uint32_t *__restrict__ intn,
                            uint32_t nspec, uint32_t base_int, uint32_t min_int, uint32_t *__restrict__ count,
                            uint32_t *__restrict__ omz, uint32_t *__restrict__ oint)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec || off[s + 1] - off[s] <= kPickCap) return;
    const uint64_t o = off[s] - off[0];
    const int n = (int)(off[s + 1] - off[s]);
    uint32_t *it = intn + o, *ms = mz + o;
    if (!key_sort(it, ms, n))
    {
        count[s] = 0xFFFFFFFFu;  // cannot happen with the stack bound above; reported as an error
        return;
    }
    const PickScale sc(it[n - 1], base_int);
    uint32_t keep = 1;
    for (int j = n - 2; j >= n - (int)HC_QALEN; j--)
        if (sc(it[j]) >= min_int) keep++;
    for (uint32_t i = 0; i < keep; i++)
    {
        const int j = n - (int)keep + (int)i;
        omz[(size_t)s * HC_QALEN + i] = ms[j];
        oint[(size_t)s * HC_QALEN + i] = j == n - 1 ? base_int : sc(it[j]);
    }
    count[s] = keep;
}

// In-place inclusive prefix sum of the kept counts in one block: on entry
// idx[1..n] holds the counts, on exit idx[s] is where spectrum s starts.
// Sets idx[n+1] = 1 when a sort reported failure.
__global__ void k_scan(uint32_t *__restrict__ idx, uint32_t n)
{
    __shared__ uint32_t warp_sum[32];
    __shared__ uint32_t carry;
    __shared__ uint32_t bad;
    const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0)
    {
        carry = 0;
        bad = 0;
        idx[0] = 0;
    }
    __syncthreads();
    for (uint32_t base = 0; base < n; base += blockDim.x)
    {
        const uint32_t s = base + t;
        uint32_t v = s < n ? idx[s + 1] : 0u;
        if (v == 0xFFFFFFFFu)
        {
            bad = 1;
            v = 0;
        }
        uint32_t x = v;
        for (int d = 1; d < 32; d <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
            if (lane >= (uint32_t)d) x += y;
        }
        if (lane == 31) warp_sum[w] = x;
        __syncthreads();
        if (w == 0)
        {
            uint32_t ws = lane < (blockDim.x >> 5) ? warp_sum[lane] : 0u;
            for (int d = 1; d < 32; d <<= 1)
            {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, ws, d);
                if (lane >= (uint32_t)d) ws += y;
            }
            warp_sum[lane] = ws;
        }
        __syncthreads();
        const uint32_t incl = carry + (w ? warp_sum[w - 1] : 0u) + x;
        if (s < n) idx[s + 1] = incl;
        __syncthreads();
        if (t == blockDim.x - 1) carry = incl;
        __syncthreads();
    }
    if (t == 0) idx[n + 1] = bad;
}

// the kept peaks of each spectrum into the CSR batch, one warp per spectrum
__global__ void k_pick_copy(const uint32_t *__restrict__ mz, const uint32_t *__restrict__ intn, uint32_t nspec,
                            const uint32_t *__restrict__ idx, uint32_t *__restrict__ omz, uint32_t *__restrict__ oint)
{
    const uint32_t s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= nspec) return;
    const uint32_t k = idx[s + 1] - idx[s];
    const size_t src = (size_t)s * HC_QALEN;
    for (uint32_t t = threadIdx.x & 31; t < k; t += 32)
    {
        omz[idx[s] + t] = mz[src + t];
        oint[idx[s] + t] = intn[src + t];
    }
}

// ---- the file's lines on the device ------------------------------------------
// A CTA takes kTxt bytes: it lists the lines that start there, in order, then
// takes them a thread each. Peak lines of the plain form (spaces, a decimal
// number, spaces, a decimal number, then a space or the line's end) are parsed
// here; any other peak line sets *odd and the host parser takes the whole file. A
// number of at most 15 digits is its digits as an integer divided by a power of
// ten, both exact doubles, so the one rounding of the division gives what atof
// gives (W. D. Clinger, "How to read floating point numbers accurately", 1990).
// The lines of S, and those of Z and I, are listed by position: they are few, and the
// host reads them. The first pass (mz null) counts, the second writes at the
// counts' prefix sums. 28 MB (1.5 M peak lines): 95 us for both.
constexpr uint32_t kTxt = 8192, kTxtHalo = 256;
constexpr int kTxtThreads = 256;

__device__ const double kPow10[16] = {1e0, 1e1, 1e2,  1e3,  1e4,  1e5,  1e6,  1e7,
                                      1e8, 1e9, 1e10, 1e11, 1e12, 1e13, 1e14, 1e15};

struct LineCounts
{
    uint32_t peaks, spectra, attrs;
};

// the decimal number at tx[p, end); false unless it is plain
__device__ __forceinline__ bool plain_number(const uint8_t *tx, uint32_t &p, uint32_t end, double &v)
{
    unsigned long long m = 0;
    uint32_t digits = 0, frac = 0, seen = 0;
    bool point = false;
    for (; p < end; p++)
    {
        const uint32_t c = tx[p], d = c - '0';
        if (d < 10u)
        {
            m = m * 10 + d;
            digits += m != 0;
            frac += point;
            seen++;
            if (digits > 15 || frac > 15) return false;
        }
        else if (c == '.' && !point) point = true;
        else break;
    }
    v = (double)m;
    if (frac) v = __ddiv_rn(v, kPow10[frac]);
    return seen != 0;
}

// exclusive prefix sum over the block's threads; *total of all
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t *ws, uint32_t *total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int i = 0; i < kTxtThreads / 32; i++)
    {
        const uint32_t t = ws[i];
        before += i < w ? t : 0u;
        all += t;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

__global__ void __launch_bounds__(kTxtThreads) k_ms2_lines(const uint8_t *__restrict__ text, uint64_t size, double scale,
                                                          LineCounts *__restrict__ counts, uint32_t *__restrict__ mz,
                                                          uint32_t *__restrict__ intn, uint64_t *__restrict__ spos,
                                                          uint32_t *__restrict__ soff, uint64_t *__restrict__ apos,
                                                          uint32_t *__restrict__ odd)
{
    __shared__ __align__(16) uint8_t tx[kTxt + kTxtHalo];
    __shared__ uint16_t starts[kTxt];
    __shared__ uint32_t ws[kTxtThreads / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kTxt;
    const int t = threadIdx.x;
    for (uint32_t i = (uint32_t)t; i < (kTxt + kTxtHalo) / 16; i += kTxtThreads)
        reinterpret_cast<uint4 *>(tx)[i] = __ldg(reinterpret_cast<const uint4 *>(text + base) + i);
    __syncthreads();
    // lines start after a newline (or at the file's start), a mask bit per byte of this thread's 32
    const uint32_t left = (uint32_t)min((uint64_t)kTxt, size - base);
    uint32_t nl = 0;
#pragma unroll
    for (int i = 0; i < 8; i++)
    {
        const uint32_t m = __vcmpeq4(reinterpret_cast<const uint32_t *>(tx)[8 * t + i], 0x0A0A0A0Au) & 0x01010101u;
        nl |= ((m * 0x01020408u) >> 24) << (4 * i);
    }
    const uint8_t prev = t ? tx[32 * t - 1] : (base ? text[base - 1] : (uint8_t)'\n');
    uint32_t st = (nl << 1) | (prev == '\n' ? 1u : 0u);
    const uint32_t b0 = 32u * (uint32_t)t;
    if (b0 + 32 > left) st &= b0 < left ? (1u << (left - b0)) - 1u : 0u;
    uint32_t nlines;
    uint32_t at = block_prefix((uint32_t)__popc(st), ws, &nlines);
    for (; st; st &= st - 1) starts[at++] = (uint16_t)(b0 + (uint32_t)__ffs(st) - 1u);
    __syncthreads();
    const uint32_t end = (uint32_t)min((uint64_t)(kTxt + kTxtHalo), size - base);
    LineCounts n = mz ? counts[blockIdx.x] : LineCounts{0, 0, 0};
    for (uint32_t l0 = 0; l0 < nlines; l0 += kTxtThreads)
    {
        const uint32_t l = l0 + (uint32_t)t;
        uint32_t p = 0, kind = 0;  // 1: a peak, 1 << 10: S, 1 << 20: Z or I
        if (l < nlines)
        {
            p = starts[l];
            const uint32_t c = tx[p];
            kind = c == '\n' || c == 'H' || c == 'D' ? 0u : c == 'S' ? 1u << 10 : c == 'Z' || c == 'I' ? 1u << 20 : 1u;
        }
        uint32_t all;
        const uint32_t before = block_prefix(kind, ws, &all);
        if (mz && kind)
        {
            const uint32_t pk = n.peaks + (before & 1023u);
            if (kind == 1u)
            {
                double a = 0.0, b = 0.0;
                while (p < end && tx[p] == ' ') p++;
                bool ok = plain_number(tx, p, end, a) && p < end && tx[p] == ' ';
                while (p < end && tx[p] == ' ') p++;
                ok = ok && plain_number(tx, p, end, b);
                if (p < end) ok = ok && (tx[p] == ' ' || tx[p] == '\n' || tx[p] == '\r');
                else ok = ok && base + p >= size;  // the file's end, not this CTA's
                a = __dmul_rn(a, scale);
                b = __dmul_rn(b, 1000.0);
                if (!ok || !(a < 4294967296.0) || !(b < 4294967296.0)) atomicOr(odd, 1u);
                else
                {
                    mz[pk] = (uint32_t)a;
                    intn[pk] = (uint32_t)b;
                }
            }
            else if (kind == 1u << 10)
            {
                const uint32_t k = n.spectra + ((before >> 10) & 1023u);
                spos[k] = base + p;
                soff[k] = pk;
            }
            else
                apos[n.attrs + (before >> 20)] = base + p;
        }
        n.peaks += all & 1023u;
        n.spectra += (all >> 10) & 1023u;
        n.attrs += all >> 20;
    }
    if (!mz && t == 0) counts[blockIdx.x] = n;
}

// One line of the file: [p, e), cut at its first NUL byte as the reference's
// strtok on c_str() cuts it. The '\n' is not part of it; a '\r' before it is
// (std::getline keeps it).
struct Line
{
    const char *p, *e;
};

// strtok_r on a line: the next token after runs of ' ' (and '\t' if `tab`)
bool next_tok(const char *&p, const char *e, bool tab, const char *&tb, const char *&te)
{
    while (p < e && (*p == ' ' || (tab && *p == '\t'))) p++;
    if (p >= e) return false;
    tb = p;
    while (p < e && *p != ' ' && !(tab && *p == '\t')) p++;
    te = p;
    return true;
}

// atof / atoi of a token (the token is copied so the conversion cannot read past it)
double tok_atof(const char *tb, const char *te, double dflt, bool have)
{
    if (!have) return dflt;
    char buf[64];
    const size_t n = (size_t)(te - tb);
    if (n < sizeof(buf))
    {
        std::memcpy(buf, tb, n);
        buf[n] = 0;
        return std::atof(buf);
    }
    return std::atof(std::string(tb, n).c_str());
}

int tok_atoi(const char *tb, const char *te, int dflt, bool have)
{
    if (!have) return dflt;
    char buf[64];
    const size_t n = (size_t)(te - tb);
    if (n < sizeof(buf))
    {
        std::memcpy(buf, tb, n);
        buf[n] = 0;
        return std::atoi(buf);
    }
    return std::atoi(std::string(tb, n).c_str());
}

// part(0) .. part(n - 1), which throw nothing, by a thread each as far as there are
// threads to be had.
template <class F>
void in_threads(unsigned n, const F &part)
{
    std::vector<std::thread> th;
    th.reserve(n);
    unsigned k = 1;
    try
    {
        for (; k < n; k++) th.emplace_back(part, k);
    }
    catch (const std::system_error &)
    {
    }
    part(0);
    for (; k < n; k++) part(k);
    for (auto &t : th) t.join();
}

// What a spectrum's own 'Z' and 'I RTime' lines set.
struct Attrs
{
    uint8_t zs = 0, rs = 0;
    uint32_t z = 0;
    double prec = 0.0, rt = 0.0;
};

// The spectra of one stretch of the file. Every stretch but the first starts
// at an 'S' line; the first holds the file's first 'S' line. A spectrum's
// charge / precursor (a 'Z' line) and retention time (an 'I RTime' line) are
// recorded only when one of its lines sets them: the others inherit the
// previous spectrum's values, which are known once the stretches are joined.
struct Stretch
{
    std::vector<Attrs> at;
    std::vector<uint64_t> npk;
    std::vector<uint32_t> mz, intn;
    uint64_t peak_lines = 0;
};

// a 'Z' or 'I' line, [q, ee)
void attr_line(char c, const char *q, const char *ee, Attrs &a)
{
    const char *tb = nullptr, *te = nullptr;
    next_tok(q, ee, true, tb, te);
    if (c == 'Z')
    {
        bool h = next_tok(q, ee, true, tb, te);
        a.z = (uint32_t)tok_atoi(tb, te, 1, h);
        h = next_tok(q, ee, true, tb, te);
        a.prec = tok_atof(tb, te, 0.01, h);
        a.zs = 1;
    }
    else if (next_tok(q, ee, true, tb, te) && te - tb == 5 && std::memcmp(tb, "RTime", 5) == 0)
    {
        const bool h = next_tok(q, ee, true, tb, te);
        a.rt = tok_atof(tb, te, 0.00, h);
        a.rs = 1;
    }
}

// appends a spectrum's attributes; what its own lines do not set it inherits
// from the spectrum before (the reference's spectrum_t starts zeroed, msquery.cpp:27-42)
void push_attrs(hc_ms2 *m, const Attrs &a, Attrs &inh)
{
    if (a.zs)
    {
        inh.z = a.z;
        inh.prec = a.prec;
    }
    if (a.rs) inh.rt = a.rt;
    m->z.push_back(inh.z);
    m->prec.push_back(inh.prec);
    m->rtime.push_back(inh.rt);
}

void parse_stretch(const char *b, const char *e, bool first, double scale, Stretch &out)
{
    bool started = false;
    Attrs at;
    uint64_t cur = 0;
    auto close = [&]() {
        out.at.push_back(at);
        out.npk.push_back(cur);
        at.zs = at.rs = 0;
        cur = 0;
    };
    const char *p = b;
    while (p < e)
    {
        const char *nl = static_cast<const char *>(std::memchr(p, '\n', (size_t)(e - p)));
        const char *le = nl ? nl : e;
        Line ln{p, le};
        p = nl ? nl + 1 : e;
        if (ln.p == ln.e) continue;  // empty line
        const char c = *ln.p;
        const char *zero = static_cast<const char *>(std::memchr(ln.p, 0, (size_t)(ln.e - ln.p)));
        const char *ee = zero ? zero : ln.e;
        const char *q = ln.p, *tb = nullptr, *te = nullptr;
        if (c == 'H' || c == 'D') continue;
        if (c == 'Z' || c == 'I') attr_line(c, q, ee, at);
        else if (c == 'S')
        {
            if (started) close();
            started = true;
        }
        else
        {
            // a peak: tokens split on ' ' only (msquery.cpp:388-404, 478-498); a
            // missing token reads "0.01" in the file's first spectrum, "0.0" after
            const double dflt = (first && out.npk.empty()) ? 0.01 : 0.0;
            bool h = next_tok(q, ee, false, tb, te);
            const double mzv = tok_atof(tb, te, dflt, h);
            h = next_tok(q, ee, false, tb, te);
            const double iv = tok_atof(tb, te, dflt, h);
            out.mz.push_back((uint32_t)(mzv * scale));
            out.intn.push_back((uint32_t)(iv * 1000));
            cur++;
            out.peak_lines++;
        }
    }
    if (started) close();
}

// position of the next line start at or after p that begins with 'S' (or e)
const char *next_s_line(const char *base, const char *p, const char *e)
{
    if (p > base && p[-1] != '\n')
    {
        const char *nl = static_cast<const char *>(std::memchr(p, '\n', (size_t)(e - p)));
        if (!nl) return e;
        p = nl + 1;
    }
    while (p < e)
    {
        if (*p == 'S') return p;
        const char *nl = static_cast<const char *>(std::memchr(p, '\n', (size_t)(e - p)));
        if (!nl) return e;
        p = nl + 1;
    }
    return e;
}

}  // namespace
}  // namespace hc

using namespace hc;

// The text [base, end) parsed by all host threads.
static int parse_host(const char *base, const char *end, double scale, hc_ms2 **out)
{
    // stretches: the first runs from the file start through its first 'S'
    // line; the others start at 'S' lines, about equal in size
    const char *s0 = next_s_line(base, base, end);
    const unsigned hw = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
    const size_t span = (size_t)(end - s0);
    const unsigned nt = s0 < end ? (unsigned)std::max<size_t>(1, std::min<size_t>(hw, span / (1u << 20) + 1)) : 1u;
    std::vector<const char *> cut{base};
    for (unsigned k = 1; k < nt; k++)
    {
        const char *c = next_s_line(base, s0 + 1 + span * k / nt, end);
        if (c > cut.back() && c < end) cut.push_back(c);
    }
    cut.push_back(end);
    const size_t ns_ = cut.size() - 1;
    std::vector<Stretch> parts(ns_);
    std::atomic<bool> full{false};
    in_threads((unsigned)ns_, [&](unsigned k) {
        try
        {
            parse_stretch(cut[k], cut[k + 1], k == 0, scale, parts[k]);
        }
        catch (const std::bad_alloc &)
        {
            full = true;
        }
    });
    if (full) return HC_ERR_BAD_MEM_ALLOC;

    // join: inherit charge / precursor / retention time in file order (the
    // reference's spectrum_t starts zeroed, msquery.cpp:27-42)
    std::unique_ptr<hc_ms2> m(new hc_ms2());
    uint64_t peak_lines = 0, nsp = 0, npk = 0;
    for (const Stretch &st : parts)
    {
        peak_lines += st.peak_lines;
        nsp += st.npk.size();
        npk += st.mz.size();
    }
    m->off.reserve(nsp + 1);
    m->prec.reserve(nsp);
    m->z.reserve(nsp);
    m->rtime.reserve(nsp);
    m->mz.reserve(npk);
    m->intn.reserve(npk);
    m->off.push_back(0);
    Attrs inh;
    for (const Stretch &st : parts)
    {
        for (size_t i = 0; i < st.npk.size(); i++)
        {
            push_attrs(m.get(), st.at[i], inh);
            m->off.push_back(m->off.back() + st.npk[i]);
            if (st.npk[i] > m->maxslen) m->maxslen = (uint32_t)std::min<uint64_t>(st.npk[i], 0xFFFFFFFFu);
        }
        // peaks of a stretch without an 'S' line (only possible with no 'S' at all) belong to no spectrum
        const uint64_t used = m->off.back() - m->mz.size();
        m->mz.insert(m->mz.end(), st.mz.begin(), st.mz.begin() + (ptrdiff_t)used);
        m->intn.insert(m->intn.end(), st.intn.begin(), st.intn.begin() + (ptrdiff_t)used);
    }
    // MSQuery::initialize: no peak line at all is ERR_INVLD_SIZE (msquery.cpp:143-147)
    if (peak_lines == 0 || m->mz.size() >= 0xFFFFFFFFull || m->off.size() > 0xFFFFFFFFull) return HC_ERR_INVLD_SIZE;
    *out = m.release();
    return HC_SUCCESS;
}

// `rc` with what the caller of an open or a read asked for
static int opened(int rc, hc_ms2 *const *out, uint32_t *nspec, uint32_t *maxslen)
{
    if (rc != HC_SUCCESS) return rc;
    if (nspec) *nspec = (uint32_t)(*out)->prec.size();
    if (maxslen) *maxslen = (*out)->maxslen;
    return rc;
}

extern "C" int hc_ms2_read(const char *path, uint32_t scale_u, hc_ms2 **out, uint32_t *nspec, uint32_t *maxslen)
try
{
    if (!path || !out) return HC_ERR_INVLD_PTR;
    *out = nullptr;
    const std::unique_ptr<FILE, int (*)(FILE *)> f(std::fopen(path, "rb"), std::fclose);
    struct stat sb;  // (a directory opens, and seeks to an end past all memory)
    if (!f || ::fstat(::fileno(f.get()), &sb) != 0 || S_ISDIR(sb.st_mode)) return HC_ERR_FILE_ERROR;
    if (std::fseek(f.get(), 0, SEEK_END) != 0) return HC_ERR_FILE_ERROR;
    const long fsz = std::ftell(f.get());
    if (fsz < 0 || std::fseek(f.get(), 0, SEEK_SET) != 0) return HC_ERR_FILE_ERROR;
    std::vector<char> buf((size_t)fsz);
    if (std::fread(buf.data(), 1, (size_t)fsz, f.get()) != (size_t)fsz) return HC_ERR_FILE_ERROR;
    return opened(parse_host(buf.data(), buf.data() + buf.size(), (double)scale_u, out), out, nspec, maxslen);
}
catch (const std::exception &)  // no memory for the file or its peaks
{
    return HC_ERR_BAD_MEM_ALLOC;
}

namespace hc {
namespace {

// Files from this size on are parsed on the device: opening takes 120 us there and 76 us
// on the host at 8 KB, 131 and 158 us at 21 KB, 0.5 and 6.4 ms at 5.7 MB, 1.5 and 13.9 ms
// at 28 MB.
constexpr uint64_t kDeviceText = 1u << 14;

// The whole file, by up to eight threads; false when it is small or cannot be read.
bool read_file(const char *path, std::unique_ptr<char[]> &buf, uint64_t &size)
{
    struct Fd
    {
        const int fd;
        ~Fd()
        {
            if (fd >= 0) ::close(fd);
        }
    } const file{::open(path, O_RDONLY)};
    const int fd = file.fd;
    if (fd < 0) return false;
    struct stat sb;
    bool ok = ::fstat(fd, &sb) == 0 && S_ISREG(sb.st_mode) && (uint64_t)sb.st_size >= kDeviceText;
    if (ok)
    {
        size = (uint64_t)sb.st_size;
        buf.reset(new char[size]);  // not zeroed
        const unsigned nt =
            (unsigned)std::max<uint64_t>(1, std::min<uint64_t>({8, std::thread::hardware_concurrency(), size >> 20}));
        std::vector<uint8_t> good(nt, 1);
        auto part = [&](unsigned k) {
            uint64_t a = size * k / nt;
            const uint64_t b = size * (k + 1) / nt;
            while (a < b)
            {
                const ssize_t r = ::pread(fd, buf.get() + a, (size_t)(b - a), (off_t)a);
                if (r <= 0)
                {
                    good[k] = 0;
                    return;
                }
                a += (uint64_t)r;
            }
        };
        in_threads(nt, part);
        for (uint8_t g : good) ok = ok && g;
    }
    return ok;
}

// Parses the text on the device: HC_SUCCESS with *out set, an error, or 1 when it
// is the host parser's (4 GB or more, a peak line that is not plain).
int parse_device(hc_ctx *ctx, const std::unique_ptr<char[]> &buf, uint64_t size, hc_ms2 **out)
{
    if (size >= 0xFFFFFFFFull) return 1;
    cudaStream_t st = ctx->stream;
    const uint32_t nb = (uint32_t)((size + kTxt - 1) / kTxt);
    const uint64_t room = (uint64_t)nb * kTxt + kTxtHalo;
    PoolScratch scr(ctx);
    uint8_t *d_text;
    LineCounts *d_counts;
    uint32_t *d_odd;
    HC_CUDA(ctx, scr.alloc(&d_text, room));
    HC_CUDA(ctx, scr.alloc(&d_counts, nb));
    HC_CUDA(ctx, scr.alloc(&d_odd, 1));
    HC_CUDA(ctx, cudaMemcpyAsync(d_text, buf.get(), size, cudaMemcpyHostToDevice, st));
    HC_CUDA(ctx, cudaMemsetAsync(d_text + size, 0, room - size, st));
    HC_CUDA(ctx, cudaMemsetAsync(d_odd, 0, 4, st));
    const double scale = (double)ctx->p.scale;
    k_ms2_lines<<<nb, kTxtThreads, 0, st>>>(d_text, size, scale, d_counts, nullptr, nullptr, nullptr, nullptr, nullptr,
                                            d_odd);
    HC_CUDA(ctx, cudaGetLastError());
    std::vector<LineCounts> counts(nb);
    HC_CUDA(ctx, cudaMemcpyAsync(counts.data(), d_counts, sizeof(LineCounts) * nb, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    LineCounts tot{0, 0, 0};  // (a line takes a byte at least, so 32 bits hold them)
    for (LineCounts &c : counts)
    {
        const LineCounts n = c;
        c = tot;
        tot.peaks += n.peaks;
        tot.spectra += n.spectra;
        tot.attrs += n.attrs;
    }
    if (tot.peaks == 0 || tot.spectra == 0) return 1;
    std::unique_ptr<hc_ms2, int (*)(hc_ms2 *)> m(new hc_ms2(), hc_ms2_close);
    m->device = ctx->device;
    HC_CUDA(ctx, dalloc(ctx, &m->d_mz, 2 * (size_t)tot.peaks));
    m->d_int = m->d_mz + tot.peaks;
    uint64_t *d_spos, *d_apos;
    uint32_t *d_soff;
    HC_CUDA(ctx, scr.alloc(&d_spos, tot.spectra));
    HC_CUDA(ctx, scr.alloc(&d_soff, tot.spectra));
    HC_CUDA(ctx, scr.alloc(&d_apos, tot.attrs));
    HC_CUDA(ctx, cudaMemcpyAsync(d_counts, counts.data(), sizeof(LineCounts) * nb, cudaMemcpyHostToDevice, st));
    k_ms2_lines<<<nb, kTxtThreads, 0, st>>>(d_text, size, scale, d_counts, m->d_mz, m->d_int, d_spos, d_soff, d_apos,
                                            d_odd);
    HC_CUDA(ctx, cudaGetLastError());
    uint32_t odd = 0;
    const uint32_t ns = tot.spectra;
    std::vector<uint64_t> spos(ns), apos(tot.attrs);
    std::vector<uint32_t> soff(ns);
    HC_CUDA(ctx, cudaMemcpyAsync(spos.data(), d_spos, 8ull * ns, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaMemcpyAsync(soff.data(), d_soff, 4ull * ns, cudaMemcpyDeviceToHost, st));
    if (tot.attrs)
        HC_CUDA(ctx, cudaMemcpyAsync(apos.data(), d_apos, 8ull * tot.attrs, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaMemcpyAsync(&odd, d_odd, 4, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    if (odd) return 1;
    // what precedes the first S line belongs to the first spectrum
    m->off.resize((size_t)ns + 1);
    for (uint32_t s = 0; s < ns; s++) m->off[s] = s ? soff[s] : 0u;
    m->off[ns] = tot.peaks;
    std::vector<Attrs> at(ns);
    auto lines = [&](uint32_t s0, uint32_t s1) {
        const uint64_t from = s0 ? spos[s0] : 0, to = s1 < ns ? spos[s1] : size;
        size_t i = (size_t)(std::lower_bound(apos.begin(), apos.end(), from) - apos.begin());
        for (uint32_t s = s0; i < apos.size() && apos[i] < to; i++)
        {
            while (s + 1 < ns && spos[s + 1] < apos[i]) s++;
            const char *p = buf.get() + apos[i], *e = buf.get() + size;
            if (const void *x = std::memchr(p, '\n', (size_t)(e - p))) e = static_cast<const char *>(x);
            if (const void *x = std::memchr(p, 0, (size_t)(e - p))) e = static_cast<const char *>(x);
            attr_line(*p, p, e, at[s]);
        }
    };
    const unsigned nt = std::max(1u, std::min({8u, std::thread::hardware_concurrency(), ns / 512 + 1}));
    {
        // (not in_threads, with which the lines took 0.55 ms of 10,000 instead of 0.46)
        std::vector<std::thread> th;
        th.reserve(nt);
        unsigned k = 1;
        try
        {
            for (; k < nt; k++)
                th.emplace_back(lines, (uint32_t)((uint64_t)ns * k / nt), (uint32_t)((uint64_t)ns * (k + 1) / nt));
        }
        catch (const std::system_error &)
        {
            lines((uint32_t)((uint64_t)ns * k / nt), ns);
        }
        lines(0, (uint32_t)((uint64_t)ns / nt));
        for (auto &x : th) x.join();
    }
    m->prec.reserve(ns);
    m->z.reserve(ns);
    m->rtime.reserve(ns);
    Attrs inh;
    for (uint32_t s = 0; s < ns; s++)
    {
        push_attrs(m.get(), at[s], inh);
        m->maxslen = std::max(m->maxslen, (uint32_t)(m->off[s + 1] - m->off[s]));
    }
    *out = m.release();
    return HC_SUCCESS;
}

// the raw peaks on the host (for a device other than theirs)
int peaks_to_host(hc_ctx *ctx, hc_ms2 *m)
{
    if (!m->d_mz || !m->mz.empty()) return HC_SUCCESS;
    const size_t n = (size_t)m->off.back();
    m->mz.resize(n);
    m->intn.resize(n);
    HC_CUDA(ctx, cudaMemcpy(m->mz.data(), m->d_mz, 4 * n, cudaMemcpyDefault));
    HC_CUDA(ctx, cudaMemcpy(m->intn.data(), m->d_int, 4 * n, cudaMemcpyDefault));
    return HC_SUCCESS;
}

}  // namespace
}  // namespace hc

extern "C" int hc_ms2_open(hc_ctx *ctx, const char *path, hc_ms2 **out, uint32_t *nspec, uint32_t *maxslen)
try
{
    if (!ctx || !path || !out) return HC_ERR_INVLD_PTR;
    *out = nullptr;
    std::unique_ptr<char[]> buf;
    uint64_t size = 0;
    int rc = 1;
    if (read_file(path, buf, size))
    {
        const BesideCapture beside;
        HC_CUDA(ctx, cudaSetDevice(ctx->device));
        // (a device at work would do it when it has ended what it does)
        if (device_idle(ctx)) rc = parse_device(ctx, buf, size, out);
        if (rc < 0 && rc != HC_ERR_BAD_MEM_ALLOC) return rc;
        // (no room on the device: the host's arrays do)
        if (rc != HC_SUCCESS) rc = parse_host(buf.get(), buf.get() + size, (double)ctx->p.scale, out);
        rc = opened(rc, out, nspec, maxslen);
    }
    else
        rc = hc_ms2_read(path, ctx->p.scale, out, nspec, maxslen);
    if (rc == HC_ERR_FILE_ERROR) return set_error(ctx, rc, std::string("cannot read ") + path);
    if (rc == HC_ERR_INVLD_SIZE) return set_error(ctx, rc, std::string("no peaks (or 2^32 or more) in ") + path);
    return rc;
}
catch (const std::exception &)
{
    return set_error(ctx, HC_ERR_BAD_MEM_ALLOC, "no memory for the file or its peaks");
}

extern "C" int hc_ms2_raw(const hc_ms2 *m, uint32_t first, uint32_t count, uint64_t *off, uint32_t *mz,
                          uint32_t *intensity, double *prec, uint32_t *z, double *rtime)
{
    if (!m || !off) return HC_ERR_INVLD_PTR;
    const uint64_t total = m->prec.size();
    if ((uint64_t)first + count > total) return HC_ERR_INVLD_SIZE;
    const uint64_t a = m->off[first];
    for (uint32_t k = 0; k <= count; k++) off[k] = m->off[first + k] - a;
    const uint64_t n = m->off[first + count] - a;
    if (m->d_mz && n && (mz || intensity))
    {
        const BesideCapture beside;
        const cudaStream_t st = cudaStreamPerThread;
        cudaError_t e = cudaSetDevice(m->device);
        if (e == cudaSuccess && mz) e = cudaMemcpyAsync(mz, m->d_mz + a, 4 * n, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && intensity)
            e = cudaMemcpyAsync(intensity, m->d_int + a, 4 * n, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return HC_ERR_CUDA;
    }
    else if (n)
    {
        if (mz) std::memcpy(mz, m->mz.data() + a, 4 * n);
        if (intensity) std::memcpy(intensity, m->intn.data() + a, 4 * n);
    }
    for (uint32_t k = 0; k < count; k++)
    {
        if (prec) prec[k] = m->prec[first + k];
        if (z) z[k] = m->z[first + k];
        if (rtime) rtime[k] = m->rtime[first + k];
    }
    return HC_SUCCESS;
}

extern "C" int hc_ms2_close(hc_ms2 *m)
{
    if (!m) return HC_SUCCESS;
    if (m->d_mz)
    {
        // (no call on m leaves work that reads it behind)
        const BesideCapture beside;
        cudaSetDevice(m->device);
        cudaFree(m->d_mz);
    }
    delete m;
    return HC_SUCCESS;
}

extern "C" int hc_ms2_extract(hc_ctx *ctx, hc_ms2 *m, uint32_t first, uint32_t count, uint32_t *idx, uint32_t *moz,
                              uint32_t *intensity, float *precurse, int32_t *charges, float *rtimes, uint32_t *nout,
                              uint64_t *npeaks)
{
    if (!ctx || !m || !idx) return HC_ERR_INVLD_PTR;
    const uint32_t total = (uint32_t)m->prec.size();
    if (first > total) return set_error(ctx, HC_ERR_INVLD_SIZE, "hc_ms2_extract: first spectrum past the end");
    const uint32_t n = count < total - first ? count : total - first;  // extractbatch clamps (msquery.cpp:254-258)
    if (nout) *nout = n;
    if (npeaks) *npeaks = 0;
    for (uint32_t k = 0; k < n; k++)
    {
        const uint32_t s = first + k;
        const uint32_t zu = m->z[s];
        if (precurse) precurse[k] = (float)m->prec[s];
        if (charges) charges[k] = (int32_t)(1u > zu ? 1u : zu);                  // MAX(1, Z), unsigned compare
        if (rtimes) rtimes[k] = (float)(0.0 > m->rtime[s] ? 0.0 : m->rtime[s]);  // MAX(0.0, rtime)
    }
    idx[0] = 0;
    if (n == 0) return HC_SUCCESS;
    const BesideCapture beside;
    cudaSetDevice(ctx->device);
    cudaStream_t st = ctx->stream;
    const uint64_t r0 = m->off[first], r1 = m->off[first + n];
    const size_t nraw = (size_t)(r1 - r0), room = (size_t)n * HC_QALEN;
    bool longer = false;
    for (uint32_t k = 0; k < n && !longer; k++) longer = m->off[first + k + 1] - m->off[first + k] > kPickCap;
    const bool there = m->d_mz && m->device == ctx->device;  // parsed on this device
    if (!there)
    {
        const int rc = peaks_to_host(ctx, m);
        if (rc) return rc;
    }
    PoolScratch scr(ctx);
    uint64_t *d_off;
    uint32_t *d_mz = nullptr, *d_int = nullptr, *d_idx, *d_kmz, *d_kint, *d_omz, *d_oint;
    HC_CUDA(ctx, scr.alloc(&d_off, (size_t)n + 1));
    HC_CUDA(ctx, scr.alloc(&d_idx, (size_t)n + 2));
    // (k_pick_long sorts in place: a copy)
    if (!there || longer)
    {
        HC_CUDA(ctx, scr.alloc(&d_mz, nraw));
        HC_CUDA(ctx, scr.alloc(&d_int, nraw));
    }
    HC_CUDA(ctx, scr.alloc(&d_kmz, room));
    HC_CUDA(ctx, scr.alloc(&d_kint, room));
    HC_CUDA(ctx, scr.alloc(&d_omz, room));
    HC_CUDA(ctx, scr.alloc(&d_oint, room));
    HC_CUDA(ctx, cudaMemcpyAsync(d_off, m->off.data() + first, 8ull * (n + 1), cudaMemcpyHostToDevice, st));
    if (nraw && d_mz)
    {
        HC_CUDA(ctx, cudaMemcpyAsync(d_mz, there ? m->d_mz + r0 : m->mz.data() + r0, 4ull * nraw, cudaMemcpyDefault, st));
        HC_CUDA(ctx, cudaMemcpyAsync(d_int, there ? m->d_int + r0 : m->intn.data() + r0, 4ull * nraw, cudaMemcpyDefault, st));
    }
    const uint32_t *r_mz = there ? m->d_mz + r0 : d_mz, *r_int = there ? m->d_int + r0 : d_int;
    const uint32_t base_int = (uint32_t)ctx->p.base_int, min_int = (uint32_t)ctx->p.min_int;
    constexpr int kPickSmem = kPickWarps * (int)sizeof(PickSmem);
    HC_CUDA(ctx, cudaFuncSetAttribute(k_pick, cudaFuncAttributeMaxDynamicSharedMemorySize, kPickSmem));
    k_pick<<<(n + kPickWarps - 1) / kPickWarps, kPickWarps * 32, kPickSmem, st>>>(d_off, r_mz, r_int, n, base_int, min_int,
                                                                               d_idx + 1, d_kmz, d_kint);
    if (longer)
        k_pick_long<<<(n + 127) / 128, 128, 0, st>>>(d_off, d_mz, d_int, n, base_int, min_int, d_idx + 1, d_kmz, d_kint);
    k_scan<<<1, 1024, 0, st>>>(d_idx, n);
    k_pick_copy<<<(n + 7) / 8, 256, 0, st>>>(d_kmz, d_kint, n, d_idx, d_omz, d_oint);
    HC_CUDA(ctx, cudaGetLastError());
    uint32_t bad = 0;
    HC_CUDA(ctx, cudaMemcpyAsync(idx, d_idx, 4ull * (n + 1), cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaMemcpyAsync(&bad, d_idx + n + 1, 4, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    if (bad) return set_error(ctx, HC_ERR_CUDA, "hc_ms2_extract: peak sort stack exhausted");
    const uint32_t kept = idx[n];
    if (kept && moz) HC_CUDA(ctx, cudaMemcpyAsync(moz, d_omz, 4ull * kept, cudaMemcpyDeviceToHost, st));
    if (kept && intensity) HC_CUDA(ctx, cudaMemcpyAsync(intensity, d_oint, 4ull * kept, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    if (npeaks) *npeaks = kept;
    return HC_SUCCESS;
}
