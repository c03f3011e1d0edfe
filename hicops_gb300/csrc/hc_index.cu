// Device construction of the SLM index of one peptide length
// (DSLIM_Construct, source/core/dslim.cpp:46-138):
//   0. entries (base peptides, then their variable-mod variants) enumerated
//      on the device (LBE_GeneratePeps, lbe_internal.cpp:204-229, and
//      MODS_GenerateMods, mods.cpp:448-496),
//   1. entries sorted by mass on the device (stable LSD radix sort; the
//      reference uses std::sort, lbe_internal.cpp:184-187),
//   2. ion keys of every entry from integer tables (UTILS_GenerateSpectrum /
//      UTILS_GenerateModSpectrum, utils.cpp:231-505, with the legality rules
//      of DSLIM_ConstructChunk, dslim.cpp:296-323),
//   3. postings iA = ion ids stably sorted by key (the reference's key/value
//      quicksort + per-bucket sort, dslim.cpp:361-388 and 452-482, leave ids
//      ascending inside every bucket: a stable sort gives exactly that),
//   4. bucket offsets bA from the sorted keys (the exclusive scan of
//      dslim.cpp:97-125).
//
// A length of a small database takes some 30 launches, of a large one 45, of 2 to
// 40 us each, every one after the other. Each starts under the end of the one before
// (launch_after), which shortens the gap between two from some 2 us: 34 lengths of
// 20,000 peptides 9.0 -> 7.6 ms, of 500,000 with variable M-oxidation 25.0 -> 22.9.
#include <cstdio>

#include <algorithm>
#include <vector>

#include "hc_device.cuh"
#include "hc_internal.h"

namespace hc {
namespace {

constexpr int kRsThreads = 512;
constexpr int kRsLong = 16, kRsShort = 4;  // items a thread of a long and of a short sort
constexpr int kRsMaxBits = 11;
constexpr int kRsWarps = kRsThreads / 32;

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---- stable LSD radix sort, digits of 8 to 11 bits -------------------------
// Bound by its bytes: a pass reads the keys twice and moves 8 bytes an item. The
// ion keys' 19 bits take two passes of 10 instead of three of 8, and a CTA puts
// its 8192 items in digit order in shared memory before it writes them, so that a
// digit's items leave as one run (32 bytes on average at 10 bits) instead of a
// 4-byte write each: 7.0 ms of sorting for a 500,000-peptide database (115 M postings
// in 34 lengths, entries' masses included), against 10.6 ms with 8-bit digits written
// item by item and a scan of three launches. With the ranking and the tile sizes below
// its build takes 21.8 ms against 22.7.

template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kRsThreads) k_rs_upsweep(const uint32_t *__restrict__ keys, size_t n, int shift,
                                                          uint32_t *__restrict__ tile_hist, uint32_t ntiles)
{
    after_predecessor();
    release_successor();
    constexpr int R = 1 << BITS, kTile = kRsThreads * ITEMS;
    __shared__ uint32_t h[R];
    for (int i = threadIdx.x; i < R; i += kRsThreads) h[i] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kTile;
#pragma unroll
    for (int i = 0; i < ITEMS; i++)
    {
        size_t idx = base + (size_t)i * kRsThreads + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & (R - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < R; d += kRsThreads) tile_hist[(size_t)d * ntiles + blockIdx.x] = h[d];
}

template <int BITS, int ITEMS>
struct RsSmem
{
    uint16_t whist[kRsWarps][1 << BITS];  // a warp's items per digit so far, then what precedes them in the tile
    uint32_t goff[1 << BITS];             // from a place in the tile's digit order to its place in the output
    uint32_t wsum[kRsWarps];
    uint32_t key[kRsThreads * ITEMS], val[kRsThreads * ITEMS];  // the tile in digit order
};

// Stable ranking: warp w owns items [w*32*ITEMS, (w+1)*32*ITEMS) of the tile in order;
// inside a round of 32 items, lanes with equal digits are ranked by lane id (a ballot
// a bit of the digit; with a match instruction, slow where a warp's 32 digits differ,
// a pass over 3.4 M ion keys took 47 us against 41), rounds advance a per-warp digit counter, and the
// warps' counters are scanned per digit, then over the digits.
template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kRsThreads) k_rs_downsweep(const uint32_t *__restrict__ keys_in,
                                                            const uint32_t *__restrict__ vals_in,
                                                            uint32_t *__restrict__ keys_out,
                                                            uint32_t *__restrict__ vals_out, size_t n, int shift,
                                                            const uint32_t *__restrict__ tile_off, uint32_t ntiles,
                                                            int write_keys)
{
    after_predecessor();
    release_successor();
    constexpr int R = 1 << BITS, kTile = kRsThreads * ITEMS;
    constexpr int kPer = (R + kRsThreads - 1) / kRsThreads;  // digits per thread (consecutive)
    extern __shared__ __align__(16) unsigned char rsm[];
    RsSmem<BITS, ITEMS> &S = *reinterpret_cast<RsSmem<BITS, ITEMS> *>(rsm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < kRsWarps * R / 2; i += kRsThreads) reinterpret_cast<uint32_t *>(&S.whist[0][0])[i] = 0;
    __syncthreads();
    const size_t tile0 = (size_t)blockIdx.x * kTile;
    const size_t base = tile0 + (size_t)warp * (ITEMS * 32);
    uint32_t k[ITEMS], v[ITEMS];
    uint16_t rank[ITEMS];
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int r = 0; r < ITEMS; r++)
    {
        const size_t idx = base + (size_t)r * 32 + lane;
        const bool ok = idx < n;
        k[r] = ok ? keys_in[idx] : 0u;
        v[r] = ok ? (vals_in ? vals_in[idx] : (uint32_t)idx) : 0u;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; r++)
    {
        const bool ok = base + (size_t)r * 32 + lane < n;
        const uint32_t d = (k[r] >> shift) & (R - 1);
        uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
        for (int b = 0; b < BITS; b++)
        {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? m : ~m;
        }
        const uint32_t before = ok ? S.whist[warp][d] : 0u;
        rank[r] = (uint16_t)(before + __popc(peers & lt));
        __syncwarp();
        if (ok && (peers >> lane) == 1u)  // highest lane of the group
            S.whist[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // per digit: what precedes each warp's items; over the digits: where each starts
    uint32_t cnt[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; j++)
    {
        const int d = tid * kPer + j;
        cnt[j] = 0;
        if (d < R)
            for (int w = 0; w < kRsWarps; w++)
            {
                const uint32_t c = S.whist[w][d];
                S.whist[w][d] = (uint16_t)cnt[j];
                cnt[j] += c;
            }
        sum += cnt[j];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) S.wsum[warp] = x;
    __syncthreads();
    uint32_t at = x - sum;
    for (int w = 0; w < warp; w++) at += S.wsum[w];
#pragma unroll
    for (int j = 0; j < kPer; j++)
    {
        const int d = tid * kPer + j;
        if (d < R)
        {
            S.goff[d] = tile_off[(size_t)d * ntiles + blockIdx.x] - at;
            for (int w = 0; w < kRsWarps; w++) S.whist[w][d] = (uint16_t)(S.whist[w][d] + at);
        }
        at += cnt[j];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++)
        if (base + (size_t)r * 32 + lane < n)
        {
            const uint32_t p = (uint32_t)S.whist[warp][(k[r] >> shift) & (R - 1)] + rank[r];
            S.key[p] = k[r];
            S.val[p] = v[r];
        }
    __syncthreads();
    const uint32_t items = (uint32_t)min((size_t)kTile, n - tile0);
    for (uint32_t i = tid; i < items; i += kRsThreads)
    {
        const uint32_t key = S.key[i], dst = S.goff[(key >> shift) & (R - 1)] + i;
        if (write_keys) keys_out[dst] = key;
        vals_out[dst] = S.val[i];
    }
}

// Up to kSmallSort masses in one CTA: their positions in ascending order (of the
// float total order, then of position: stable). Three passes of the sort above are
// nine launches or more; 600 masses take 11 us here, four 8-bit passes took 58.
constexpr uint32_t kSmallSort = 8192;

__device__ __forceinline__ uint32_t mass_key(float m)
{
    const uint32_t b = __float_as_uint(m);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);  // total order of floats
}

__global__ void __launch_bounds__(1024) k_sort_masses(const float *__restrict__ mass, uint32_t n, uint32_t *__restrict__ perm)
{
    after_predecessor();
    release_successor();
    extern __shared__ __align__(16) unsigned char msm[];
    unsigned long long *key = reinterpret_cast<unsigned long long *>(msm);
    uint32_t P = 2;
    while (P < n) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x)
        key[i] = i < n ? ((unsigned long long)mass_key(mass[i]) << 32) | i : ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1)
        {
            for (uint32_t t = threadIdx.x; t < P / 2; t += blockDim.x)
            {
                const uint32_t a = 2 * t - (t & (j - 1)), b = a + j;
                const unsigned long long x = key[a], y = key[b];
                if ((x > y) == ((a & k) == 0u))
                {
                    key[a] = y;
                    key[b] = x;
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) perm[i] = (uint32_t)key[i];
}

// ---- exclusive scan of u32 (in place), recursive over block sums ----------
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

// four words from a + i on (as one load where `a` is 16-byte aligned), 0 past n
__device__ __forceinline__ uint4 load4(const uint32_t *a, size_t i, size_t n, bool al)
{
    if (al && i + 4 <= n) return *reinterpret_cast<const uint4 *>(a + i);
    return make_uint4(i < n ? a[i] : 0u, i + 1 < n ? a[i + 1] : 0u, i + 2 < n ? a[i + 2] : 0u, i + 3 < n ? a[i + 3] : 0u);
}

__device__ __forceinline__ void store4(uint32_t *a, size_t i, size_t n, bool al, const uint4 &v)
{
    if (al && i + 4 <= n)
    {
        *reinterpret_cast<uint4 *>(a + i) = v;
        return;
    }
    if (i < n) a[i] = v.x;
    if (i + 1 < n) a[i + 1] = v.y;
    if (i + 2 < n) a[i + 2] = v.z;
    if (i + 3 < n) a[i + 3] = v.w;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(uint32_t *__restrict__ a, size_t n, uint32_t *__restrict__ sums)
{
    after_predecessor();
    release_successor();
    __shared__ uint32_t wsum[32];
    static_assert(kScanItems == 4, "four words a thread");
    const size_t at = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    const bool al = ((uintptr_t)a & 15) == 0;
    const uint4 x = load4(a, at, n, al);
    const uint32_t t = x.x + x.y + x.z + x.w;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t s = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    if (warp == 0)
    {
        uint32_t w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        wsum[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = s - t + (warp ? wsum[warp - 1] : 0u);
    store4(a, at, n, al, make_uint4(excl, excl + x.x, excl + x.x + x.y, excl + x.x + x.y + x.z));
    if (threadIdx.x == kScanThreads - 1 && sums) sums[blockIdx.x] = excl + t;
}

// adds to a tile what precedes it: its scanned sum, or, up to kScanTile tiles
// (raw), the sums of the tiles before it, added up here (one launch less)
__global__ void __launch_bounds__(kScanThreads) k_scan_add(uint32_t *__restrict__ a, size_t n,
                                                          const uint32_t *__restrict__ sums, int raw)
{
    after_predecessor();
    release_successor();
    __shared__ uint32_t part[kScanThreads / 32];
    const size_t at = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    const bool al = ((uintptr_t)a & 15) == 0;
    const uint4 x = load4(a, at, n, al);
    uint32_t off = 0;
    if (raw)
    {
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kScanThreads) off += sums[i];
        off = __reduce_add_sync(0xFFFFFFFFu, off);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = off;
        __syncthreads();
        off = __reduce_add_sync(0xFFFFFFFFu, part[threadIdx.x & 31]);
    }
    else
        off = sums[blockIdx.x];
    store4(a, at, n, al, make_uint4(x.x + off, x.y + off, x.z + off, x.w + off));
}

// Words of one level's sums, to whole 128-byte lines: the next level's lie behind them, and
// a level is scanned in place under a successor that has started (see after_predecessor).
constexpr size_t scan_level_words(size_t n) { return (n + 31) / 32 * 32; }

cudaError_t scan_exclusive(uint32_t *a, size_t n, uint32_t *tmp, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const size_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 1)
    {
        launch_after(k_scan_tiles, 1, kScanThreads, 0, st, a, n, nullptr);
        return cudaGetLastError();
    }
    launch_after(k_scan_tiles, (unsigned)nb, kScanThreads, 0, st, a, n, tmp);
    const bool raw = nb <= (size_t)kScanTile;
    if (!raw)
    {
        const cudaError_t e = scan_exclusive(tmp, nb, tmp + scan_level_words(nb), st);
        if (e != cudaSuccess) return e;
    }
    launch_after(k_scan_add, (unsigned)nb, kScanThreads, 0, st, a, n, tmp, raw ? 1 : 0);
    return cudaGetLastError();
}

size_t scan_tmp_words(size_t n)
{
    size_t t = 0;
    while (n > (size_t)kScanTile)
    {
        n = (n + kScanTile - 1) / kScanTile;
        t += scan_level_words(n);
    }
    return t + 16;
}

// Items a thread sorts. The long sort's 8192-item tiles leave SMs idle below one a
// SM, and what a CTA does once per digit is then all there is: 45,000 masses are six
// tiles, 12.7 us a pass against 6.8 in 2048-item tiles, a small database's 34 lengths
// 7.3 ms against 6.7. Up to a short tile for every SM the sort is short (twice as many,
// or long tiles of 4096 or 6144: no faster).
int radix_items(const hc_ctx *ctx, size_t n)
{
    return n > (size_t)ctx->sm_count * kRsThreads * kRsShort ? kRsLong : kRsShort;
}

template <int BITS, int ITEMS>
cudaError_t radix_pass_of(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, size_t n, int shift,
                          uint32_t *hist, uint32_t *scan_tmp, int write_keys, cudaStream_t st)
{
    const uint32_t ntiles = (uint32_t)((n + kRsThreads * ITEMS - 1) / (kRsThreads * ITEMS));
    constexpr size_t smem = sizeof(RsSmem<BITS, ITEMS>);
    cudaError_t e = cudaFuncSetAttribute(k_rs_downsweep<BITS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    launch_after(k_rs_upsweep<BITS, ITEMS>, ntiles, kRsThreads, 0, st, kin, n, shift, hist, ntiles);
    if ((e = scan_exclusive(hist, (size_t)ntiles << BITS, scan_tmp, st)) != cudaSuccess) return e;
    launch_after(k_rs_downsweep<BITS, ITEMS>, ntiles, kRsThreads, smem, st, kin, vin, kout, vout, n, shift, hist,
                 ntiles, write_keys);
    return cudaGetLastError();
}

template <int BITS, class... A>
cudaError_t radix_pass(int items, A... args)
{
    return items == kRsLong ? radix_pass_of<BITS, kRsLong>(args...) : radix_pass_of<BITS, kRsShort>(args...);
}

// words of `hist` a sort of up to n items needs
size_t radix_hist_words(const hc_ctx *ctx, size_t n)
{
    const size_t shortest = std::min(n, (size_t)ctx->sm_count * kRsThreads * kRsShort);
    return std::max((n + kRsThreads * kRsLong - 1) / (kRsThreads * kRsLong),
                    (shortest + kRsThreads * kRsShort - 1) / (kRsThreads * kRsShort))
           << kRsMaxBits;
}

// Sorts (keys, vals) by the low `bits` bits of the keys, stably. Ping-pongs
// between the given buffers (all four must be valid, n words each); returns
// which pair holds the result (0 or 1). With positions_as_values the input
// values are not read: value i is the input position i.
cudaError_t radix_sort(const hc_ctx *ctx, uint32_t *keys0, uint32_t *keys1, uint32_t *vals0, uint32_t *vals1, size_t n,
                       int bits, uint32_t *hist, uint32_t *scan_tmp, cudaStream_t st, int *which,
                       int *launches, bool keys_out, bool positions_as_values)
{
    int cur = 0;
    const uint32_t *vin = positions_as_values ? nullptr : vals0;
    const int items = radix_items(ctx, n);
    const int passes = (bits + kRsMaxBits - 1) / kRsMaxBits, digit = std::max(8, (bits + passes - 1) / passes);
    for (int shift = 0; shift < bits; shift += digit)
    {
        uint32_t *kin = cur ? keys1 : keys0, *kout = cur ? keys0 : keys1;
        uint32_t *vout = cur ? vals0 : vals1;
        if (n)
        {
            const int write_keys = shift + digit >= bits && !keys_out ? 0 : 1;
            const cudaError_t e =
                digit == 8    ? radix_pass<8>(items, kin, vin, kout, vout, n, shift, hist, scan_tmp, write_keys, st)
                : digit == 9  ? radix_pass<9>(items, kin, vin, kout, vout, n, shift, hist, scan_tmp, write_keys, st)
                : digit == 10 ? radix_pass<10>(items, kin, vin, kout, vout, n, shift, hist, scan_tmp, write_keys, st)
                              : radix_pass<11>(items, kin, vin, kout, vout, n, shift, hist, scan_tmp, write_keys, st);
            if (e != cudaSuccess) return e;
            *launches += 3;
        }
        vin = vout;
        cur ^= 1;
    }
    *which = cur;
    return cudaGetLastError();
}

// ---- entries ---------------------------------------------------------------

// Entry enumeration on the device, one thread per peptide. The base entry of
// peptide i (LBE_GeneratePeps, lbe_internal.cpp:204-229) is entry i; its
// variable-mod variants (MODS_GenerateMods, mods.cpp:448-496) follow all base
// entries, peptide by peptide, in the order of MODS_ModList's depth-first walk
// (mods.cpp:333-384): at each modifiable position the branch that modifies it
// comes before the one that skips it, and a variant is emitted as each mod is
// added. Here the walk is a loop over a stack of chosen positions. The first
// pass (mass == nullptr) counts the variants per peptide; the second writes
// them at npep + voff[i].
constexpr int kEnumThreads = 128;

__global__ void __launch_bounds__(kEnumThreads) k_enum_entries(const uint8_t *__restrict__ seqs, uint32_t L, uint32_t npep, EnumConst ec,
                               const uint32_t *__restrict__ voff, uint32_t *__restrict__ vcount,
                               float *__restrict__ mass, uint32_t *__restrict__ seqid,
                               uint64_t *__restrict__ sites, uint32_t *__restrict__ modnum)
{
    after_predecessor();
    release_successor();
    // the block's sequences, read together (a thread's own are L bytes apart)
    __shared__ uint8_t sh[kEnumThreads * 64];
    const size_t at0 = (size_t)blockIdx.x * kEnumThreads * L, all = (size_t)npep * L;
    const uint32_t bytes = at0 < all ? (uint32_t)min((size_t)kEnumThreads * L, all - at0) : 0u;
    for (uint32_t b = threadIdx.x; b < bytes; b += kEnumThreads) sh[b] = __ldg(seqs + at0 + b);
    // the residue tables too: lanes index them apart, which kernel parameters serialise
    __shared__ float2 mtab[26];  // residue, static mod
    __shared__ int8_t cond[26];
    if (threadIdx.x < 26)
    {
        mtab[threadIdx.x] = make_float2(ec.aa[threadIdx.x], ec.stat[threadIdx.x]);
        cond[threadIdx.x] = ec.cond_of[threadIdx.x];
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * kEnumThreads + threadIdx.x;
    if (i == npep && vcount) vcount[i] = 0;  // the scan makes it the total
    if (i >= npep) return;
    const uint8_t *s = sh + threadIdx.x * L;
    // UTILS_CalculatePepMass: two float additions per residue, in order
    // (and a bit per modifiable virtual position, see below)
    float pm = ec.h2o;
    uint64_t can = ec.nterm >= 0 ? 1ull : 0ull;
    for (uint32_t l = 0; l < L; l++)
    {
        can |= (uint64_t)(cond[s[l] - 'A'] >= 0) << (l + 1);
        const float2 m = mtab[s[l] - 'A'];
        pm += m.x;
        pm += m.y;
    }
    const bool write = mass != nullptr;
    if (write)
    {
        mass[i] = pm;
        seqid[i] = i;
        sites[i] = 0;
        modnum[i] = 0;
    }
    uint32_t k = 0;
    if (ec.vmods > 0 && ec.nmods > 0)
    {
        int cap[HC_MAX_MODS];
        for (int m = 0; m < HC_MAX_MODS; m++) cap[m] = (int)ec.limit[m];
        uint8_t pos[64];
        uint32_t d = 0, mn = 0;
        uint64_t st = 0;
        uint32_t start = 0;
        const uint64_t at = write ? (uint64_t)npep + voff[i] : 0;  // (read only with mods)
        for (;;)
        {
            // virtual positions: q = 0 is the N-terminus (a '^' mod, an
            // extension; site bit kNtermBit), q >= 1 is residue q - 1
            int p = -1;
            if (d < ec.vmods && d < 64)
                for (uint64_t t = can & (~0ull << start); t; t &= t - 1)
                {
                    const int q = __ffsll((long long)t) - 1;
                    if (cap[q == 0 ? ec.nterm : cond[s[q - 1] - 'A']] > 0)
                    {
                        p = q;
                        break;
                    }
                }
            if (p >= 0)
            {
                const int c = p == 0 ? ec.nterm : cond[s[p - 1] - 'A'];
                cap[c] -= 1;
                pos[d] = (uint8_t)p;
                mn += (1u << ((4u * d) & 31u)) * (uint32_t)(1 + c);  // shift count taken mod 32, as the CPU does
                st |= 1ull << (p == 0 ? kNtermBit : p - 1);
                d++;
                if (write)
                {
                    // UTILS_CalculateModMass: only the first mod's mass is added
                    const uint64_t e = at + k;
                    mass[e] = pm + ec.modadd[(mn & 0xF) - 1];
                    seqid[e] = i;
                    sites[e] = st;
                    modnum[e] = mn;
                }
                k++;
                start = (uint32_t)p + 1;
            }
            else
            {
                if (d == 0) break;
                d--;
                const uint32_t q = pos[d];
                const int c = q == 0 ? ec.nterm : cond[s[q - 1] - 'A'];
                cap[c] += 1;
                mn -= (1u << ((4u * d) & 31u)) * (uint32_t)(1 + c);
                st &= ~(1ull << (q == 0 ? kNtermBit : q - 1));
                start = q + 1;
            }
        }
    }
    if (!write) vcount[i] = k;
}

__global__ void k_mass_keys(const float *__restrict__ mass, uint32_t n, uint32_t *__restrict__ keys)
{
    after_predecessor();
    release_successor();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        keys[i] = mass_key(mass[i]);
}

__global__ void k_gather_entries(const uint32_t *__restrict__ perm, uint32_t n, const float *mass_in,
                                 const uint32_t *seqid_in, const uint64_t *sites_in,
                                 const uint32_t *modnum_in, float *mass, uint32_t *seqid,
                                 uint64_t *sites, uint32_t *modnum)
{
    after_predecessor();
    release_successor();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        const uint32_t j = perm[i];
        mass[i] = mass_in[j];
        seqid[i] = seqid_in[j];
        sites[i] = sites_in[j];
        modnum[i] = modnum_in[j];
    }
}

// ---- ion keys ----------------------------------------------------------------
// One thread per (entry, series, charge): writes the L-1 keys of one b or y
// series. Layout per entry: [b z=1][b z=2]..[y z=1][y z=2].., each L-1 long
// (utils.cpp:251-252).
__global__ void k_ion_keys(const IonTables *__restrict__ gt, uint32_t L, uint32_t n,
                           const float *__restrict__ mass, const uint32_t *__restrict__ seqid,
                           const uint64_t *__restrict__ sites, const uint32_t *__restrict__ modnum,
                           const uint8_t *__restrict__ seqs, uint32_t *__restrict__ keys)
{
    after_predecessor();
    release_successor();
    __shared__ IonTables t;
    for (int i = threadIdx.x; i < (int)(sizeof(IonTables) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t *>(&t)[i] = reinterpret_cast<const uint32_t *>(gt)[i];
    __syncthreads();
    const uint32_t maxz = t.maxz, nser = 2 * maxz;
    const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (uint64_t)n * nser) return;
    const uint32_t k = (uint32_t)(gid / nser), s = (uint32_t)(gid % nser);
    const bool isY = s >= maxz;
    const uint32_t z = isY ? s - maxz : s;
    const uint32_t Lm1 = L - 1, speclen = nser * Lm1;
    uint32_t *out = keys + (size_t)k * speclen + (isY ? maxz * Lm1 : 0) + z * Lm1;
    const uint8_t *seq = seqs + (size_t)seqid[k] * L;
    const double m = mass[k];
    const double minm = t.min_mass, maxm = t.max_mass;
    const uint32_t top = t.max_mass * t.scale;
    const uint32_t mn = modnum[k];
    bool legal = (m >= minm && m <= maxm);
    // mass exactly on a bound: the reference reads an uninitialised spectrum
    if (mn != 0 && legal && !(m > minm && m < maxm)) legal = false;
    if (!legal)
    {
        for (uint32_t l = 0; l < Lm1; l++) out[l] = 0;
        return;
    }
    if (mn == 0)
    {
        uint32_t v = isY ? t.yf[seq[L - 1] - 'A'][z] : t.bf[seq[0] - 'A'][z];
        out[0] = v >= top ? top - 1 : v;
        for (uint32_t l = 1; l < Lm1; l++)
        {
            const uint8_t a = isY ? seq[L - 1 - l] : seq[l];
            v += t.inc[a - 'A'][z];
            out[l] = v >= top ? top - 1 : v;
        }
        return;
    }
    // variable mods (utils.cpp:407-500): undivided running sums, plus the
    // masses of the first `counter` mods (b) or last `counter` mods (y),
    // then integer division by the charge
    uint32_t mods[16];
    int seen = 0;
    {
        uint32_t bm = mn;
        for (int i = 0; i < 8; i++)
        {
            int q = (int)(bm & 0xF) - 1;
            bm >>= 4;
            if (q != -1) mods[seen++] = t.mod_mass[q & 15];
        }
    }
    const uint64_t st = sites[k];
    uint32_t v = isY ? t.yfm[seq[L - 1] - 'A'][z] : t.bfm[seq[0] - 'A'][z];
    uint32_t madd = 0;
    int cnt = 0;
    // an N-terminal mod (extension) is the first mod and part of every b ion
    if (!isY && ((st >> kNtermBit) & 1ull) && seen > 0)
    {
        madd = mods[0];
        cnt = 1;
    }
    for (uint32_t l = 0; l < Lm1; l++)
    {
        const uint32_t pos = isY ? (L - 1 - l) : l;
        if (l > 0) v += t.incm[seq[pos] - 'A'];
        if (((st >> pos) & 1ull) && cnt < seen)
        {
            madd += isY ? mods[seen - 1 - cnt] : mods[cnt];
            cnt++;
        }
        uint32_t o = (v + madd) / (z + 1);
        out[l] = o >= top ? top - 1 : o;
    }
}

// bA[b] = first position of the sorted keys whose key is >= b, b in [0, nb]
// (the exclusive scan of the bucket counts, dslim.cpp:97-125): one thread per
// bucket, a lower bound over the keys. Neighbouring buckets search the same
// stretch of keys, so the probes share cache lines.
__global__ void k_bucket_bounds(const uint32_t *__restrict__ skeys, size_t M, uint32_t nb,
                                uint32_t *__restrict__ bA)
{
    after_predecessor();
    release_successor();
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= nb;
         b += (uint64_t)gridDim.x * blockDim.x)
    {
        size_t lo = 0, hi = M;
        while (lo < hi)
        {
            const size_t m = lo + ((hi - lo) >> 1);
            if (__ldg(skeys + m) < (uint32_t)b) lo = m + 1;
            else hi = m;
        }
        bA[b] = (uint32_t)lo;
    }
}

// Row table over the query postings: rows[b * stride + k] = first position in
// bucket b whose entry is >= k * kRowG (a lower bound on k * kRowG << 3).
// Column 0 is qA[b], column stride-1 is qA[b+1] (padding decodes past every
// entry, so it never precedes a lower bound).
__global__ void k_row_table(const uint32_t *__restrict__ qA, const uint32_t *__restrict__ qp, uint32_t nb,
                            uint32_t stride, uint32_t n, uint32_t *__restrict__ rows)
{
    after_predecessor();
    release_successor();
    const uint64_t total = (uint64_t)nb * stride;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t b = (uint32_t)(t / stride), k = (uint32_t)(t - (uint64_t)b * stride);
        uint32_t lo = __ldg(qA + b), hi = __ldg(qA + b + 1);
        if (k == stride - 1) lo = hi;
        else if (k > 0)
        {
            const uint32_t v = min(k * kRowG, n) << kQpEntryShift;
            while (lo < hi)
            {
                const uint32_t m = lo + ((hi - lo) >> 1);
                if (__ldg(qp + m) < v) lo = m + 1;
                else hi = m;
            }
        }
        rows[t] = lo;
    }
}

// padded bucket sizes: ceil4(bA[b+1] - bA[b]); entry nb is 0 (the scan makes it the total)
__global__ void k_pad_counts(const uint32_t *__restrict__ bA, uint32_t nb, uint32_t *__restrict__ pc)
{
    after_predecessor();
    release_successor();
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x)
        pc[b] = b < nb ? ((bA[b + 1] - bA[b] + 3u) & ~3u) : 0u;
}

// Division of the ids by the postings of an entry: multiply and shift below
// 2^31 ids (division_magic), the plain quotient past it.
struct IdDiv
{
    uint32_t d, magic, sh;
    bool fast;
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const { return fast ? __umulhi(x, magic) >> sh : x / d; }
};

// the charge of a query posting's ion when it is a y1 ion, else -1;
// ion = series * half + charge * (L - 1) + position
__device__ __forceinline__ int y1_charge(uint32_t ion, uint32_t Lm1, uint32_t half)
{
    int z = -1;
    for (uint32_t y = half, k = 0; y < 2 * half; y += Lm1, k++)
        if (ion == y) z = (int)k;
    return z;
}

// The query postings, a thread per posting: `ids` (entry * speclen + ion) and
// their buckets `keys` in bucket order; posting j of the order goes to
// qA[b] + (j - bA[b]). Bound by its bytes (8 read, 6 written a posting): the
// same with a thread per bucket took 24 ms for 115 M postings (the buckets of the
// y1 ions hold a large share each, walked by one thread), 0.6 ms so.
// Every y1 posting of a classed entry must lie in its class's key bucket;
// bad[e] = 1 marks the entries where one does not (they lose their class).
// A padding id (kQpostPad) is skipped: every posting in front of the first bucket is
// one. qp null: the check only.
__global__ void k_qpost(const uint32_t *__restrict__ ids, const uint32_t *__restrict__ keys, uint32_t total,
                        const uint32_t *__restrict__ bA, const uint32_t *__restrict__ qA, IdDiv div, uint32_t half,
                        uint32_t Lm1, const uint8_t *__restrict__ cls, const ClassKeys *__restrict__ ck,
                        uint8_t *__restrict__ bad, uint32_t *__restrict__ qp, uint16_t *__restrict__ qion)
{
    after_predecessor();
    release_successor();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t id = ids[j];
        if (id == kQpostPad) continue;
        const uint32_t b = keys[j], entry = div(id), ion = id - entry * div.d;
        if (qp)
        {
            const uint32_t q = qA[b] + ((uint32_t)j - bA[b]);
            qp[q] = (entry << kQpEntryShift) | ((ion >= half ? 1u : 0u) << 2);
            qion[q] = (uint16_t)ion;
        }
        const int z = y1_charge(ion, Lm1, half);
        if (z >= 0)
        {
            const uint32_t c = cls[entry];
            if (c != kClassNone && ck->key[c][z] != b) bad[entry] = 1;
        }
    }
}

// the padding after each bucket's postings and after the last bucket
__global__ void k_qpost_pads(const uint32_t *__restrict__ bA, const uint32_t *__restrict__ qA, uint32_t nb,
                             uint32_t *__restrict__ qp, uint16_t *__restrict__ qion)
{
    after_predecessor();
    release_successor();
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x)
    {
        const uint32_t q0 = b < nb ? qA[b] + (bA[b + 1] - bA[b]) : qA[nb], q1 = b < nb ? qA[b + 1] : qA[nb] + (uint32_t)kIaPad;
        for (uint32_t q = q0; q < q1; q++)
        {
            qp[q] = kQpostPad;
            qion[q] = 0;
        }
    }
}

// The last bucket that starts at or before i: start[b] <= i < start[b + 1]; 0 where i lies in
// front of every bucket.
__device__ __forceinline__ uint32_t bucket_of(const uint32_t *__restrict__ start, uint32_t nb, uint32_t i)
{
    uint32_t lo = 0, hi = nb - 1;
    while (lo < hi)
    {
        const uint32_t m = (lo + hi + 1) >> 1;
        if (__ldg(start + m) <= i) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// the bucket of every posting (postings that were not sorted here)
__global__ void k_bucket_keys(const uint32_t *__restrict__ start, uint32_t nb, uint32_t total, uint32_t *__restrict__ keys)
{
    after_predecessor();
    release_successor();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (uint64_t)gridDim.x * blockDim.x)
        keys[j] = bucket_of(start, nb, (uint32_t)j);
}

// query postings -> ids, position by position (padding: kQpostPad)
__global__ void k_qpost_to_ids(const uint32_t *__restrict__ qp, const uint16_t *__restrict__ qion, uint32_t total,
                               uint32_t speclen, uint32_t *__restrict__ ids)
{
    after_predecessor();
    release_successor();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t x = qp[j];
        ids[j] = x == kQpostPad ? kQpostPad : (x >> kQpEntryShift) * speclen + qion[j];
    }
}

// counts query-posting words that are neither padding nor an (entry < n, ion < speclen)
// pair whose b/y bit matches its ion
__global__ void k_check_qpost(const uint32_t *__restrict__ qp, const uint16_t *__restrict__ qion, size_t total,
                              uint32_t n, uint32_t speclen, uint32_t half, uint32_t *__restrict__ bad)
{
    after_predecessor();
    release_successor();
    uint32_t b = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
    {
        const uint32_t x = qp[i];
        if (x == kQpostPad) continue;
        const uint32_t ion = qion[i];
        if ((x & 3u) || (x >> kQpEntryShift) >= n || ion >= speclen || ((x >> 2) & 1u) != (ion >= half ? 1u : 0u)) b++;
    }
    if (b) atomicAdd(bad, b);
}

// query postings -> ids (the reference's iA), one thread per posting; 0 in front of the first
// bucket (such postings are not kept)
__global__ void k_qpost_ids(const uint32_t *__restrict__ bA, const uint32_t *__restrict__ qA,
                            const uint32_t *__restrict__ qp, const uint16_t *__restrict__ qion, uint32_t nb,
                            uint32_t npost, uint32_t speclen, uint32_t *__restrict__ ids)
{
    after_predecessor();
    release_successor();
    const uint32_t qtotal = qA[nb];
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < npost; j += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t b = bucket_of(bA, nb, (uint32_t)j), s = bA[b], q = qA[b] + ((uint32_t)j - s);
        if ((uint32_t)j < s) ids[j] = 0;
        else if (q < qtotal) ids[j] = (qp[q] >> kQpEntryShift) * speclen + qion[q];
    }
}

// ---- entry classes and the search postings ------------------------------------
// (see ClassKeys in hc_internal.h)

// The class code of one entry: the facts k_ion_keys reads for the first y
// ion (legal mass, mod path, last residue, the mod there); kCodes - 1 for an
// illegal mass, and for a residue byte outside 'A'..'Z' a code no entry's
// postings can match (the build check then leaves it unclassed).
__device__ __forceinline__ uint32_t entry_code(double minm, double maxm, uint32_t L, const uint8_t *seq, double m,
                                               uint32_t mn, uint64_t st)
{
    bool legal = (m >= minm && m <= maxm);
    if (mn != 0 && legal && !(m > minm && m < maxm)) legal = false;
    if (!legal) return kCodes - 1;
    const uint32_t rl = (uint32_t)seq[L - 1] - 'A';
    if (rl >= 26u) return kCodes - 2;
    if (mn == 0) return rl;
    // the last mod, when the last residue carries one (utils.cpp:480-500)
    uint32_t last = 0;
    for (int i = 0; i < 8; i++)
    {
        const uint32_t q = (mn >> (4 * i)) & 0xFu;
        if (q) last = q;
    }
    const uint32_t qy = ((st >> (L - 1)) & 1ull) ? last : 0u;
    return 0x200u | (rl << 4) | qy;
}

__global__ void k_entry_codes(double minm, double maxm, uint32_t L, uint32_t n, const float *__restrict__ mass,
                              const uint32_t *__restrict__ seqid, const uint64_t *__restrict__ sites,
                              const uint32_t *__restrict__ modnum, const uint8_t *__restrict__ seqs,
                              uint16_t *__restrict__ code, uint8_t *__restrict__ used, uint8_t *__restrict__ bad)
{
    after_predecessor();
    release_successor();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t c = entry_code(minm, maxm, L, seqs + (size_t)seqid[k] * L, (double)mass[k], modnum[k], sites[k]);
    code[k] = (uint16_t)c;
    used[c] = 1;
    bad[k] = 0;
}

// (and the 4 bytes past the last entry, which the search reads in fours)
__global__ void k_entry_classes(const uint16_t *__restrict__ code, uint32_t n, const uint8_t *__restrict__ class_of,
                                uint8_t *__restrict__ cls)
{
    after_predecessor();
    release_successor();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n + 4) cls[k] = k < n ? class_of[code[k]] : (uint8_t)kClassNone;
}

__global__ void k_class_fix(uint8_t *__restrict__ cls, const uint8_t *__restrict__ bad, uint32_t n)
{
    after_predecessor();
    release_successor();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n && bad[k]) cls[k] = (uint8_t)kClassNone;
}

// Which postings stay in the search postings (all but padding and the y1
// postings of classed entries): a bit each, in words of 32, and each word's
// count. With the counts scanned, the kept postings before position i are one
// word's sum and a population count, so the flags cost a thirty-second of a
// scan over the postings themselves (three passes of 4 bytes a posting).
__global__ void k_spost_mask(const uint32_t *__restrict__ ids, uint32_t total, IdDiv div, uint32_t half, uint32_t Lm1,
                             const uint8_t *__restrict__ cls, uint32_t nwords, uint32_t *__restrict__ mask,
                             uint32_t *__restrict__ sum)
{
    after_predecessor();
    release_successor();
    const int lane = threadIdx.x & 31;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwords;
         w += ((uint64_t)gridDim.x * blockDim.x) >> 5)
    {
        const uint64_t j = 32 * w + (uint64_t)lane;
        const uint32_t id = j < total ? ids[j] : kQpostPad;
        bool keep = false;
        if (id != kQpostPad)
        {
            const uint32_t entry = div(id), ion = id - entry * div.d;
            keep = y1_charge(ion, Lm1, half) < 0 || cls[entry] == kClassNone;
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, keep);
        if (lane == 0)
        {
            mask[w] = m;
            sum[w] = (uint32_t)__popc(m);
        }
    }
}

// kept postings before position i (sum scanned)
__device__ __forceinline__ uint32_t kept_before(const uint32_t *__restrict__ mask, const uint32_t *__restrict__ sum,
                                                uint32_t i)
{
    return sum[i >> 5] + (uint32_t)__popc(mask[i >> 5] & ((1u << (i & 31u)) - 1u));
}

// the padded size of each bucket's search postings; entry nb is 0 (the scan
// makes it the total)
__global__ void k_spost_counts(const uint32_t *__restrict__ start, const uint32_t *__restrict__ mask,
                               const uint32_t *__restrict__ sum, uint32_t nb, uint32_t *__restrict__ qAs)
{
    after_predecessor();
    release_successor();
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x)
        qAs[b] = b < nb ? ((kept_before(mask, sum, start[b + 1]) - kept_before(mask, sum, start[b]) + 3u) & ~3u) : 0u;
}

// per bucket: what takes a kept posting's rank to its place (off), and the
// padding after the bucket's postings (and after the last bucket)
__global__ void k_spost_pads(const uint32_t *__restrict__ start, const uint32_t *__restrict__ mask,
                             const uint32_t *__restrict__ sum, uint32_t nb, const uint32_t *__restrict__ qAs,
                             uint32_t *__restrict__ off, uint32_t *__restrict__ qps)
{
    after_predecessor();
    release_successor();
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x)
    {
        if (b == nb)
        {
            for (uint32_t q = 0; q < kIaPad; q++) qps[qAs[nb] + q] = kQpostPad;
            break;
        }
        const uint32_t k0 = kept_before(mask, sum, start[b]), k1 = kept_before(mask, sum, start[b + 1]);
        off[b] = qAs[b] - k0;
        for (uint32_t q = qAs[b] + (k1 - k0); q < qAs[b + 1]; q++) qps[q] = kQpostPad;
    }
}

// every kept posting to its place, a thread per posting
__global__ void k_spost_scatter(const uint32_t *__restrict__ ids, const uint32_t *__restrict__ keys, uint32_t total,
                                IdDiv div, uint32_t half, const uint32_t *__restrict__ mask,
                                const uint32_t *__restrict__ sum, const uint32_t *__restrict__ off,
                                uint32_t *__restrict__ qps)
{
    after_predecessor();
    release_successor();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint32_t m = mask[j >> 5];
        if (!((m >> (j & 31u)) & 1u)) continue;
        const uint32_t rank = sum[j >> 5] + (uint32_t)__popc(m & ((1u << (j & 31u)) - 1u));
        const uint32_t id = ids[j], entry = div(id), ion = id - entry * div.d;
        qps[off[keys[j]] + rank] = (entry << kQpEntryShift) | ((ion >= half ? 1u : 0u) << 2);
    }
}

}  // namespace

// The class code of every entry, and room for a mark on those that lose their class.
struct EntryCodes
{
    uint16_t *code;
    uint8_t *bad;
};

static int build_search(hc_ctx *ctx, LenHost &lh, const EntryCodes &ec, const uint32_t *d_ids, const uint32_t *d_keys,
                        uint32_t total, const uint32_t *start, bool write);

// The entries of one length enumerated on the device (k_enum_entries, two
// passes around a scan of the per-peptide variant counts) into fresh SoA
// arrays in generation order; sets lh.n.
static int enumerate_entries(hc_ctx *ctx, LenHost &lh, PoolScratch &out, float **d_m, uint32_t **d_s,
                             uint64_t **d_si, uint32_t **d_mo, int *launches)
{
    cudaStream_t st = ctx->stream;
    const uint32_t npep = lh.npep, L = lh.L;
    EnumConst ec;
    make_enum_const(ctx->p, &ec);
    PoolScratch tmp(ctx);
    uint32_t *cnt = nullptr, *stmp = nullptr;
    uint32_t nvar = 0;
    const unsigned grid = npep / kEnumThreads + 1;
    if (ec.vmods > 0 && ec.nmods > 0 && npep)  // without variable mods there is nothing to count
    {
        HC_CUDA(ctx, tmp.alloc(&cnt, (size_t)npep + 1));
        HC_CUDA(ctx, tmp.alloc(&stmp, scan_tmp_words((size_t)npep + 1)));
        launch_after(k_enum_entries, grid, kEnumThreads, 0, st, lh.d_seqs, L, npep, ec, nullptr, cnt, nullptr,
                     nullptr, nullptr, nullptr);
        (*launches)++;
        HC_CUDA(ctx, scan_exclusive(cnt, (size_t)npep + 1, stmp, st));
        HC_CUDA(ctx, cudaMemcpyAsync(ctx->h_read, cnt + npep, 4, cudaMemcpyDeviceToHost, st));
        HC_CUDA(ctx, cudaStreamSynchronize(st));
        nvar = *static_cast<const uint32_t *>(ctx->h_read);
    }
    const uint64_t n = (uint64_t)npep + nvar;
    if (n >= (1u << 24)) return set_error(ctx, HC_ERR_INVLD_SIZE, "more than 2^24 entries in one length");
    lh.n = (uint32_t)n;
    HC_CUDA(ctx, out.alloc(d_m, n));
    HC_CUDA(ctx, out.alloc(d_s, n));
    HC_CUDA(ctx, out.alloc(d_si, n));
    HC_CUDA(ctx, out.alloc(d_mo, n));
    if (npep)
    {
        launch_after(k_enum_entries, grid, kEnumThreads, 0, st, lh.d_seqs, L, npep, ec, cnt, nullptr, *d_m, *d_s,
                     *d_si, *d_mo);
        (*launches)++;
    }
    HC_CUDA(ctx, cudaGetLastError());
    return HC_SUCCESS;
}

int build_length_device(hc_ctx *ctx, LenHost &lh, const hc_entry *h_entries, bool sort_by_mass)
{
    cudaStream_t st = ctx->stream;
    int launches = 0;
    // entries in generation order: enumerated here, or uploaded from the host
    PoolScratch scr(ctx);
    float *d_m0 = nullptr;
    uint32_t *d_s0 = nullptr, *d_mod0 = nullptr;
    uint64_t *d_site0 = nullptr;
    if (!h_entries)
    {
        const int rc = enumerate_entries(ctx, lh, scr, &d_m0, &d_s0, &d_site0, &d_mod0, &launches);
        if (rc) return rc;
    }
    const uint32_t n = lh.n, L = lh.L;
    const uint32_t speclen = 2 * ctx->p.maxz * (L - 1);
    const size_t M = (size_t)n * speclen;
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale;
    if (M >= 0x80000000ull) return set_error(ctx, HC_ERR_INVLD_SIZE, "more than 2^31 ions in one length");
    if (h_entries && (sort_by_mass && n > 1))
    {
        std::vector<float> hm(n);
        std::vector<uint32_t> hs(n), hmod(n);
        std::vector<uint64_t> hsite(n);
        for (uint32_t i = 0; i < n; i++)
        {
            hm[i] = h_entries[i].mass;
            hs[i] = h_entries[i].seqid;
            hsite[i] = h_entries[i].sites;
            hmod[i] = h_entries[i].modnum;
        }
        HC_CUDA(ctx, scr.alloc(&d_m0, n));
        HC_CUDA(ctx, scr.alloc(&d_s0, n));
        HC_CUDA(ctx, scr.alloc(&d_mod0, n));
        HC_CUDA(ctx, scr.alloc(&d_site0, n));
        HC_CUDA(ctx, cudaMemcpyAsync(d_m0, hm.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(d_s0, hs.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(d_mod0, hmod.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(d_site0, hsite.data(), 8ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaStreamSynchronize(st));
    }
    HC_CUDA(ctx, dalloc(ctx, &lh.d_mass, n));
    HC_CUDA(ctx, dalloc(ctx, &lh.d_seqid, n));
    HC_CUDA(ctx, dalloc(ctx, &lh.d_sites, n));
    HC_CUDA(ctx, dalloc(ctx, &lh.d_modnum, n));
    HC_CUDA(ctx, dalloc(ctx, &lh.d_bA, (size_t)nb + 1));

    // scratch: keys/vals ping-pong, radix histograms, scan temp
    const size_t items = M > n ? M : n;
    uint32_t *k0, *k1, *v0, *v1, *hist, *stmp;
    HC_CUDA(ctx, scr.alloc(&k0, items));
    HC_CUDA(ctx, scr.alloc(&k1, items));
    HC_CUDA(ctx, scr.alloc(&v0, items));
    HC_CUDA(ctx, scr.alloc(&v1, items));
    HC_CUDA(ctx, scr.alloc(&hist, radix_hist_words(ctx, items)));
    HC_CUDA(ctx, scr.alloc(&stmp, scan_tmp_words(radix_hist_words(ctx, items))));

    if (sort_by_mass && n > 1)
    {
        uint32_t *perm = v0;
        if (n <= kSmallSort)
        {
            HC_CUDA(ctx, cudaFuncSetAttribute(k_sort_masses, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              8 * (int)kSmallSort));
            uint32_t room = 2;
            while (room < n) room <<= 1;
            launch_after(k_sort_masses, 1, 1024, 8 * room, st, d_m0, n, perm);
            launches++;
        }
        else
        {
            launch_after(k_mass_keys, (n + 255) / 256, 256, 0, st, d_m0, n, k0);
            int which = 0;
            HC_CUDA(ctx, radix_sort(ctx, k0, k1, v0, v1, n, 32, hist, stmp, st, &which, &launches, false, true));
            perm = which ? v1 : v0;
        }
        launch_after(k_gather_entries, (n + 255) / 256, 256, 0, st, perm, n, d_m0, d_s0, d_site0, d_mod0, lh.d_mass,
                     lh.d_seqid, lh.d_sites, lh.d_modnum);
        launches += 2;
    }
    else if (d_m0)
    {
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_mass, d_m0, 4ull * n, cudaMemcpyDeviceToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_seqid, d_s0, 4ull * n, cudaMemcpyDeviceToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_modnum, d_mod0, 4ull * n, cudaMemcpyDeviceToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_sites, d_site0, 8ull * n, cudaMemcpyDeviceToDevice, st));
    }
    else
    {
        std::vector<float> hm(n);
        std::vector<uint32_t> hs(n), hmod(n);
        std::vector<uint64_t> hsite(n);
        for (uint32_t i = 0; i < n; i++)
        {
            hm[i] = h_entries[i].mass;
            hs[i] = h_entries[i].seqid;
            hsite[i] = h_entries[i].sites;
            hmod[i] = h_entries[i].modnum;
        }
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_mass, hm.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_seqid, hs.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_modnum, hmod.data(), 4ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaMemcpyAsync(lh.d_sites, hsite.data(), 8ull * n, cudaMemcpyHostToDevice, st));
        HC_CUDA(ctx, cudaStreamSynchronize(st));
    }

    // ion keys -> (k0), sorted with ids -> iA, bucket bounds -> bA
    if (M > 0)
    {
        const uint64_t threads = (uint64_t)n * 2 * ctx->p.maxz;
        launch_after(k_ion_keys, (unsigned)((threads + 127) / 128), 128, 0, st, ctx->d_tables, L, n, lh.d_mass,
                     lh.d_seqid, lh.d_sites, lh.d_modnum, lh.d_seqs, k0);
        launches++;
        int bits = 1;
        while ((1ull << bits) < nb) bits++;
        int which = 0;
        HC_CUDA(ctx, radix_sort(ctx, k0, k1, v0, v1, M, bits, hist, stmp, st, &which, &launches, true, true));
        uint32_t *skeys = which ? k1 : k0;
        uint32_t *svals = which ? v1 : v0;
        launch_after(k_bucket_bounds, (unsigned)std::min<uint64_t>((nb + 256) / 256, (uint64_t)ctx->sm_count * 32),
                     256, 0, st, skeys, M, nb, lh.d_bA);
        launches += 1;
        lh.npost = M;
        const int rq = build_query_postings(ctx, lh, svals, skeys);
        if (rq) return rq;
        launches += 4;
    }
    else
    {
        HC_CUDA(ctx, cudaMemsetAsync(lh.d_bA, 0, 4ull * (nb + 1), st));
        lh.npost = 0;
        const int rq = build_query_postings(ctx, lh, nullptr, nullptr);
        if (rq) return rq;
    }
    lh.built = true;
    ctx->lens_dirty = true;
    ctx->epoch++;
    ctx->last_launches = launches + 1;
    return HC_SUCCESS;
}

static IdDiv id_div(uint32_t speclen, uint64_t ids)
{
    IdDiv d{speclen, 0, 0, ids < 0x80000000ull};
    if (d.fast) division_magic(speclen, &d.magic, &d.sh);
    return d;
}

// Where the build reads back to, in pinned memory: the codes seen, a total.
static uint8_t *read_used(hc_ctx *ctx) { return static_cast<uint8_t *>(ctx->h_read); }
static uint32_t *read_total(hc_ctx *ctx) { return reinterpret_cast<uint32_t *>(read_used(ctx) + kCodes); }
static_assert(kCodes + 4 <= kReadBytes, "read-back words");

// The entries' class codes; waits for the codes seen and for the query
// postings' total (qA scanned), read back together.
static int entry_codes(hc_ctx *ctx, LenHost &lh, PoolScratch &scr, EntryCodes *ec)
{
    cudaStream_t st = ctx->stream;
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale, n = lh.n;
    if (n > 0)
    {
        uint8_t *used;
        HC_CUDA(ctx, scr.alloc(&ec->code, n));
        HC_CUDA(ctx, scr.alloc(&used, (size_t)kCodes));
        HC_CUDA(ctx, scr.alloc(&ec->bad, (size_t)n));
        HC_CUDA(ctx, cudaMemsetAsync(used, 0, kCodes, st));
        launch_after(k_entry_codes, (n + 255) / 256, 256, 0, st, (double)ctx->p.min_mass, (double)ctx->p.max_mass,
                     lh.L, n, lh.d_mass, lh.d_seqid, lh.d_sites, lh.d_modnum, lh.d_seqs, ec->code, used, ec->bad);
        HC_CUDA(ctx, cudaGetLastError());
        HC_CUDA(ctx, cudaMemcpyAsync(read_used(ctx), used, kCodes, cudaMemcpyDeviceToHost, st));
    }
    HC_CUDA(ctx, cudaMemcpyAsync(read_total(ctx), lh.d_qA + nb, 4, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    return HC_SUCCESS;
}

static unsigned flat_blocks(const hc_ctx *ctx, uint64_t items)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + 255) / 256, (uint64_t)ctx->sm_count * 64));
}

// The query postings (padded buckets), their bucket starts and the search side,
// from bA (on the device) and the ids in bucket order (d_ids; null when the
// length has no postings) with their buckets (d_keys; null: found here).
// Leaves d_ids untouched.
int build_query_postings(hc_ctx *ctx, LenHost &lh, const uint32_t *d_ids, const uint32_t *d_keys)
{
    cudaStream_t st = ctx->stream;
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale;
    // entry << 3 must stay below 2^32 and below the padding word
    if (lh.n > kQpMaxEntries)
        return set_error(ctx, HC_ERR_INVLD_SIZE, "too many entries of one length for the query postings");
    dfree(ctx, lh.d_qA);
    dfree(ctx, lh.d_qp);
    dfree(ctx, lh.d_qion);
    lh.d_qA = lh.d_qp = nullptr;
    lh.d_qion = nullptr;
    HC_CUDA(ctx, dalloc(ctx, &lh.d_qA, (size_t)nb + 1));
    uint32_t *stmp = nullptr, *keys = nullptr;
    PoolScratch scr(ctx);
    HC_CUDA(ctx, scr.alloc(&stmp, scan_tmp_words((size_t)nb + 1)));
    const uint32_t npost = d_ids ? (uint32_t)lh.npost : 0u;
    if (npost && !d_keys)
    {
        HC_CUDA(ctx, scr.alloc(&keys, npost));
        launch_after(k_bucket_keys, flat_blocks(ctx, npost), 256, 0, st, lh.d_bA, nb, npost, keys);
        d_keys = keys;
    }
    launch_after(k_pad_counts, flat_blocks(ctx, (uint64_t)nb + 1), 256, 0, st, lh.d_bA, nb, lh.d_qA);
    HC_CUDA(ctx, scan_exclusive(lh.d_qA, (size_t)nb + 1, stmp, st));
    EntryCodes ec{};
    const int rc = entry_codes(ctx, lh, scr, &ec);
    if (rc) return rc;
    const uint32_t total = *read_total(ctx);
    HC_CUDA(ctx, dalloc(ctx, &lh.d_qp, (size_t)total + kIaPad));
    HC_CUDA(ctx, dalloc(ctx, &lh.d_qion, (size_t)total + kIaPad));
    launch_after(k_qpost_pads, flat_blocks(ctx, (uint64_t)nb + 1), 256, 0, st, lh.d_bA, lh.d_qA, nb, lh.d_qp,
                 lh.d_qion);
    HC_CUDA(ctx, cudaGetLastError());
    return build_search(ctx, lh, ec, d_ids, d_keys, npost, lh.d_bA, true);
}

// Classes for the codes seen in `used` that have none yet (ids are only ever
// added, so the lengths built before keep theirs), and the device copies.
static int add_classes(hc_ctx *ctx, const uint8_t *used)
{
    bool changed = false;
    for (uint32_t code = 0; code < kCodes; code++)
    {
        if (!used[code] || code == kCodes - 2 || ctx->class_of[code] != kClassNone || ctx->classes.n >= kMaxClasses)
            continue;
        const uint32_t id = ctx->classes.n++;
        ctx->class_of[code] = (uint8_t)id;
        class_keys_of(ctx->p, ctx->tables, code, ctx->classes.key[id]);
        for (uint32_t z = 0; z < ctx->p.maxz; z++)
            ctx->classes.maxkey = std::max(ctx->classes.maxkey, ctx->classes.key[id][z]);
        changed = true;
    }
    if (!ctx->d_classes)
    {
        HC_CUDA(ctx, cudaMalloc((void **)&ctx->d_classes, sizeof(ClassKeys)));
        HC_CUDA(ctx, cudaMalloc((void **)&ctx->d_class_of, kCodes));
        changed = true;
    }
    if (changed)
    {
        HC_CUDA(ctx, overwrite(ctx->d_classes, &ctx->classes, sizeof(ClassKeys)));
        HC_CUDA(ctx, overwrite(ctx->d_class_of, ctx->class_of.data(), kCodes));
    }
    return HC_SUCCESS;
}

// The search side of a length: each entry's class (checked against its own y1
// postings), the search postings (the query postings less the y1 postings of
// classed entries, buckets padded to 4 words) and their row table. From `total`
// ids (entry * speclen + ion, kQpostPad: none) in bucket order, their buckets
// and the buckets' starts among them; `write`: the query postings too.
static int build_search(hc_ctx *ctx, LenHost &lh, const EntryCodes &ec, const uint32_t *d_ids, const uint32_t *d_keys,
                        uint32_t total, const uint32_t *start, bool write)
{
    cudaStream_t st = ctx->stream;
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale, n = lh.n, Lm1 = lh.L - 1;
    const uint32_t half = ctx->p.maxz * Lm1;
    const IdDiv div = id_div(2 * half, (uint64_t)n * 2 * half);
    dfree(ctx, lh.d_rows);
    dfree(ctx, lh.d_qAs);
    dfree(ctx, lh.d_qps);
    dfree(ctx, lh.d_cls);
    lh.d_rows = lh.d_qAs = lh.d_qps = nullptr;
    lh.d_cls = nullptr;
    HC_CUDA(ctx, dalloc(ctx, &lh.d_cls, (size_t)n + 4));  // +4: the search reads class bytes in fours
    HC_CUDA(ctx, dalloc(ctx, &lh.d_qAs, (size_t)nb + 1));
    const unsigned eblocks = (n + 255) / 256, bblocks = flat_blocks(ctx, (uint64_t)nb + 1);
    const unsigned pblocks = flat_blocks(ctx, total);
    PoolScratch scr(ctx);
    if (n > 0)
    {
        const int rc = add_classes(ctx, read_used(ctx));
        if (rc) return rc;
        launch_after(k_entry_classes, n / 256 + 2, 256, 0, st, ec.code, n, ctx->d_class_of, lh.d_cls);
        if (total)
            launch_after(k_qpost, pblocks, 256, 0, st, d_ids, d_keys, total, start, lh.d_qA, div, half, Lm1,
                         lh.d_cls, ctx->d_classes, ec.bad, write ? lh.d_qp : nullptr, write ? lh.d_qion : nullptr);
        launch_after(k_class_fix, eblocks, 256, 0, st, lh.d_cls, ec.bad, n);
        HC_CUDA(ctx, cudaGetLastError());
    }
    // the kept postings' bits and counts, the padded bucket sizes from them and
    // their scan (qAs), then every kept posting to its place
    const uint32_t nwords = total / 32 + 1;  // (position `total` has one too)
    uint32_t *mask = nullptr, *sum = nullptr, *stmp = nullptr, *off = nullptr;
    HC_CUDA(ctx, scr.alloc(&mask, nwords));
    HC_CUDA(ctx, scr.alloc(&sum, nwords));
    HC_CUDA(ctx, scr.alloc(&off, (size_t)nb));
    HC_CUDA(ctx, scr.alloc(&stmp, scan_tmp_words(std::max<size_t>(nwords, (size_t)nb + 1))));
    launch_after(k_spost_mask, flat_blocks(ctx, 32ull * nwords), 256, 0, st, d_ids, total, div, half, Lm1, lh.d_cls,
                 nwords, mask, sum);
    HC_CUDA(ctx, cudaGetLastError());
    HC_CUDA(ctx, scan_exclusive(sum, nwords, stmp, st));
    launch_after(k_spost_counts, bblocks, 256, 0, st, start, mask, sum, nb, lh.d_qAs);
    HC_CUDA(ctx, cudaGetLastError());
    HC_CUDA(ctx, scan_exclusive(lh.d_qAs, (size_t)nb + 1, stmp, st));
    HC_CUDA(ctx, cudaMemcpyAsync(read_total(ctx), lh.d_qAs + nb, 4, cudaMemcpyDeviceToHost, st));
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    lh.nsearch = *read_total(ctx);
    HC_CUDA(ctx, dalloc(ctx, &lh.d_qps, (size_t)lh.nsearch + kIaPad));
    launch_after(k_spost_pads, bblocks, 256, 0, st, start, mask, sum, nb, lh.d_qAs, off, lh.d_qps);
    if (total)
        launch_after(k_spost_scatter, pblocks, 256, 0, st, d_ids, d_keys, total, div, half, mask, sum, off, lh.d_qps);
    HC_CUDA(ctx, cudaGetLastError());
    lh.stride = (n + kRowG - 1) / kRowG + 1;
    HC_CUDA(ctx, dalloc(ctx, &lh.d_rows, (size_t)nb * lh.stride));
    const uint64_t rt = (uint64_t)nb * lh.stride;
    const unsigned blocks = (unsigned)std::min<uint64_t>((rt + 255) / 256, (uint64_t)ctx->sm_count * 64);
    launch_after(k_row_table, blocks, 256, 0, st, lh.d_qAs, lh.d_qps, nb, lh.stride, n, lh.d_rows);
    HC_CUDA(ctx, cudaGetLastError());
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    return HC_SUCCESS;
}

// The same from query postings that are there already (an index file's, in
// padded order): qA, qp, qion and the entries set and checked.
int build_rows(hc_ctx *ctx, LenHost &lh)
{
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale;
    PoolScratch scr(ctx);
    EntryCodes ec{};
    const int rc = entry_codes(ctx, lh, scr, &ec);
    if (rc) return rc;
    const uint32_t qtotal = *read_total(ctx);
    uint32_t *ids = nullptr, *keys = nullptr;
    HC_CUDA(ctx, scr.alloc(&ids, qtotal));
    HC_CUDA(ctx, scr.alloc(&keys, qtotal));
    if (qtotal)
    {
        launch_after(k_qpost_to_ids, flat_blocks(ctx, qtotal), 256, 0, ctx->stream, lh.d_qp, lh.d_qion, qtotal,
                     2 * ctx->p.maxz * (lh.L - 1), ids);
        launch_after(k_bucket_keys, flat_blocks(ctx, qtotal), 256, 0, ctx->stream, lh.d_qA, nb, qtotal, keys);
        HC_CUDA(ctx, cudaGetLastError());
    }
    return build_search(ctx, lh, ec, ids, keys, qtotal, lh.d_qA, false);
}

// Checks query postings read from outside (an index file): bucket starts
// ascending multiples of 4 ending at the total, and every word padding or a
// valid (entry, ion). Returns HC_ERR_FILE_ERROR otherwise.
int check_query_postings(hc_ctx *ctx, const LenHost &lh, uint64_t qtotal)
{
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale;
    const uint32_t speclen = 2 * ctx->p.maxz * (lh.L - 1);
    if (lh.n > kQpMaxEntries)
        return set_error(ctx, HC_ERR_FILE_ERROR, "index file: too many entries of one length");
    std::vector<uint32_t> qa(nb + 1);
    HC_CUDA(ctx, cudaMemcpy(qa.data(), lh.d_qA, 4ull * (nb + 1), cudaMemcpyDeviceToHost));
    for (uint32_t b = 0; b <= nb; b++)
        if ((qa[b] & 3u) || (b && qa[b] < qa[b - 1]))
            return set_error(ctx, HC_ERR_FILE_ERROR, "index file: bucket starts out of order");
    if (qa[0] != 0 || qa[nb] != qtotal) return set_error(ctx, HC_ERR_FILE_ERROR, "index file: bucket starts");
    uint32_t *d_bad = nullptr;
    HC_CUDA(ctx, cudaMalloc((void **)&d_bad, 4));
    uint32_t bad = 0;
    cudaError_t e = cudaMemsetAsync(d_bad, 0, 4, ctx->stream);
    if (e == cudaSuccess && qtotal)
    {
        const unsigned blocks = (unsigned)std::min<uint64_t>((qtotal + 255) / 256, (uint64_t)ctx->sm_count * 32);
        launch_after(k_check_qpost, blocks, 256, 0, ctx->stream, lh.d_qp, lh.d_qion, qtotal, lh.n, speclen,
                     speclen / 2, d_bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpy(&bad, d_bad, 4, cudaMemcpyDeviceToHost);
    cudaFree(d_bad);
    HC_CUDA(ctx, e);
    if (bad) return set_error(ctx, HC_ERR_FILE_ERROR, "index file: invalid postings");
    return HC_SUCCESS;
}

// The reference's iA (ids entry*speclen + ion, bucket order) from the query postings.
int export_ids(hc_ctx *ctx, const LenHost &lh, uint32_t *d_ids)
{
    const uint32_t nb = ctx->p.max_mass * ctx->p.scale;
    const uint32_t speclen = 2 * ctx->p.maxz * (lh.L - 1);
    if (lh.npost)
        launch_after(k_qpost_ids, flat_blocks(ctx, lh.npost), 256, 0, ctx->stream, lh.d_bA, lh.d_qA, lh.d_qp,
                     lh.d_qion, nb, (uint32_t)lh.npost, speclen, d_ids);
    HC_CUDA(ctx, cudaGetLastError());
    HC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return HC_SUCCESS;
}

}  // namespace hc
