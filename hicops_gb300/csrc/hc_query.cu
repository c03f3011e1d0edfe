// DSLIM query on the device (DSLIM_QuerySpectrum, source/core/dslim_query.cpp:515-842).
//
// Kernels, in launch order (each starts under the end of the one before, see launch_after):
//   k_windows   one thread per (spectrum, length): the precursor window
//               [minlimit, maxlimit] of DSLIM_BinarySearch (dslim_query.cpp:854-994).
//   k_search    persistent CTAs, one spectrum at a time (work stealing):
//               for every length with a non-empty window, the candidate range
//               is cut into shared-memory scorecard tiles; the postings of every
//               (peak, bin) pair (dslim_query.cpp:617-676) are streamed with
//               coalesced loads, and each posting adds (count, intensity) to its
//               candidate's packed b or y word with one shared-memory atomic. Then
//               the tile is scanned, and the candidates whose shared-peak count
//               reaches min_shp are scored (dslim_query.cpp:679-725)
//               into the 1002-bin histogram, cpsms and the top hit.
//   k_search_small the same for spectra whose windows hold few candidates: all
//               their windows in one scorecard.
//   k_search<WIDE> the same for spectra whose packed words could overflow
//               (a count past 127): 2 x 64-bit words per candidate, exact FP64.
//   k_tailfit   expeRT::ModelTailFit (expeRT.cpp:572-718) and
//               e(x) = 10^(mu*maxhyp + beta) * cpsms (dslim_query.cpp:773-799):
//               a warp per spectrum for its curve, then a lane per spectrum.
//
// Hyperscore. The reference evaluates h = lgfact[bc] + lgfact[yc] +
// log10(1+ibc) + log10(1+iyc) - 6 in double and stores it as float. Here it is
// first evaluated in float; the float value lies within 1.1e-4 of the
// reference's (table rounding 2 x 7.6e-6, three float additions 3 x 1.6e-5,
// log10f within 2 ulp, the final rounding 4e-6), and a score below 50 within
// 1.5e-5 (its terms and sums stay below 64: table roundings 2 x 1.9e-6, the sums
// 3 x 1.9e-6, the logarithm 2 ulp of a log2 below 48, x 0.301: 2.3e-6, its factor
// and product 1.2e-6, the reference's rounding 1.9e-6). Wherever that bound leaves
// a decision open (sign, histogram bin, or a candidate that can still be the
// top hit) the reference's double expression is evaluated, so cpsms, the
// histogram and the top hit equal the reference's double evaluation.
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <cstdio>
#include <type_traits>

#include "hc_device.cuh"
#include "hc_internal.h"

namespace hc {
namespace {

constexpr int kDefer = HC_DEFER_MAX;  // undecided candidates per spectrum, resolved at its end
constexpr uint32_t kWQ = 64;         // per-warp ring of qualifying candidates' words (power of two, >= 31 + 32)
constexpr uint32_t kNoJob = 0xFFFFFFFFu;
constexpr float kApproxErr = 1.1e-4f;
// A score this close to a bin's edge (on the x10 scale) is open: 10 x the bound
// above and the roundings of the two products (3e-5 and 6e-5 below 512; 2.4e-4 in all
// for scores below 50). The wider margin took in 420 candidates of an open-search
// spectrum, more than its queue holds, and the rest were evaluated on the spot, some
// warp of almost every job waiting on double arithmetic; the narrow one takes in 60.
constexpr float kBinMargin = 4e-4f, kBinMarginHigh = 2.5e-3f, kLowScore = 50.0f;
__device__ __forceinline__ bool bin_open(float ha, float fr)
{
    return fabsf(fr - 0.5f) > 0.5f - (ha < kLowScore ? kBinMargin : kBinMarginHigh);
}
constexpr float kNear = 3.5e-4f;       // > 2 * kApproxErr: candidates that may be the top
static_assert(HC_DEFER_MAX >= 128, "the scan's last step may read 127 packed words past the tile, into the queue");

// What the tile loop reads of a length's record: kept in the kernel's
// parameters (the constant cache; the length index is warp-uniform)
struct LenS
{
    const uint32_t *qp, *rows;  // search postings and their row table
    uint32_t stride, n;
    const uint8_t *cls;         // entry classes (4 bytes of padding past the last entry)
};

// what one of the CTAs that share a spectrum found
struct PartSum
{
    unsigned long long best, bytes;
    uint32_t best_shp, flags, cps, overflow;
};
static_assert(sizeof(PartSum) == 4 * kPartWords, "kPartWords");

struct SearchArgs
{
    const LenDev *lens;
    uint32_t nlen;
    const QueryConst *qc;
    const uint32_t *idx, *moz, *inten;
    const float *prec;
    const int2 *win;
    uint32_t nspec;
    uint32_t dF, thr, min_shp, maxbin;  // maxbin = max_mass*scale
    hc_result *out;
    uint32_t *hist;
    uint32_t *wide_list, *nwide;
    uint32_t *work;
    uint32_t tile;
    uint32_t defer_cap;     // <= kDefer
    const uint32_t *only;   // optional list of spectra to process (wide pass)
    const uint32_t *nonly_dev;  // its length, in device memory
    const uint32_t *order;  // optional processing order (longest first)
    const uint32_t *obase;  // optional (device word): the first position of the order this launch takes
    const uint32_t *olim;   // optional (device word): the position it stops at (else nspec)
    uint32_t wsplit;        // optional: k_search leaves the spectra whose windows hold fewer candidates
                            // in all, k_search_small those whose windows hold as many or more
    uint32_t parts;         // k_search: CTAs that share a spectrum at most (0, 1: none; else `hist` starts at zero)
    uint32_t part_min;      // ... candidates of a part at least
    uint32_t *arrived;      // ... per spectrum, how many of them have ended
    struct PartSum *psum;   // ... what each found, `parts` a spectrum
    uint32_t follows;       // k_search_small: 1 when the launch before it writes what it reads
    uint32_t persistent;    // 1: CTAs loop over a work counter; 0: one spectrum per CTA
    uint32_t maxz;
    const ClassKeys *classes;   // entry classes (null: none built)
    unsigned long long *phase;  // optional: SM cycles per phase, summed over CTAs (kPhases)
    LenS len[HC_MAX_LENGTHS];
};

// phases of k_search timed when SearchArgs::phase is set
constexpr int kPhases = 6;  // bucket setup | postings stream | score pass 1 | pass 2 | tile clear | rest

// The reference's double-precision hyperscore, rounded to float
// (dslim_query.cpp:695-698). Additions only: no contraction possible.
__device__ __forceinline__ float exact_h(const QueryConst *__restrict__ qc, uint32_t bc, uint32_t yc,
                                        uint64_t ib, uint64_t iy)
{
    const double h1 = __dadd_rn(qc->lgfact[bc < kLgTable ? bc : kLgTable - 1],
                                qc->lgfact[yc < kLgTable ? yc : kLgTable - 1]);
    // log10 of the intensity sums from the host-built table (the device's
    // double log10 is very slow on this part); beyond it, the device log10
    const double lb = (1 + ib < kLog10Tab) ? __ldg(qc->log10_tab + 1 + ib) : log10((double)(1 + ib));
    const double ly = (1 + iy < kLog10Tab) ? __ldg(qc->log10_tab + 1 + iy) : log10((double)(1 + iy));
    double h = __dadd_rn(h1, lb);
    h = __dadd_rn(h, ly);
    h = __dadd_rn(h, -6.0);
    return __double2float_rn(h);
}

template <bool WIDE>
struct Card;

template <>
struct Card<false>
{
    // b word [bc:8 | ibc:24] and y word [yc:8 | iyc:24]: a posting is a b or
    // a y ion, so it adds to one 32-bit word (native shared-memory atomic).
    // Every atomic returns the word before the add; a count that passes 128
    // shows as a returned top bit, and the spectrum is redone wide. Below
    // that, with intensities < 2^17, the sums stay below 2^24.
    using word = uint32_t;
    static constexpr int kWords = 2;
};

template <>
struct Card<true>
{
    // b word and y word: [count:24 | sum:40]
    using word = unsigned long long;
    static constexpr int kWords = 2;
};

// histogram bins kept in shared memory; candidates of the bins past them
// (hyperscores of 25.6 and more: a few per spectrum) add to the spectrum's
// output histogram directly
constexpr int kHistSm = 256;
// float log-factorials kept in shared memory: a packed count stays below 128
// (a spectrum whose count reaches 128 is redone with wide words)
constexpr int kLgSm = 128;

struct SmemTail
{
    union
    {
        // while the spectrum's candidates are scored; lgf first: an
        // overflowing packed count (up to 255, redone wide) reads histogram
        // words, inside the block's memory
        struct
        {
            float lgf[kLgSm];
            uint32_t hist[kHistSm];
        } run;
        // during the spectrum's set-up: per entry class, what its y1 keys
        // collect from the valid peaks as a wide word [count:24 | sum:40]
        // (kept apart for wide words, whose scorecard start reads it); the
        // valid peaks that can reach a class key
        struct
        {
            unsigned long long ucls[kMaxClasses + 1];
            uint32_t low[HC_QALEN];
        } setup;
    } u;
    unsigned long long best;   // (exact h bits << 32) | ~(ixx << 24 | psid)
    uint32_t best_shp;
    uint32_t maxbits;          // running max of the float estimate
    uint32_t cpsms;
    uint32_t flags;
    uint32_t overflow;
    uint32_t spec;
    uint32_t nv;
    uint32_t noret;            // the stream's atomics need not return the old words (see k_search)
    uint32_t pnext;            // next 16-byte chunk (of the tile's lists laid end to end) to hand out
    uint32_t ndefer;           // undecided candidates queued for the exact evaluation
    uint32_t cchunks;          // 16-byte chunks (all lists) of the job
    uint32_t ncl;              // its non-empty lists
    unsigned long long bytes;
    unsigned long long ph[kPhases];
    unsigned long long ph_last;
    unsigned long long cnt[4];  // tiles | tiles scanned whole | listed candidates | exact evaluations
    int2 win[HC_MAX_LENGTHS];  // the spectrum's window per length
    // per entry class: what its y1 keys collect from the spectrum's valid
    // peaks, packed [count:8 | sum:24]; entry kClassNone stays zero
    uint32_t upk[kMaxClasses + 1];
    uint32_t ncu, cu;          // how many of them are not zero; one that is not
    uint32_t nlow;
};

// adds the cycles since the last mark to phase k (thread 0 only, after a barrier)
#define HC_PHASE(k)                                               \
    do {                                                          \
        if (a.phase && tid == 0)                                  \
        {                                                         \
            const unsigned long long _t = clock64();              \
            T.ph[(k)] += _t - T.ph_last;                          \
            T.ph_last = _t;                                       \
        }                                                         \
    } while (0)

struct SmemLayout
{
    size_t defer, lnext, lend, loff, coff, kinfo, pmoz, pint, wq, ucls, sink, tail, total;
    uint32_t maxpairs;  // lists: valid peaks x bins
};

__host__ __device__ inline SmemLayout smem_layout(uint32_t tile, uint32_t dF, bool wide, uint32_t nwarps)
{
    const size_t maxpairs = (size_t)HC_QALEN * (2 * dF + 1);
    SmemLayout o;
    // the scorecard, then the undecided queue: the scan reads whole
    // 128-candidate steps, and a window's last step may read up to 127 words
    // past the tile's end (masked), inside the queue
    o.defer = wide ? (size_t)tile * 16 : (size_t)tile * 8;
    o.maxpairs = (uint32_t)maxpairs;
    // per list (of the next job: written while the job streams): its first
    // posting, the end of its list, its chunk count; per non-empty list of
    // the job: its first chunk and {first posting, intensity} (the next
    // job's written after the job's stream)
    o.lnext = o.defer + 8ull * kDefer;
    o.lend = o.lnext + 4 * maxpairs;
    o.loff = o.lend + 4 * maxpairs;
    o.coff = o.loff + 4 * (maxpairs + 4);
    o.kinfo = (o.coff + 4 * (maxpairs + 4) + 7) & ~(size_t)7;
    o.pmoz = (o.kinfo + 8 * maxpairs + 15) & ~(size_t)15;
    o.pint = o.pmoz + 4ull * HC_QALEN;
    o.wq = (o.pint + 4ull * HC_QALEN + 15) & ~(size_t)15;
    size_t end = o.wq + 4ull * kWQ * nwarps;
    // wide words: the class adds, read by every job's scorecard start
    o.ucls = (end + 15) & ~(size_t)15;
    if (wide) end = o.ucls + 8ull * (kMaxClasses + 1);
    o.sink = (end + 15) & ~(size_t)15;
    o.tail = o.sink + 4 * 32;
    // right after the tail: per group of 32 lists of the next job, its chunks
    // and non-empty lists
    o.total = o.tail + sizeof(SmemTail) + 8 * ((maxpairs + 31) / 32);
    return o;
}

// float estimate of the hyperscore; the packed sums are < 2^24, so the
// integer-to-float conversions stay 32-bit (exact, full-rate). The two
// logarithms are one of the product (< 2^48, rounded by 2^-24 relative) with
// the fast hardware log2: together about 1e-6 off, well inside kApproxErr,
// which the callers' sign and bin margins are built on.
__device__ __forceinline__ float approx_h(const float *lgf, uint32_t bc, uint32_t yc, uint64_t ib, uint64_t iy)
{
    const float fb = __uint2float_rn((uint32_t)ib + 1u), fy = __uint2float_rn((uint32_t)iy + 1u);
    return (lgf[bc] + lgf[yc]) + __log2f(fb * fy) * 0.30102999566f - 6.0f;  // one log of the product
}

__device__ __forceinline__ void decode_packed(uint32_t wb, uint32_t wy, uint32_t &bc, uint32_t &yc, uint32_t &shp,
                                              uint64_t &ib, uint64_t &iy)
{
    bc = wb >> 24;
    yc = wy >> 24;
    ib = wb & 0xFFFFFFu;
    iy = wy & 0xFFFFFFu;
    shp = (uint32_t)(uint16_t)(bc + yc);
}

template <bool WIDE>
__device__ __forceinline__ void decode(const typename Card<WIDE>::word *card, uint32_t loc, uint32_t &bc,
                                       uint32_t &yc, uint32_t &shp, uint64_t &ib, uint64_t &iy)
{
    if constexpr (!WIDE)
    {
        const uint2 w = *reinterpret_cast<const uint2 *>(card + 2 * loc);
        decode_packed(w.x, w.y, bc, yc, shp, ib, iy);
        return;
    }
    else
    {
        const unsigned long long wb = card[2 * loc], wy = card[2 * loc + 1];
        bc = (uint32_t)(wb >> 40);
        yc = (uint32_t)(wy >> 40);
        ib = wb & 0xFFFFFFFFFFull;
        iy = wy & 0xFFFFFFFFFFull;
    }
    // the reference reads bc/yc through short/ushort (dslim_query.cpp:684-686)
    shp = (uint32_t)(uint16_t)(bc + yc);
}

// byte k's top bit of x (S = 0x8888 + k * 0x1111) in every bit
template <uint32_t S>
__device__ __forceinline__ uint32_t byte_sign(uint32_t x)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "n"(S));
    return r;
}

// 32-bit adds to a shared-memory word given by its shared-window address.
// No memory clobber: the scorecard is read only after a block barrier.
__device__ __forceinline__ void red_shared_add(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v));
}

__device__ __forceinline__ uint32_t atom_shared_add(uint32_t addr, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v));
    return old;
}

// A word to which an add came with this in it has a count of 128 or more: more than
// a count byte's compare, and the score's table, hold.
__device__ __forceinline__ bool count_full(uint32_t before) { return before >= 127u << 24; }

// Bounds of a bucket's postings for candidates [c0, c1), widened to row-table
// boundaries (multiples of kRowG entries): the postings of entries outside
// the range are read but fail the scorecard's index test, so no search is
// needed. Tile boundaries inside a window are multiples of kRowG already.
__device__ __forceinline__ uint32_t row_lo(const uint32_t *__restrict__ col, uint32_t c0)
{
    return __ldg(col + c0 / kRowG);
}

__device__ __forceinline__ uint32_t row_hi(const uint32_t *__restrict__ col, uint32_t c1)
{
    return __ldg(col + (c1 + kRowG - 1) / kRowG);
}

// Chunk offsets of a job's lists, in two steps around a block barrier, with
// the lists in groups of 32 (group g = lists 32g .. 32g + 31).
// Step 1, by the warp that computed the group's chunk counts (cnt = this
// lane's list, 0 past the last list): the group's totals of chunks and of
// non-empty lists.
__device__ __forceinline__ void group_totals(uint32_t cnt, uint32_t g, int lane, uint2 *gt)
{
    const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, cnt);
    const uint32_t z = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, cnt != 0u));
    if (lane == 0) gt[g] = make_uint2(c, z);
}

// Step 2, one warp per group, any warp: from the chunk counts lo[0, np) and
// the group totals, the job's non-empty lists in order: coff[k] = its first
// chunk (of all lists laid end to end), kinfo[k] = {its first posting, its
// peak's intensity} (list pr = peak pr / nbin, bin pr % nbin); the warp of
// the last group (of ng) writes coff[ncl] = *total and the counts.
__device__ __forceinline__ void group_offsets(uint32_t g, uint32_t ng, const uint32_t *lo, uint32_t np, int lane,
                                              const uint2 *gt, const uint32_t *first, const uint32_t *pint,
                                              uint32_t nbin, uint32_t *coff, uint2 *kinfo, uint32_t *total,
                                              uint32_t *ncl)
{
    uint32_t pc = 0, pz = 0;
    for (uint32_t i = (uint32_t)lane; i < g; i += 32)
    {
        const uint2 t = gt[i];
        pc += t.x;
        pz += t.y;
    }
    pc = __reduce_add_sync(0xFFFFFFFFu, pc);
    pz = __reduce_add_sync(0xFFFFFFFFu, pz);
    const uint32_t pr = 32 * g + (uint32_t)lane;
    const uint32_t cnt = pr < np ? lo[pr] : 0u;
    uint32_t c = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, c, o);
        if (lane >= o) c += y;
    }
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cnt != 0u);
    if (cnt)
    {
        const uint32_t k = pz + (uint32_t)__popc(bal & ((1u << lane) - 1u));
        coff[k] = pc + c - cnt;
        kinfo[k] = make_uint2(first[pr], pint[pr / nbin]);
    }
    if (g + 1 == ng && lane == 31)
    {
        const uint32_t nz = pz + (uint32_t)__popc(bal);
        coff[nz] = pc + c;
        *total = pc + c;
        *ncl = nz;
    }
}

// One unit of a spectrum's work: the candidates [c0, c1) of length l, at
// most one scorecard tile. A window's first tile ends one tile past the
// window start rounded down to a row-table boundary (kRowG); every later
// boundary is a multiple of kRowG, so only a window's two ends widen the
// postings bounds.
struct Job
{
    uint32_t l, c0, c1;
};

__device__ __forceinline__ Job job_from(const int2 *win, uint32_t nlen, uint32_t tile, uint32_t l)
{
    for (; l < nlen; l++)
    {
        const int2 w = win[l];
        if (w.x <= w.y)
        {
            const uint32_t c0 = (uint32_t)w.x;
            return Job{l, c0, min((uint32_t)w.y + 1, (c0 / kRowG) * kRowG + tile)};
        }
    }
    return Job{kNoJob, 0u, 0u};
}

__device__ __forceinline__ Job first_job(const int2 *win, uint32_t nlen, uint32_t tile)
{
    return job_from(win, nlen, tile, 0);
}

__device__ __forceinline__ Job next_job(const Job &j, const int2 *win, uint32_t nlen, uint32_t tile)
{
    const uint32_t end = (uint32_t)win[j.l].y + 1;
    if (j.c1 < end) return Job{j.l, j.c1, min(end, j.c1 + tile)};
    return job_from(win, nlen, tile, j.l + 1);
}

// A job whose bounds are both row-table boundaries inside the length's
// entries: its lists hold the postings of the job's entries and nothing else
// (no padding, no neighbours), so their lengths are its visited postings.
__device__ __forceinline__ bool job_interior(const Job &j, uint32_t n)
{
    return (j.c0 % kRowG) == 0 && (j.c1 % kRowG) == 0 && j.c1 < n;
}

// The last list i in [0, n) with off[i] <= q (off ascending, off[0] = 0):
// a 32-way search, one shared-memory read per lane per round.
__device__ __forceinline__ uint32_t find_list(const uint32_t *off, uint32_t n, uint32_t q, int lane)
{
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1)
    {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t i = lo + (uint32_t)lane * step;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, i < hi && off[i] <= q);
        lo += (uint32_t)(31 - __clz(m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// a spectrum's result, its e-value left open
__device__ __forceinline__ void write_result(const SearchArgs &a, uint32_t s, uint32_t cpsms, uint32_t flags,
                                             unsigned long long bytes, unsigned long long best, uint32_t best_shp)
{
    hc_result r;
    r.cpsms = cpsms;
    r.flags = flags;
    r.post_bytes = bytes;
    if (cpsms > 0 && best != 0)
    {
        const uint32_t tie = ~(uint32_t)(best & 0xFFFFFFFFu);
        r.idxoffset = (int32_t)(tie >> 24);
        r.psid = (int32_t)(tie & 0xFFFFFF);
        r.hyperscore = __uint_as_float((uint32_t)(best >> 32));
        r.sharedions = (uint16_t)best_shp;
        r.totalions = (uint16_t)a.lens[r.idxoffset].speclen;
    }
    else
    {
        r.idxoffset = -1;
        r.psid = -1;
        r.hyperscore = 0.0f;
        r.sharedions = 0;
        r.totalions = 0;
    }
    r.mu = r.beta = r.minhyp = r.nexthyp = r.maxhyp = 0;
    r.reported = 0;
    r.evalue = 0.0;
    a.out[s] = r;
}

// the candidates of a spectrum's windows, by one warp
__device__ __forceinline__ uint32_t window_sum(const int2 *win, uint32_t nlen, int lane)
{
    uint32_t c = 0;
    for (uint32_t l = lane; l < nlen; l += 32)
        if (win[l].x <= win[l].y) c += (uint32_t)(win[l].y - win[l].x) + 1u;
    return __reduce_add_sync(0xFFFFFFFFu, c);
}

// The windows of part `part` of `parts`, by one warp: the row-table steps (kRowG
// entries) that the spectrum's windows touch, laid end to end, are dealt out in equal runs.
__device__ __forceinline__ void part_windows(int2 *win, uint32_t nlen, uint32_t part, uint32_t parts, int lane)
{
    uint32_t rows[2], sum = 0;
    int2 w[2];
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const uint32_t l = 2 * (uint32_t)lane + h;
        w[h] = l < nlen ? win[l] : make_int2(1, 0);
        rows[h] = w[h].x <= w[h].y ? (uint32_t)w[h].y / kRowG - (uint32_t)w[h].x / kRowG + 1u : 0u;
        sum += rows[h];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    const unsigned long long total = __shfl_sync(0xFFFFFFFFu, x, 31);
    const uint32_t g0 = (uint32_t)(total * part / parts), g1 = (uint32_t)(total * (part + 1) / parts);
    uint32_t base = x - sum;  // of the rows before this length
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        const uint32_t l = 2 * (uint32_t)lane + h;
        const uint32_t r0 = max(base, g0), r1 = min(base + rows[h], g1);  // its rows of this part
        int2 p = make_int2(1, 0);
        if (r0 < r1)
        {
            const uint32_t first = (uint32_t)w[h].x / kRowG - base;
            p.x = max(w[h].x, (int)((first + r0) * kRowG));
            p.y = min(w[h].y, (int)((first + r1) * kRowG) - 1);
        }
        if (l < nlen) win[l] = p;
        base += rows[h];
    }
}

// Leaves what a part found; the last of the spectrum's parts writes its result, or
// lists it for the wide search. By one thread.
__device__ __forceinline__ void end_part(const SearchArgs &a, uint32_t s, uint32_t part, uint32_t parts,
                                         const PartSum &mine)
{
    PartSum *p = a.psum + (size_t)s * a.parts;
    p[part] = mine;
    __threadfence();
    if (atomicAdd(&a.arrived[s], 1u) + 1u != parts) return;
    __threadfence();
    PartSum t{};
    for (uint32_t i = 0; i < parts; i++)
    {
        const unsigned long long best = __ldcg(&p[i].best);
        if (best > t.best)
        {
            t.best = best;
            t.best_shp = __ldcg(&p[i].best_shp);
        }
        t.bytes += __ldcg(&p[i].bytes);
        t.flags |= __ldcg(&p[i].flags);
        t.cps += __ldcg(&p[i].cps);
        t.overflow |= __ldcg(&p[i].overflow);
    }
    if (t.overflow) a.wide_list[atomicAdd(a.nwide, 1u)] = s;
    else write_result(a, s, t.cps, t.flags, t.bytes, t.best, t.best_shp);
}

template <bool WIDE, int G, bool PARTS = false>
__global__ void __launch_bounds__(G >= 4 ? 512 : 1024, G == 4 ? 2 : 1) k_search(SearchArgs a)
{
    using W = typename Card<WIDE>::word;
    constexpr int NW = Card<WIDE>::kWords;
    // lists per thread whose bucket is kept and whose next-job row-table
    // words are loaded early (two for blocks of up to 512 threads, one for
    // 1024: 300 lists at dF = 1 either way; the rest are computed directly)
    constexpr int kPf = G >= 4 ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t tile = a.tile;
    const uint32_t nbin = 2 * a.dF + 1;
    const SmemLayout L = smem_layout(tile, a.dF, WIDE, blockDim.x >> 5);
    W *card = reinterpret_cast<W *>(smem);
    uint32_t *coff = reinterpret_cast<uint32_t *>(smem + L.coff);    // first chunk of each non-empty list
    uint2 *kinfo = reinterpret_cast<uint2 *>(smem + L.kinfo);         // {first posting, intensity} of each
    uint2 *defer = reinterpret_cast<uint2 *>(smem + L.defer);  // undecided candidates: {b word, y word}
    uint32_t *lnext = reinterpret_cast<uint32_t *>(smem + L.lnext);  // per list: first posting (next job)
    uint32_t *lend = reinterpret_cast<uint32_t *>(smem + L.lend);  // per list: end of the current job's list
    uint32_t *loff = reinterpret_cast<uint32_t *>(smem + L.loff);
    uint32_t *pmoz = reinterpret_cast<uint32_t *>(smem + L.pmoz);
    uint32_t *pint = reinterpret_cast<uint32_t *>(smem + L.pint);
    SmemTail &T = *reinterpret_cast<SmemTail *>(smem + L.tail);
    uint2 *gt = reinterpret_cast<uint2 *>(&T + 1);
    unsigned long long *ucls = WIDE ? reinterpret_cast<unsigned long long *>(smem + L.ucls) : T.u.setup.ucls;
    uint32_t *low = T.u.setup.low;

    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, wid = tid >> 5;
    // one word per lane that postings outside the tile add to (never read);
    // the stream addresses the scorecard and the sinks as shared-window offsets
    const uint32_t card_s = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t sink_s = (uint32_t)__cvta_generic_to_shared(smem + L.sink) + 4u * (uint32_t)lane;
    uint32_t *wq = reinterpret_cast<uint32_t *>(smem + L.wq) + wid * kWQ;  // this warp's candidate ring

    // The next launch's CTAs may take SMs as they fall free: the tail fit's, which
    // wait for this one's end, or k_search_small's, which read only what was
    // complete before this kernel's wait.
    if constexpr (WIDE)
    {
        after_predecessor();
        release_successor();
        if (blockIdx.x >= *a.nonly_dev) return;  // most batches list no spectrum
    }
    for (uint32_t i = tid; i < tile * NW; i += nthr) card[i] = 0;
    [[maybe_unused]] uint32_t parts = 1;  // that the spectrum is searched in
    if constexpr (!WIDE)
    {
        after_predecessor();
        release_successor();
        if constexpr (PARTS)
        {
            // CTA i takes part i % parts of spectrum i / parts, and nothing else; most of a
            // batch of small windows leave here
            const uint32_t s = blockIdx.x / a.parts;
            if (s >= a.nspec) return;
            const uint32_t c = window_sum(a.win + (size_t)s * a.nlen, a.nlen, lane);
            parts = min(a.parts, max(c / a.part_min, 1u));
            if (c < a.wsplit || blockIdx.x % a.parts >= parts) return;
        }
    }
    if (tid == 0)
    {
        for (int k = 0; k < kPhases; k++) T.ph[k] = 0;
        for (int k = 0; k < 4; k++) T.cnt[k] = 0;
        T.ph_last = clock64();
        T.pnext = 0;   // reset again after every tile
    }

    // Scores one candidate (the float estimate; undecided ones are queued):
    // cpsms, histogram, flags. A candidate whose estimate comes within kNear
    // of the running maximum (all candidates of the spectrum so far) gets the
    // reference's double hyperscore and competes for the top hit. The true top
    // hit's estimate is within 2*kApproxErr < kNear of the final maximum, so it
    // is always among them, whatever the order candidates are scored in.
    // (cpsms is the histogram's sum: T.cpsms counts only what goes past kHistSm)
    auto count_psm = [&](uint32_t bc, uint32_t yc, int bin) {
        if (max(bc, yc) >= (uint32_t)kRefMaxShp) atomicOr(&T.flags, HC_FLAG_LGFACT_OOB);
        if ((uint32_t)bin < (uint32_t)kHistSm) atomicAdd(&T.u.run.hist[bin], 1u);
        else
        {
            if (bin >= HC_HIST_BINS || bin < 0)
            {
                atomicOr(&T.flags, HC_FLAG_HIST_OOB);
                bin = bin < 0 ? 0 : HC_HIST_BINS - 1;
            }
            atomicAdd(&T.cpsms, 1u);
            atomicAdd(&a.hist[(size_t)T.spec * HC_HIST_BINS + (uint32_t)bin], 1u);
        }
    };
    auto exact_done = [&]() {
        if (a.phase) atomicAdd(&T.cnt[3], 1ull);
    };
    unsigned long long my_best = 0;
    uint32_t my_shp = 0;
    auto score_one = [&](uint32_t bc, uint32_t yc, uint64_t ib, uint64_t iy, uint32_t shp, uint32_t key_lo) {
        float ha;
        if constexpr (!WIDE) ha = approx_h(T.u.run.lgf, bc, yc, ib, iy);
        else ha = exact_h(a.qc, bc, yc, ib, iy);
        const float runmax = __uint_as_float(*(volatile uint32_t *)&T.maxbits);
        if (ha >= runmax - kNear)
        {
            if (ha > runmax) atomicMax(&T.maxbits, __float_as_uint(ha));
            const float he = WIDE ? ha : exact_h(a.qc, bc, yc, ib, iy);
            if (he > 0.0f)
            {
                const unsigned long long key = ((unsigned long long)__float_as_uint(he) << 32) | key_lo;
                if (key > my_best)
                {
                    my_best = key;
                    my_shp = shp;
                }
                atomicMax(&T.best, key);
            }
        }
        float h;
        int bin;
        if constexpr (!WIDE)
        {
            const float tt = ha * 10.0f + 0.5f;
            const float fr = tt - floorf(tt);
            if (fabsf(ha) <= kApproxErr * 4.0f || bin_open(ha, fr))
            {
                const uint32_t di = atomicAdd(&T.ndefer, 1u);
                if (di < a.defer_cap)
                {
                    defer[di] = make_uint2((uint32_t)ib | (bc << 24), (uint32_t)iy | (yc << 24));
                    return;
                }
                exact_done();  // queue full: exact now
                h = exact_h(a.qc, bc, yc, ib, iy);
                bin = hist_bin(h);
                if (!(h > 0.0f)) return;
            }
            else
            {
                if (!(ha > 0.0f)) return;
                h = ha;
                bin = (int)floorf(tt);
            }
        }
        else
        {
            exact_done();
            h = ha;
            bin = hist_bin(h);
            if (!(h > 0.0f)) return;
        }
        count_psm(bc, yc, bin);
    };

    for (uint32_t iter = 0;; iter++)
    {
        __syncthreads();
        if (tid == 0)
        {
            const uint32_t w = a.persistent ? atomicAdd(a.work, 1u) : (iter == 0 ? blockIdx.x : 0xFFFFFFFFu);
            uint32_t sp = 0xFFFFFFFFu;
            if (a.only) sp = w < *a.nonly_dev ? a.only[w] : 0xFFFFFFFFu;
            else if (PARTS)
            {
                if (iter == 0) sp = blockIdx.x / a.parts;
            }
            else
            {
                const uint32_t o = (a.obase ? *a.obase : 0u) + w;
                if (w < a.nspec && o < (a.olim ? *a.olim : a.nspec)) sp = a.order ? a.order[o] : o;
            }
            T.spec = sp;
        }
        __syncthreads();
        const uint32_t s = T.spec;
        if (s == 0xFFFFFFFFu) break;
        if (tid == 0)
        {
            T.best = 0;
            T.best_shp = 0;
            T.maxbits = 0;
            T.cpsms = 0;
            T.ndefer = 0;
            T.flags = WIDE ? HC_FLAG_WIDE : 0u;
            T.overflow = 0;
            T.bytes = 0;
            T.nv = 0;
            T.nlow = 0;
            T.ncu = 0;
        }
        for (uint32_t l = tid; l < a.nlen; l += nthr) T.win[l] = a.win[(size_t)s * a.nlen + l];
        for (uint32_t i = tid; i < kMaxClasses + 1; i += nthr) ucls[i] = 0ull;
        __syncthreads();
        if (!WIDE && !PARTS && a.wsplit && window_sum(T.win, a.nlen, lane) < a.wsplit) continue;  // k_search_small's
        const bool shared = PARTS && parts > 1;
        if (shared)
        {
            if (wid == 0) part_windows(T.win, a.nlen, blockIdx.x % a.parts, parts, lane);
        }
        else
            for (int i = kHistSm + tid; i < HC_HIST_BINS; i += nthr) a.hist[(size_t)s * HC_HIST_BINS + i] = 0;
        // valid peaks (dslim_query.cpp:625): dF < qion < max*scale - 1 - dF
        {
            const uint32_t lowlim = a.classes ? __ldg(&a.classes->maxkey) + a.dF : 0u;
            const uint32_t p0 = a.idx[s], p1 = a.idx[s + 1];
            for (uint32_t k = p0 + tid; k < p1; k += nthr)
            {
                const uint32_t q = a.moz[k];
                if (q > a.dF && (uint64_t)q + 1 + a.dF < a.maxbin)
                {
                    // packed sums stay exact only for intensities below 2^17
                    if (!WIDE && a.inten[k] >= (1u << 17)) T.overflow = 1;
                    const uint32_t slot = atomicAdd(&T.nv, 1u);
                    if (slot < HC_QALEN)
                    {
                        pmoz[slot] = q;
                        pint[slot] = a.inten[k];
                        if (q <= lowlim) low[atomicAdd(&T.nlow, 1u)] = slot;
                    }
                }
            }
        }
        __syncthreads();
        const uint32_t nv = T.nv < HC_QALEN ? T.nv : HC_QALEN;
        // The stream's atomics need not return the old words when no word can
        // reach a count of 128: if every list of the spectrum has a bucket of
        // its own (valid peaks more than 2*dF bins apart), a candidate's b (y)
        // count is at most its number of b (y) ions, (L-1)*maxz, below 128 for
        // every length; with intensities below 2^17 the sums stay below 2^24.
        if constexpr (!WIDE)
        {
            // warp w takes peaks i = w, w + nw, ...; its lanes the peaks j > i
            bool close = false;
            for (uint32_t i = (uint32_t)wid; i < nv; i += (uint32_t)(nthr >> 5))
            {
                const uint32_t x = pmoz[i];
                for (uint32_t j = i + 1 + (uint32_t)lane; j < nv; j += 32)
                {
                    const uint32_t y = pmoz[j];
                    close |= (x > y ? x - y : y - x) <= 2 * a.dF;
                }
            }
            close = __syncthreads_or(close);
            if (tid == 0) T.noret = (!close && a.lens[a.nlen - 1].half < 128u) ? 1u : 0u;
        }
        // the class adds: for each class, charge and valid peak whose bins
        // (q - dF .. q + dF) hold the class's y1 key, what the left-out
        // posting of every entry of the class would add there
        if (a.classes)
        {
            const uint32_t nz = a.maxz, tot = a.classes->n * nz, nlow = T.nlow;
            for (uint32_t i = tid; i < tot; i += nthr)
            {
                const uint32_t c = i / nz, z = i - c * nz;
                const uint32_t key = a.classes->key[c][z];
                unsigned long long acc = 0;
                for (uint32_t t = 0; t < nlow; t++)
                {
                    const uint32_t sl = low[t], q = pmoz[sl];
                    if (q <= key + a.dF && q + a.dF >= key) acc += (1ull << 40) | pint[sl];
                }
                if (acc) atomicAdd(&ucls[c], acc);
            }
        }
        __syncthreads();
        for (uint32_t i = tid; i < kMaxClasses + 1; i += nthr)
        {
            // packed: a count of 64 or more from a class alone is redone wide
            const unsigned long long u = ucls[i];
            if (!WIDE && (u >> 40) >= 64u) T.overflow = 1;
            T.upk[i] = ((uint32_t)(u >> 40) << 24) | (uint32_t)(u & 0xFFFFFFull);
            if (u)
            {
                T.cu = i;
                atomicAdd(&T.ncu, 1u);
            }
        }
        __syncthreads();
        // the set-up's tables are read: their space takes the scoring's (seen
        // by the scan after the first job's barriers)
        for (int i = tid; i < kLgSm; i += nthr) T.u.run.lgf[i] = a.qc->lgfact_f[i];
        for (int i = tid; i < kHistSm; i += nthr) T.u.run.hist[i] = 0;
        const uint32_t np = nv * nbin;
        my_best = 0;
        my_shp = 0;
        if (tid == 0)
            for (uint32_t l = 0; l < a.nlen; l++)
                // the reference's bA reads (of a window in parts, with its first)
                if (T.win[l].x <= T.win[l].y && (!shared || T.win[l].x == a.win[(size_t)s * a.nlen + l].x))
                    atomicAdd(&T.bytes, 4ull * (2 * a.dF + 2) * nv);

        // The spectrum's work is a sequence of jobs (length l, scorecard tile
        // t). Interior tile boundaries are row-table entries; a window's own
        // ends are widened to the nearest ones (see row_lo / row_hi). The
        // per-list bounds are pipelined: while job j streams, the row-table
        // words of job j+1's boundaries are in flight; right after its own
        // stream each thread turns them into job j+1's bounds (lnext, lend,
        // loff), and after the barrier that ends the stream the warps turn
        // those into job j+1's chunk offsets and {first posting, intensity}
        // per non-empty list, which only job j+1's stream reads. (Asking L2
        // for job j+1's postings at that point was measured: it cost more
        // issue slots than the latency it hid.)
        Job jb = first_job(T.win, a.nlen, tile);
        uint32_t pf_hi[kPf], ps_lo[kPf];
        // the bucket and the intensity of this thread's lists tid + m * nthr
        // (list = (valid peak, bin)): the same for every job of the spectrum
        uint32_t my_bkt[kPf];
#pragma unroll
        for (int m = 0; m < kPf; m++)
        {
            const uint32_t pr = tid + m * nthr;
            my_bkt[m] = 0u;
            if (pr < np)
            {
                const uint32_t k = pr / nbin, j = pr - k * nbin;
                my_bkt[m] = pmoz[k] - a.dF + j;
            }
        }
        uint32_t npass = 0;  // postings of entries inside the window (the reference visits exactly these)
        const uint32_t nw = (uint32_t)nthr >> 5, ng = (np + 31) >> 5;
        if (jb.l != kNoJob)
        {
            // the first job's boundaries, directly
            const LenS d = a.len[jb.l];
            const bool inter = !WIDE && job_interior(jb, d.n);
            for (uint32_t base = 0; base < np; base += (uint32_t)nthr)
            {
                const uint32_t pr = base + (uint32_t)tid;
                uint32_t cnt = 0;
                if (pr < np)
                {
                    const uint32_t k = pr / nbin, j = pr - k * nbin;
                    const uint32_t *col = d.rows + (size_t)(pmoz[k] - a.dF + j) * d.stride;
                    const uint32_t st = row_lo(col, jb.c0), en = row_hi(col, jb.c1);
                    if (inter && st < en) npass += en - st;
                    lnext[pr] = st;
                    lend[pr] = en;
                    cnt = st < en ? ((en + 3) >> 2) - (st >> 2) : 0u;
                    loff[pr] = cnt;
                }
                if (base + 32 * (uint32_t)wid < np) group_totals(cnt, (pr >> 5), lane, gt);
            }
            // the first job's scorecard: each candidate's y word starts with its class's adds
            {
                const uint32_t nt0 = jb.c1 - jb.c0;
                const uint8_t *cl0 = d.cls + jb.c0;
                for (uint32_t c = tid; c < nt0; c += nthr)
                {
                    const uint32_t k = __ldg(cl0 + c);
                    if constexpr (!WIDE)
                    {
                        const uint32_t wy = T.upk[k];
                        card[2 * c + 1] = wy;
                        npass += wy >> 24;
                    }
                    else
                    {
                        const W wy = ucls[k];
                        card[2 * c + 1] = wy;
                        npass += (uint32_t)(wy >> 40);
                    }
                }
            }
            __syncthreads();
            for (uint32_t g = nw - 1 - (uint32_t)wid; g < ng; g += nw)
                group_offsets(g, ng, loff, np, lane, gt, lnext, pint, nbin, coff, kinfo, &T.cchunks, &T.ncl);
            if (ng == 0 && tid == 0) T.cchunks = T.ncl = coff[0] = 0;
        }
        __syncthreads();
        while (jb.l != kNoJob)
        {
            const LenS d = a.len[jb.l];
            const uint32_t c0 = jb.c0, ntile = jb.c1 - jb.c0;
            const uint32_t C = T.cchunks;
            const uint32_t ncl = T.ncl;
            const uint32_t *co = coff;
            HC_PHASE(0);
            // ---- row-table words of the next job's boundaries, in flight ----
            const Job nj = next_job(jb, T.win, a.nlen, tile);
            const bool same = nj.l == jb.l;
            LenS dn;
            if (nj.l != kNoJob)
            {
                dn = same ? d : a.len[nj.l];
#pragma unroll
                for (int m = 0; m < kPf; m++)
                {
                    const uint32_t pr = tid + m * nthr;
                    if (pr < np)
                    {
                        const uint32_t *col = dn.rows + (size_t)my_bkt[m] * dn.stride;
                        pf_hi[m] = row_hi(col, nj.c1);
                        if (!same) ps_lo[m] = row_lo(col, nj.c0);
                    }
                }
            }
            // ---- stream the job's postings into the scorecard ----
            // A warp takes 32*G consecutive chunks; lane j handles chunks
            // q0 + j + 32g. All G loads are issued before any is used. A
            // posting is the byte offset of its scorecard word counted from
            // entry 0, so one subtraction gives its place in the tile and one
            // unsigned compare rejects entries outside the tile and padding.
            // Visited postings are counted per posting only in a window's end
            // tiles; an interior tile's lists hold exactly the tile's entries,
            // and their lengths were added when its bounds were set.
            uint32_t ovf = 0;  // largest word that an atomic returned (see count_full)
            auto stream = [&](auto no_return, auto count) {
            constexpr bool NR = decltype(no_return)::value;
            constexpr bool CNT = decltype(count)::value;
            (void)NR;
            (void)CNT;
            // packed: byte offsets of the tile's words; wide: word indexes
            [[maybe_unused]] const uint32_t base8 = c0 << kQpEntryShift, lim8 = ntile << kQpEntryShift;
            [[maybe_unused]] const uint32_t base2 = 2 * c0, lim2 = 2 * ntile;
            for (;;)
            {
                uint32_t q0 = 0;
                if (lane == 0) q0 = atomicAdd(&T.pnext, 32u * G);
                q0 = __shfl_sync(0xFFFFFFFFu, q0, 0);
                if (q0 >= C) break;
                uint4 v[G];
                uint32_t inte[G];
                // the list holding chunk q0, then for each group of 32 chunks the
                // list of every lane's chunk: lists that start inside the group
                // set one bit each at their first lane, and a lane's list is the
                // one before plus the bits at or below it
                uint32_t k0 = find_list(co, ncl, q0, lane);
                if (co[k0 + 1u] >= q0 + 32u * G)  // warp-uniform: the whole grab lies in list k0
                {
                    const uint2 ki = kinfo[k0];
                    const uint32_t p0 = (ki.x & ~3u) + 4u * (q0 + (uint32_t)lane - co[k0]);
                    const uint32_t li = ki.y;
#pragma unroll
                    for (int g = 0; g < G; g++)
                    {
                        inte[g] = li;
                        v[g] = __ldg(reinterpret_cast<const uint4 *>(d.qp + p0 + 128u * g));
                    }
                }
                else
#pragma unroll
                for (int g = 0; g < G; g++)
                {
                    const uint32_t kb = q0 + 32u * g;
                    const uint32_t kc = kb + (uint32_t)lane;
                    inte[g] = 0u;
                    v[g] = make_uint4(kQpostPad, kQpostPad, kQpostPad, kQpostPad);
                    if (kb < C && co[k0 + 1u] >= kb + 32u)  // warp-uniform
                    {
                        // the group's 32 chunks all lie in list k0 (most
                        // postings sit in long lists): one lookup for the warp
                        const uint2 ki = kinfo[k0];
                        const uint32_t pos = (ki.x & ~3u) + 4u * (kc - co[k0]);
                        inte[g] = ki.y;
                        v[g] = __ldg(reinterpret_cast<const uint4 *>(d.qp + pos));
                    }
                    else if (kb < C)  // warp-uniform
                    {
                        const uint32_t j1 = k0 + 1u + (uint32_t)lane;
                        const uint32_t u = (j1 <= ncl ? co[j1] : 0xFFFFFFFFu) - kb;  // >= 1
                        const uint32_t msk = __reduce_or_sync(0xFFFFFFFFu, u < 32u ? (1u << u) : 0u);
                        const uint32_t k = k0 + (uint32_t)__popc(msk & ((2u << lane) - 1u));
                        if (kc < C)
                        {
                            const uint2 ki = kinfo[k];
                            // a chunk never leaves its bucket (buckets start at
                            // multiples of 4, padded to them); its postings
                            // outside [first, end) belong to entries outside
                            // the tile and fail the index test below
                            const uint32_t pos = (ki.x & ~3u) + 4u * (kc - co[k]);
                            inte[g] = ki.y;
                            v[g] = __ldg(reinterpret_cast<const uint4 *>(d.qp + pos));
                        }
                        k0 = __shfl_sync(0xFFFFFFFFu, k, 31);  // the list holding chunk kb + 31
                    }
                }
#pragma unroll
                for (int g = 0; g < G; g++)
                {
                    const uint32_t xs[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
                    if constexpr (!WIDE)
                    {
                        const uint32_t add = (1u << 24) | inte[g];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                        {
                            // byte offset of the word in the tile; a posting
                            // outside the tile (or padding) adds to the lane's
                            // own sink word instead, so the atomic is not
                            // behind a branch
                            const uint32_t o = xs[e] - base8;
                            const bool in = o < lim8;
                            const uint32_t wa = in ? card_s + o : sink_s;
                            if constexpr (NR) red_shared_add(wa, add);
                            else
                            {
                                const uint32_t old = atom_shared_add(wa, add);
                                ovf = max(ovf, in ? old : 0u);
                            }
                            if constexpr (CNT) npass += in ? 1u : 0u;
                        }
                    }
                    else
                    {
                        const W add = (1ull << 40) | (W)inte[g];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                        {
                            const uint32_t w = (xs[e] >> 2) - base2;  // 2*(entry - c0) + isY
                            if (w < lim2)
                            {
                                atomicAdd(&card[w], add);
                                npass++;
                            }
                        }
                    }
                }
            }
            };
            if constexpr (WIDE) stream(std::false_type{}, std::true_type{});
            else
            {
                const bool cnt = !job_interior(jb, d.n);
                if (T.noret)
                {
                    if (cnt) stream(std::true_type{}, std::true_type{});
                    else stream(std::true_type{}, std::false_type{});
                }
                else
                {
                    if (cnt) stream(std::false_type{}, std::true_type{});
                    else stream(std::false_type{}, std::false_type{});
                }
            }
            if (!WIDE && count_full(__reduce_max_sync(0xFFFFFFFFu, ovf)) && lane == 0) T.overflow = 1;
            // ---- the next job's list bounds ----
            if (nj.l != kNoJob)
            {
                const bool inter = !WIDE && job_interior(nj, dn.n);
#pragma unroll
                for (int m = 0; m < kPf; m++)
                {
                    const uint32_t pr = tid + m * nthr;
                    uint32_t cnt = 0, st = 0, en = 0;
                    if (pr < np)
                    {
                        st = same ? lend[pr] : ps_lo[m];
                        en = pf_hi[m];
                        if (inter && st < en) npass += en - st;
                        lnext[pr] = st;
                        lend[pr] = en;
                        cnt = st < en ? ((en + 3) >> 2) - (st >> 2) : 0u;
                        loff[pr] = cnt;
                    }
                    if (m * nthr + 32 * wid < np) group_totals(cnt, pr >> 5, lane, gt);
                }
                // lists past kPf * nthr (small blocks, wide bin windows): directly
                for (uint32_t base = kPf * nthr; base < np; base += (uint32_t)nthr)
                {
                    const uint32_t pr = base + (uint32_t)tid;
                    uint32_t cnt = 0, st = 0, en = 0;
                    if (pr < np)
                    {
                        const uint32_t k = pr / nbin, j = pr - k * nbin;
                        const uint32_t *col = dn.rows + (size_t)(pmoz[k] - a.dF + j) * dn.stride;
                        st = same ? lend[pr] : row_lo(col, nj.c0);
                        en = row_hi(col, nj.c1);
                        if (inter && st < en) npass += en - st;
                        lnext[pr] = st;
                        lend[pr] = en;
                        cnt = st < en ? ((en + 3) >> 2) - (st >> 2) : 0u;
                        loff[pr] = cnt;
                    }
                    if (base + 32 * (uint32_t)wid < np) group_totals(cnt, pr >> 5, lane, gt);
                }
            }
            __syncthreads();
            HC_PHASE(1);
            // ---- the next job's chunk offsets (one group of 32 lists per warp,
            // the last warps first: the first warps computed the bounds) ----
            if (nj.l != kNoJob)
            {
                for (uint32_t g = nw - 1 - (uint32_t)wid; g < ng; g += nw)
                    group_offsets(g, ng, loff, np, lane, gt, lnext, pint, nbin, coff, kinfo, &T.cchunks, &T.ncl);
                if (ng == 0 && tid == 0) T.cchunks = T.ncl = coff[0] = 0;
            }
            // ---- every candidate that reached min_shp ----
            // cpsms, histogram and the top hit (see score_one). The packed tile
            // is scanned four candidates per lane and step; a warp collects its
            // qualifying candidates in its own ring and scores them 32 at a
            // time (all lanes busy), then clears the words it scanned.
            const uint32_t key_l = jb.l << 24;
            if constexpr (!WIDE)
            {
                const uint4 *c4 = reinterpret_cast<const uint4 *>(card);
                // the warp's ring: an entry is one lane's four candidates of a
                // step, (first candidate << 4) | the ones that qualify, so a step
                // takes one ballot and one store whatever it finds (an entry a
                // candidate, placed by a returning shared-memory atomic and a
                // loop over the lane's candidates, took 27 instructions more a
                // step). A pop scores one candidate of each of 32 entries and
                // puts back those that hold another (one in eight).
                uint32_t fill = 0, head = 0;  // warp-uniform
                const uint32_t lt = (1u << lane) - 1u;
                auto put = [&](bool any, uint32_t e) {
                    const uint32_t b = __ballot_sync(0xFFFFFFFFu, any);
                    if (any) wq[(head + fill + (uint32_t)__popc(b & lt)) & (kWQ - 1)] = e;
                    fill += (uint32_t)__popc(b);
                };
                auto pop_score = [&](uint32_t cnt) {
                    __syncwarp();
                    uint32_t rest = 0;
                    if ((uint32_t)lane < cnt)
                    {
                        const uint32_t e = wq[(head + lane) & (kWQ - 1)];
                        const uint32_t k = (uint32_t)__ffs(e) - 1u;
                        rest = e & (e - 1u);
                        const uint32_t loc = (e >> 4) + (k & 1u) + ((k & 2u) << 5);
                        uint32_t bc, yc, shp;
                        uint64_t ib, iy;
                        decode<false>(card, loc, bc, yc, shp, ib, iy);
                        score_one(bc, yc, ib, iy, shp, ~(key_l | ((c0 + loc) & 0xFFFFFF)));
                    }
                    head += cnt;
                    fill -= cnt;
                    put((rest & 15u) != 0u, rest);
                    __syncwarp();
                };
                const uint32_t first = 4 * (tid - (uint32_t)lane), step = 4 * nthr;
                const uint32_t thr4 = min(a.thr, 255u) * 0x01010101u;
                const bool thr7 = a.thr <= 127u;
                for (uint32_t base = first; base < ntile; base += step)
                {
                    // words past ntile are zero up to the tile's end (the clear
                    // leaves every word past the next job's end zero) and past
                    // it belong to the queue: a window's last step is masked
                    const uint32_t ca = base + 2 * (uint32_t)lane, cb = ca + 64;
                    const uint4 wa = c4[ca >> 1];
                    const uint4 wb = c4[cb >> 1];
                    // the four candidates' counts (the top bytes of their b and y
                    // words) summed and compared as bytes: candidates ca, ca + 1,
                    // cb, cb + 1 in bytes 0..3 (each count < 128, so no carry)
                    const uint32_t bw = __byte_perm(__byte_perm(wa.x, wa.z, 0x0073u), __byte_perm(wb.x, wb.z, 0x0073u),
                                                    0x5410u);
                    const uint32_t yw = __byte_perm(__byte_perm(wa.y, wa.w, 0x0073u), __byte_perm(wb.y, wb.w, 0x0073u),
                                                    0x5410u);
                    // (a plain add: each sum is below 256). Byte k's top bit of m:
                    // its sum reaches thr; for thr <= 127, (sum | 0x80) - thr
                    // keeps the top bit exactly when sum >= thr, with no borrow
                    // between bytes, and a sum of 128 or more has it already
                    const uint32_t sw = bw + yw;
                    uint32_t m = thr7 ? (((sw | 0x80808080u) - thr4) | sw) & 0x80808080u
                                      : (__vcmpgeu4(sw, thr4) & 0x01010101u) << 7;
                    if (base + 128u > ntile)  // warp-uniform
                        m &= (ca < ntile ? 0x80u : 0u) | (ca + 1u < ntile ? 0x8000u : 0u) |
                             (cb < ntile ? 0x800000u : 0u) | (cb + 1u < ntile ? 0x80000000u : 0u);
                    // bytes' top bits to bits 0..3 (the products land apart)
                    const uint32_t nib = ((m >> 7) * 0x01020408u) >> 24;
                    if (!__any_sync(0xFFFFFFFFu, m)) continue;
                    put(m != 0u, (ca << 4) | nib);
                    while (fill >= 32) pop_score(32);
                }
                while (fill) pop_score(min(fill, 32u));
                // the next job's candidates and their classes (its scorecard start)
                const uint32_t nn = nj.l != kNoJob ? nj.c1 - nj.c0 : 0u;
                const uint8_t *ncls = nn ? a.len[nj.l].cls + nj.c0 : nullptr;
                // the warp's own words, now read: the next job's start there,
                // four consecutive candidates per lane (b word zero, y word
                // its class's adds; zero past the next job's end)
                uint4 *z4 = reinterpret_cast<uint4 *>(card);
                const uint32_t lim = max(ntile, nn);
                const bool al4 = (nj.c0 & 3u) == 0u;  // class bytes readable as one word (warp-uniform)
                uint32_t base = first;
                // The steps that lie in the next job. Most spectra have a peak at the
                // y1 keys of one class (K or R at the end) or of none: a compare
                // takes the place of the table, and with none the classes are
                // not read at all; without the edges' checks, and with stores that
                // meet no bank twice, a step takes half the instructions
                // (2,432 open-search spectra: 6.26 -> 6.06 ms).
                const uint32_t ncu = T.ncu;
                if (ncu == 0u)
                    for (; base + 128u <= nn; base += step)
                        z4[(base >> 1) + (uint32_t)lane] = z4[(base >> 1) + 32u + (uint32_t)lane] =
                            make_uint4(0u, 0u, 0u, 0u);
                else if (ncu == 1u && al4)
                {
                    const uint32_t cu4 = T.cu * 0x01010101u, cu_y = T.upk[T.cu];
                    const uint16_t *cp = reinterpret_cast<const uint16_t *>(ncls) + lane;
                    uint32_t hits = 0;
                    for (; base + 128u <= nn; base += step)
                    {
                        const uint32_t k4 = __ldg(cp + (base >> 1)) | (uint32_t)__ldg(cp + (base >> 1) + 32) << 16;
                        // class ids stay below 128: a byte's top bit is set where it is the class
                        const uint32_t e = (0x80808080u - (k4 ^ cu4)) & 0x80808080u;
                        hits += (uint32_t)__popc(e);
                        uint4 *z = z4 + (base >> 1) + lane;
                        z[0] = make_uint4(0u, cu_y & byte_sign<0x8888>(e), 0u, cu_y & byte_sign<0x9999>(e));
                        z[32] = make_uint4(0u, cu_y & byte_sign<0xAAAA>(e), 0u, cu_y & byte_sign<0xBBBB>(e));
                    }
                    npass += hits * (cu_y >> 24);
                }
                for (; base < lim; base += step)
                {
                    const uint32_t c = base + 4 * (uint32_t)lane;
                    uint32_t k4 = kClassNone * 0x01010101u;
                    if (c < nn)
                    {
                        if (al4) k4 = __ldg(reinterpret_cast<const uint32_t *>(ncls + c));
                        else
                            k4 = (uint32_t)__ldg(ncls + c) | ((uint32_t)__ldg(ncls + c + 1) << 8) |
                                 ((uint32_t)__ldg(ncls + c + 2) << 16) | ((uint32_t)__ldg(ncls + c + 3) << 24);
                        if (c + 4 > nn)
                        {
                            const uint32_t keep = (1u << (8 * (nn - c))) - 1u;  // bytes of candidates < nn
                            k4 = (k4 & keep) | (kClassNone * 0x01010101u & ~keep);
                        }
                    }
                    const uint32_t y0 = T.upk[k4 & 0xFFu], y1 = T.upk[(k4 >> 8) & 0xFFu];
                    const uint32_t y2 = T.upk[(k4 >> 16) & 0xFFu], y3 = T.upk[k4 >> 24];
                    if (c < lim)  // words from lim on are zero already (and past the tile not its own)
                    {
                        z4[c >> 1] = make_uint4(0u, y0, 0u, y1);
                        z4[(c >> 1) + 1] = make_uint4(0u, y2, 0u, y3);
                    }
                    npass = __dp4a(__byte_perm(__byte_perm(y0, y1, 0x0073u), __byte_perm(y2, y3, 0x0073u), 0x5410u),
                                   0x01010101u, npass);  // + the four counts (top bytes)
                }
            }
            else
            {
                // wide words: one candidate per thread, every one checked, then
                // set to the next job's start (y word: class adds; zero past its end)
                const uint32_t nn = nj.l != kNoJob ? nj.c1 - nj.c0 : 0u;
                const uint8_t *ncls = nn ? a.len[nj.l].cls + nj.c0 : nullptr;
                const uint32_t lim = max(ntile, nn);
                for (uint32_t c = tid; c < lim; c += nthr)
                {
                    if (c < ntile)
                    {
                        uint32_t bc, yc, shp;
                        uint64_t ib, iy;
                        decode<WIDE>(card, c, bc, yc, shp, ib, iy);
                        if (shp >= a.min_shp && shp != 0)
                            score_one(bc, yc, ib, iy, shp, ~(key_l | ((c0 + c) & 0xFFFFFF)));
                    }
                    W wy = 0;
                    if (c < nn)
                    {
                        wy = ucls[__ldg(ncls + c)];
                        npass += (uint32_t)(wy >> 40);
                    }
                    card[2 * c] = 0;
                    card[2 * c + 1] = wy;
                }
            }
            if (a.phase && tid == 0) T.cnt[0] += 1;
            HC_PHASE(2);
            if (tid == 0) T.pnext = 0;
            __syncthreads();
            HC_PHASE(3);
            jb = nj;
        }
        // ---- candidates whose sign or bin the float estimate left open ----
        if (!WIDE)
        {
            const uint32_t nd = min(T.ndefer, a.defer_cap);
            for (uint32_t i = tid; i < nd; i += nthr)
            {
                uint32_t bc, yc, shp;
                uint64_t ib, iy;
                const uint2 w = defer[i];
                decode_packed(w.x, w.y, bc, yc, shp, ib, iy);
                exact_done();
                const float h = exact_h(a.qc, bc, yc, ib, iy);
                if (h > 0.0f) count_psm(bc, yc, hist_bin(h));
            }
        }
        // postings visited: those of entries inside the window
        npass = __reduce_add_sync(0xFFFFFFFFu, npass);
        if (lane == 0 && npass) atomicAdd(&T.bytes, 4ull * npass);
        // the top hit's shared ions come from the thread that found it
        if (my_best != 0 && my_best == T.best) T.best_shp = my_shp;
        __syncthreads();
        HC_PHASE(5);
        // ---- write the spectrum's results ----
        if (shared)
        {
            for (int i = tid; i < kHistSm; i += nthr)
                if (T.u.run.hist[i]) atomicAdd(&a.hist[(size_t)s * HC_HIST_BINS + i], T.u.run.hist[i]);
            if (wid == 0)
            {
                uint32_t cps = 0;
#pragma unroll
                for (int i = 0; i < kHistSm; i += 32) cps += T.u.run.hist[i + lane];
                cps = __reduce_add_sync(0xFFFFFFFFu, cps) + T.cpsms;
                if (lane == 0)
                    end_part(a, s, blockIdx.x % a.parts, parts, PartSum{T.best, T.bytes, T.best_shp, T.flags, cps, T.overflow});
            }
            continue;
        }
        if (!WIDE && T.overflow)
        {
            if (tid == 0)
            {
                const uint32_t wi = atomicAdd(a.nwide, 1u);
                a.wide_list[wi] = s;
            }
            continue;
        }
        for (int i = tid; i < kHistSm; i += nthr) a.hist[(size_t)s * HC_HIST_BINS + i] = T.u.run.hist[i];
        if (wid == 0)
        {
            uint32_t cps = 0;
#pragma unroll
            for (int i = 0; i < kHistSm; i += 32) cps += T.u.run.hist[i + lane];
            cps = __reduce_add_sync(0xFFFFFFFFu, cps) + T.cpsms;
            if (lane == 0) write_result(a, s, cps, T.flags, T.bytes, T.best, T.best_shp);
        }
    }
    if (a.phase && tid == 0)
    {
        for (int k = 0; k < kPhases; k++) atomicAdd(&a.phase[k], T.ph[k]);
        for (int k = 0; k < 4; k++) atomicAdd(&a.phase[kPhases + k], T.cnt[k]);
    }
}

// ---- the search of small windows ------------------------------------------------
// k_search gives a length of a spectrum's windows a job of its own: list bounds,
// chunk offsets, two barriers, whatever the window holds. Where windows hold a few
// hundred candidates (a small database, a narrow tolerance) that fixed work is all
// there is: 34 jobs a spectrum, most of their lists empty, some 2,500 warp
// instructions each. k_search_small packs the windows of all lengths into one
// scorecard instead (each from a multiple of 128 candidates on, so that a step of the
// scan lies in one length) and walks the (length, list) pairs flat, a thread a
// pair: its two row-table words say whether the list holds anything; the non-empty
// ones (a tenth, in a database of 20,000 peptides) go through a ring of the warp's
// and are read 32 at a time, a lane a list, long ones by the whole warp. A spectrum
// whose windows together exceed the scorecard takes it as often as it needs.
// The same results as k_search: the same words, the same scoring.
constexpr int kSmThreads = 256;      // threads of a CTA
constexpr uint32_t kSmTile = 3584;   // candidates of the scorecard (a multiple of 128, < 2^16): four CTAs an SM
                                     // then leave it the 60 KB of L1 (see kSmemKeepL1)
constexpr uint32_t kSmRing = 64;     // lists waiting per warp (a power of two, >= 31 + 32)
constexpr uint32_t kSmLong = 8;      // chunks from which the warp reads a list together
constexpr uint32_t kSmStep = 128;
constexpr uint32_t kSmWQ = 128;      // candidates waiting per warp (a power of two, >= 31 + 64)
constexpr uint32_t kSmCtas = 4;
// launch shapes picked for a context that chose none (see launch_packed)
constexpr uint32_t kWideWindows = 512;  // (spectrum, length) pairs per SM up to which windows are searched four ways
constexpr uint32_t kMaxParts = 32, kPartMin = 32768, kPartMinFew = 4096;  // see auto_parts
constexpr uint32_t kAutoSmallLog2 = 15, kAutoAllSmall = 1u << 16, kAutoOrder = 1024;

struct SmSeg
{
    const uint32_t *rows;  // of the first bucket, at the segment's first row-table entry
    const uint32_t *qp;
    uint32_t stride, drow;  // ... and how far its last one is
    uint32_t off, lim;      // byte offset of its first entry's words, bytes of its words
    uint32_t card;          // where they lie in the scorecard (shared-window address)
};

struct SmSmem
{
    uint32_t card[2 * kSmTile];
    uint2 ring[kSmThreads / 32][kSmRing];
    uint16_t wq[kSmThreads / 32][kSmWQ];
    uint2 defer[kDefer];
    unsigned long long ucls[kMaxClasses + 1];
    SmSeg seg[HC_MAX_LENGTHS];
    uint32_t low[HC_QALEN];
    uint32_t pmoz[HC_QALEN], pint[HC_QALEN];
    uint32_t upk[kMaxClasses + 1];
    float lgf[kLgTable];  // (all of it: an overflowing count, redone wide, reads inside)
    uint32_t hist[kHistSm];
    int2 win[HC_MAX_LENGTHS];
    uint32_t vbase[HC_MAX_LENGTHS + 1];  // first packed candidate of each length
    uint32_t sink[32];
    uint8_t stepl[kSmTile / kSmStep];    // the length a step of the scan lies in (0xFF: none)
    unsigned long long best, bytes;
    uint32_t best_shp, maxbits, cpsms, flags, overflow, spec, nv, nlow, ndefer, nseg, cand;
};

static size_t small_smem(uint32_t dF) { return sizeof(SmSmem) + 4 * (size_t)HC_QALEN * (2 * dF + 1); }

__global__ void __launch_bounds__(kSmThreads, 4) k_search_small(SearchArgs a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SmSmem &S = *reinterpret_cast<SmSmem *>(smem);
    uint32_t *lbkt = reinterpret_cast<uint32_t *>(smem + sizeof(SmSmem));  // bucket of each list
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int nthr = kSmThreads;
    const uint32_t nbin = 2 * a.dF + 1;
    const uint32_t card_s = (uint32_t)__cvta_generic_to_shared(S.card);
    const uint32_t sink_s = (uint32_t)__cvta_generic_to_shared(S.sink) + 4u * (uint32_t)lane;
    uint16_t *wq = S.wq[wid];
    uint2 *ring = S.ring[wid];
    for (int i = tid; i < kLgTable; i += nthr) S.lgf[i] = a.qc->lgfact_f[i];
    if (a.follows) after_predecessor();
    release_successor();

    uint32_t my_cps = 0, my_fl = 0, my_shp = 0;
    unsigned long long my_best = 0;
    auto hist_add = [&](int bin) {
        if (bin < kHistSm) atomicAdd(&S.hist[bin], 1u);
        else atomicAdd(&a.hist[(size_t)S.spec * HC_HIST_BINS + (uint32_t)bin], 1u);
    };
    auto count_psm = [&](uint32_t bc, uint32_t yc, int bin) {
        my_cps++;
        if (bc >= (uint32_t)kRefMaxShp || yc >= (uint32_t)kRefMaxShp) my_fl |= HC_FLAG_LGFACT_OOB;
        if (bin >= HC_HIST_BINS || bin < 0) { my_fl |= HC_FLAG_HIST_OOB; bin = bin < 0 ? 0 : HC_HIST_BINS - 1; }
        hist_add(bin);
    };
    // one candidate, as k_search scores it
    auto score_one = [&](uint32_t wb, uint32_t wy, uint32_t key_lo) {
        uint32_t bc, yc, shp;
        uint64_t ib, iy;
        decode_packed(wb, wy, bc, yc, shp, ib, iy);
        const float ha = approx_h(S.lgf, bc, yc, ib, iy);
        const float runmax = __uint_as_float(*(volatile uint32_t *)&S.maxbits);
        if (ha >= runmax - kNear)
        {
            if (ha > runmax) atomicMax(&S.maxbits, __float_as_uint(ha));
            const float he = exact_h(a.qc, bc, yc, ib, iy);
            if (he > 0.0f)
            {
                const unsigned long long key = ((unsigned long long)__float_as_uint(he) << 32) | key_lo;
                if (key > my_best)
                {
                    my_best = key;
                    my_shp = shp;
                }
                atomicMax(&S.best, key);
            }
        }
        const float tt = ha * 10.0f + 0.5f;
        const float fr = tt - floorf(tt);
        if (fabsf(ha) <= kApproxErr * 4.0f || bin_open(ha, fr))
        {
            const uint32_t di = atomicAdd(&S.ndefer, 1u);
            if (di < a.defer_cap)
            {
                S.defer[di] = make_uint2(wb, wy);
                return;
            }
            const float h = exact_h(a.qc, bc, yc, ib, iy);
            if (h > 0.0f) count_psm(bc, yc, hist_bin(h));
        }
        else if (ha > 0.0f) count_psm(bc, yc, (int)floorf(tt));
    };

    for (uint32_t iter = 0;; iter++)
    {
        __syncthreads();
        if (tid == 0)
        {
            const uint32_t w = atomicAdd(a.work, 1u);
            const uint32_t o = (a.obase ? *a.obase : 0u) + w;
            S.spec = w < a.nspec && o < a.nspec ? (a.order ? a.order[o] : o) : 0xFFFFFFFFu;
            S.best = 0;
            S.best_shp = 0;
            S.maxbits = 0;
            S.cpsms = 0;
            S.ndefer = 0;
            S.flags = 0;
            S.overflow = 0;
            S.bytes = 0;
            S.nv = 0;
            S.nlow = 0;
        }
        for (uint32_t i = tid; i < kMaxClasses + 1; i += nthr) S.ucls[i] = 0ull;
        __syncthreads();
        const uint32_t s = S.spec;
        if (s == 0xFFFFFFFFu) break;
        // the windows' places in the packed candidates, by warp 0 (two lengths a lane)
        if (wid == 0)
        {
            uint32_t sz[2], tot = 0, cand = 0;
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                const uint32_t l = 2 * (uint32_t)lane + h;
                const int2 w = l < a.nlen ? a.win[(size_t)s * a.nlen + l] : make_int2(1, 0);
                S.win[l] = w;
                sz[h] = w.x <= w.y ? ((uint32_t)(w.y - w.x) + kSmStep) / kSmStep * kSmStep : 0u;
                tot += sz[h];
                cand += w.x <= w.y ? (uint32_t)(w.y - w.x) + 1u : 0u;
            }
            cand = __reduce_add_sync(0xFFFFFFFFu, cand);
            if (lane == 0) S.cand = cand;
            uint32_t x = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            S.vbase[2 * lane] = x - tot;
            S.vbase[2 * lane + 1] = x - tot + sz[0];
            if (lane == 31) S.vbase[HC_MAX_LENGTHS] = x;
        }
        // valid peaks (dslim_query.cpp:625): dF < qion < max*scale - 1 - dF
        else
        {
            const uint32_t lowlim = a.classes ? __ldg(&a.classes->maxkey) + a.dF : 0u;
            const uint32_t p1 = a.idx[s + 1];
            for (uint32_t k = a.idx[s] + tid - 32; k < p1; k += nthr - 32)
            {
                const uint32_t q = a.moz[k];
                if (q > a.dF && (uint64_t)q + 1 + a.dF < a.maxbin)
                {
                    const uint32_t in = a.inten[k];
                    // packed sums stay exact only for intensities below 2^17
                    if (in >= (1u << 17)) S.overflow = 1;
                    const uint32_t slot = atomicAdd(&S.nv, 1u);
                    if (slot < HC_QALEN)
                    {
                        S.pmoz[slot] = q;
                        S.pint[slot] = in;
                        if (q <= lowlim) S.low[atomicAdd(&S.nlow, 1u)] = slot;
                    }
                }
            }
        }
        __syncthreads();
        if (a.wsplit && S.cand >= a.wsplit) continue;  // k_search's
        for (int i = tid; i < HC_HIST_BINS; i += nthr)
        {
            if (i < kHistSm) S.hist[i] = 0;
            else a.hist[(size_t)s * HC_HIST_BINS + i] = 0;
        }
        const uint32_t nv = S.nv < HC_QALEN ? S.nv : HC_QALEN;
        const uint32_t np = nv * nbin, vtot = S.vbase[HC_MAX_LENGTHS];
        // the class adds (see k_search), the lists' buckets
        if (a.classes)
        {
            const uint32_t nz = a.maxz, tot = a.classes->n * nz, nlow = S.nlow;
            for (uint32_t i = tid; i < tot; i += nthr)
            {
                const uint32_t c = i / nz, z = i - c * nz;
                const uint32_t key = a.classes->key[c][z];
                unsigned long long acc = 0;
                for (uint32_t t = 0; t < nlow; t++)
                {
                    const uint32_t sl = S.low[t], q = S.pmoz[sl];
                    if (q <= key + a.dF && q + a.dF >= key) acc += (1ull << 40) | S.pint[sl];
                }
                if (acc) atomicAdd(&S.ucls[c], acc);
            }
        }
        for (uint32_t i = tid; i < np; i += nthr)
        {
            const uint32_t k = i / nbin;
            lbkt[i] = S.pmoz[k] - a.dF + (i - k * nbin);
        }
        __syncthreads();
        for (uint32_t i = tid; i < kMaxClasses + 1; i += nthr)
        {
            // packed: a count of 64 or more from a class alone is redone wide
            const unsigned long long u = S.ucls[i];
            if ((u >> 40) >= 64u) S.overflow = 1;
            S.upk[i] = ((uint32_t)(u >> 40) << 24) | (uint32_t)(u & 0xFFFFFFull);
        }
        if (tid < (int)a.nlen && S.win[tid].x <= S.win[tid].y)
            atomicAdd(&S.bytes, 4ull * (2 * a.dF + 2) * nv);  // the reference's bA reads
        my_best = 0;
        my_shp = my_cps = my_fl = 0;
        uint32_t npass = 0, ovf = 0;
        for (uint32_t v0 = 0; v0 < vtot; v0 += kSmTile)
        {
            const uint32_t v1 = min(vtot, v0 + kSmTile), used = v1 - v0;
            // the steps' lengths and the lengths' pieces of this scorecard
            if (tid < (int)(kSmTile / kSmStep))
            {
                const uint32_t v = v0 + kSmStep * (uint32_t)tid;
                uint32_t l = 0xFFu;
                if (v < v1)
                {
                    uint32_t lo = 0, hi = HC_MAX_LENGTHS - 1;  // the last length with vbase <= v
                    while (lo < hi)
                    {
                        const uint32_t m = (lo + hi + 1) >> 1;
                        if (S.vbase[m] <= v) lo = m;
                        else hi = m - 1;
                    }
                    l = lo;
                }
                S.stepl[tid] = (uint8_t)l;
            }
            // (lengths in order: the pieces' list is the range [l0, l1] of those not empty here)
            if (wid == kSmThreads / 32 - 1)
            {
                uint32_t n = 0;
                for (int h = 0; h < 2; h++)
                {
                    const uint32_t l = 32 * h + (uint32_t)lane;
                    const uint32_t b0 = S.vbase[l], b1 = S.vbase[l + 1];
                    const bool in = b0 < b1 && b0 < v1 && b1 > v0;
                    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, in);
                    if (in)
                    {
                        const int2 w = S.win[l];
                        const uint32_t skip = v0 > b0 ? v0 - b0 : 0u;  // candidates of earlier scorecards
                        const uint32_t c0 = (uint32_t)w.x + skip, c1 = min((uint32_t)w.y + 1u, c0 + (v1 - max(b0, v0)));
                        const LenS d = a.len[l];
                        SmSeg g;
                        g.rows = d.rows + c0 / kRowG;
                        g.qp = d.qp;
                        g.stride = d.stride;
                        g.drow = (c1 + kRowG - 1) / kRowG - c0 / kRowG;
                        g.off = c0 << kQpEntryShift;
                        g.lim = (c1 - c0) << kQpEntryShift;
                        g.card = card_s + 8u * (max(b0, v0) - v0);
                        S.seg[n + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = g;
                    }
                    n += (uint32_t)__popc(bal);
                }
                if (lane == 0) S.nseg = n;
            }
            __syncthreads();
            const uint32_t nseg = S.nseg;
            // every candidate's start: b word zero, y word its class's adds (zero past its window)
            for (uint32_t c = 4 * (uint32_t)tid; c < used; c += 4 * nthr)
            {
                const uint32_t l = S.stepl[c / kSmStep];
                const int2 w = S.win[l];
                const uint32_t e = (uint32_t)w.x + (v0 + c - S.vbase[l]);  // entry of the first of four
                const uint8_t *cl = a.len[l].cls + e;
                const uint32_t left = (uint32_t)w.y + 1u > e ? (uint32_t)w.y + 1u - e : 0u;
                uint32_t y[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                {
                    y[i] = (uint32_t)i < left ? S.upk[__ldg(cl + i)] : 0u;
                    npass += y[i] >> 24;
                }
                uint4 *z4 = reinterpret_cast<uint4 *>(S.card);
                z4[c >> 1] = make_uint4(0u, y[0], 0u, y[1]);
                z4[(c >> 1) + 1] = make_uint4(0u, y[2], 0u, y[3]);
            }
            __syncthreads();
            // ---- the lists: (piece, list) pairs, a thread a pair ----
            auto add4 = [&](const uint4 v, const SmSeg &g, uint32_t inten) {
                const uint32_t add = (1u << 24) | inten;
                const uint32_t xs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                {
                    const uint32_t o = xs[e] - g.off;
                    const bool in = o < g.lim;
                    const uint32_t old = atom_shared_add(in ? g.card + o : sink_s, add);
                    ovf = max(ovf, in ? old : 0u);
                    npass += in ? 1u : 0u;
                }
            };
            uint32_t qn = 0, qh = 0;  // ring fill and head (warp-uniform)
            auto drain = [&](uint32_t cnt) {
                __syncwarp();
                if ((uint32_t)lane < cnt)
                {
                    const uint2 r = ring[(qh + (uint32_t)lane) & (kSmRing - 1)];
                    const SmSeg g = S.seg[r.y >> 20];
                    const uint32_t pr = (r.y >> 4) & 0xFFFFu, nch = r.y & 0xFu;
                    const uint4 *p = reinterpret_cast<const uint4 *>(g.qp) + r.x;
                    const uint32_t inten = S.pint[pr / nbin];
                    uint4 v = __ldg(p);
                    for (uint32_t c = 1; c < nch; c++)
                    {
                        const uint4 nx = __ldg(p + c);
                        add4(v, g, inten);
                        v = nx;
                    }
                    add4(v, g, inten);
                }
                __syncwarp();
                qh += cnt;
                qn -= cnt;
            };
            constexpr int U = 4;  // pairs whose row-table words are in flight
            uint32_t sg = np ? (uint32_t)tid / np : 0u, pr = (uint32_t)tid - sg * np;
            const uint32_t dsg = np ? nthr / np : 0u, dpr = nthr - dsg * np;
            const uint32_t pairs = nseg * np, iters = (pairs + nthr * U - 1) / (nthr * U);
            for (uint32_t it = 0; it < iters; it++)
            {
                uint32_t st[U], en[U], id[U];
#pragma unroll
                for (int u = 0; u < U; u++)
                {
                    st[u] = en[u] = 0;
                    id[u] = (sg << 20) | (pr << 4);
                    if (sg < nseg)
                    {
                        const SmSeg &g = S.seg[sg];
                        const uint32_t *col = g.rows + (size_t)lbkt[pr] * g.stride;
                        st[u] = __ldg(col);
                        en[u] = __ldg(col + g.drow);
                    }
                    sg += dsg;
                    pr += dpr;
                    if (pr >= np) { pr -= np; sg++; }
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                {
                    const uint32_t nch = st[u] < en[u] ? ((en[u] + 3) >> 2) - (st[u] >> 2) : 0u;
                    const bool shrt = nch != 0u && nch < kSmLong;
                    const uint32_t b = __ballot_sync(0xFFFFFFFFu, shrt);
                    if (shrt)
                        ring[(qh + qn + (uint32_t)__popc(b & ((1u << lane) - 1u))) & (kSmRing - 1)] =
                            make_uint2(st[u] >> 2, id[u] | nch);
                    qn += (uint32_t)__popc(b);
                    if (qn >= 32) drain(32);
                    for (uint32_t lb = __ballot_sync(0xFFFFFFFFu, nch >= kSmLong); lb; lb &= lb - 1)
                    {
                        const int src = __ffs(lb) - 1;
                        const uint32_t q0 = __shfl_sync(0xFFFFFFFFu, st[u] >> 2, src);
                        const uint32_t n = __shfl_sync(0xFFFFFFFFu, nch, src), i = __shfl_sync(0xFFFFFFFFu, id[u], src);
                        const SmSeg g = S.seg[i >> 20];
                        const uint32_t inten = S.pint[((i >> 4) & 0xFFFFu) / nbin];
                        for (uint32_t c = (uint32_t)lane; c < n; c += 32)
                            add4(__ldg(reinterpret_cast<const uint4 *>(g.qp) + q0 + c), g, inten);
                    }
                }
            }
            if (qn) drain(qn);
            __syncthreads();
            // ---- every candidate that reached min_shp (see k_search's scan) ----
            const uint4 *c4 = reinterpret_cast<const uint4 *>(S.card);
            uint32_t fill = 0, head = 0;
            auto pop_score = [&](uint32_t cnt) {
                __syncwarp();
                if ((uint32_t)lane < cnt)
                {
                    const uint32_t loc = wq[(head + (uint32_t)lane) & (kSmWQ - 1)];
                    const uint32_t l = S.stepl[loc / kSmStep];
                    const uint32_t e = (uint32_t)S.win[l].x + (v0 + loc - S.vbase[l]);
                    const uint2 w = reinterpret_cast<const uint2 *>(S.card)[loc];
                    score_one(w.x, w.y, ~((l << 24) | (e & 0xFFFFFFu)));
                }
                __syncwarp();
                head += cnt;
                fill -= cnt;
            };
            for (uint32_t base = 64 * (uint32_t)wid; base < used; base += 64 * (nthr / 32))
            {
                const uint32_t c = base + 2 * (uint32_t)lane;
                const uint4 w = c4[c >> 1];
                const uint32_t s0 = (w.x >> 24) + (w.y >> 24), s1 = (w.z >> 24) + (w.w >> 24);
                const bool q0 = s0 >= a.thr, q1 = s1 >= a.thr;  // (words past a window are zero; thr >= 1)
                const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, q0), b1 = __ballot_sync(0xFFFFFFFFu, q1);
                if ((b0 | b1) == 0) continue;
                const uint32_t lt = (1u << lane) - 1u;
                const uint32_t r = head + fill + (uint32_t)(__popc(b0 & lt) + __popc(b1 & lt));
                if (q0) wq[r & (kSmWQ - 1)] = (uint16_t)c;
                if (q1) wq[(r + (q0 ? 1u : 0u)) & (kSmWQ - 1)] = (uint16_t)(c + 1);
                fill += (uint32_t)(__popc(b0) + __popc(b1));
                while (fill >= 32) pop_score(32);
            }
            if (fill) pop_score(fill);
            __syncthreads();
        }
        if (count_full(__reduce_max_sync(0xFFFFFFFFu, ovf)) && lane == 0) S.overflow = 1;
        // ---- candidates whose sign or bin the float estimate left open ----
        for (uint32_t i = tid; i < min(S.ndefer, a.defer_cap); i += nthr)
        {
            uint32_t bc, yc, shp;
            uint64_t ib, iy;
            const uint2 w = S.defer[i];
            decode_packed(w.x, w.y, bc, yc, shp, ib, iy);
            const float h = exact_h(a.qc, bc, yc, ib, iy);
            if (h > 0.0f) count_psm(bc, yc, hist_bin(h));
        }
        my_cps = __reduce_add_sync(0xFFFFFFFFu, my_cps);
        my_fl = __reduce_or_sync(0xFFFFFFFFu, my_fl);
        npass = __reduce_add_sync(0xFFFFFFFFu, npass);
        if (lane == 0)
        {
            if (my_cps) atomicAdd(&S.cpsms, my_cps);
            if (my_fl) atomicOr(&S.flags, my_fl);
            if (npass) atomicAdd(&S.bytes, 4ull * npass);  // postings visited: those of entries inside the windows
        }
        // the top hit's shared ions come from the thread that found it
        if (my_best != 0 && my_best == S.best) S.best_shp = my_shp;
        __syncthreads();
        if (S.overflow)
        {
            if (tid == 0) a.wide_list[atomicAdd(a.nwide, 1u)] = s;
            continue;
        }
        for (int i = tid; i < kHistSm; i += nthr) a.hist[(size_t)s * HC_HIST_BINS + i] = S.hist[i];
        if (tid == 0) write_result(a, s, S.cpsms, S.flags, S.bytes, S.best, S.best_shp);
    }
    // what follows this kernel follows the k_search it may have overlapped too
    after_predecessor();
}

// ---- windows: DSLIM_BinarySearch (dslim_query.cpp:854-994) -----------------
// The first of m's n sorted masses that is not below x1, and the first that is
// above x2: a search in P + 1 parts for each, P loads of either in flight at a time.
// The limits are the reference's (its binary search and the walks at its end find the
// same places), and a NaN limit finds no window.
//
// A batch waits for this kernel before it can search anything. What bounds it is
// the chain of dependent loads while all pairs run at once (two halving searches one
// after the other, with a walk over the last 20 masses each, took 9 us for 8 spectra
// against 34 lengths of 600 masses; four ways this takes 4 us), and the loads
// themselves in larger batches, of which four ways take half as many again. +-500 Da
// against 34 lengths of up to 60,000 masses, four ways / two / as it was: 8 spectra 4.4 /
// 5.2 / 11.6 us, 2,000 8.2 / 11.0 / 19.7, 8,000 23 / 21 / 21, 100,000 189 / 172 / 148;
// +-1 ppm, 60,000 spectra: 65 / 66 / 99.
template <int P>
__device__ __forceinline__ int2 find_limits(const float *__restrict__ m, int n, float x1, float x2)
{
    // many windows end at, or miss, the length's masses
    const float lo = __ldg(m), hi = __ldg(m + n - 1);
    if (!(x1 <= hi && x2 >= lo)) return make_int2(0, 0);
    int b1 = 0, b2 = x2 >= hi ? n : 0, n1 = x1 <= lo ? 0 : n, n2 = x2 >= hi ? 0 : n;
    while (n1 > 0 || n2 > 0)
    {
        const int s1 = (n1 + P) / (P + 1), s2 = (n2 + P) / (P + 1);
        int c1 = 0, c2 = 0;
#pragma unroll
        for (int k = 1; k <= P; k++)
        {
            if (k * s1 <= n1 && n1 > 0) c1 += __ldg(m + b1 + k * s1 - 1) < x1;
            if (k * s2 <= n2 && n2 > 0) c2 += __ldg(m + b2 + k * s2 - 1) <= x2;
        }
        b1 += c1 * s1;
        b2 += c2 * s2;
        // a probe that fails ends the range before it
        n1 = c1 == P ? n1 - P * s1 : min(n1 - c1 * s1, s1 - 1);
        n2 = c2 == P ? n2 - P * s2 : min(n2 - c2 * s2, s2 - 1);
    }
    return make_int2(b1, b2);
}

template <int P>
__global__ void k_windows(const LenDev *__restrict__ lens, uint32_t nlen, const float *__restrict__ prec,
                          const double *__restrict__ dMs, double dM0, uint32_t nspec, int2 *__restrict__ win,
                          uint32_t *__restrict__ zero)
{
    release_successor();
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (zero)  // the histograms that several CTAs will add to
        for (uint64_t i = g; i < (uint64_t)nspec * HC_HIST_BINS; i += (uint64_t)gridDim.x * blockDim.x) zero[i] = 0u;
    if (g >= (uint64_t)nspec * nlen) return;
    const uint32_t s = (uint32_t)(g / nlen), l = (uint32_t)(g % nlen);
    const double dM = dMs ? dMs[s] : dM0;
    const float pm = prec[s];
    // float pmass1 = precmass - params.dM: double difference rounded to float
    const float pm1 = __double2float_rn(__dadd_rn((double)pm, -dM));
    const float pm2 = __double2float_rn(__dadd_rn((double)pm, dM));
    const int n = (int)lens[l].n;
    const float *m = lens[l].mass;
    int2 r = make_int2(1, 0);
    if (n > 0 && !(dM < 0.0))
    {
        const int2 f = find_limits<P>(m, n, pm1, pm2);
        if (f.x < f.y) r = make_int2(f.x, f.y - 1);
    }
    win[g] = r;
}

// ---- tail fit + e-value ------------------------------------------------------
// The plain form, for the spectra whose result k_tailfit's shorter arithmetic
// leaves open: expeRT::ModelTailFit (expeRT.cpp:572-718) and e(x) (dslim_query.cpp:773-799)
// of spectrum s, by one warp. Elementwise steps run across lanes; the sums
// whose rounding depends on order (ybar, top, bot of LinearFit) run on lane 0
// in the reference's order. Cumulative sums are exact integers either way.
// sx: the warp's HC_HIST_BINS + 2 doubles of shared memory.
__device__ void tailfit_one(uint32_t s, hc_result *__restrict__ out, const uint32_t *__restrict__ hist,
                            uint32_t min_cpsm, double expect_max, int32_t *__restrict__ fitstart, double *sx,
                            int lane)
{
    hc_result r = out[s];
    r.mu = r.beta = r.minhyp = r.nexthyp = r.maxhyp = 0;
    r.evalue = 0.0;
    r.reported = 0;
    if (r.cpsms < min_cpsm || r.cpsms == 0)
    {
        if (lane == 0)
        {
            out[s] = r;
            fitstart[s] = -1;
        }
        return;
    }
    int fit_first = -1;  // first regression bin (the learned tail's third target)
    const uint32_t *yy = hist + (size_t)s * HC_HIST_BINS;
    const int hyp = hist_bin(r.hyperscore);  // maxhypscore (dslim_query.cpp:778)
    const int cps = (int)r.cpsms;
    // expeRT.cpp:590-598: end1 = last bin below hyp holding >= 1, stt1 = first
    int stt1, end1;
    const int n = tail_bins(yy, hyp, HC_HIST_BINS, lane, stt1, end1);
    double mu_t = 0.0, beta_t = 0.0;
    uint32_t fl = 0;
    if (n == 0)
    {
        fl |= HC_FLAG_TAILFIT_EMPTY;  // LinearFit of 0 points: 0/0
        mu_t = beta_t = __longlong_as_double(0x7FF8000000000000ll);
    }
    else
    {
        // s(x) = -(cumsum/cpsms + -1), values > 1 -> 0.999 (expeRT.cpp:625-636)
        unsigned long long carry = 0;
        for (int i0 = 0; i0 < n; i0 += 32)
        {
            const int i = i0 + lane;
            unsigned long long v = (i < n) ? yy[stt1 + i] : 0ull;
            for (int o = 1; o < 32; o <<= 1)
            {
                const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, v, o);
                if (lane >= o) v += t;
            }
            if (i < n)
            {
                double d = __ddiv_rn((double)(carry + v), (double)cps);
                d = -__dadd_rn(d, -1.0);
                if (d > 1.0) d = 0.999;
                sx[i + 1] = d;
            }
            carry += __shfl_sync(0xFFFFFFFFu, v, 31);
        }
        if (lane == 0) sx[0] = 0.0;
        __syncwarp();
        // values <= 0 take the last value >= 1e-4 (expeRT.cpp:639-640), then log10
        int repl = n - 1;
        for (int q0 = n - 1; q0 >= 0; q0 -= 32)
        {
            const int q = q0 - lane;
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && sx[q + 1] >= 1e-4);
            if (b) { repl = q0 - (__ffs(b) - 1); break; }
        }
        const double rv = sx[repl + 1];
        __syncwarp();
        for (int i = lane; i < n; i += 32)
        {
            double v = sx[i + 1];
            if (v <= 0.0) v = rv;
            sx[i + 1] = log10(v);
        }
        __syncwarp();
        // regression window (expeRT.cpp:646-684)
        int mark = 0, mark2 = n - 1;
        const double hgt = __dadd_rn(sx[n], -sx[1]);
        if (n >= 3)
        {
            const double t1 = __dadd_rn(sx[1], __dmul_rn(hgt, 0.22));
            int lm = 0;
            for (int q0 = 0; q0 < n; q0 += 32)
            {
                const int q = q0 + lane;
                const uint32_t b = __ballot_sync(0xFFFFFFFFu, q < n && sx[q + 1] <= t1);
                if (b) { lm = q0 + __ffs(b) - 1; break; }
            }
            mark = lm - 1;
            if (n > 3)
            {
                const double t2 = __dadd_rn(sx[1], __dmul_rn(hgt, 0.87));
                for (int q0 = n - 1; q0 >= 0; q0 -= 32)
                {
                    const int q = q0 - lane;
                    const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && sx[q + 1] >= t2);
                    if (b) { mark2 = q0 - (__ffs(b) - 1); break; }
                }
            }
            if (mark >= mark2) mark = mark2 - 1;
        }
        if (mark < 0) fl |= HC_FLAG_TAILFIT_OOB;  // reads element -1 (sx[0] = +0.0)
        fit_first = stt1 + mark;
        const int m = mark2 - mark + 1;
        const double *y = sx + 1 + mark;
        // LinearFit (expeRT.cpp:1297-1345) on lane 0, in the reference's order
        if (lane == 0)
        {
            if (m == 1)
            {
                mu_t = 0.0;
                beta_t = y[0];
            }
            else
            {
                double xbar = 0.0, ybar = 0.0, top = 0.0, bot = 0.0;
                for (int i = 0; i < m; i++)
                {
                    xbar = __dadd_rn(xbar, (double)(stt1 + mark + i));
                    ybar = __dadd_rn(ybar, y[i]);
                }
                xbar = __ddiv_rn(xbar, (double)m);
                ybar = __ddiv_rn(ybar, (double)m);
                for (int i = 0; i < m; i++)
                {
                    const double dx = __dadd_rn((double)(stt1 + mark + i), -xbar);
                    top = __dadd_rn(top, __dmul_rn(dx, __dadd_rn(y[i], -ybar)));
                    bot = __dadd_rn(bot, __dmul_rn(dx, dx));
                }
                mu_t = __ddiv_rn(top, bot);
                beta_t = __dadd_rn(ybar, -__dmul_rn(mu_t, xbar));
            }
        }
    }
    if (lane == 0)
    {
        fitstart[s] = fit_first;
        r.flags |= fl;
        r.mu = x86_d2i(__dmul_rn(mu_t, 1e6));
        r.beta = x86_d2i(__dmul_rn(beta_t, 1e6));
        r.minhyp = stt1;
        r.nexthyp = end1;
        r.maxhyp = hyp;
        // e(x) = 10^(w*maxhyp + b) * cpsms (dslim_query.cpp:786-799)
        const double wv = __ddiv_rn((double)r.mu, 1e6), bv = __ddiv_rn((double)r.beta, 1e6);
        const double lgs = __dadd_rn(__dmul_rn(wv, (double)hyp), bv);
        double e = pow(10.0, lgs);
        e = __dmul_rn(e, (double)r.cpsms);
        r.evalue = e;
        r.reported = e < expect_max ? 1u : 0u;
        out[s] = r;
    }
}

// Every spectrum by tailfit_one: what k_tailfit's results are compared with.
constexpr int kTfPlainWarps = 4;

__global__ void __launch_bounds__(kTfPlainWarps * 32) k_tailfit_plain(hc_result *__restrict__ out,
                                                                     const uint32_t *__restrict__ hist, uint32_t n,
                                                                     uint32_t min_cpsm, double expect_max,
                                                                     int32_t *__restrict__ fitstart)
{
    __shared__ double sx[kTfPlainWarps][HC_HIST_BINS + 2];
    const uint32_t s = blockIdx.x * kTfPlainWarps + (threadIdx.x >> 5);
    if (s < n) tailfit_one(s, out, hist, min_cpsm, expect_max, fitstart, sx[threadIdx.x >> 5], threadIdx.x & 31);
}

// k_tailfit. This part's FP64 rate is 1/64 of its FP32 rate (a warp's FP64
// instruction takes the SM's pipe 16 clocks, whatever its active lanes), so
// the fit is arranged around it:
//   - the regression window is found on an FP32 curve; FP64 decides only the
//     points that lie within kTfNear of a level;
//   - FP64 logarithms are taken of the window's points alone, with a table
//     and a degree-6 polynomial (P. T. P. Tang, "Table-driven implementation of
//     the logarithm function in IEEE floating-point arithmetic", 1990), and the
//     quotients by one reciprocal per spectrum and a corrected product
//     (P. Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", 1990: the correctly rounded quotient);
//   - the abscissae are consecutive integers, so their sums are closed forms,
//     and the two sums left run across the lanes;
//   - what follows once per spectrum (the quotients, the power) runs with a
//     lane per spectrum, sixteen spectra at a time.
// The line is (mu, beta) x 1e6 truncated to integers, so a result that differs
// in its last bits is the same result unless a value lies near an integer (or
// a point on a level): those spectra, about 1 in 10^5, are fitted again by
// tailfit_one, in the reference's own order of operations. Results are therefore
// tailfit_one's, bit for bit. 2,000 spectra of an open search: 23 us,
// against 183 us with every point in FP64 and the sums on one lane.
constexpr int kTfWarps = 16;
constexpr float kTfNear = 5e-5f;      // FP32 curve and level: together within 5e-6 of FP64's
constexpr double kTfLevel = 1e-9;     // the short FP64 logarithm: within 1e-14
// How far the values x 1e6 may be from tailfit_one's. Two logarithms of a point differ by
// 4e-15 at most (the short one within 2e-15, log10's 2 ulp below 8), the slope of m points by
// 3 / m times that and twice it for two, so by 8e-15 and its own rounding: below 1.5e-8 x 1e-6.
// The intercept is the points' mean less the slope times the window's middle x: 8.5e-15 x, the
// product's roundings (2.3e-13 each where x is 1000) and the mean's, below 5e-13: 1.1e-8 x and
// 5e-7 x 1e-6. Each margin is more than twice its bound, and what is next to an integer is refitted
// by one warp in 10 us: with 3e-5 for every intercept a batch of 129 spectra had one more often.
constexpr double kTfSlope = 1e-6, kTfIntercept = 2e-6, kTfMiddle = 3e-8;

struct TfJob
{
    double sy, sxy, yf;   // sums of y - yf and of (x - xbar) y over the window, yf its first point
    uint32_t s, fl;
    int status, m, first, stt1, end1, hyp;
};

enum TfStatus
{
    kTfNone = 0,   // nothing (left) to do
    kTfFit = 1,    // the window's sums are there
    kTfAgain = 2,  // to be fitted by tailfit_one
    kTfEmpty = 3,  // no point
};

struct TfSmem
{
    double sx[HC_HIST_BINS + 2];  // tailfit_one's
    double2 tab[kLgTab];
    TfJob job[kTfWarps];
    alignas(16) uint32_t cum[kTfWarps][kCumRow];
};

// log10 of a positive normal double up to 1, within 4e-15
__device__ __forceinline__ double lg10_short(double d, const double2 *tab)
{
    const int hi = __double2hiint(d);
    const double2 t = tab[(hi >> 13) & (kLgTab - 1)];
    const double mant = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(d));
    const double r = fma(mant, t.x, -1.0);  // |r| < 2^-8 (1 + 2^-7)
    double p = fma(r, -0.07238241365054197128, 0.08685889638065036553);
    p = fma(r, p, -0.10857362047581295691);
    p = fma(r, p, 0.14476482730108394255);
    p = fma(r, p, -0.21714724095162591383);
    p = fma(r, p, 0.43429448190325182765);
    return fma(r, p, fma((double)((hi >> 20) - 1023), 0.30102999566398119521, t.y));
}

// A spectrum's survival curve, s(i) = 1 - cum / cpsms (expeRT.cpp:625-636), its
// values of 0 replaced by the last one of 1e-4 or more (639-640).
struct TfCurve
{
    const uint32_t *c;  // cumulative counts of the points
    uint32_t cps, crep; // crep: the count whose value replaces those at or past cps
    float invf;
    double cd, inv;
    __device__ __forceinline__ double value(uint32_t x) const
    {
        const double xd = (double)x;
        double q = __dmul_rn(xd, inv);
        q = fma(fma(-q, cd, xd), inv, q);  // the correctly rounded x / cps
        return __dadd_rn(1.0, -q);
    }
    __device__ __forceinline__ uint32_t count(int i) const { return c[i] < cps ? c[i] : crep; }
    __device__ __forceinline__ float lgf(int i) const
    {
        return __log2f((float)(cps - count(i)) * invf) * 0.30102999566f;
    }
    __device__ __forceinline__ double lg(int i, const double2 *tab) const { return lg10_short(value(count(i)), tab); }
};

// The sums of spectrum s's regression window, by one warp (see k_tailfit).
__device__ __forceinline__ void tailfit_sums(uint32_t s, const hc_result &r, const uint32_t *__restrict__ hist, int hyp,
                                             uint32_t *cum, const double2 *tab, TfJob &job, int lane)
{
    int stt1, end1;
    const int n = tail_curve(hist + (size_t)s * HC_HIST_BINS, hyp, HC_HIST_BINS, lane, cum, stt1, end1);
    int status = kTfFit, mark = 0, mark2 = n - 1, m = 0;
    double sy = 0.0, sxy = 0.0, yf = 0.0;
    if (n == 0) status = kTfEmpty;
    else
    {
        TfCurve cv;
        cv.c = cum + stt1;
        cv.cps = r.cpsms;
        cv.crep = 0;
        cv.invf = 1.0f / (float)r.cpsms;
        cv.cd = (double)r.cpsms;
        cv.inv = __drcp_rn(cv.cd);
        if (cv.c[n - 1] >= cv.cps)  // the counts ascend: the only case with a value of 0 (or below)
        {
            status = kTfAgain;
            for (int q0 = n - 1; q0 >= 0; q0 -= 32)
            {
                const int q = q0 - lane;
                const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && cv.c[q] < cv.cps && cv.value(cv.c[q]) >= 1e-4);
                if (b)
                {
                    cv.crep = cv.c[q0 - (__ffs(b) - 1)];
                    status = kTfFit;
                    break;
                }
            }
        }
        // regression window (expeRT.cpp:646-684)
        if (status == kTfFit && n >= 3)
        {
            const double ye = lane < 2 ? cv.lg(lane ? n - 1 : 0, tab) : 0.0;
            const double y0 = __shfl_sync(0xFFFFFFFFu, ye, 0), hgt = __dadd_rn(__shfl_sync(0xFFFFFFFFu, ye, 1), -y0);
            const double t1 = __dadd_rn(y0, __dmul_rn(hgt, 0.22));
            const float t1f = (float)t1;
            bool open = false;
            int lm = 0;
            for (int q0 = 0; q0 < n; q0 += 32)
            {
                const int q = q0 + lane;
                const float y = q < n ? cv.lgf(q) : 1.0f;
                bool in = y <= t1f;
                if (__any_sync(0xFFFFFFFFu, fabsf(y - t1f) < kTfNear) && fabsf(y - t1f) < kTfNear)
                {
                    const double yd = cv.lg(q, tab);
                    in = yd <= t1;
                    open |= fabs(yd - t1) < kTfLevel;
                }
                const uint32_t b = __ballot_sync(0xFFFFFFFFu, q < n && in);
                if (b)
                {
                    lm = q0 + __ffs(b) - 1;
                    break;
                }
            }
            mark = lm - 1;
            if (n > 3)
            {
                const double t2 = __dadd_rn(y0, __dmul_rn(hgt, 0.87));
                const float t2f = (float)t2;
                for (int q0 = n - 1; q0 >= 0; q0 -= 32)
                {
                    const int q = q0 - lane;
                    const float y = q >= 0 ? cv.lgf(q) : -1e9f;
                    bool in = y >= t2f;
                    if (fabsf(y - t2f) < kTfNear)
                    {
                        const double yd = cv.lg(q, tab);
                        in = yd >= t2;
                        open |= fabs(yd - t2) < kTfLevel;
                    }
                    const uint32_t b = __ballot_sync(0xFFFFFFFFu, q >= 0 && in);
                    if (b)
                    {
                        mark2 = q0 - (__ffs(b) - 1);
                        break;
                    }
                }
            }
            if (mark >= mark2) mark = mark2 - 1;
            if (__any_sync(0xFFFFFFFFu, open)) status = kTfAgain;
        }
        m = mark2 - mark + 1;
        if (status == kTfFit)
        {
            // element -1 reads as 0 (see tailfit_one)
            double dx = (double)(2 * lane - (m - 1)) * 0.5;
            for (int j0 = 0; j0 < m; j0 += 32)
            {
                const int j = j0 + lane;
                const double y = j < m && mark + j >= 0 ? cv.lg(mark + j, tab) : 0.0;
                if (j0 == 0) yf = __shfl_sync(0xFFFFFFFFu, y, 0);
                if (j < m)
                {
                    const double v = y - yf;
                    sy += v;
                    sxy = fma(dx, v, sxy);
                }
                dx += 32.0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                sy += __shfl_xor_sync(0xFFFFFFFFu, sy, o);
                sxy += __shfl_xor_sync(0xFFFFFFFFu, sxy, o);
            }
        }
    }
    if (lane == 0)
    {
        job.sy = sy;
        job.sxy = sxy;
        job.yf = yf;
        job.s = s;
        job.fl = status == kTfEmpty ? HC_FLAG_TAILFIT_EMPTY : (mark < 0 ? HC_FLAG_TAILFIT_OOB : 0u);
        job.status = status;
        job.m = m;
        job.first = n ? stt1 + mark : -1;
        job.stt1 = stt1;
        job.end1 = end1;
        job.hyp = hyp;
    }
}

// The line and the e-value of a job, one lane each; false when a value's
// truncation is left open (nothing is written then).
__device__ __forceinline__ bool tailfit_line(const TfJob &j, hc_result *__restrict__ out, double expect_max,
                                             int32_t *__restrict__ fitstart)
{
    double mu_t, beta_t;  // x 1e6
    if (j.status == kTfEmpty) mu_t = beta_t = __longlong_as_double(0x7FF8000000000000ll);  // LinearFit of 0 points: 0/0
    else
    {
        const double m = (double)j.m, xbar = (double)j.first + 0.5 * (m - 1.0);
        const double ybar = j.yf + j.sy / m;
        // sum of (x - xbar)^2 over m consecutive integers: m (m^2 - 1) / 12
        const double bot = 0.25 * (double)(((uint32_t)j.m * ((uint32_t)j.m * (uint32_t)j.m - 1u)) / 3u);
        const double mu = j.m == 1 ? 0.0 : j.sxy / bot;
        mu_t = mu * 1e6;
        beta_t = (ybar - mu * xbar) * 1e6;
        // (a value that truncates to 0 from either side is not open)
        const bool open = !(fabs(mu_t) < 1e9) || !(fabs(beta_t) < 1e9) ||
                          (fabs(mu_t) > 0.5 && fabs(mu_t - rint(mu_t)) < kTfSlope) ||
                          (fabs(beta_t) > 0.5 && fabs(beta_t - rint(beta_t)) < fma(kTfMiddle, xbar, kTfIntercept));
        if (open) return false;
    }
    hc_result r = out[j.s];
    fitstart[j.s] = j.first;
    r.flags |= j.fl;
    r.mu = x86_d2i(mu_t);
    r.beta = x86_d2i(beta_t);
    r.minhyp = j.stt1;
    r.nexthyp = j.end1;
    r.maxhyp = j.hyp;
    // e(x) = 10^(w*maxhyp + b) * cpsms (dslim_query.cpp:786-799)
    const double wv = __ddiv_rn((double)r.mu, 1e6), bv = __ddiv_rn((double)r.beta, 1e6);
    const double lgs = __dadd_rn(__dmul_rn(wv, (double)j.hyp), bv);
    double e = pow(10.0, lgs);
    e = __dmul_rn(e, (double)r.cpsms);
    r.evalue = e;
    r.reported = e < expect_max ? 1u : 0u;
    out[j.s] = r;
    return true;
}

// One warp per spectrum, then one lane per spectrum: every spectrum of
// [0, nspec), or those of `list` (its length *nlist read on the device) when a
// list is given.
__global__ void __launch_bounds__(kTfWarps * 32, 2) k_tailfit(const QueryConst *__restrict__ qc,
                                                             hc_result *__restrict__ out,
                                                             const uint32_t *__restrict__ hist, uint32_t nspec,
                                                             uint32_t min_cpsm, double expect_max,
                                                             int32_t *__restrict__ fitstart,
                                                             const uint32_t *__restrict__ list,
                                                             const uint32_t *__restrict__ nlist)
{
    extern __shared__ __align__(16) unsigned char tsm[];
    TfSmem &S = *reinterpret_cast<TfSmem *>(tsm);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kLgTab; i += kTfWarps * 32) S.tab[i] = make_double2(qc->lg_tab[2 * i], qc->lg_tab[2 * i + 1]);
    after_predecessor();
    const uint32_t cnt = list ? min(*nlist, nspec) : nspec;
    if (blockIdx.x * kTfWarps >= cnt) return;
    __syncthreads();
    for (uint32_t w0 = blockIdx.x * kTfWarps; w0 < cnt; w0 += gridDim.x * kTfWarps)
    {
        TfJob &job = S.job[warp];
        if (lane == 0) job.status = kTfNone;
        if (w0 + warp < cnt)
        {
            const uint32_t s = list ? list[w0 + warp] : w0 + warp;
            hc_result r = out[s];
            if (r.cpsms < min_cpsm || r.cpsms == 0)
            {
                if (lane == 0)
                {
                    r.mu = r.beta = r.minhyp = r.nexthyp = r.maxhyp = 0;
                    r.evalue = 0.0;
                    r.reported = 0;
                    out[s] = r;
                    fitstart[s] = -1;
                }
            }
            else
                tailfit_sums(s, r, hist, hist_bin(r.hyperscore), S.cum[warp], S.tab, job, lane);
        }
        __syncthreads();
        if (warp == 0)
        {
            bool again = false;
            if (lane < kTfWarps)
            {
                const TfJob &j = S.job[lane];
                again = j.status == kTfAgain;
                if (j.status == kTfFit || j.status == kTfEmpty) again = !tailfit_line(j, out, expect_max, fitstart);
            }
            for (uint32_t b = __ballot_sync(0xFFFFFFFFu, again); b; b &= b - 1)
            {
                tailfit_one(S.job[__ffs(b) - 1].s, out, hist, min_cpsm, expect_max, fitstart, S.sx, lane);
                __syncwarp();
            }
        }
        __syncthreads();
    }
}

// ---- longest-first order for the batched schedule --------------------------
// cost class of a spectrum = bit length of its total window size (candidates)
constexpr int kCostClasses = 64;

__global__ void k_cost(const int2 *__restrict__ win, uint32_t nspec, uint32_t nlen, uint32_t *__restrict__ cls,
                       uint32_t *__restrict__ cnt)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    unsigned long long c = 0;
    for (uint32_t l = 0; l < nlen; l++)
    {
        const int2 w = win[(size_t)s * nlen + l];
        if (w.y >= w.x) c += (unsigned long long)(w.y - w.x + 1);
    }
    const uint32_t k = c ? 64u - (uint32_t)__clzll(c) : 0u;
    cls[s] = k;
    atomicAdd(&cnt[k], 1u);
}

// split (optional): the number of spectra whose cost class exceeds
// split_class, i.e. whose windows hold 2^split_class candidates or more in all
// (they come first in the order)
__global__ void k_order(const uint32_t *__restrict__ cls, uint32_t nspec, const uint32_t *__restrict__ cnt,
                        uint32_t *__restrict__ cursor, uint32_t *__restrict__ order, uint32_t split_class,
                        uint32_t *__restrict__ split)
{
    __shared__ uint32_t off[kCostClasses];
    if (threadIdx.x == 0)
    {
        uint32_t run = 0;
        for (int k = kCostClasses - 1; k >= 0; k--)
        {
            off[k] = run;
            run += cnt[k];
        }
        if (split && blockIdx.x == 0) *split = off[split_class];
    }
    __syncthreads();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    const uint32_t k = cls[s];
    order[off[k] + atomicAdd(&cursor[k], 1u)] = s;
}

}  // namespace

size_t search_smem(uint32_t tile, uint32_t dF, bool wide, uint32_t threads)
{
    return smem_layout(tile, dF, wide, threads / 32).total;
}

template <class T>
static int grow(hc_ctx *ctx, T **p, size_t *cap, size_t need);

// the largest tile (a multiple of kRowG) whose whole layout fits in `budget` bytes
static uint32_t fit_tile(size_t budget, uint32_t dF, uint32_t threads)
{
    uint32_t t = (uint32_t)std::min<size_t>(budget / 8, 32768) / kRowG * kRowG;  // ring entries are 16-bit
    while (t > kRowG && smem_layout(t, dF, false, threads / 32).total > budget) t -= kRowG;
    return t < kRowG ? kRowG : t;
}

// Stage timing event; inside a stream capture it becomes an external event
// record node, so a replayed graph still times its stages.
cudaError_t record_stage(hc_ctx *ctx, int i, cudaStream_t st)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const cudaError_t e = cudaStreamIsCapturing(st, &cs);
    if (e != cudaSuccess) return e;
    return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ctx->ev[i], st, cudaEventRecordExternal)
                                               : cudaEventRecord(ctx->ev[i], st);
}

// Shared memory the resident CTAs take at most when a tile is picked, so that
// the SM keeps 60 KB of its 256 KB as L1 (the next configuration down keeps
// 28 KB): the search reads its jobs' class codes and row-table words through
// L1, and with 28 KB it runs 9-10 % slower at the same tile.
constexpr size_t kSmemKeepL1 = 196 * 1024;

uint32_t max_tile(const hc_ctx *ctx, uint32_t dF, uint32_t threads)
{
    return max_tile_for(ctx, dF, 1, threads);
}

uint32_t max_tile_for(const hc_ctx *ctx, uint32_t dF, uint32_t ctas_per_sm, uint32_t threads)
{
    if (ctas_per_sm < 1) ctas_per_sm = 1;
    // the SM's shared memory is split; each CTA also keeps a reserve for the system
    const size_t full = std::min(ctx->smem_optin, ctx->smem_sm / ctas_per_sm - ctx->smem_reserved);
    const size_t keep = std::min(full, kSmemKeepL1 / ctas_per_sm - ctx->smem_reserved);
    for (const size_t per : {keep, full})
    {
        const uint32_t t = fit_tile(per, dF, threads);
        if (smem_layout(t, dF, false, threads / 32).total <= per) return t;
    }
    return 0u;
}

int prepare_query(hc_ctx *ctx, uint32_t nspec)
{
    int rc = sync_lengths(ctx);
    if (rc) return rc;
    const uint32_t nlen = (uint32_t)ctx->lens.size();
    QueryScratch &q = ctx->qs;
    if ((rc = grow(ctx, &q.d_win, &q.win_cap, (size_t)nspec * nlen))) return rc;
    if ((rc = grow(ctx, &q.d_wide, &q.wide_cap, (size_t)nspec + 4))) return rc;
    if ((rc = grow(ctx, &q.d_order, &q.order_cap, 2 * (size_t)nspec))) return rc;
    if ((rc = grow(ctx, &q.d_fitstart, &q.fit_cap, (size_t)nspec))) return rc;
    if (!q.d_work) HC_CUDA(ctx, cudaMalloc((void **)&q.d_work, 4 * kWorkWords));
    return HC_SUCCESS;
}

namespace {

template <bool WIDE, int G, bool PARTS = false>
int launch_g(hc_ctx *ctx, const SearchArgs &a, int grid, uint32_t threads, size_t smem, cudaStream_t st)
{
    if (G >= 4 && threads > 512) threads = 512;
    HC_CUDA(ctx, cudaFuncSetAttribute(k_search<WIDE, G, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HC_CUDA(ctx, launch_after(k_search<WIDE, G, PARTS>, (unsigned)grid, threads, smem, st, a));
    return HC_SUCCESS;
}

template <bool WIDE>
int launch_search(hc_ctx *ctx, const SearchArgs &a, int grid, uint32_t threads, size_t smem, uint32_t g,
                  cudaStream_t st)
{
    switch (g)
    {
    case 1: return launch_g<WIDE, 1>(ctx, a, grid, threads, smem, st);
    case 2: return launch_g<WIDE, 2>(ctx, a, grid, threads, smem, st);
    case 8: return launch_g<WIDE, 8>(ctx, a, grid, threads, smem, st);
    default: return launch_g<WIDE, 4>(ctx, a, grid, threads, smem, st);
    }
}

}  // namespace

// the device record of one length
static void fill_lendev(const hc_ctx *ctx, const LenHost &lh, LenDev &d)
{
    std::memset(&d, 0, sizeof(d));
    d.L = lh.L;
    d.n = lh.built ? lh.n : 0;
    d.npep = lh.npep;
    d.speclen = 2 * ctx->p.maxz * (lh.L - 1);
    d.half = d.speclen / 2;
    division_magic(d.speclen, &d.magic, &d.msh);
    d.stride = lh.stride;
    d.mass = lh.d_mass;
    d.seqid = lh.d_seqid;
    d.sites = lh.d_sites;
    d.modnum = lh.d_modnum;
    d.seqs = lh.d_seqs;
    d.bA = lh.d_bA;
    d.qA = lh.d_qA;
    d.qp = lh.d_qp;
    d.qps = lh.d_qps;
    d.rows = lh.d_rows;
    d.cls = lh.d_cls;
}

// the length records the search kernel keeps in its parameters
static void fill_lens(const hc_ctx *ctx, SearchArgs &a)
{
    for (size_t i = 0; i < ctx->lens.size(); i++)
    {
        const LenHost &lh = ctx->lens[i];
        a.len[i] = LenS{lh.d_qps, lh.d_rows, lh.stride, lh.built ? lh.n : 0u, lh.d_cls};
    }
}

int sync_lengths(hc_ctx *ctx)
{
    if (!ctx->lens_dirty) return HC_SUCCESS;
    const uint32_t nlen = (uint32_t)ctx->lens.size();
    std::vector<LenDev> h(nlen);
    for (uint32_t i = 0; i < nlen; i++)
    {
        fill_lendev(ctx, ctx->lens[i], h[i]);
    }
    if (!ctx->d_lens) HC_CUDA(ctx, cudaMalloc((void **)&ctx->d_lens, sizeof(LenDev) * HC_MAX_LENGTHS));
    HC_CUDA(ctx, overwrite(ctx->d_lens, h.data(), sizeof(LenDev) * nlen));
    ctx->lens_dirty = false;
    return HC_SUCCESS;
}

template <class T>
static int grow(hc_ctx *ctx, T **p, size_t *cap, size_t need)
{
    if (*cap >= need) return HC_SUCCESS;
    ctx->epoch++;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    HC_CUDA(ctx, cudaMalloc((void **)p, sizeof(T) * need));
    *cap = need;
    return HC_SUCCESS;
}

// The windows of a batch: four-way searches in small batches, halving ones in large
// ones; the two meet between 2,000 and 6,000 spectra of 34 lengths (find_limits).
static int launch_windows(hc_ctx *ctx, const LenDev *lens, uint32_t nlen, const float *d_prec, const double *d_dM,
                          uint32_t nspec, int2 *win, uint32_t *zero, cudaStream_t st)
{
    const uint64_t nw = (uint64_t)nspec * nlen;
    const unsigned blocks = (unsigned)((nw + 255) / 256);
    if (nw <= kWideWindows * (uint64_t)ctx->sm_count)
        k_windows<3><<<blocks, 256, 0, st>>>(lens, nlen, d_prec, d_dM, ctx->p.dM, nspec, win, zero);
    else
        k_windows<1><<<blocks, 256, 0, st>>>(lens, nlen, d_prec, d_dM, ctx->p.dM, nspec, win, zero);
    HC_CUDA(ctx, cudaGetLastError());
    return HC_SUCCESS;
}

// The search of small windows: the spectra of the order from *obase on (null: all, in
// batch order). `after`: it was preceded by k_search on the same order, which it
// does not depend on; its CTAs start as k_search's leave SMs free.
static int launch_small(hc_ctx *ctx, SearchArgs s, uint32_t nspec, const uint32_t *obase, uint32_t *work, bool after,
                        cudaStream_t st)
{
    s.obase = obase;
    s.olim = nullptr;
    s.work = work + kWkSmall;
    s.follows = after ? 0u : 1u;
    const size_t smem = small_smem(s.dF);
    HC_CUDA(ctx, cudaFuncSetAttribute(k_search_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HC_CUDA(ctx, launch_after(k_search_small, std::min<uint32_t>(nspec, (uint32_t)ctx->sm_count * kSmCtas), kSmThreads,
                              smem, st, s));
    return HC_SUCCESS;
}

static uint64_t index_entries(const hc_ctx *ctx)
{
    uint64_t n = 0;
    for (const LenHost &lh : ctx->lens) n += lh.built ? lh.n : 0u;
    return n;
}

// The CTAs that share a spectrum in k_search, at most. With at most half as many spectra as
// SMs, in a context whose launch shape nobody chose, the windows are cut so that every SM
// (one 1024-thread CTA each) has a part, up to kMaxParts: one CTA a spectrum left the
// others idle. A part costs its CTA some 8 us of set-up, so it holds kPartMin candidates at
// least, kPartMinFew while one spectrum in eight SMs is all there is. Whole / in parts:
// +-500 Da against 2 M peptides, 1 spectrum 539 / 71 us, 8 586 / 94, 32 755 / 257, 76 780 /
// 435; against 500,000, 8 spectra 186 / 66, 76 286 / 175. (Four parts an SM for two 512-thread
// CTAs: 76 spectra 321 and 165, but 40 spectra of 44 k candidates 137 us against 117 whole,
// 152 of 54 k 175 against 138.)
static uint32_t auto_parts(const hc_ctx *ctx, uint32_t nspec)
{
    const uint32_t items = std::min((uint32_t)ctx->sm_count, kMaxPartItems);
    if (!ctx->auto_shape || 2 * (uint64_t)nspec > items || index_entries(ctx) < kAutoAllSmall) return 1;
    return std::min(items / nspec, kMaxParts);
}

// The packed search of a batch: with schedule 2 the longest-first order first,
// then the tuned shape, or, when small windows have their own launch, two: the
// tuned shape takes the order up to the split point and k_search_small the rest.
// Both read their range of the order on the device.
//
// A context whose launch shape nobody chose (neither hc_tune nor
// hc_ctx_set_tuning) gets one by what is searched. k_search_small takes the
// spectra whose windows hold fewer than 2^15 candidates: search times of 3,000
// spectra, all in k_search_small / all in two 512-thread k_search CTAs per SM, at
// about 2 k candidates a spectrum 191 / 455 us, 9 k 358 / 692, 45 k 908 / 926 and,
// in a larger index, 1,013 / 862, 220 k 3,833 / 2,377. An index of fewer than 2^16
// entries has next to no others. Else both kernels are launched: up to kAutoOrder
// spectra each passes over the other's (the order's two kernels take longer than
// that), beyond it the order splits the batch. k_search runs as one 1024-thread CTA
// per SM while a CTA has at most one spectrum (8 spectra of 220 k candidates 199 us
// against 257), as two of 512 beyond that (3,000 spectra 2,380 us against 2,946).
static int launch_packed(hc_ctx *ctx, SearchArgs &a, uint32_t nspec, uint32_t nlen, const int2 *win, uint32_t *order,
                         uint32_t *work, cudaStream_t st, int &launches, bool stages)
{
    hc_tuning t = ctx->tuning;
    bool all_small = false;
    a.wsplit = 0;
    if (ctx->auto_shape)
    {
        all_small = index_entries(ctx) < kAutoAllSmall;
        const uint32_t tile = max_tile_for(ctx, a.dF, 2, 512);
        if (nspec > (uint32_t)ctx->sm_count && tile >= kRowG)
        {
            t.threads = 512;
            t.ctas_per_sm = 2;
            t.pairs_per_warp = 4;
            t.tile = tile;
        }
        if (nspec > kAutoOrder)
        {
            t.schedule = 2;
            t.small_log2 = kAutoSmallLog2;
        }
        else
            a.wsplit = 1u << kAutoSmallLog2;
    }
    a.tile = t.tile;
    a.persistent = t.schedule != 1;
    a.obase = a.olim = nullptr;
    a.arrived = work + kWkArrived;
    a.part_min = nspec <= (uint32_t)ctx->sm_count / 8 ? kPartMinFew : kPartMin;
    a.psum = reinterpret_cast<PartSum *>(work + kWkPart);
    const bool split = t.schedule == 2 && t.small_log2 != 0;
    if (t.schedule == 2 && !all_small)
    {
        uint32_t *cls = order + nspec;
        k_cost<<<(nspec + 255) / 256, 256, 0, st>>>(win, nspec, nlen, cls, work + kWkCnt);
        k_order<<<(nspec + 255) / 256, 256, 0, st>>>(cls, nspec, work + kWkCnt, work + kWkCur, order,
                                                     split ? t.small_log2 : 0u, split ? work + kWkSplit : nullptr);
        HC_CUDA(ctx, cudaGetLastError());
        a.order = order;
        launches += 2;
        if (split) a.olim = work + kWkSplit;
    }
    // the search stage: the packed launches
    if (stages) HC_CUDA(ctx, record_stage(ctx, 1, st));
    if (all_small)
    {
        a.wsplit = 0;
        return launch_small(ctx, a, nspec, nullptr, work, false, st);
    }
    const size_t smem = search_smem(t.tile, a.dF, false, t.threads);
    const int grid = t.schedule == 1 ? (int)nspec : ctx->sm_count * (int)t.ctas_per_sm;
    const int rc = a.parts > 1 ? launch_g<false, 2, true>(ctx, a, grid, t.threads, smem, st)
                               : launch_search<false>(ctx, a, grid, t.threads, smem, t.pairs_per_warp, st);
    if (rc || !(split || a.wsplit)) return rc;
    launches++;
    return launch_small(ctx, a, nspec, split ? work + kWkSplit : nullptr, work, true, st);
}

// the tail fit of spectra [0, n), or of a list of at most n
static int launch_tailfit(hc_ctx *ctx, hc_result *out, const uint32_t *hist, uint32_t n, int32_t *fitstart,
                          const uint32_t *list, const uint32_t *nlist, cudaStream_t st)
{
    HC_CUDA(ctx, cudaFuncSetAttribute(k_tailfit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TfSmem)));
    const uint32_t blocks = std::min<uint32_t>((n + kTfWarps - 1) / kTfWarps, 2u * (uint32_t)ctx->sm_count);
    HC_CUDA(ctx, launch_after(k_tailfit, blocks, kTfWarps * 32, sizeof(TfSmem), st, ctx->d_qconst, out, hist, n,
                              ctx->p.min_cpsm, ctx->p.expect_max, fitstart, list, nlist));
    return HC_SUCCESS;
}

int query_device(hc_ctx *ctx, const uint32_t *d_idx, const uint32_t *d_moz, const uint32_t *d_int,
                 const float *d_prec, const double *d_dM, uint32_t nspec, uint32_t npeaks,
                 hc_result *d_out, uint32_t *d_hist, cudaStream_t st, bool tailfit)
{
    (void)npeaks;
    int rc = sync_lengths(ctx);
    if (rc) return rc;
    ctx->last_launches = 0;
    ctx->last_learned = !tailfit;
    if (nspec == 0) return HC_SUCCESS;
    const uint32_t nlen = (uint32_t)ctx->lens.size();
    QueryScratch &q = ctx->qs;
    if ((rc = grow(ctx, &q.d_win, &q.win_cap, (size_t)nspec * nlen))) return rc;
    if ((rc = grow(ctx, &q.d_wide, &q.wide_cap, (size_t)nspec + 4))) return rc;
    if ((ctx->tuning.schedule == 2 || ctx->auto_shape) && (rc = grow(ctx, &q.d_order, &q.order_cap, 2 * (size_t)nspec)))
        return rc;
    if ((rc = grow(ctx, &q.d_fitstart, &q.fit_cap, (size_t)nspec))) return rc;
    if (!q.d_work) HC_CUDA(ctx, cudaMalloc((void **)&q.d_work, 4 * kWorkWords));
    q.d_nwide = q.d_work + kWkNwide;
    HC_CUDA(ctx, cudaMemsetAsync(q.d_work, 0, 4 * kWkPart, st));
    const uint32_t parts = auto_parts(ctx, nspec);

    if (ctx->profiling) HC_CUDA(ctx, record_stage(ctx, 0, st));
    rc = launch_windows(ctx, ctx->d_lens, nlen, d_prec, d_dM, nspec, q.d_win, parts > 1 ? d_hist : nullptr, st);
    if (rc) return rc;

    SearchArgs a{};
    a.lens = ctx->d_lens;
    fill_lens(ctx, a);
    a.nlen = nlen;
    a.qc = ctx->d_qconst;
    a.idx = d_idx;
    a.moz = d_moz;
    a.inten = d_int;
    a.prec = d_prec;
    a.win = q.d_win;
    a.nspec = nspec;
    a.dF = ctx->p.dF;
    a.min_shp = ctx->p.min_shp;
    a.thr = ctx->p.min_shp > 0 ? ctx->p.min_shp : 1;
    a.maxbin = ctx->p.max_mass * ctx->p.scale;
    a.out = d_out;
    a.hist = d_hist;
    a.wide_list = q.d_wide;
    a.nwide = q.d_nwide;
    a.work = q.d_work;
    a.parts = parts;
    a.defer_cap = ctx->tuning.defer_cap;
    a.maxz = ctx->p.maxz;
    a.classes = ctx->d_classes;
    a.phase = ctx->d_phase;
    int launches = 4;
    int rc2 = launch_packed(ctx, a, nspec, nlen, q.d_win, q.d_order, q.d_work, st, launches, ctx->profiling);
    if (rc2) return rc2;
    if (ctx->profiling) HC_CUDA(ctx, record_stage(ctx, 2, st));
    // spectra whose packed scorecard could overflow are redone wide; the
    // list length is read on the device (no host synchronisation)
    SearchArgs b = a;
    b.persistent = 1;
    b.phase = nullptr;
    b.order = nullptr;
    b.only = q.d_wide;
    b.nonly_dev = q.d_nwide;
    b.work = q.d_work + kWkWide;
    b.obase = b.olim = nullptr;
    b.parts = 0;
    b.tile = std::max(kRowG, ctx->tuning.tile / 2 / kRowG * kRowG);  // same shared memory, 16-byte words
    const size_t smem2 = search_smem(b.tile, b.dF, true, ctx->tuning.threads);
    rc2 = launch_search<true>(ctx, b, ctx->sm_count, ctx->tuning.threads, smem2, 2, st);
    if (rc2) return rc2;
    if (ctx->profiling) HC_CUDA(ctx, record_stage(ctx, 3, st));
    if (tailfit)
    {
        if ((rc2 = launch_tailfit(ctx, d_out, d_hist, nspec, q.d_fitstart, nullptr, nullptr, st))) return rc2;
    }
    else
        launches--;
    if (ctx->profiling) HC_CUDA(ctx, record_stage(ctx, 4, st));
    ctx->last_launches = launches;
    return HC_SUCCESS;
}

namespace {

// The length table of one query, passed by value as a kernel parameter
// (7 KB, inside the 32 KB parameter space), so that writing it to device
// scratch needs neither a host copy nor a host buffer that must outlive the call.
struct LenTable
{
    LenDev l[HC_MAX_LENGTHS];
};

__global__ void k_put_lens(const LenTable t, uint32_t nlen, LenDev *__restrict__ dst)
{
    if (threadIdx.x < nlen) dst[threadIdx.x] = t.l[threadIdx.x];
}

template <class F>
cudaError_t load_one(F *f)
{
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, f);
}

}  // namespace

// Loads every kernel launch_query_scratch can launch into the current
// context. With lazy module loading (the default) a kernel's code is loaded,
// and device memory allocated for it, at its first launch; asking for its
// attributes loads it now instead.
int preload_query_kernels(hc_ctx *ctx)
{
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    chk(load_one(k_put_lens));
    chk(load_one(k_windows<1>));
    chk(load_one(k_windows<3>));
    chk(load_one(k_cost));
    chk(load_one(k_order));
    chk(load_one(k_tailfit));
    chk(load_one(k_search<false, 1>));
    chk(load_one(k_search<false, 2>));
    chk(load_one(k_search<false, 2, true>));
    chk(load_one(k_search<false, 4>));
    chk(load_one(k_search<false, 8>));
    chk(load_one(k_search<true, 2>));
    chk(load_one(k_search_small));
    HC_CUDA(ctx, e);
    return HC_SUCCESS;
}

// The expeRT tail fit of the spectra in `list` (its length *d_nlist on the
// device, at most nmax): the fallback of the learned tail.
int tailfit_list(hc_ctx *ctx, hc_result *d_out, const uint32_t *d_hist, const uint32_t *list,
                 const uint32_t *d_nlist, uint32_t nmax, cudaStream_t st)
{
    if (nmax == 0) return HC_SUCCESS;
    QueryScratch &q = ctx->qs;
    int rc = grow(ctx, &q.d_fitstart, &q.fit_cap, (size_t)nmax);
    if (rc) return rc;
    return launch_tailfit(ctx, d_out, d_hist, nmax, q.d_fitstart, list, d_nlist, st);
}

// The query pipeline of query_device with every scratch buffer supplied by
// the caller (used by the allocation-free entry point): the length table is
// written into s.lens by a kernel that takes it as a parameter, nothing is
// allocated and the host does not wait.
int launch_query_scratch(hc_ctx *ctx, const uint32_t *d_idx, const uint32_t *d_moz, const uint32_t *d_int,
                         const float *d_prec, const double *d_dM, uint32_t nspec, hc_result *d_out,
                         uint32_t *d_hist, const ScratchPtrs &s, cudaStream_t st)
{
    const uint32_t nlen = (uint32_t)ctx->lens.size();
    LenTable t;
    std::memset(&t, 0, sizeof(t));
    for (uint32_t i = 0; i < nlen; i++)
    {
        fill_lendev(ctx, ctx->lens[i], t.l[i]);
    }
    k_put_lens<<<1, HC_MAX_LENGTHS, 0, st>>>(t, nlen, s.lens);
    HC_CUDA(ctx, cudaGetLastError());
    ctx->last_launches = 0;
    if (nspec == 0) return HC_SUCCESS;
    uint32_t *nwide = s.work + kWkNwide;
    HC_CUDA(ctx, cudaMemsetAsync(s.work, 0, 4 * kWkPart, st));
    const uint32_t parts = auto_parts(ctx, nspec);
    int rc = launch_windows(ctx, s.lens, nlen, d_prec, d_dM, nspec, s.win, parts > 1 ? d_hist : nullptr, st);
    if (rc) return rc;
    SearchArgs a{};
    a.lens = s.lens;
    fill_lens(ctx, a);
    a.nlen = nlen;
    a.qc = ctx->d_qconst;
    a.idx = d_idx;
    a.moz = d_moz;
    a.inten = d_int;
    a.prec = d_prec;
    a.win = s.win;
    a.nspec = nspec;
    a.dF = ctx->p.dF;
    a.min_shp = ctx->p.min_shp;
    a.thr = ctx->p.min_shp > 0 ? ctx->p.min_shp : 1;
    a.maxbin = ctx->p.max_mass * ctx->p.scale;
    a.out = d_out;
    a.hist = d_hist;
    a.wide_list = s.wide;
    a.nwide = nwide;
    a.work = s.work;
    a.parts = parts;
    a.defer_cap = ctx->tuning.defer_cap;
    a.maxz = ctx->p.maxz;
    a.classes = ctx->d_classes;
    int launches = 4;
    rc = launch_packed(ctx, a, nspec, nlen, s.win, s.order, s.work, st, launches, false);
    if (rc) return rc;
    SearchArgs b = a;
    b.persistent = 1;
    b.order = nullptr;
    b.only = s.wide;
    b.nonly_dev = nwide;
    b.work = s.work + kWkWide;
    b.obase = b.olim = nullptr;
    b.parts = 0;
    b.tile = std::max(kRowG, ctx->tuning.tile / 2 / kRowG * kRowG);  // same shared memory, 16-byte words
    rc = launch_search<true>(ctx, b, ctx->sm_count, ctx->tuning.threads, search_smem(b.tile, b.dF, true, ctx->tuning.threads), 2, st);
    if (rc) return rc;
    if ((rc = launch_tailfit(ctx, d_out, d_hist, nspec, s.fitstart, nullptr, nullptr, st))) return rc;
    ctx->last_launches = launches + 1;
    return HC_SUCCESS;
}

}  // namespace hc

using namespace hc;

extern "C" int hc_check_tailfit(hc_ctx *ctx, const uint32_t *d_hist, hc_result *d_res, uint32_t n, int plain,
                                int32_t *d_first)
{
    if (!ctx || (n && (!d_hist || !d_res || !d_first))) return HC_ERR_INVLD_PTR;
    if (n == 0) return HC_SUCCESS;
    HC_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    if (plain)
    {
        k_tailfit_plain<<<(n + kTfPlainWarps - 1) / kTfPlainWarps, kTfPlainWarps * 32, 0, st>>>(
            d_res, d_hist, n, ctx->p.min_cpsm, ctx->p.expect_max, d_first);
        HC_CUDA(ctx, cudaGetLastError());
    }
    else if (const int rc = launch_tailfit(ctx, d_res, d_hist, n, d_first, nullptr, nullptr, st))
        return rc;
    HC_CUDA(ctx, cudaStreamSynchronize(st));
    return HC_SUCCESS;
}
