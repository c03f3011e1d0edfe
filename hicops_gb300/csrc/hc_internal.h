// Internal declarations shared by the host API (hc_api.cpp) and the device
// code (hc_index.cu, hc_query.cu). Not installed; not part of the C ABI.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "hicops_gb300.h"

namespace hc {

constexpr int kMaxZ = 8;           // fragment charges handled (the reference clamps maxz <= 5)
constexpr int kLgTable = 256;      // lgfact entries kept on the device (flagged past 80)
constexpr int kRefMaxShp = 81;     // MAX_SHDPEAKS + 1 (utils.h:110)
constexpr size_t kIaPad = 128;     // postings arrays are padded: the query reads aligned 16-byte groups
// Row table: for every bucket, the position of its first posting whose entry
// is >= k * kRowG, for k = 0 .. ceil(n / kRowG). Scorecard tiles are whole
// multiples of kRowG entries, so every interior tile boundary is a lookup.
constexpr uint32_t kRowG = 2048;
// Query postings: the same postings as the reference's iA (ids entry*speclen
// + ion, ascending inside each bucket), stored as
//   (entry << 3) | (isY << 2)
// which is the byte offset of the candidate's scorecard word (two 32-bit
// words per candidate, b then y) counted from entry 0: a tile starting at
// entry c0 finds a posting's word at x - (c0 << 3) with no further decoding.
// The ion of each posting (needed only to give the reference's ids back)
// sits in a parallel u16 array. Every bucket starts at a multiple of 4 words;
// the gaps hold kQpostPad, which lies past every tile.
constexpr uint32_t kQpostPad = 0xFFFFFFFFu;
constexpr uint32_t kQpEntryShift = 3;
constexpr uint32_t kQpMaxEntries = (1u << 29) - 2;  // entries of one length the encoding holds

// Entry classes. An entry's first y ion (y1), at every fragment charge, is
// fixed by a few facts about the entry: whether its mass is legal, whether it
// takes the mod-spectrum path (utils.cpp:378-505 when it carries mods), its
// last residue and the mod there. Those facts form a small "code"; entries
// with the same code share their y1 keys (a tryptic database has a few dozen
// codes, and y1 postings are about half of all the postings a search
// visits). Every code seen gets a class id with the class's keys; the search
// postings leave out the y1 postings of classed entries, and the search
// starts each candidate's y word with what its class's keys collect from the
// spectrum's peaks (the same count and intensity sum the left-out postings
// would have added). The index build checks every left-out posting against
// its class's key, so the code only has to be right for an entry to be
// classed, never for the results to be right. (The first b ion has as few
// codes, but its postings are a tenth of the total: classing it costs the
// search more per candidate than its postings do.)
constexpr uint32_t kMaxClasses = 127;   // class ids 0 .. 126
constexpr uint32_t kClassNone = 127;    // an entry without a class (adds nothing)
constexpr uint32_t kCodes = 1u << 10;   // codes: legal, path, last residue, mod at the last residue

// The class keys, per class and charge.
struct ClassKeys
{
    uint32_t n;         // classes
    uint32_t maxkey;    // the largest key of any class (peaks above it + dF cannot reach one)
    uint32_t key[kMaxClasses][kMaxZ];
};

// One peptide length's device-resident index. All arrays are device pointers.
struct LenDev
{
    uint32_t L, speclen, half, n;  // n = entries
    uint32_t npep;
    uint32_t magic, msh;           // floor(x / speclen) = umulhi(x, magic) >> msh, x < 2^31
    uint32_t stride;               // row-table entries per bucket: ceil(n / kRowG) + 1
    const float *mass;
    const uint32_t *seqid;
    const uint64_t *sites;
    const uint32_t *modnum;
    const uint8_t *seqs;
    const uint32_t *bA;
    const uint32_t *qA;            // bucket starts in qp (multiples of 4)
    const uint32_t *qp;            // query postings (see kQpostPad)
    const uint32_t *qps;           // search postings: qp without the y1 postings of classed entries
    const uint32_t *rows;          // row table over qps, [bucket][k] with `stride` entries per bucket
    const uint8_t *cls;            // per entry: its class (kClassNone: none)
};

// Integer ion-key tables, derived on the host with the reference's double
// arithmetic (utils.cpp:231-276 and 378-505; see hc_host.cpp).
struct IonTables
{
    uint32_t bf[26][kMaxZ];   // (uint)((GETAA(a, z+1) * scale) / (z+1))
    uint32_t yf[26][kMaxZ];   // (uint)(((GETAA(a, z+1) + H2O) * scale) / (z+1))
    uint32_t inc[26][kMaxZ];  // (uint)((GETAA(a, 0) * scale) / (z+1))
    uint32_t bfm[26][kMaxZ];  // (uint)(GETAA(a, z+1) * scale)          (mod spectra)
    uint32_t yfm[26][kMaxZ];  // (uint)((GETAA(a, z+1) + H2O) * scale)  (mod spectra)
    uint32_t incm[26];        // (uint)(GETAA(a, 0) * scale)             (mod spectra)
    uint32_t mod_mass[16];
    uint32_t maxz, scale, min_mass, max_mass;
};

constexpr uint32_t kLog10Tab = 1u << 24;  // log10(n) for every n the packed sums can reach

// Table of the tail fit's logarithm: for 128 intervals of the mantissa the
// reciprocal of the midpoint and minus its log10.
constexpr int kLgTab = 128;

struct QueryConst
{
    double lgfact[kLgTable];   // log10(n!) exactly as utils.h:115-131 builds it
    float lgfact_f[kLgTable];  // the same, rounded to float (fast path)
    double lg_tab[2 * kLgTab];
    const double *log10_tab;   // device table: log10_tab[n] = log10(n), n < kLog10Tab (host libm values)
};

// Host-side record of one length.
struct LenHost
{
    uint32_t L = 0, npep = 0, n = 0;
    uint64_t npost = 0;
    float *d_mass = nullptr;
    uint32_t *d_seqid = nullptr;
    uint64_t *d_sites = nullptr;
    uint32_t *d_modnum = nullptr;
    uint8_t *d_seqs = nullptr;
    uint32_t *d_bA = nullptr;
    uint32_t *d_qA = nullptr;    // padded bucket starts (max_mass*scale + 1)
    uint32_t *d_qp = nullptr;    // query postings, qA[nb] words (+ kIaPad)
    uint16_t *d_qion = nullptr;  // ion of each query posting (same positions as d_qp)
    uint32_t *d_qAs = nullptr;   // search postings: bucket starts (multiples of 4)
    uint32_t *d_qps = nullptr;   // search postings (query postings less the classed y1 ones)
    uint8_t *d_cls = nullptr;    // per entry: its class
    uint64_t nsearch = 0;        // search postings (without padding)
    uint32_t *d_rows = nullptr;  // row table over the search postings (max_mass*scale buckets x stride)
    uint32_t stride = 0;
    bool built = false;
};

// Device scratch for one query call; grown on demand.
struct QueryScratch
{
    int2 *d_win = nullptr;        // nspec * nlen windows [minl, maxl]
    uint32_t *d_wide = nullptr;   // spectra that overflowed the packed scorecard
    uint32_t *d_nwide = nullptr;
    uint32_t *d_work = nullptr;   // work counters | cost-class counts | cursors
    uint32_t *d_order = nullptr;  // longest-first order | cost classes
    int32_t *d_fitstart = nullptr;  // first regression bin of each spectrum's tail fit (-1: none)
    size_t fit_cap = 0;
    size_t win_cap = 0, wide_cap = 0, order_cap = 0;
    // host-path staging
    void *d_in = nullptr;
    size_t in_cap = 0;
    void *d_outbuf = nullptr;
    size_t out_cap = 0;
};

// Caller-supplied scratch of one query (see launch_query_scratch).
struct ScratchPtrs
{
    int2 *win;          // nspec * nlen
    uint32_t *wide;     // nspec + 4
    uint32_t *work;     // kWorkWords
    uint32_t *order;    // 2 * nspec
    int32_t *fitstart;  // nspec
    LenDev *lens;       // HC_MAX_LENGTHS
};

// Per-query counters (device words): the searches' work counters, the
// overflow list's length, the small-window split point of the longest-first
// order, then its per-class counts and cursors.
constexpr uint32_t kWkSearch = 0, kWkWide = 1, kWkNwide = 2, kWkSmall = 3, kWkSplit = 4;
constexpr uint32_t kWkCnt = 8, kWkCur = kWkCnt + 64, kWkArrived = kWkCur + 64;
// spectra searched in parts (k_search): per spectrum the parts that have ended, then
// (not zeroed) each part's sums
constexpr uint32_t kMaxPartItems = 256, kPartWords = 8;
constexpr uint32_t kWkPart = kWkArrived + kMaxPartItems / 2, kWorkWords = kWkPart + kPartWords * kMaxPartItems;
static_assert(kWkPart % 4 == 0, "16-byte aligned");

// What a captured query graph was recorded with; a call that differs re-captures.
struct GraphKey
{
    uint64_t epoch;             // of the index and of the scratch that the graph's kernels name
    const void *idx, *moz, *inten, *prec, *dM, *out, *hist;
    const void *mlp, *learned;  // the learned form: network, learned log10 e-values (else null)
    float gate_resid;           // ... and its gate (kernel parameters of the captured graph)
    uint32_t gate_radius;
    uint64_t net_serial;        // ... and the network's buffers, and its context's scratch
    uint64_t net_epoch;
    uint32_t nspec, npeaks;
    hc_tuning tuning;
    uint32_t auto_shape;
    uint32_t profiling;  // stage events captured or not
};

struct StreamStage;  // staging slots of hc_dslim_query_stream (hc_stream.cpp)
void free_stream_stage(StreamStage *s);

struct Launch
{
    uint32_t threads, tile, ctas_per_sm, pairs_per_warp;
    size_t smem;
    int grid;
};

}  // namespace hc

struct hc_ctx
{
    int device = 0;
    // Index arrays and build scratch come from this pool, ordered on `stream`:
    // building a length takes some 25 buffers, and cudaMalloc / cudaFree at 10-25 us
    // each were two thirds of a build. At a wait for the stream the pool gives free memory
    // back to the device until it holds kPoolKeep bytes, the index's arrays among them: a
    // small index keeps a build's scratch for the next length and the next build (45 MB
    // beside 20,000 peptides' 340 MB, 170 MB beside 660), one past kPoolKeep maps it anew.
    // The pool goes with the context.
    cudaMemPool_t pool = nullptr;
    void *h_read = nullptr;  // pinned words the build reads counts back through
    int sm_count = 0;
    size_t smem_optin = 0;     // per CTA, opt-in maximum
    size_t smem_sm = 0;        // per SM
    size_t smem_reserved = 0;  // per CTA, kept by the system
    hc_params p{};
    cudaStream_t stream = nullptr;
    cudaEvent_t searched = nullptr;  // after the last search on a stream other than `stream`
    bool elsewhere = false;          // ... which has not been seen to have ended
    hc_tuning tuning{}, initial{};  // the shape, and a new context's
    bool auto_shape = true;  // nobody chose a launch shape: picked by what is searched (launch_packed)
    std::vector<hc::LenHost> lens;
    hc::LenDev *d_lens = nullptr;
    hc::IonTables tables{};
    hc::IonTables *d_tables = nullptr;
    // entry classes (shared by all lengths; ids are only ever added)
    std::vector<uint8_t> class_of;     // code -> class id
    hc::ClassKeys classes{};
    hc::ClassKeys *d_classes = nullptr;
    uint8_t *d_class_of = nullptr;
    hc::QueryConst *d_qconst = nullptr;
    hc::QueryScratch qs;
    std::string last_error;
    int last_launches = 0;
    bool lens_dirty = true;
    // Counts what a captured graph does not outlive: a length's arrays freed or built
    // (a graph holds their addresses, sizes and the launches picked for them), and
    // every buffer of the pipeline allocated again.
    uint64_t epoch = 0;
    bool profiling = false;
    bool last_learned = false;  // the last query ran the learned tail (stage 5 recorded)
    cudaEvent_t ev[6] = {};  // windows | search | wide | tailfit | learned tail boundaries
    unsigned long long *d_phase = nullptr;  // per-phase SM cycles of the search kernel (diagnostics)
    double *d_log10 = nullptr;              // log10 table of the exact hyperscore path
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t graph_exec = nullptr;
    hc::GraphKey graph_key{};
    int graph_launches = 0;
    float *d_grad_part = nullptr;  // training: the CTAs' shares of a minibatch's gradients (hc_mlp.cu)
    uint32_t grad_part_cap = 0;
    hc::StreamStage *stage = nullptr;  // kept between streaming calls, grown on demand
};

namespace hc {

// What the device entry enumeration needs (passed by value to its kernels):
// the float residue and static-mod masses of UTILS_CalculatePepMass
// (utils.cpp:290-303), the residue -> mod-condition map and per-condition
// limits of MODS_ModList (mods.cpp:333-384), and each mod's mass as
// UTILS_CalculateModMass adds it (float(scaled mass) / float(scale)).
// Site bit of an N-terminal mod (an extension without a reference
// counterpart: a mod whose residue code is '^'); residues use bits 0..L-1.
constexpr int kNtermBit = 63;

struct EnumConst
{
    float aa[26];
    float stat[26];
    float h2o;
    int8_t cond_of[26];  // mod condition of a residue, -1 if none
    int8_t nterm;        // mod condition of the N-terminus ('^'), -1 if none
    uint32_t limit[HC_MAX_MODS];
    float modadd[HC_MAX_MODS];
    uint32_t vmods, nmods;
};

// hc_host.cpp
void make_enum_const(const hc_params &p, EnumConst *e);
void make_ion_tables(const hc_params &p, IonTables *t);
void make_query_const(QueryConst *q);
void make_log10_table(double *t, uint32_t n);
int64_t make_entries(const hc_params &p, uint32_t L, const uint8_t *seqs, uint32_t npep,
                     hc_entry *out, int64_t cap);
void division_magic(uint32_t d, uint32_t *magic, uint32_t *sh);

// hc_index.cu
int build_length_device(hc_ctx *ctx, LenHost &lh, const hc_entry *h_entries, bool sort_by_mass);
int build_query_postings(hc_ctx *ctx, LenHost &lh, const uint32_t *d_ids, const uint32_t *d_keys);
int build_rows(hc_ctx *ctx, LenHost &lh);  // from query postings: entry classes, search postings and their row table
void class_keys_of(const hc_params &p, const IonTables &t, uint32_t code, uint32_t *keys);
int check_query_postings(hc_ctx *ctx, const LenHost &lh, uint64_t qtotal);
void free_len(hc_ctx *ctx, LenHost &lh);
int export_ids(hc_ctx *ctx, const LenHost &lh, uint32_t *d_ids);

// hc_query.cu
uint32_t max_tile(const hc_ctx *ctx, uint32_t dF, uint32_t threads);
uint32_t max_tile_for(const hc_ctx *ctx, uint32_t dF, uint32_t ctas_per_sm, uint32_t threads);
int prepare_query(hc_ctx *ctx, uint32_t nspec);
size_t search_smem(uint32_t tile, uint32_t dF, bool wide, uint32_t threads);
// tailfit = false leaves the e-values to the learned tail (learned_pipeline)
int query_device(hc_ctx *ctx, const uint32_t *d_idx, const uint32_t *d_moz, const uint32_t *d_int,
                 const float *d_prec, const double *d_dM, uint32_t nspec, uint32_t npeaks,
                 hc_result *d_out, uint32_t *d_hist, cudaStream_t stream, bool tailfit = true);
// profiling: stage event i on st (a graph node when st is capturing)
cudaError_t record_stage(hc_ctx *ctx, int i, cudaStream_t st);
int tailfit_list(hc_ctx *ctx, hc_result *d_out, const uint32_t *d_hist, const uint32_t *list,
                 const uint32_t *d_nlist, uint32_t nmax, cudaStream_t st);
int sync_lengths(hc_ctx *ctx);
int preload_query_kernels(hc_ctx *ctx);
int launch_query_scratch(hc_ctx *ctx, const uint32_t *d_idx, const uint32_t *d_moz, const uint32_t *d_int,
                         const float *d_prec, const double *d_dM, uint32_t nspec, hc_result *d_out,
                         uint32_t *d_hist, const ScratchPtrs &s, cudaStream_t st);

// hc_mlp.cu: the learned tail after a search without tail fit
int learned_prepare(hc_mlp *m, uint32_t n);
void learned_key(const hc_mlp *m, GraphKey *key);
int learned_pipeline(hc_mlp *m, const uint32_t *d_hist, hc_result *d_res, uint32_t n, float *lg, cudaStream_t st,
                     int *launches);

constexpr uint64_t kPoolKeep = 1ull << 30;  // hc_ctx::pool's release threshold
constexpr size_t kReadBytes = 4096;  // hc_ctx::h_read

// hc_api.cpp: device memory of the index and its builds, n elements (at least one)
cudaError_t pool_alloc(hc_ctx *ctx, void **p, size_t bytes);
template <class T>
cudaError_t dalloc(hc_ctx *ctx, T **p, size_t n)
{
    return pool_alloc(ctx, (void **)p, sizeof(T) * (n ? n : 1));
}
template <class T>
void dfree(hc_ctx *ctx, T *&p)
{
    if (p) cudaFreeAsync(p, ctx->stream);
    p = nullptr;
}

// Copies to the device that have ended, for any stream, when they return. (The runtime's
// blocking copy of pageable memory may end after the call, on the legacy stream, which neither
// the context's stream nor a caller's non-blocking one waits for.) upload: to a buffer that
// nothing has read yet; overwrite: behind what a caller's blocking streams still read there.
inline cudaError_t upload(hc_ctx *ctx, void *d, const void *h, size_t bytes)
{
    const cudaError_t e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, ctx->stream);
    return e != cudaSuccess ? e : cudaStreamSynchronize(ctx->stream);
}
inline cudaError_t overwrite(void *d, const void *h, size_t bytes)
{
    const cudaError_t e = cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice);
    return e != cudaSuccess ? e : cudaStreamSynchronize(cudaStreamLegacy);
}

// For calls that touch no stream under capture (reading a file is a host call to its
// caller): they may come while a thread of the program captures a graph, in a mode that
// forbids all others most calls until it has ended.
struct BesideCapture
{
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~BesideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    BesideCapture(const BesideCapture &) = delete;
};

// Device scratch of one call or build step, given back when it goes out of
// scope (also on error paths); the work enqueued on the context's stream until
// then still has it.
struct PoolScratch
{
    hc_ctx *ctx;
    std::vector<void *> ptrs;
    explicit PoolScratch(hc_ctx *c) : ctx(c) {}
    PoolScratch(const PoolScratch &) = delete;
    template <class T>
    cudaError_t alloc(T **p, size_t n)
    {
        const cudaError_t e = dalloc(ctx, p, n);
        if (e == cudaSuccess) ptrs.push_back(*p);
        return e;
    }
    ~PoolScratch()
    {
        for (void *p : ptrs) dfree(ctx, p);
    }
};

// A search was enqueued on st and may be left running there.
int left_running(hc_ctx *ctx, cudaStream_t st);
// No search of the context is running (as far as one can see that is not part of a
// graph of the caller's own).
bool device_idle(hc_ctx *ctx);

int set_error(hc_ctx *ctx, int code, const std::string &msg);
int cuda_check(hc_ctx *ctx, cudaError_t e, const char *what);

}  // namespace hc

#define HC_CUDA(ctx, call)                                          \
    do {                                                            \
        cudaError_t _e = (call);                                    \
        if (_e != cudaSuccess) return hc::cuda_check((ctx), _e, #call); \
    } while (0)
