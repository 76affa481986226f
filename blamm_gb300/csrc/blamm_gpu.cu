// blamm_gpu.cu -- libblamm_gpu.so: the C ABI declared in include/blamm_gpu.h.
//
// Host half of the GB300 scan: motif-bank planning (length-sorted motif tiles,
// fixed-point BF16 hi/lo split, per-column guard band), device buffers, and
// the drivers that chain pack -> fused tcgen05 scan -> FP32 rescoring (or the
// plain FP32 kernel) on the context's stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "blamm_gpu.h"
#include "scan_kernels.cuh"
#include "scan_tc.cuh"
#include "hist_kernels.cuh"
#include "hist_tc.cuh"
#include "ingest_kernels.cuh"
#include "plan_kernels.cuh"

#include <nvtx3/nvToolsExt.h>

// A named range on the profiler timeline (nsys, ncu --nvtx) around each entry point;
// NVTX calls do nothing unless a tool is attached.
namespace {
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};
}  // namespace

using namespace blamm;

static_assert(sizeof(blamm_hit) == sizeof(HitRec), "hit record layout");

// A synchronous scan's counters, and behind them the times that its kernels note (KernelTimes).
constexpr int kCounts = 4, kTimes = 4;

// Default scan window (positions): see launch_tc_windows.
constexpr int64_t kEWindowDefault = int64_t(16) << 20;

struct blamm_ctx {
    int device = 0;
    int sm_count = 0;
    int max_smem = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};  // the kernels' start and end, the plain scan's start
    std::string err;
    int mode = BLAMM_MODE_AUTO;
    int auto_terms = 1;  // BLAMM_MODE_AUTO: the form in use, 1 or 2 BF16 terms or kE4M3 (1 until tuned)
    int lower_scores = 0;  // soft-masked bases add their PWM value (simple scan) when 1
    long long wait_limit = 4000000000LL;  // clock64 cycles (about 2 s)
    int debug_stall = 0;                  // test hook: make the scan kernel's first wait run out
    int64_t ewindow = 0;                  // positions per tensor-core scan window (one-hot entry array)

    // motif bank (host copy); `active` lists the columns scanned (all when empty)
    int ncols = 0, p_rows = 0, lmax = 0;
    std::vector<int32_t> active;
    int32_t *d_active = nullptr;
    size_t cap_active = 0;
    bool active_dirty = false;
    std::vector<float> P;
    std::vector<int32_t> len;
    std::vector<float> thr;
    float *d_P = nullptr;
    int32_t *d_len = nullptr;
    float *d_thr = nullptr;

    // tensor-core plan (valid for plan_terms; rebuilt on mode/threshold change)
    int plan_terms = 0;
    bool plan_valid = false;
    int ntiles = 0;
    std::vector<TileDesc> tiles;  // ntiles + 1: the last one holds the end offset
    int erows = 0;               // one-hot entries per E stage
    int plan_tg = 1;             // most tiles per group whose A fits in shared memory (evened out)
    bool plan_stream = false;    // not even one tile fits: A is streamed
    TileDesc *d_tiles = nullptr;
    uint8_t *d_abuf = nullptr;
    int32_t *d_slot_col = nullptr;
    float *d_slot_thr = nullptr;
    size_t cap_tiles = 0, cap_abuf = 0, cap_slot_col = 0, cap_slot_thr = 0;
    std::vector<int32_t> slot_col;  // (the upload's source)
    // per-column fixed-point BF16 terms and guard bands of the bank (for colq_terms terms)
    bool colq_valid = false;
    int colq_terms = 0;
    std::vector<int> colq_k;
    std::vector<double> colq_guard;
    std::vector<uint32_t> colq_off;  // column c's 4L values start at colq_off[c]
    std::vector<uint16_t> colq_hi, colq_lo;
    std::vector<uint8_t> colq_e8;  // E4M3 codes of P(c) x 2^colq_k[c] (the E4M3 form)
    uint8_t *d_colq = nullptr;     // on the device: guards, exponents, offsets, terms (colq_at: their places)
    size_t cap_colq = 0, colq_at[5] = {0, 0, 0, 0, 0};
    // planner knobs: widest tile (columns beyond a tile's 128 rows have no effect) and the
    // fixed cycles per job (kept for callers that set and read it; no plan depends on it)
    int plan_nmax = 256;
    double plan_job_cost = 700.0;

    // stream buffers
    char *d_bases = nullptr;
    size_t cap_bases = 0;
    uint32_t *d_seq2 = nullptr, *d_zmask = nullptr;
    size_t cap_words32 = 0, cap_zmask = 0;
    uint4 *d_e16 = nullptr;  // one-hot entries of the packed stream (tensor-core A operand windows)
    size_t cap_e16 = 0;
    int64_t *d_runs = nullptr;
    size_t cap_runs = 0;
    uint4 *d_cand = nullptr;  // candidate record slots (scan_tc.cuh: blocks of kRecBlock)
    int64_t cand_cap = 0;     // record slots
    int64_t cand_spare = 0;   // spare ones behind them
    blamm_hit *d_hits = nullptr;
    int64_t hits_cap = 0;
    unsigned long long *d_counters = nullptr;  // record slots, hits, status (bit 0: a wait timed out), candidates; times
    // hit filtering of one chunk of a pipelined blamm_scan: hits at chunk positions >=
    // keep_below are dropped (0: none), pos_base is added to the positions written
    int64_t keep_below = 0, pos_base = 0;
    // blamm_scan's copy pipeline: a second stream and double-buffered chunk inputs
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t chunk_ev[2] = {nullptr, nullptr};
    char *d_chunk_bases[2] = {nullptr, nullptr};
    size_t cap_chunk_bases[2] = {0, 0};
    int64_t *d_chunk_runs[2] = {nullptr, nullptr};
    size_t cap_chunk_runs[2] = {0, 0};
    int64_t *h_chunk_runs[2] = {nullptr, nullptr};  // pinned: their copies stay asynchronous
    size_t cap_h_chunk_runs = 0;
    cudaEvent_t done_ev[2] = {nullptr, nullptr};  // per input buffer: its chunk's kernels are done
    unsigned long long *h_chunk_counts = nullptr;  // pinned, 4 per chunk: candidates, hits, status
    size_t cap_h_chunk_counts = 0;
    // resident stream (blamm_stream_load_fasta): FASTA text, filtered bases, run table
    // (stream position, sequence index, position in the sequence), header offsets
    char *d_raw = nullptr, *d_stream = nullptr;
    size_t cap_raw = 0, cap_stream = 0;
    int64_t *d_srun[3] = {nullptr, nullptr, nullptr}, *d_shdr = nullptr;
    size_t cap_srun[3] = {0, 0, 0}, cap_shdr = 0;
    int64_t stream_n = 0, stream_nruns = 0, stream_nseqs = 0;
    uint8_t *d_theo = nullptr;  // theoretical histograms: bank, tables, results of a call
    size_t cap_theo = 0;
    // FASTA parsing: tile summaries, the parser before each tile, totals (4,704 bytes per 32 KB of text)
    uint4 *d_ing_tiles = nullptr;  // the tiles' sums (IngTile)
    IngPrefix *d_ing_prefix = nullptr;
    unsigned long long *d_ing_totals = nullptr;
    size_t cap_ing_tiles = 0, cap_ing_prefix = 0, cap_ing_totals = 0;
    bool prof_on = false;
    long long *d_prof = nullptr;
    std::vector<long long> prof;  // last scan's role timing, 32 counters per CTA
    int prof_ctas = 0;

    blamm_stats stats{};
    int64_t rec_slots = 0;  // record slots the last tensor-core scan reserved
    uint8_t *h_stage = nullptr;  // pinned: inputs of short host scans, counters and first hits on their way back
    size_t cap_stage = 0;
};

// ------------------------------------------------------------------ errors
static int fail(blamm_ctx *c, int code, const char *fmt, ...)
{
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    return code;
}

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? BLAMM_ERR_NOMEM : BLAMM_ERR_CUDA, \
                        "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

// Grow a context buffer to at least `need` elements.  The stream-ordered
// allocator keeps a growing buffer from synchronising the whole device (other
// contexts' work keeps running); every use of these buffers is on ctx->stream.
template <typename T>
static int ensure(blamm_ctx *ctx, T **ptr, size_t *cap, size_t need)
{
    if (need <= *cap && *ptr) return BLAMM_OK;
    if (*ptr) CK(cudaFreeAsync(*ptr, ctx->stream));
    *ptr = nullptr;
    *cap = 0;
    size_t n = std::max<size_t>(need, 1);
    CK(cudaMallocAsync((void **)ptr, n * sizeof(T), ctx->stream));
    *cap = n;
    return BLAMM_OK;
}

// Pinned staging of at least `bytes` (nothing may be in flight on it: every user waits).
static int ensure_stage(blamm_ctx *ctx, size_t bytes)
{
    if (bytes <= ctx->cap_stage) return BLAMM_OK;
    if (ctx->h_stage) CK(cudaFreeHost(ctx->h_stage));
    ctx->h_stage = nullptr;
    ctx->cap_stage = 0;
    CK(cudaHostAlloc((void **)&ctx->h_stage, bytes, 0));
    ctx->cap_stage = bytes;
    return BLAMM_OK;
}

// memcpy, from a few threads where it is long (most of it is the destination's page faults).
static void copy_out(void *dst, const void *src, size_t bytes)
{
    constexpr size_t kPart = size_t(2) << 20;
    uint8_t *d = static_cast<uint8_t *>(dst);
    const uint8_t *s = static_cast<const uint8_t *>(src);
    std::thread help[3];
    const size_t parts = std::min<size_t>(4, bytes / kPart);
    size_t done = bytes;  // [done, bytes) is with the helpers
    try {
        for (size_t k = 1; k < parts; ++k) {
            const size_t at = bytes / parts * (parts - k);
            help[k - 1] = std::thread([=] { std::memcpy(d + at, s + at, done - at); });
            done = at;
        }
    } catch (...) {  // no more threads: the rest is copied here
    }
    std::memcpy(d, s, done);
    for (auto &t : help)
        if (t.joinable()) t.join();
}

// Spare record slots of an enqueued scan, two blocks per drain warp: its counts say how many
// candidates there were, also of records that did not fit.
static int64_t spare_slots(const blamm_ctx *ctx) { return (int64_t)ctx->sm_count * kEpiWarps * 2 * kRecBlock; }

// Candidate record slots: `need` rounded up to whole blocks (the scan counts on it), and behind
// them spare ones, where the scan puts what does not fit.
static int ensure_cand(blamm_ctx *ctx, int64_t need, int64_t spare = kRecBlock)
{
    need = std::max<int64_t>(1, (need + kRecBlock - 1) / kRecBlock) * kRecBlock;
    if (ctx->d_cand && need <= ctx->cand_cap && spare <= ctx->cand_spare) return BLAMM_OK;
    need = std::max(need, ctx->cand_cap);
    spare = std::max(spare, ctx->cand_spare);
    size_t cap = (size_t)(ctx->cand_cap + ctx->cand_spare);
    ctx->cand_cap = ctx->cand_spare = 0;
    if (int rc = ensure(ctx, &ctx->d_cand, &cap, (size_t)(need + spare))) return rc;
    ctx->cand_cap = need;
    ctx->cand_spare = spare;
    return BLAMM_OK;
}

static int scanned_columns(const blamm_ctx *ctx)
{
    return ctx->active.empty() ? ctx->ncols : (int)ctx->active.size();
}

// ------------------------------------------------------------------ planning
namespace {

// Fixed-point BF16 split of one column: hi on the grid 2^-k, lo on 2^-(k+8),
// with k chosen so |hi| <= 128 * 2^-k.  Every partial sum of such values over
// up to 256 motif positions is an integer multiple of 2^-(k+8) below 2^24 of
// those units, i.e. exactly representable in FP32: the tensor-core
// accumulation is exact, whatever its internal rounding.
int column_exponent(const float *col, int L)
{
    double mx = 0.0;
    for (int r = 0; r < 4 * L; ++r) mx = std::max(mx, (double)std::fabs(col[r]));
    if (!(mx > 0.0) || !std::isfinite(mx)) return -30;
    int e;
    double f = std::frexp(mx, &e);  // mx = f * 2^e, f in [0.5, 1)
    if (f == 0.5) e -= 1;           // mx is a power of two: mx <= 2^(e-1)
    return std::max(-30, std::min(40, e));
}

inline double q_hi(double v, int k) { return std::nearbyint(std::ldexp(v, k)) * std::ldexp(1.0, -k); }
inline double q_lo(double r, int k) { return std::nearbyint(std::ldexp(r, k + 8)) * std::ldexp(1.0, -(k + 8)); }

inline uint16_t bf16_bits_exact(double v)
{
    float f = (float)v;
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return (uint16_t)(u >> 16);  // exact: v has <= 8 significant bits
}

// E4M3 (sign, 4 exponent bits with bias 7, 3 mantissa bits; exponent 0 subnormal, largest
// finite 448).  In units of 2^-9 every E4M3 value is an integer: m (subnormal, m < 8) or
// (8 + m) 2^(e-1).
// The E4M3 value nearest to v (ties to even mantissa), as its code; |v| <= 448.
inline uint8_t e4m3_round(double v)
{
    const uint8_t sign = v < 0 ? 0x80 : 0;
    const double a = std::fabs(v) * 512.0;  // in units of 2^-9
    if (a < 7.5) {  // subnormal: nearest integer, 8 rounds up to the smallest normal
        const double r = std::nearbyint(a);
        return (uint8_t)(sign | (r >= 8.0 ? 0x08 : (uint8_t)r));
    }
    int e = 1;
    while (e < 15 && a >= 16.0 * std::ldexp(1.0, e - 1)) ++e;  // (8+m) 2^(e-1) with m < 8
    double m = std::nearbyint(a / std::ldexp(1.0, e - 1)) - 8.0;  // ties to even (FE_TONEAREST)
    if (m >= 8.0) {  // carried into the next binade
        m = 0.0;
        ++e;
    }
    if (e > 15 || (e == 15 && m > 6.0)) {  // beyond 448 (callers keep |v| <= 256)
        e = 15;
        m = 6.0;
    }
    return (uint8_t)(sign | (uint8_t)(e << 3) | (uint8_t)m);
}

// value of an E4M3 code in units of 2^-9
inline int64_t e4m3_units(uint8_t code)
{
    const int e = (code >> 3) & 15, m = code & 7;
    const int64_t a = e == 0 ? m : (int64_t)(8 + m) << (e - 1);
    return code & 0x80 ? -a : a;
}

}  // namespace

// The quantised bank on the device.
static int upload_colq(blamm_ctx *ctx)
{
    const size_t nc = (size_t)ctx->ncols;
    const void *src[5] = {ctx->colq_guard.data(), ctx->colq_k.data(), ctx->colq_off.data(),
                          ctx->colq_e8.empty() ? (const void *)ctx->colq_hi.data() : ctx->colq_e8.data(),
                          ctx->colq_lo.data()};
    const size_t bytes[5] = {8 * nc, 4 * nc, 4 * nc, ctx->colq_e8.size() + 2 * ctx->colq_hi.size(), 2 * ctx->colq_lo.size()};
    size_t total = 0;
    for (int i = 0; i < 5; ++i) {
        ctx->colq_at[i] = total;
        total += (bytes[i] + 255) & ~size_t(255);
    }
    if (int rc = ensure(ctx, &ctx->d_colq, &ctx->cap_colq, total)) return rc;
    for (int i = 0; i < 5; ++i)
        if (bytes[i]) CK(cudaMemcpyAsync(ctx->d_colq + ctx->colq_at[i], src[i], bytes[i], cudaMemcpyHostToDevice, ctx->stream));
    return BLAMM_OK;
}

static int build_plan(blamm_ctx *ctx, int terms)
{
    // an earlier plan's uploads may still read the host tables that this one rewrites
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->plan_valid = false;
    // the scanned columns, sorted by length (a stable counting sort)
    const int nsel = scanned_columns(ctx);
    std::vector<int> first(kMaxMotifLen + 2, 0), order(nsel);
    auto col_at = [&](int i) { return ctx->active.empty() ? i : (int)ctx->active[i]; };
    for (int i = 0; i < nsel; ++i) ++first[ctx->len[col_at(i)] + 1];
    for (int l = 0; l <= kMaxMotifLen; ++l) first[l + 1] += first[l];
    for (int i = 0; i < nsel; ++i) {
        const int c = col_at(i);
        order[first[ctx->len[c]]++] = c;
    }
    const int lmax_sel = nsel ? ctx->len[order.back()] : 1;
    if (lmax_sel > kMaxTcLen)
        return fail(ctx, BLAMM_ERR_UNSUPPORTED,
                    "motif length %d exceeds the tensor-core limit %d (use BLAMM_MODE_FP32)", lmax_sel,
                    kMaxTcLen);

    // the E4M3 form: one B term, 8 motif positions per k-step (K = 32); BF16: 4 (K = 16)
    const bool e8 = terms == kE4M3;
    const int kpos = e8 ? 8 : 4, nterm = e8 ? 1 : terms;
    if (e8 && lmax_sel > kMaxE4M3Len)
        return fail(ctx, BLAMM_ERR_UNSUPPORTED, "motif length %d exceeds the E4M3 form's limit %d", lmax_sel,
                    kMaxE4M3Len);
    const int gmax = std::max(1, (lmax_sel + kpos - 1) / kpos);
    // Tiles: at most 128 columns each, longest motifs first, cut from the long end, so that
    // only the tile of the shortest motifs is partly empty.  A job of a tile costs its
    // k-steps whatever its number of columns, so no other cut is cheaper.
    const int width = std::min(kTileCols, std::max(32, std::min(256, ctx->plan_nmax / 32 * 32)));
    std::vector<std::pair<int, int>> spans;
    for (int j = nsel; j > 0; j -= width) spans.push_back({std::max(0, j - width), j});
    const int ncols = ctx->ncols;

    // per-column quantisation and guard band: computed once per bank and number of terms
    // (thresholds only move the bias), reused by every later plan (column subsets,
    // threshold sets of the scan service)
    if (!(ctx->colq_valid && ctx->colq_terms == terms)) {
        ctx->colq_k.assign(ncols, 0);
        ctx->colq_guard.assign(ncols, 0.0);
        ctx->colq_off.assign(ncols + 1, 0);
        for (int c = 0; c < ncols; ++c) ctx->colq_off[c + 1] = ctx->colq_off[c] + 4 * (uint32_t)ctx->len[c];
        ctx->colq_hi.assign(e8 ? 0 : ctx->colq_off[ncols], 0);
        ctx->colq_lo.assign(terms == 2 ? ctx->colq_off[ncols] : 0, 0);
        ctx->colq_e8.assign(e8 ? ctx->colq_off[ncols] : 0, 0);
        for (int c = 0; c < ncols; ++c) {
            const float *col = &ctx->P[(size_t)c * ctx->p_rows];
            const int L = ctx->len[c];
            // BF16: grid 2^-k with |P| <= 128 * 2^-k; E4M3: scale 2^k with max|P| 2^k in (32, 64]
            const int k = (e8 ? 6 : 7) - column_exponent(col, L);
            ctx->colq_k[c] = k;
            double eq = 0.0, a = 0.0;
            for (int j = 0; j < L; ++j) {
                double mres = 0.0, mabs = 0.0;
                for (int b = 0; b < 4; ++b) {
                    const double v = col[4 * j + b];
                    double q;
                    if (e8) {
                        const uint8_t code = e4m3_round(std::ldexp(v, k));
                        ctx->colq_e8[ctx->colq_off[c] + 4 * j + b] = code;
                        q = std::ldexp((double)e4m3_units(code), -9 - k);
                    } else {
                        const double hi = q_hi(v, k);
                        const double lo = terms == 2 ? q_lo(v - hi, k) : 0.0;
                        ctx->colq_hi[ctx->colq_off[c] + 4 * j + b] = bf16_bits_exact(hi);
                        if (terms == 2) ctx->colq_lo[ctx->colq_off[c] + 4 * j + b] = bf16_bits_exact(lo);
                        q = hi + lo;
                    }
                    // only P > q can put a reference hit below T: sum(q) = sum(P) - sum(P - q)
                    mres = std::max(mres, v - q);
                    mabs = std::max(mabs, std::fabs(v));
                }
                eq += mres;
                a += mabs;
            }
            // guard = sum_j max_b (P - q)^+ (mres starts at 0) + the bound on the reference's
            // own rounding, |fl(sequential sum) - exact sum| <= gamma_{L-1} * sum|terms|
            const double u = std::ldexp(1.0, -24);
            const double nl = std::max(0, L - 1);
            const double gamma = nl * u / (1.0 - nl * u);
            ctx->colq_guard[c] = (eq + gamma * a) * (1.0 + 1e-9) + std::ldexp(1.0, -60);
        }
        if (int rc = upload_colq(ctx)) return rc;
        ctx->colq_terms = terms;
        ctx->colq_valid = true;
    }

    // Tiles and slots; the thresholds and A are built on the device from the quantised bank.
    // A of one k-step of one term is kStepBytes; a tile's terms follow one another.
    std::vector<TileDesc> &tiles = ctx->tiles;
    tiles.clear();
    const size_t nslots = spans.size() * kTileCols;
    ctx->slot_col.assign(nslots, -1);
    int nsteps = 0;
    for (size_t t = 0; t < spans.size(); ++t) {
        const auto &sp = spans[t];
        const int g = std::max(1, (ctx->len[order[sp.second - 1]] + kpos - 1) / kpos);
        tiles.push_back(TileDesc{g, nsteps});
        nsteps += g * nterm;
        std::copy(order.begin() + sp.first, order.begin() + sp.second, ctx->slot_col.begin() + t * kTileCols);
    }
    tiles.push_back(TileDesc{0, nsteps});
    int rc = ensure(ctx, &ctx->d_tiles, &ctx->cap_tiles, tiles.size());
    if (!rc) rc = ensure(ctx, &ctx->d_abuf, &ctx->cap_abuf, (size_t)nsteps * kStepBytes);
    if (!rc) rc = ensure(ctx, &ctx->d_slot_col, &ctx->cap_slot_col, nslots);
    if (!rc) rc = ensure(ctx, &ctx->d_slot_thr, &ctx->cap_slot_thr, nslots);
    if (rc) return rc;
    // (their sources live in the context, unchanged until the stream has been waited for)
    CK(cudaMemcpyAsync(ctx->d_tiles, tiles.data(), sizeof(TileDesc) * tiles.size(), cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(cudaMemcpyAsync(ctx->d_slot_col, ctx->slot_col.data(), sizeof(int32_t) * nslots, cudaMemcpyHostToDevice,
                       ctx->stream));
    if (!spans.empty()) {
        PlanParams p{};
        p.tiles = ctx->d_tiles;
        p.ntiles = (int32_t)spans.size();
        p.slot_col = ctx->d_slot_col;
        p.slot_thr = ctx->d_slot_thr;
        p.abuf = ctx->d_abuf;
        p.nsteps = nsteps;
        p.terms = terms;
        p.P = ctx->d_P;
        p.p_rows = ctx->p_rows;
        p.col_len = ctx->d_len;
        p.thr = ctx->d_thr;
        p.guard = reinterpret_cast<const double *>(ctx->d_colq + ctx->colq_at[0]);
        p.k = reinterpret_cast<const int32_t *>(ctx->d_colq + ctx->colq_at[1]);
        p.off = reinterpret_cast<const uint32_t *>(ctx->d_colq + ctx->colq_at[2]);
        p.hi = reinterpret_cast<const uint16_t *>(ctx->d_colq + ctx->colq_at[3]);
        p.lo = reinterpret_cast<const uint16_t *>(ctx->d_colq + ctx->colq_at[4]);
        p.e8 = ctx->d_colq + ctx->colq_at[3];
        plan_thr_kernel<<<(unsigned)((nslots + 7) / 8), 256, 0, ctx->stream>>>(p);
        CK(cudaGetLastError());
        plan_fill_kernel<<<(unsigned)nsteps, 256, 0, ctx->stream>>>(p);
        CK(cudaGetLastError());
    }
    ctx->ntiles = (int)spans.size();
    ctx->erows = kBlockPos + kpos * gmax + 8;
    // groups: as many of the first (longest) tiles as fit beside the E stages, then evened out
    const TcSmem L0 = tc_smem_layout(0, ctx->erows);
    const int room = (ctx->max_smem - (int)L0.total) / kStepBytes;
    int tg = 0;
    while (tg < ctx->ntiles && tiles[tg + 1].off <= room) ++tg;
    ctx->plan_stream = ctx->ntiles > 0 && tg == 0;
    const int ng = tg > 0 ? (ctx->ntiles + tg - 1) / tg : std::max(1, ctx->ntiles);
    ctx->plan_tg = std::max(1, (ctx->ntiles + ng - 1) / ng);
    ctx->plan_terms = terms;
    ctx->plan_valid = true;
    return BLAMM_OK;
}

// ------------------------------------------------------------------ API
extern "C" {

int blamm_version(void) { return 10000; }

int blamm_ctx_create(int device, blamm_ctx **out)
{
    if (!out) return BLAMM_ERR_ARG;
    *out = nullptr;
    blamm_ctx *ctx = new blamm_ctx();
    ctx->device = device;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || device < 0 || device >= ndev) {
        delete ctx;
        return BLAMM_ERR_CUDA;
    }
    int rc = BLAMM_OK;
    auto init = [&]() -> int {
        CK(cudaSetDevice(device));
        cudaDeviceProp prop;
        CK(cudaGetDeviceProperties(&prop, device));
        if (prop.major != 10)
            return fail(ctx, BLAMM_ERR_UNSUPPORTED, "compute capability %d.%d is not sm_100-class",
                        prop.major, prop.minor);
        ctx->sm_count = prop.multiProcessorCount;
        // scan window (positions, a multiple of 256): BLAMM_SCAN_WINDOW overrides the default
        ctx->ewindow = kEWindowDefault;
        if (const char *w = std::getenv("BLAMM_SCAN_WINDOW"))
            ctx->ewindow = std::max<int64_t>(kBlockPos, std::atoll(w) / kBlockPos * kBlockPos);
        ctx->max_smem = (int)prop.sharedMemPerBlockOptin;
        cudaFuncAttributes fa;
        // fails if no sm_103a image fits
        // (the raw-score and role-timing instances are set up when they are launched)
        for (const void *k : {(const void *)scan_tc_kernel<false, false, 1, false, false>,
                              (const void *)scan_tc_kernel<false, false, 2, false, false>,
                              (const void *)scan_tc_kernel<false, false, kE4M3, false, false>,
                              (const void *)scan_tc_kernel<false, false, 1, true, false>,
                              (const void *)scan_tc_kernel<false, false, 2, true, false>,
                              (const void *)scan_tc_kernel<false, false, 1, false, true>,
                              (const void *)scan_tc_kernel<false, false, 2, false, true>,
                              (const void *)scan_tc_kernel<false, false, kE4M3, false, true>,
                              (const void *)scan_tc_kernel<false, false, 1, true, true>,
                              (const void *)scan_tc_kernel<false, false, 2, true, true>}) {
            CK(cudaFuncGetAttributes(&fa, k));
            if (fa.maxThreadsPerBlock < kTcThreads)
                return fail(ctx, BLAMM_ERR_UNSUPPORTED,
                            "scan kernel: %d registers allow only %d threads per block (< %d)", fa.numRegs,
                            fa.maxThreadsPerBlock, kTcThreads);
            CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem));
        }
        CK(cudaFuncSetAttribute(plain_scores_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                ctx->max_smem));
        CK(cudaFuncSetAttribute(plain_scores_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                ctx->max_smem));
        CK(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
        for (auto &ev : ctx->ev) CK(cudaEventCreate(&ev));
        CK(cudaMalloc(&ctx->d_counters, (kCounts + kTimes) * sizeof(unsigned long long)));
        return BLAMM_OK;
    };
    rc = init();
    if (rc != BLAMM_OK) {
        fprintf(stderr, "blamm_ctx_create: %s\n", ctx->err.c_str());
        blamm_ctx_destroy(ctx);
        return rc;
    }
    *out = ctx;
    return BLAMM_OK;
}

void blamm_ctx_destroy(blamm_ctx *ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    void *bufs[] = {ctx->d_P,      ctx->d_len,   ctx->d_thr,      ctx->d_tiles, ctx->d_abuf,
                    ctx->d_slot_col, ctx->d_slot_thr, ctx->d_colq, ctx->d_prof, ctx->d_bases, ctx->d_seq2, ctx->d_zmask, ctx->d_e16,
                    ctx->d_runs,   ctx->d_cand,  ctx->d_hits,     ctx->d_counters,
                    ctx->d_active, ctx->d_chunk_bases[0], ctx->d_chunk_bases[1], ctx->d_chunk_runs[0],
                    ctx->d_chunk_runs[1], ctx->d_raw, ctx->d_stream, ctx->d_srun[0], ctx->d_srun[1],
                    ctx->d_srun[2], ctx->d_shdr, ctx->d_ing_tiles, ctx->d_ing_prefix, ctx->d_ing_totals, ctx->d_theo};
    if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
    for (void *b : bufs)
        if (b) cudaFree(b);
    for (auto &ev : ctx->ev)
        if (ev) cudaEventDestroy(ev);
    for (auto &ev : ctx->chunk_ev)
        if (ev) cudaEventDestroy(ev);
    for (auto &ev : ctx->done_ev)
        if (ev) cudaEventDestroy(ev);
    for (auto &h : ctx->h_chunk_runs)
        if (h) cudaFreeHost(h);
    if (ctx->h_chunk_counts) cudaFreeHost(ctx->h_chunk_counts);
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}

// Device bytes of the per-call buffers (stream, packed stream, one-hot window, run table,
// candidate records, hits, pipeline chunks, resident stream); the motif bank and its plan
// are not counted.
static int64_t call_buffer_bytes(const blamm_ctx *ctx)
{
    return (int64_t)(ctx->cap_bases + 4 * ctx->cap_words32 + 4 * ctx->cap_zmask + 16 * ctx->cap_e16 +
                     8 * ctx->cap_runs + 8 * (ctx->cap_chunk_runs[0] + ctx->cap_chunk_runs[1]) +
                     ctx->cap_chunk_bases[0] + ctx->cap_chunk_bases[1] + ctx->cap_raw + ctx->cap_stream +
                     8 * (ctx->cap_srun[0] + ctx->cap_srun[1] + ctx->cap_srun[2] + ctx->cap_shdr) +
                     16 * ctx->cap_ing_tiles + sizeof(IngPrefix) * ctx->cap_ing_prefix +
                     8 * ctx->cap_ing_totals + ctx->cap_theo) +
           16 * (ctx->cand_cap + ctx->cand_spare) + (int64_t)sizeof(blamm_hit) * ctx->hits_cap;
}

int blamm_ctx_call_bytes(const blamm_ctx *ctx, int64_t *bytes)
{
    if (!ctx || !bytes) return BLAMM_ERR_ARG;
    *bytes = call_buffer_bytes(ctx);
    return BLAMM_OK;
}

int blamm_release_buffers(blamm_ctx *ctx)
{
    if (!ctx) return BLAMM_ERR_ARG;
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->stream));
    if (ctx->copy_stream) CK(cudaStreamSynchronize(ctx->copy_stream));
    auto drop = [&](auto **ptr, auto *cap) {
        if (*ptr) cudaFreeAsync(*ptr, ctx->stream);
        *ptr = nullptr;
        *cap = 0;
    };
    drop(&ctx->d_bases, &ctx->cap_bases);
    drop(&ctx->d_seq2, &ctx->cap_words32);
    drop(&ctx->d_zmask, &ctx->cap_zmask);
    drop(&ctx->d_e16, &ctx->cap_e16);
    drop(&ctx->d_runs, &ctx->cap_runs);
    for (int b = 0; b < 2; ++b) {
        drop(&ctx->d_chunk_bases[b], &ctx->cap_chunk_bases[b]);
        drop(&ctx->d_chunk_runs[b], &ctx->cap_chunk_runs[b]);
    }
    drop(&ctx->d_raw, &ctx->cap_raw);
    drop(&ctx->d_stream, &ctx->cap_stream);
    for (int k = 0; k < 3; ++k) drop(&ctx->d_srun[k], &ctx->cap_srun[k]);
    drop(&ctx->d_shdr, &ctx->cap_shdr);
    drop(&ctx->d_ing_tiles, &ctx->cap_ing_tiles);
    drop(&ctx->d_ing_prefix, &ctx->cap_ing_prefix);
    drop(&ctx->d_ing_totals, &ctx->cap_ing_totals);
    drop(&ctx->d_theo, &ctx->cap_theo);
    ctx->stream_n = ctx->stream_nruns = ctx->stream_nseqs = 0;
    if (ctx->d_cand) cudaFreeAsync(ctx->d_cand, ctx->stream);
    ctx->d_cand = nullptr;
    ctx->cand_cap = ctx->cand_spare = 0;
    if (ctx->d_hits) cudaFreeAsync(ctx->d_hits, ctx->stream);
    ctx->d_hits = nullptr;
    ctx->hits_cap = 0;
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    ctx->h_stage = nullptr;
    ctx->cap_stage = 0;
    CK(cudaStreamSynchronize(ctx->stream));
    // give the freed memory back to the device: the stream-ordered pool would keep it
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, ctx->device) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
    return BLAMM_OK;
}

const char *blamm_last_error(const blamm_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int blamm_set_mode(blamm_ctx *ctx, int mode)
{
    if (!ctx) return BLAMM_ERR_ARG;
    if (mode != BLAMM_MODE_FP32 && mode != BLAMM_MODE_BF16 && mode != BLAMM_MODE_BF16X2 && mode != BLAMM_MODE_AUTO &&
        mode != BLAMM_MODE_E4M3)
        return fail(ctx, BLAMM_ERR_ARG, "unknown mode %d", mode);
    ctx->mode = mode;
    return BLAMM_OK;
}

int blamm_set_motifs(blamm_ctx *ctx, const float *P, int p_rows, int ncols, const int32_t *col_len,
                     const float *thr)
{
    const NvtxRange nvtx_range("blamm_set_motifs");
    if (!ctx) return BLAMM_ERR_ARG;
    if (!P || !col_len || !thr || ncols <= 0 || p_rows <= 0 || p_rows % 4)
        return fail(ctx, BLAMM_ERR_ARG, "invalid motif bank arguments");
    if (ncols >= (1 << kColBits)) return fail(ctx, BLAMM_ERR_ARG, "too many motif columns");
    int lmax = 0;
    for (int c = 0; c < ncols; ++c) {
        if (col_len[c] <= 0 || 4 * col_len[c] > p_rows)
            return fail(ctx, BLAMM_ERR_ARG, "column %d: length %d does not fit %d rows", c, col_len[c],
                        p_rows);
        if (col_len[c] > kMaxMotifLen)
            return fail(ctx, BLAMM_ERR_UNSUPPORTED, "column %d: length %d > %d", c, col_len[c], kMaxMotifLen);
        lmax = std::max(lmax, (int)col_len[c]);
    }
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->stream));  // (what is enqueued may still read the old bank)
    ctx->ncols = ncols;
    ctx->p_rows = p_rows;
    ctx->lmax = lmax;
    ctx->P.assign(P, P + (size_t)p_rows * ncols);
    ctx->len.assign(col_len, col_len + ncols);
    ctx->thr.assign(thr, thr + ncols);
    ctx->active.clear();
    ctx->colq_valid = false;
    if (ctx->d_P) cudaFree(ctx->d_P);
    if (ctx->d_len) cudaFree(ctx->d_len);
    if (ctx->d_thr) cudaFree(ctx->d_thr);
    ctx->d_P = nullptr;
    ctx->d_len = nullptr;
    ctx->d_thr = nullptr;
    CK(cudaMalloc(&ctx->d_P, sizeof(float) * ctx->P.size()));
    CK(cudaMalloc(&ctx->d_len, sizeof(int32_t) * ncols));
    CK(cudaMalloc(&ctx->d_thr, sizeof(float) * ncols));
    // On the context's stream, ahead of the plan and scan kernels that read these: a plain
    // cudaMemcpy from pageable memory may return before the data is on the device, and nothing
    // orders this non-blocking stream behind it.  (The sources stay until the stream is waited for.)
    CK(cudaMemcpyAsync(ctx->d_P, ctx->P.data(), sizeof(float) * ctx->P.size(), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->d_len, ctx->len.data(), sizeof(int32_t) * ncols, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(ctx->d_thr, ctx->thr.data(), sizeof(float) * ncols, cudaMemcpyHostToDevice, ctx->stream));
    ctx->plan_valid = false;
    return BLAMM_OK;
}

int blamm_set_columns(blamm_ctx *ctx, const int32_t *cols, int n)
{
    if (!ctx || n < 0 || (n > 0 && !cols)) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "no motif bank");
    if (n > ctx->ncols) return fail(ctx, BLAMM_ERR_ARG, "%d columns > bank size %d", n, ctx->ncols);
    std::vector<int32_t> act;
    if (n > 0) {
        std::vector<char> seen(ctx->ncols, 0);
        act.reserve(n);
        for (int i = 0; i < n; ++i) {
            const int c = cols[i];
            if (c < 0 || c >= ctx->ncols) return fail(ctx, BLAMM_ERR_ARG, "column %d is not in the bank", c);
            if (seen[c]) return fail(ctx, BLAMM_ERR_ARG, "column %d is listed twice", c);
            seen[c] = 1;
            act.push_back(c);
        }
    }
    CK(cudaSetDevice(ctx->device));
    ctx->active.swap(act);
    if (!ctx->active.empty()) {
        int rc = ensure(ctx, &ctx->d_active, &ctx->cap_active, ctx->active.size());
        if (rc) return rc;
        CK(cudaMemcpyAsync(ctx->d_active, ctx->active.data(), sizeof(int32_t) * ctx->active.size(),
                           cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    ctx->plan_valid = false;
    return BLAMM_OK;
}

int blamm_set_thresholds(blamm_ctx *ctx, const float *thr)
{
    if (!ctx || !thr) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "no motif bank");
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->stream));  // (an earlier upload may still read the host copy)
    ctx->thr.assign(thr, thr + ctx->ncols);
    CK(cudaMemcpyAsync(ctx->d_thr, ctx->thr.data(), sizeof(float) * ctx->ncols, cudaMemcpyHostToDevice, ctx->stream));
    ctx->plan_valid = false;
    return BLAMM_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ drivers
// BF16 terms of the tensor-core modes
static int mode_terms(const blamm_ctx *ctx)
{
    return ctx->mode == BLAMM_MODE_BF16X2 ? 2
           : ctx->mode == BLAMM_MODE_E4M3  ? kE4M3
           : ctx->mode == BLAMM_MODE_AUTO  ? ctx->auto_terms
                                           : 1;
}

static int ensure_plan(blamm_ctx *ctx)
{
    const int terms = mode_terms(ctx);
    if (ctx->plan_valid && ctx->plan_terms == terms) return BLAMM_OK;
    return build_plan(ctx, terms);
}

// The tensor-core scan runs over windows of at most ctx->ewindow positions (16 Mi by
// default): per window its packed bases and one-hot entries (prep_kernel, 16 B per entry) and
// one scan launch, so the entry array holds one window (256 MB) whatever the stream
// length.  A window's scan copies up to entry (its positions rounded up to 256) + 4 * 64 (BF16)
// or + 8 * 8 (E4M3): positions + kStreamPad - 64 entries hold that.
static int64_t e16_entries(const blamm_ctx *ctx, int64_t n) { return std::min(n, ctx->ewindow) + kStreamPad - 64; }

// One launch of prep_kernel: form 0 (packing only), 1 (BF16 entries) or kE4M3.
static cudaError_t launch_prep(const PrepParams &a, int form, cudaStream_t st)
{
    const int64_t span = std::max(a.pack_end - a.base, form ? a.ne : 0);
    const unsigned grid = (unsigned)((span + kPrepTile - 1) / kPrepTile);
    if (form == 0) prep_kernel<0><<<grid, kPrepThreads, 0, st>>>(a);
    else if (form == kE4M3) prep_kernel<8><<<grid, kPrepThreads, 0, st>>>(a);
    else prep_kernel<1><<<grid, kPrepThreads, 0, st>>>(a);
    return cudaGetLastError();
}

// Parameters of the preparation of n bases: counts[i] is set to zero where bit i of zero is set.
static PrepParams prep_params(const blamm_ctx *ctx, const char *d_bases, int64_t n, uint32_t *seq2, uint32_t *zmask,
                              unsigned long long *counts, uint32_t zero)
{
    PrepParams a{};
    a.bases = d_bases;
    a.n = n;
    a.pack_end = (n + kStreamPad + 31) / 32 * 32;
    a.seq2 = seq2;
    a.zmask = zmask;
    a.lower_scores = ctx->lower_scores;
    a.counts = counts;
    a.zero = zero;
    return a;
}

// Buffers of the packed stream (and one window's entries) for n positions.
static int ensure_packed(blamm_ctx *ctx, int64_t n, bool entries)
{
    const int64_t nwords32 = (n + kStreamPad + 31) / 32;
    int rc = ensure(ctx, &ctx->d_seq2, &ctx->cap_words32, (size_t)(2 * nwords32));
    if (!rc) rc = ensure(ctx, &ctx->d_zmask, &ctx->cap_zmask, (size_t)nwords32);
    if (!rc && entries) rc = ensure(ctx, &ctx->d_e16, &ctx->cap_e16, (size_t)e16_entries(ctx, n));
    return rc;
}

// Pack n bases into the context's packed stream (no entries).
static int launch_pack(blamm_ctx *ctx, const char *d_bases, int64_t n, unsigned long long *counts = nullptr,
                       uint32_t zero = 0)
{
    if (int rc = ensure_packed(ctx, n, false)) return rc;
    CK(launch_prep(prep_params(ctx, d_bases, n, ctx->d_seq2, ctx->d_zmask, counts, zero), 0, ctx->stream));
    return BLAMM_OK;
}

// Kernel parameters of the current plan over a packed stream of n positions
// (the caller adds candidates, counters, status and the test hooks).
static TcParams tc_params(const blamm_ctx *ctx, int64_t n)
{
    TcParams p{};
    p.n = n;
    p.tiles = ctx->d_tiles;
    p.ntiles = (int32_t)ctx->ntiles;
    p.terms = ctx->plan_terms;
    p.abuf = ctx->d_abuf;
    p.slot_col = ctx->d_slot_col;
    p.slot_thr = ctx->d_slot_thr;
    p.erows = ctx->erows;
    p.wait_limit = ctx->wait_limit;
    p.dump_ncols = ctx->ncols;
    return p;
}

static int64_t scan_blocks(int64_t n) { return (n + kBlockPos - 1) / kBlockPos; }

// The scan kernel counts jobs and record slots in 32 bits.
constexpr int64_t kMaxJobs = 0x7fffffff;
constexpr int64_t kMaxRecordSlots = (int64_t(1) << 31) - 1024;

static int check_jobs(blamm_ctx *ctx, int64_t n)
{
    const long long njobs = (long long)ctx->ntiles * scan_blocks(n);
    return njobs > kMaxJobs ? fail(ctx, BLAMM_ERR_UNSUPPORTED,
                                   "%lld scan jobs (tiles x 256-position blocks) exceed one launch's %lld; "
                                   "scan the stream in parts", njobs, (long long)kMaxJobs)
                            : BLAMM_OK;
}

// Record slots a scan with this grid reserves beyond its records: every drain warp holds
// one block it fills and one reserved ahead.
static int64_t record_slots_reserved(int grid) { return (int64_t)grid * kEpiWarps * 2 * kRecBlock; }

// Record slots for a first scan of n positions (about one candidate per 1000 position x
// column pairs, the thresholds' p-values being small) on a full grid.
static int64_t record_slots_guess(const blamm_ctx *ctx, int64_t n, double per = 1000.0)
{
    const double est = (double)n * scanned_columns(ctx) / per + (double)record_slots_reserved(ctx->sm_count);
    return (int64_t)std::min(std::max(est, (double)(1 << 20)), 512.0 * 1024 * 1024);
}

// Rescoring of the candidate records of one scan: the context's bank and chunk filter.
static RescoreParams rescore_params(const blamm_ctx *ctx, const uint4 *cand, const unsigned long long *cand_count,
                                    int64_t cand_cap, const uint32_t *seq2,
                                    const uint32_t *zmask, int64_t n, const int64_t *d_runs, int64_t nruns,
                                    blamm_hit *d_hits, unsigned long long *hit_count, int64_t hit_cap,
                                    unsigned long long *ncand)
{
    RescoreParams r{};
    r.ncand = ncand;
    r.cand = cand;
    r.slot_col = ctx->d_slot_col;
    r.cand_count = cand_count;
    r.cand_cap = cand_cap;
    r.seq2 = seq2;
    r.zmask = zmask;
    r.n = n;
    r.run_start = d_runs;
    r.nruns = nruns;
    r.P = ctx->d_P;
    r.p_rows = ctx->p_rows;
    r.col_len = ctx->d_len;
    r.thr = ctx->d_thr;
    r.hits = d_hits;
    r.hit_count = hit_count;
    r.hit_cap = hit_cap;
    r.keep_below = ctx->keep_below;
    r.pos_base = ctx->pos_base;
    return r;
}

// One launch of the scan kernel instance that p asks for.
template <bool kDump, bool kProf, bool kStream, bool kCount>
static void launch_tc_as(const TcParams &p, int grid, uint32_t smem, cudaStream_t st)
{
    auto go = [&](auto *kernel) {
        if (kDump || kProf)
            cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kernel<<<grid, kTcThreads, smem, st>>>(p);
    };
    if (p.terms == 2) go(scan_tc_kernel<kDump, kProf, 2, kStream, kCount>);
    else if (!kStream && p.terms == kE4M3) go(scan_tc_kernel<kDump, kProf, kE4M3, false, kCount>);
    else go(scan_tc_kernel<kDump, kProf, 1, kStream, kCount>);
}

template <bool kStream>
static void launch_tc(const TcParams &p, bool dump, int grid, uint32_t smem, cudaStream_t st)
{
    if (dump) launch_tc_as<true, false, kStream, false>(p, grid, smem, st);
    else if (p.prof) launch_tc_as<false, true, kStream, false>(p, grid, smem, st);
    else if (p.ncand) launch_tc_as<false, false, kStream, true>(p, grid, smem, st);
    else launch_tc_as<false, false, kStream, false>(p, grid, smem, st);
}

// The scan of n bases (p: the plan, candidates, counters, status; a: the packed stream and what
// the first window sets to zero), window by window: the window's packing and one-hot entries
// (into e16), then its scan launch.  Returns the largest grid used; adds the launches to
// *launches.
static int launch_tc_windows(blamm_ctx *ctx, TcParams p, PrepParams a, uint4 *e16, bool dump, int *launches, int *grid_out)
{
    const int64_t n = a.n, pack_end = a.pack_end;
    const int64_t nblocks = scan_blocks(n), wb = std::max<int64_t>(1, ctx->ewindow / kBlockPos);
    int gmax = 0;
    for (int64_t b0 = 0; b0 < nblocks; b0 += wb) {
        const int64_t nb = std::min(wb, nblocks - b0), base = b0 * kBlockPos;
        a.base = base;
        a.pack_end = b0 + nb < nblocks ? base + nb * kBlockPos : pack_end;
        a.e = e16;
        a.ne = std::min(nb * kBlockPos, n - base) + kStreamPad - 64;
        a.first = b0 == 0 ? 1 : 0;
        CK(launch_prep(a, p.terms == kE4M3 ? kE4M3 : 1, ctx->stream));
        a.zero = 0;
        p.e16 = e16;
        p.nblocks = (int32_t)nb;
        p.chunk0 = (uint32_t)(base / 32);
        // Tiles per group: the plan's, or fewer where a CTA would get less than about 8 units
        // (units differ by one between CTAs); blocks fewer than CTAs go out in ranges.
        const int64_t per_cta = (int64_t)ctx->ntiles * nb / ctx->sm_count;
        const int tg = ctx->plan_stream ? 1 : (int)std::max<int64_t>(1, std::min<int64_t>(ctx->plan_tg, per_cta / 8));
        const int ng = (ctx->ntiles + tg - 1) / tg;
        p.tg = (ctx->ntiles + ng - 1) / ng;
        const int grid = (int)std::min<int64_t>(ctx->sm_count, (int64_t)ng * nb);
        p.contiguous = nb < grid ? 1 : 0;
        // Two BF16 terms, a few tiles a unit, the longest of them (2 g MMAs of 128 cycles) longer than
        // the hand-off of an accumulator (about 1200 cycles): every other unit takes its tiles in
        // reverse.  Taken in one order, the short tiles follow one another on the same accumulator
        // and a unit's last job is too short to hide the hand-off of the long one before it.  30 Mbp,
        // scan kernel, ms: 130 columns of 5-30 positions 1.26 -> 1.20, 140 of 8-30 1.37 -> 1.21, 300
        // 1.89 -> 1.67; no gain from six tiles on (1024 columns: 1.157, 1.155 at 8 Mbp), a loss with
        // short motifs (130 of 8-14, 8 Mbp: 0.180, 0.207) and with one term or E4M3 (0.67, 0.82).
        p.turn = p.terms == 2 && p.tg >= 2 && p.tg <= 5 && ctx->tiles[0].g >= 6 ? 1 : 0;
        // (the longest tiles come first: the first group is the largest)
        const int steps = ctx->tiles[std::min(p.tg, ctx->ntiles)].off;
        p.a_bytes = (uint32_t)(ctx->plan_stream ? kChunks * kChunkBlocks : steps) * kStepBytes;
        // at least ~116 KB so that two CTAs never share an SM (each allocates all of TMEM)
        const uint32_t smem = std::max<uint32_t>(tc_smem_layout(p.a_bytes, p.erows).total, 116 * 1024);
        if ((int)smem > ctx->max_smem)
            return fail(ctx, BLAMM_ERR_UNSUPPORTED, "shared memory plan %u > %d", smem, ctx->max_smem);
        if (ctx->plan_stream) launch_tc<true>(p, dump, grid, smem, ctx->stream);
        else launch_tc<false>(p, dump, grid, smem, ctx->stream);
        CK(cudaGetLastError());
        gmax = std::max(gmax, grid);
        if (launches) *launches += 2;
    }
    if (grid_out) *grid_out = gmax;
    return BLAMM_OK;
}

// The plain FP32 scan of n positions of the packed stream (seq2/zmask) on the context's
// stream: parameters of the current bank and columns, hits appended through hit_count.
static PlainParams plain_params(const blamm_ctx *ctx, const uint32_t *seq2, const uint32_t *zmask, int64_t n,
                                const int64_t *d_runs, int64_t nruns, blamm_hit *d_hits, int64_t hit_cap,
                                unsigned long long *hit_count)
{
    PlainParams p{};
    p.seq2 = seq2;
    p.zmask = zmask;
    p.n = n;
    p.run_start = d_runs;
    p.nruns = nruns;
    p.P = ctx->d_P;
    p.p_rows = ctx->p_rows;
    p.ncols = scanned_columns(ctx);
    p.lmax = ctx->lmax;
    p.col_len = ctx->d_len;
    p.thr = ctx->d_thr;
    p.cols = ctx->active.empty() ? nullptr : ctx->d_active;
    p.hits = d_hits;
    p.hit_count = hit_count;
    p.hit_cap = hit_cap;
    p.keep_below = ctx->keep_below;
    p.pos_base = ctx->pos_base;
    return p;
}

// Launch it: a block's columns staged in shared memory, as many (at most 64) as leave room for
// four blocks on an SM; about four rounds of blocks, each walking over its share of the
// position tiles, so that the staging is paid rarely.
template <bool kHist>
static int launch_plain(blamm_ctx *ctx, PlainParams &p)
{
    const int bins = kHist && p.shared_bins ? p.nbins : 0;
    int cpb = std::min(64, (p.ncols + 3) / 4 * 4);
    while (cpb > 4 && plain_smem_bytes(cpb, p.lmax, bins) > (size_t)ctx->max_smem / 4) cpb -= 4;
    p.cols_per_block = cpb;
    const size_t smem = plain_smem_bytes(cpb, p.lmax, bins);
    const int64_t tiles = (p.n + kPlainThreads - 1) / kPlainThreads;
    const int by = (p.ncols + cpb - 1) / cpb;
    if (tiles > 0x7fffffff || by > 65535) return fail(ctx, BLAMM_ERR_UNSUPPORTED, "grid too large");
    if (tiles > 0) {
        const int64_t bx = std::min(tiles, std::max<int64_t>(1, (int64_t)ctx->sm_count * 16 / by));
        plain_scores_kernel<kHist><<<dim3((unsigned)bx, (unsigned)by), kPlainThreads, smem, ctx->stream>>>(p);
        CK(cudaGetLastError());
    }
    return BLAMM_OK;
}

// Rescoring behind the scan: the number of record slots is only known on the device, so the
// grid covers what the scan's warps reserve at least and the usual number of candidates.
static int launch_rescore(blamm_ctx *ctx, const RescoreParams &r, int64_t n, int scan_grid)
{
    const int64_t slots = (int64_t)((double)n * scanned_columns(ctx) / 1000.0) + record_slots_reserved(scan_grid);
    const int64_t blocks = std::min<int64_t>((slots + kRescoreThreads - 1) / kRescoreThreads, (int64_t)ctx->sm_count * 16);
    rescore_kernel<<<(unsigned)std::max<int64_t>(blocks, 1), kRescoreThreads, 0, ctx->stream>>>(r);
    CK(cudaGetLastError());
    return BLAMM_OK;
}

// A host scan's hits lie behind its counters in one buffer, so that the first of them come
// back in the same copy.
constexpr size_t kHitsAt = 64;
static_assert(kHitsAt % sizeof(blamm_hit) == 0 && kHitsAt >= (kCounts + kTimes) * sizeof(unsigned long long), "hits behind the counters");

// Raw accumulators of some positions (the raw-score hook).
struct ScanDump {
    float *out = nullptr;
    int64_t p0 = 0, npos = 0;
};

// One scan of device-resident bases, its counters back on the host: preparation, scan and
// rescoring are enqueued one behind the other and the host waits once (a candidate buffer that
// was too small grows and the scan runs again).
// fetch: bytes that come back behind the counters (to `back`, pinned: the counters, then these).
static int scan_core(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_runs, int64_t nruns,
                     blamm_hit *d_hits, int64_t hit_cap, int64_t *n_hits, const ScanDump &dump = ScanDump(),
                     unsigned long long *d_counters = nullptr, unsigned long long *back = nullptr, size_t fetch = 0)
{
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    const bool tc = ctx->mode != BLAMM_MODE_FP32;
    unsigned long long *cnt = d_counters ? d_counters : ctx->d_counters;  // record slots, hits, status, candidates; times
    ctx->stats = blamm_stats{};
    ctx->stats.positions = n;
    ctx->stats.columns = scanned_columns(ctx);
    int rc = BLAMM_OK;
    if (tc) {
        if ((rc = ensure_plan(ctx)) || (rc = check_jobs(ctx, n))) return rc;
        if (ctx->cand_cap == 0 && (rc = ensure_cand(ctx, record_slots_guess(ctx, n)))) return rc;
    }
    if ((rc = ensure_packed(ctx, n, tc))) return rc;
    unsigned long long got[kCounts + kTimes] = {0, 0, 0, 0, 0, 0, 0, 0};
    int launches = 0;
    for (int attempt = 0;; ++attempt) {
        launches = 0;
        CK(cudaEventRecord(ctx->ev[0], ctx->stream));
        if (tc) {
            TcParams p = tc_params(ctx, n);
            p.cand = ctx->d_cand;
            p.cand_count = cnt;
            p.cand_cap = ctx->cand_cap;
            p.status = reinterpret_cast<int *>(cnt + 2);
            p.debug_stall = ctx->debug_stall;
            p.dump = dump.out;
            p.dump_p0 = dump.p0;
            p.dump_npos = dump.npos;
            if (ctx->prof_on) {
                if (!ctx->d_prof) CK(cudaMalloc(&ctx->d_prof, sizeof(long long) * 32 * ctx->sm_count));
                CK(cudaMemsetAsync(ctx->d_prof, 0, sizeof(long long) * 32 * ctx->sm_count, ctx->stream));
                p.prof = ctx->d_prof;
            }
            int grid = 0;
            PrepParams a = prep_params(ctx, d_bases, n, ctx->d_seq2, ctx->d_zmask, cnt, 15u);
            a.times = p.times = cnt + kCounts;
            if ((rc = launch_tc_windows(ctx, p, a, ctx->d_e16, dump.out || ctx->debug_stall > kStallIssuers, &launches, &grid)))
                return rc;
            RescoreParams r = rescore_params(ctx, ctx->d_cand, cnt, ctx->cand_cap, ctx->d_seq2, ctx->d_zmask, n,
                                             d_runs, nruns, d_hits, cnt + 1, hit_cap, cnt + 3);
            r.times = p.times;
            if ((rc = launch_rescore(ctx, r, n, grid))) return rc;
            ctx->prof_ctas = ctx->prof_on ? grid : ctx->prof_ctas;
        } else {
            if ((rc = launch_pack(ctx, d_bases, n, cnt, 15u))) return rc;
            CK(cudaEventRecord(ctx->ev[2], ctx->stream));
            PlainParams p = plain_params(ctx, ctx->d_seq2, ctx->d_zmask, n, d_runs, nruns, d_hits, hit_cap, cnt + 1);
            if ((rc = launch_plain<false>(ctx, p))) return rc;
            ++launches;  // (packing)
        }
        ++launches;
        CK(cudaEventRecord(ctx->ev[1], ctx->stream));
        CK(cudaMemcpyAsync(back ? back : got, cnt, back ? kHitsAt + fetch : sizeof got, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        if (back) std::memcpy(got, back, sizeof got);
        if ((int)got[2]) return fail(ctx, BLAMM_ERR_TIMEOUT, "scan kernel: a device wait timed out");
        ctx->rec_slots = (int64_t)got[0];
        if (!tc || (int64_t)got[0] <= ctx->cand_cap) break;
        if ((int64_t)got[0] >= kMaxRecordSlots)
            return fail(ctx, BLAMM_ERR_OVERFLOW, "%llu candidate records exceed one launch's %lld", got[0],
                        (long long)kMaxRecordSlots);
        if (attempt == 2) return fail(ctx, BLAMM_ERR_OVERFLOW, "candidate buffer overflow");
        rc = ensure_cand(ctx, std::min<int64_t>((int64_t)(got[0] + got[0] / 4 + 1024), kMaxRecordSlots));
        if (rc) return rc;
    }
    if (tc && ctx->prof_on) {
        ctx->prof.resize((size_t)32 * ctx->prof_ctas);
        CK(cudaMemcpy(ctx->prof.data(), ctx->d_prof, sizeof(long long) * 32 * ctx->prof_ctas, cudaMemcpyDeviceToHost));
    }
    const int64_t nh = (int64_t)got[1];
    if (tc) ctx->stats.candidates = (int64_t)got[3];
    cudaEventElapsedTime(&ctx->stats.kernel_ms, ctx->ev[0], ctx->ev[1]);
    if (tc) {
        // the kernels' own clock: preparation begins, scan kernels together, -, rescoring begins
        const unsigned long long *t = got + kCounts;
        ctx->stats.scan_ms = 1e-6f * (float)t[1];
        ctx->stats.rescore_ms = std::max(0.f, ctx->stats.kernel_ms - 1e-6f * (float)(t[3] - t[0]));
    } else {
        cudaEventElapsedTime(&ctx->stats.scan_ms, ctx->ev[2], ctx->ev[1]);
    }
    ctx->stats.hits = nh;
    ctx->stats.tiles = (int32_t)(tc ? ctx->ntiles : 0);
    ctx->stats.launches = launches;
    *n_hits = nh;
    return nh > hit_cap ? fail(ctx, BLAMM_ERR_OVERFLOW, "%lld hits > capacity %lld", (long long)nh, (long long)hit_cap)
                        : BLAMM_OK;
}

extern "C" {

int blamm_scan_device(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_run_start,
                      int64_t nruns, blamm_hit *d_hits, int64_t hit_cap, int64_t *n_hits)
{
    const NvtxRange nvtx_range("blamm_scan_device");
    if (!ctx || !n_hits || n < 0 || hit_cap < 0) return BLAMM_ERR_ARG;
    *n_hits = 0;
    if (n == 0) return BLAMM_OK;
    if (!d_bases || !d_run_start || nruns <= 0 || (hit_cap > 0 && !d_hits))
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    return scan_core(ctx, d_bases, n, d_run_start, nruns, d_hits, hit_cap, n_hits);
}

// blamm_scan on a long stream: chunks of kPipeChunk positions (plus the longest motif - 1
// bases of overlap, whose window starts belong to the next chunk), each chunk's bases
// copied in on a second stream while the previous chunk is scanned, and its hits copied
// out there while the next one is scanned.
constexpr int64_t kPipeChunk = int64_t(16) << 20;

static int scan_host_pipelined_steps(blamm_ctx *ctx, const char *bases, int64_t n, const int64_t *run_start,
                                     int64_t nruns, blamm_hit *hits, int64_t hit_cap, int64_t *n_hits)
{
    const int64_t ov = std::max(ctx->lmax - 1, 0);
    const int64_t nchunks = (n + kPipeChunk - 1) / kPipeChunk;
    int rc = BLAMM_OK;
    for (int b = 0; b < 2; ++b) {
        if ((rc = ensure(ctx, &ctx->d_chunk_bases[b], &ctx->cap_chunk_bases[b], (size_t)(kPipeChunk + ov))))
            return rc;
        if ((rc = ensure(ctx, &ctx->d_chunk_runs[b], &ctx->cap_chunk_runs[b], (size_t)nruns + 1))) return rc;
    }
    size_t hc = (size_t)ctx->hits_cap;
    if ((rc = ensure(ctx, &ctx->d_hits, &hc, (size_t)std::max<int64_t>(hit_cap, 1)))) return rc;
    ctx->hits_cap = (int64_t)hc;
    if (!ctx->copy_stream) {
        CK(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
        for (auto &ev : ctx->chunk_ev) CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    }
    CK(cudaStreamSynchronize(ctx->stream));  // the buffers exist before the copy stream uses them
    if (ctx->cap_h_chunk_runs < (size_t)nruns + 1) {
        for (auto &h : ctx->h_chunk_runs) {
            if (h) CK(cudaFreeHost(h));
            h = nullptr;
        }
        ctx->cap_h_chunk_runs = 0;
        for (auto &h : ctx->h_chunk_runs) CK(cudaHostAlloc((void **)&h, sizeof(int64_t) * ((size_t)nruns + 1), 0));
        ctx->cap_h_chunk_runs = (size_t)nruns + 1;
    }
    int64_t kruns[2] = {0, 0};  // per buffer: run starts of its chunk (in h_chunk_runs)
    auto issue_in = [&](int64_t k) -> int {
        const int b = (int)(k & 1);
        const int64_t c0 = k * kPipeChunk, end = std::min(n, c0 + kPipeChunk + ov);
        int64_t *hr = ctx->h_chunk_runs[b];  // its previous copy (chunk k - 2) has landed
        int64_t m = 0;
        hr[m++] = 0;  // c0 lies inside some run
        for (const int64_t *r = std::upper_bound(run_start, run_start + nruns, c0); r < run_start + nruns && *r < end;
             ++r)
            hr[m++] = *r - c0;
        kruns[b] = m;
        CK(cudaMemcpyAsync(ctx->d_chunk_bases[b], bases + c0, (size_t)(end - c0), cudaMemcpyHostToDevice,
                           ctx->copy_stream));
        CK(cudaMemcpyAsync(ctx->d_chunk_runs[b], hr, sizeof(int64_t) * (size_t)m, cudaMemcpyHostToDevice,
                           ctx->copy_stream));
        CK(cudaEventRecord(ctx->chunk_ev[b], ctx->copy_stream));
        return BLAMM_OK;
    };
    blamm_stats total{};
    total.positions = n;
    int64_t nh_total = 0;
    if ((rc = issue_in(0))) return rc;
    for (int64_t k = 0; k < nchunks; ++k) {
        const int b = (int)(k & 1);
        // the next chunk's input buffer served chunk k - 1, whose scan has returned
        if (k + 1 < nchunks && (rc = issue_in(k + 1))) return rc;
        CK(cudaStreamWaitEvent(ctx->stream, ctx->chunk_ev[b], 0));
        const int64_t c0 = k * kPipeChunk, c1 = std::min(n, c0 + kPipeChunk), end = std::min(n, c1 + ov);
        ctx->keep_below = end > c1 ? c1 - c0 : 0;
        ctx->pos_base = c0;
        const int64_t at = std::min(nh_total, hit_cap), cap_k = hit_cap - at;
        int64_t nh = 0;
        rc = scan_core(ctx, ctx->d_chunk_bases[b], end - c0, ctx->d_chunk_runs[b], kruns[b], ctx->d_hits + at,
                       cap_k, &nh);
        if (rc && rc != BLAMM_ERR_OVERFLOW) return rc;
        // scan_core returned after its stream drained: copy this chunk's hits out beside the next scan
        const int64_t ncopy = std::min(nh, cap_k);
        if (ncopy > 0)
            CK(cudaMemcpyAsync(hits + at, ctx->d_hits + at, sizeof(blamm_hit) * ncopy, cudaMemcpyDeviceToHost,
                               ctx->copy_stream));
        nh_total += nh;
        total.columns = ctx->stats.columns;
        total.candidates += ctx->stats.candidates;
        total.tiles = ctx->stats.tiles;
        total.launches += ctx->stats.launches;
        total.kernel_ms += ctx->stats.kernel_ms;
        total.scan_ms += ctx->stats.scan_ms;
        total.rescore_ms += ctx->stats.rescore_ms;
    }
    CK(cudaStreamSynchronize(ctx->copy_stream));  // the hits are in host memory
    total.hits = nh_total;
    ctx->stats = total;
    *n_hits = nh_total;
    return nh_total > hit_cap
               ? fail(ctx, BLAMM_ERR_OVERFLOW, "%lld hits > capacity %lld", (long long)nh_total, (long long)hit_cap)
               : BLAMM_OK;
}

// One chunk's kernels, enqueued without host synchronisation (the blamm_scan_enqueue
// sequence): candidates beyond the candidate buffer are only counted, and the rescoring
// reads their number on the device.
static int enqueue_chunk(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_runs, int64_t nruns,
                         blamm_hit *d_hits, int64_t hit_cap)
{
    unsigned long long *cnt = ctx->d_counters;  // [0] record slots and [3] candidates of this chunk, [1] hits of the call
    if (ctx->mode == BLAMM_MODE_FP32) {
        if (int rc = launch_pack(ctx, d_bases, n)) return rc;
        PlainParams p = plain_params(ctx, ctx->d_seq2, ctx->d_zmask, n, d_runs, nruns, d_hits, hit_cap, cnt + 1);
        return launch_plain<false>(ctx, p);
    }
    int rc = check_jobs(ctx, n);
    if (rc) return rc;
    TcParams p = tc_params(ctx, n);
    p.cand = ctx->d_cand;
    p.cand_count = cnt;
    p.cand_cap = ctx->cand_cap;
    p.status = reinterpret_cast<int *>(cnt + 2);
    int grid = 0;
    const PrepParams a = prep_params(ctx, d_bases, n, ctx->d_seq2, ctx->d_zmask, cnt, 9u);
    if ((rc = launch_tc_windows(ctx, p, a, ctx->d_e16, false, nullptr, &grid))) return rc;
    return launch_rescore(ctx, rescore_params(ctx, ctx->d_cand, cnt, ctx->cand_cap, ctx->d_seq2, ctx->d_zmask, n, d_runs,
                                              nruns, d_hits, cnt + 1, hit_cap, cnt + 3), n, grid);
}

// The copy pipeline without host synchronisation inside a chunk: the host only waits for
// chunk k - 1 to finish (while chunk k runs) to learn how many hits to copy out.  Returns
// BLAMM_ERR_OVERFLOW with *cand_overflow set when a chunk had more candidates than the
// candidate buffer holds (its hits are then incomplete: the caller rescans).
static int scan_host_async_steps(blamm_ctx *ctx, const char *bases, int64_t n, const int64_t *run_start,
                                 int64_t nruns, blamm_hit *hits, int64_t hit_cap, int64_t *n_hits,
                                 int64_t *cand_overflow)
{
    *cand_overflow = 0;
    const int64_t ov = std::max(ctx->lmax - 1, 0);
    const int64_t nchunks = (n + kPipeChunk - 1) / kPipeChunk;
    const int64_t span = kPipeChunk + ov;  // positions of the longest chunk
    const bool tc = ctx->mode != BLAMM_MODE_FP32;
    int rc = BLAMM_OK;
    for (int b = 0; b < 2; ++b) {
        if ((rc = ensure(ctx, &ctx->d_chunk_bases[b], &ctx->cap_chunk_bases[b], (size_t)span))) return rc;
        if ((rc = ensure(ctx, &ctx->d_chunk_runs[b], &ctx->cap_chunk_runs[b], (size_t)nruns + 1))) return rc;
    }
    if ((rc = ensure_packed(ctx, span, tc))) return rc;
    if (tc) {
        if ((rc = ensure_plan(ctx))) return rc;
        // candidates: four times the usual first guess for a chunk (a chunk that still
        // overflows sends the whole call to the synchronous path)
        const double want = (double)record_slots_guess(ctx, span, 250.0);
        if ((rc = ensure_cand(ctx, (int64_t)want))) return rc;
    }
    size_t hc = (size_t)ctx->hits_cap;
    if ((rc = ensure(ctx, &ctx->d_hits, &hc, (size_t)std::max<int64_t>(hit_cap, 1)))) return rc;
    ctx->hits_cap = (int64_t)hc;
    if (!ctx->copy_stream) {
        CK(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
        for (auto &ev : ctx->chunk_ev) CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    }
    if (!ctx->done_ev[0])
        for (auto &ev : ctx->done_ev) CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    if (ctx->cap_h_chunk_runs < (size_t)nruns + 1) {
        for (auto &h : ctx->h_chunk_runs) {
            if (h) CK(cudaFreeHost(h));
            h = nullptr;
        }
        ctx->cap_h_chunk_runs = 0;
        for (auto &h : ctx->h_chunk_runs) CK(cudaHostAlloc((void **)&h, sizeof(int64_t) * ((size_t)nruns + 1), 0));
        ctx->cap_h_chunk_runs = (size_t)nruns + 1;
    }
    if (ctx->cap_h_chunk_counts < (size_t)(4 * nchunks)) {
        if (ctx->h_chunk_counts) CK(cudaFreeHost(ctx->h_chunk_counts));
        ctx->h_chunk_counts = nullptr;
        ctx->cap_h_chunk_counts = 0;
        CK(cudaHostAlloc((void **)&ctx->h_chunk_counts, sizeof(unsigned long long) * 4 * (size_t)nchunks, 0));
        ctx->cap_h_chunk_counts = (size_t)(4 * nchunks);
    }
    CK(cudaMemsetAsync(ctx->d_counters, 0, 4 * sizeof(unsigned long long), ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));  // the buffers exist before the copy stream uses them
    int64_t kruns[2] = {0, 0};
    auto issue_in = [&](int64_t k) -> int {
        const int b = (int)(k & 1);
        const int64_t c0 = k * kPipeChunk, end = std::min(n, c0 + kPipeChunk + ov);
        // the staging and device buffers served chunk k - 2: its run copy has landed, and the
        // copy stream waits for its kernels (packing reads the bases, the scans the runs)
        if (k >= 2) {
            CK(cudaEventSynchronize(ctx->chunk_ev[b]));
            CK(cudaStreamWaitEvent(ctx->copy_stream, ctx->done_ev[b], 0));
        }
        int64_t *hr = ctx->h_chunk_runs[b];
        int64_t m = 0;
        hr[m++] = 0;  // c0 lies inside some run
        for (const int64_t *r = std::upper_bound(run_start, run_start + nruns, c0); r < run_start + nruns && *r < end;
             ++r)
            hr[m++] = *r - c0;
        kruns[b] = m;
        CK(cudaMemcpyAsync(ctx->d_chunk_bases[b], bases + c0, (size_t)(end - c0), cudaMemcpyHostToDevice,
                           ctx->copy_stream));
        CK(cudaMemcpyAsync(ctx->d_chunk_runs[b], hr, sizeof(int64_t) * (size_t)m, cudaMemcpyHostToDevice,
                           ctx->copy_stream));
        CK(cudaEventRecord(ctx->chunk_ev[b], ctx->copy_stream));
        return BLAMM_OK;
    };
    unsigned long long *hc_k = ctx->h_chunk_counts;
    int64_t copied = 0;  // hits already sent to host memory
    // copy out the hits chunk k added, once it has finished (the host waits for that chunk)
    auto drain_out = [&](int64_t k) -> int {
        CK(cudaEventSynchronize(ctx->done_ev[k & 1]));
        const int64_t upto = std::min<int64_t>((int64_t)hc_k[4 * k + 1], hit_cap);
        if (upto > copied) {
            CK(cudaStreamWaitEvent(ctx->copy_stream, ctx->done_ev[k & 1], 0));
            CK(cudaMemcpyAsync(hits + copied, ctx->d_hits + copied, sizeof(blamm_hit) * (size_t)(upto - copied),
                               cudaMemcpyDeviceToHost, ctx->copy_stream));
            copied = upto;
        }
        return BLAMM_OK;
    };
    CK(cudaEventRecord(ctx->ev[0], ctx->stream));
    if ((rc = issue_in(0))) return rc;
    for (int64_t k = 0; k < nchunks; ++k) {
        const int b = (int)(k & 1);
        if (k + 1 < nchunks && (rc = issue_in(k + 1))) return rc;
        CK(cudaStreamWaitEvent(ctx->stream, ctx->chunk_ev[b], 0));
        const int64_t c0 = k * kPipeChunk, c1 = std::min(n, c0 + kPipeChunk), end = std::min(n, c1 + ov);
        ctx->keep_below = end > c1 ? c1 - c0 : 0;
        ctx->pos_base = c0;
        rc = enqueue_chunk(ctx, ctx->d_chunk_bases[b], end - c0, ctx->d_chunk_runs[b], kruns[b], ctx->d_hits,
                           hit_cap);
        ctx->keep_below = ctx->pos_base = 0;
        if (rc) return rc;
        // this chunk's record slots, the running hit count, its candidates and the status, to
        // host memory
        CK(cudaMemcpyAsync(hc_k + 4 * k, ctx->d_counters, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                           ctx->stream));
        CK(cudaEventRecord(ctx->done_ev[b], ctx->stream));
        if (k >= 1 && (rc = drain_out(k - 1))) return rc;
    }
    CK(cudaEventRecord(ctx->ev[1], ctx->stream));
    if ((rc = drain_out(nchunks - 1))) return rc;
    CK(cudaStreamSynchronize(ctx->copy_stream));  // the hits are in host memory
    blamm_stats total{};
    total.positions = n;
    total.columns = scanned_columns(ctx);
    total.tiles = (int32_t)(tc ? ctx->ntiles : 0);
    total.launches = 0;
    for (int64_t k = 0; k < nchunks; ++k) {  // preparation and scan (per window), rescoring
        const int64_t len = std::min(n, (k + 1) * kPipeChunk + ov) - k * kPipeChunk;
        total.launches += (int32_t)(tc ? 1 + 2 * ((len + ctx->ewindow - 1) / ctx->ewindow) : 2);
    }
    int status = 0;
    for (int64_t k = 0; k < nchunks; ++k) {
        const int64_t nc = (int64_t)hc_k[4 * k];
        if (tc) total.candidates += (int64_t)hc_k[4 * k + 3];
        if (tc && nc > ctx->cand_cap) *cand_overflow = std::max(*cand_overflow, nc);
        status |= (int)(hc_k[4 * k + 2] & 0xffffffffu);
    }
    cudaEventElapsedTime(&total.kernel_ms, ctx->ev[0], ctx->ev[1]);
    const int64_t nh_total = (int64_t)hc_k[4 * (nchunks - 1) + 1];
    total.hits = nh_total;
    ctx->stats = total;
    *n_hits = nh_total;
    if (status) return fail(ctx, BLAMM_ERR_TIMEOUT, "scan kernel: a device wait timed out");
    if (*cand_overflow) return BLAMM_ERR_OVERFLOW;
    return nh_total > hit_cap
               ? fail(ctx, BLAMM_ERR_OVERFLOW, "%lld hits > capacity %lld", (long long)nh_total, (long long)hit_cap)
               : BLAMM_OK;
}

// Whatever way the steps end, the chunk filter is reset and no copy into the caller's
// buffers is still in flight.  A chunk whose candidates overflowed the buffer sends the
// call to the synchronous chunked path, which grows the buffer and rescans.
static int scan_host_pipelined(blamm_ctx *ctx, const char *bases, int64_t n, const int64_t *run_start,
                               int64_t nruns, blamm_hit *hits, int64_t hit_cap, int64_t *n_hits)
{
    int64_t cand_overflow = 0;
    int rc = scan_host_async_steps(ctx, bases, n, run_start, nruns, hits, hit_cap, n_hits, &cand_overflow);
    ctx->keep_below = ctx->pos_base = 0;
    if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
    cudaStreamSynchronize(ctx->stream);
    if (rc == BLAMM_ERR_OVERFLOW && cand_overflow > 0) {
        rc = scan_host_pipelined_steps(ctx, bases, n, run_start, nruns, hits, hit_cap, n_hits);
        ctx->keep_below = ctx->pos_base = 0;
        if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
    }
    return rc;
}

// One scan with host run starts and hits, of host bases or (bases null) of device bases.  A
// short input travels through pinned staging in one copy, and the first hits come back with
// the counters: a short call is a copy, three kernels, a copy and one wait.
constexpr size_t kStageIn = size_t(256) << 10;
constexpr int64_t kStageHits = 16384;

static int scan_host_once(blamm_ctx *ctx, const char *bases, const char *d_bases, int64_t n, const int64_t *run_start,
                          int64_t nruns, blamm_hit *hits, int64_t hit_cap, int64_t *n_hits)
{
    const auto t0 = std::chrono::steady_clock::now();
    const size_t run_bytes = sizeof(int64_t) * (size_t)nruns, at = (run_bytes + 15) & ~size_t(15);
    const size_t in_bytes = at + (bases ? (size_t)n : 0);
    // hits that come back with the counters: about twice what p = 1e-4 gives
    const int64_t first = std::min<int64_t>(
        hit_cap, std::max<int64_t>(512, std::min<int64_t>(kStageHits, n * (int64_t)scanned_columns(ctx) / 5000)));
    const size_t back_at = in_bytes <= kStageIn ? (in_bytes + 63) & ~size_t(63) : 0;
    const size_t fetch = sizeof(blamm_hit) * (size_t)first;
    int rc = ensure_stage(ctx, std::max(back_at + kHitsAt + fetch, size_t(64) << 10));
    if (!rc) rc = ensure(ctx, &ctx->d_bases, &ctx->cap_bases, in_bytes);
    size_t hc = (size_t)ctx->hits_cap;
    if (!rc) rc = ensure(ctx, &ctx->d_hits, &hc, (size_t)hit_cap + kHitsAt / sizeof(blamm_hit));
    if (rc) return rc;
    ctx->hits_cap = (int64_t)hc;
    char *d_in = ctx->d_bases;
    if (in_bytes <= kStageIn) {
        std::memcpy(ctx->h_stage, run_start, run_bytes);
        if (bases) std::memcpy(ctx->h_stage + at, bases, (size_t)n);
        CK(cudaMemcpyAsync(d_in, ctx->h_stage, in_bytes, cudaMemcpyHostToDevice, ctx->stream));
    } else {
        CK(cudaMemcpyAsync(d_in, run_start, run_bytes, cudaMemcpyHostToDevice, ctx->stream));
        if (bases) CK(cudaMemcpyAsync(d_in + at, bases, (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    }
    blamm_hit *d_hits = ctx->d_hits + kHitsAt / sizeof(blamm_hit);
    rc = scan_core(ctx, bases ? d_in + at : d_bases, n, reinterpret_cast<const int64_t *>(d_in), nruns, d_hits, hit_cap,
                   n_hits, ScanDump(), reinterpret_cast<unsigned long long *>(ctx->d_hits),
                   reinterpret_cast<unsigned long long *>(ctx->h_stage + back_at), fetch);
    if (rc && rc != BLAMM_ERR_OVERFLOW) {
        // no copy out of the caller's buffers may be in flight when the call returns
        cudaStreamSynchronize(ctx->stream);
        return rc;
    }
    const int64_t ncopy = std::min<int64_t>(*n_hits, hit_cap);
    if (ncopy <= first) {
        if (ncopy > 0) std::memcpy(hits, ctx->h_stage + back_at + kHitsAt, sizeof(blamm_hit) * (size_t)ncopy);
    } else {
        // All of them in one copy: where the caller's pages are fresh, a copy behind a first part that
        // the CPU has written takes longer (6.5 M hits into a new array: the call 4.7 ms, 4.0 so).
        CK(cudaMemcpyAsync(hits, d_hits, sizeof(blamm_hit) * (size_t)ncopy, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
    }
    // (by the host's clock: a pair of events around the copies took 5 us of a 58 us call)
    ctx->stats.total_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return rc;
}

int blamm_scan(blamm_ctx *ctx, const char *bases, int64_t n, const int64_t *run_start, int64_t nruns,
               blamm_hit *hits, int64_t hit_cap, int64_t *n_hits)
{
    const NvtxRange nvtx_range("blamm_scan");
    if (!ctx || !n_hits || n < 0 || hit_cap < 0) return BLAMM_ERR_ARG;
    *n_hits = 0;
    if (n == 0) return BLAMM_OK;
    if (!bases || !run_start || nruns <= 0 || (hit_cap > 0 && !hits))
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    if (run_start[0] != 0) return fail(ctx, BLAMM_ERR_ARG, "run_start[0] must be 0");
    for (int64_t r = 1; r < nruns; ++r)
        if (run_start[r] <= run_start[r - 1] || run_start[r] >= n)
            return fail(ctx, BLAMM_ERR_ARG, "run_start must ascend strictly inside [0, n)");
    CK(cudaSetDevice(ctx->device));
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    if (n > 2 * kPipeChunk) {
        const auto t0 = std::chrono::steady_clock::now();
        const int rc = scan_host_pipelined(ctx, bases, n, run_start, nruns, hits, hit_cap, n_hits);
        ctx->stats.total_ms =
            std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
        return rc;
    }
    return scan_host_once(ctx, bases, nullptr, n, run_start, nruns, hits, hit_cap, n_hits);
}

int blamm_filter_score(blamm_ctx *ctx, float *d_R, int m, int n, const float *d_threshold, int *d_occIdx,
                       float *d_occScore, int *d_nOcc)
{
    if (!ctx || m < 0 || n < 0) return BLAMM_ERR_ARG;
    if ((long long)m * n == 0) return BLAMM_OK;
    if (!d_R || !d_threshold || !d_occIdx || !d_occScore || !d_nOcc)
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    const long long total = (long long)m * n;
    const int threads = 256;
    const long long blocks = std::min<long long>((total + threads - 1) / threads, (long long)ctx->sm_count * 32);
    filter_score_kernel<<<(unsigned)blocks, threads, 0, ctx->stream>>>(d_R, m, n, d_threshold, d_occIdx,
                                                                      d_occScore, d_nOcc);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(ctx->stream));
    return BLAMM_OK;
}

int blamm_device_count(int *n)
{
    if (!n) return BLAMM_ERR_ARG;
    *n = 0;
    int c = 0;
    if (cudaGetDeviceCount(&c) != cudaSuccess) {
        cudaGetLastError();
        return BLAMM_OK;
    }
    *n = c;
    return BLAMM_OK;
}

int blamm_device_memory(int device, int64_t *free_bytes, int64_t *total_bytes)
{
    if (!free_bytes || !total_bytes) return BLAMM_ERR_ARG;
    *free_bytes = *total_bytes = 0;
    int cur = 0;
    if (cudaGetDevice(&cur) != cudaSuccess) return BLAMM_ERR_CUDA;
    if (cudaSetDevice(device) != cudaSuccess) return BLAMM_ERR_CUDA;
    size_t f = 0, t = 0;
    const cudaError_t e = cudaMemGetInfo(&f, &t);
    cudaSetDevice(cur);
    if (e != cudaSuccess) return BLAMM_ERR_CUDA;
    *free_bytes = (int64_t)f;
    *total_bytes = (int64_t)t;
    return BLAMM_OK;
}

int blamm_set_softmask(blamm_ctx *ctx, int lowercase_scores)
{
    if (!ctx) return BLAMM_ERR_ARG;
    ctx->lower_scores = lowercase_scores ? 1 : 0;
    return BLAMM_OK;
}

// Whether the tensor-core form of the histograms takes this call, and its columns' constants.
// A tile costs it the same for one column as for 64, the plain form costs by the addition and
// by the bin (about five additions): 8 Mbp, lengths 6-20, ms: 16 columns 0.43 against 0.40,
// 32 columns 0.47 against 0.65, 64 columns 0.51 against 1.17: a tile is worth about 300
// additions a position.  And its set-up (A, rows, counts of every tile) has to be paid: the two
// meet where the additions saved reach about 90 M a tile for up to four tiles, which run side by
// side on a stream this short, and 180 M beyond (lengths 6-24, us, against the plain form: 64
// columns 79 against 72 at 64 kbp, 89 against 102 at 150 kbp; 200 columns 132 against 123 and
// 156 against 177; 800 columns 526 against 468 at 150 kbp; 4000 columns 4540 against 4416 at
// 100 kbp, 4184 against 4403 at 150 kbp).  And A, rows and counts have to fit in shared memory,
// values to be finite and of usual magnitude, and bins so wide that few scores lie too near a
// boundary to settle theirs.
static bool hist_tc_fits(const blamm_ctx *ctx, int64_t n, const float *min_score, const float *width, int nbins,
                         std::vector<float4> &scale)
{
    const int tiles = (ctx->ncols + kHistCols - 1) / kHistCols;
    int64_t adds = 0;
    for (int c = 0; c < ctx->ncols; ++c) adds += ctx->len[c] + 5;
    const double saved = (double)(adds - 300 * (int64_t)tiles) * (double)n;
    if (saved < (tiles > 4 ? 180e6 : 90e6) * tiles || n >= (int64_t(1) << 32)) return false;
    if (nbins > 1024 || ctx->lmax > 128 || hist_tc_layout(ctx->lmax, nbins).total > (uint32_t)ctx->max_smem) return false;
    scale.resize((size_t)ctx->ncols);
    for (int c = 0; c < ctx->ncols; ++c) {
        const float *P = &ctx->P[(size_t)c * ctx->p_rows];
        const int L = ctx->len[c];
        float top = 0.f;
        double sum = 0.0;
        for (int j = 0; j < L; ++j) {
            float m = 0.f;
            for (int b = 0; b < 4; ++b) m = std::max(m, std::isnan(P[4 * j + b]) ? INFINITY : std::fabs(P[4 * j + b]));
            top = std::max(top, m);
            sum += m;
        }
        const double w = width[c], mn = min_score[c];
        auto usual = [](double x) { return x > 0x1p-60 && x < 0x1p60; };  // (false for NaN)
        if (!usual(w) || !(std::fabs(mn) < 0x1p60) || !(top == 0.f || usual(top))) return false;
        const int k = top == 0.f ? 0 : 7 - column_exponent(P, L);
        if (std::ldexp((double)top, k) > 128.0) return false;  // (column_exponent stops at 2^40: hi would not be exact)
        // how far the scaled score can be off in bins: the terms' grid, the FP32 sum's own
        // rounding, the roundings of the factor, the offset and the bin's formula (generous)
        const double eps = (std::ldexp((double)L, -k - 9) + 0x1p-20 * (sum + std::fabs(mn))) / w + 0x1p-20 * nbins + L * 0x1p-24 * sum / w;
        // (the rounding to bins holds for |t| < 2^22)
        if (!(eps < 0.02) || !((sum + std::fabs(mn)) / w < 0x1p21)) return false;
        scale[c] = make_float4(std::ldexp(1.f, k), (float)(std::ldexp(1.0, -k) / w), (float)(-mn / w - 0.5), (float)(0.5 - eps));
    }
    return true;
}

// The empirical histograms of n bases already on the device (run starts on the host).
static int score_histograms_on(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *run_start,
                               int64_t nruns, const float *min_score, const float *width, int nbins,
                               uint64_t *counts)
{
    int rc = ensure(ctx, &ctx->d_runs, &ctx->cap_runs, (size_t)nruns);
    if (rc) return rc;
    CK(cudaMemcpyAsync(ctx->d_runs, run_start, sizeof(int64_t) * nruns, cudaMemcpyHostToDevice, ctx->stream));
    rc = launch_pack(ctx, d_bases, n);
    if (rc) return rc;
    const size_t nc = (size_t)ctx->ncols;
    std::vector<float4> scale;
    const bool tc = hist_tc_fits(ctx, n, min_score, width, nbins, scale);
    if ((size_t)(ctx->p_rows + nbins) * 4 + 256 + ctx->lmax + 64 > (size_t)ctx->max_smem)
        return fail(ctx, BLAMM_ERR_UNSUPPORTED, "too many bins for shared memory");
    // counts and status, columns' values: one workspace
    const size_t cbytes = sizeof(unsigned long long) * (nc * nbins + 1);
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    rc = ensure(ctx, &ctx->d_theo, &ctx->cap_theo, up(cbytes) + 2 * up(sizeof(float) * nc) + sizeof(float4) * nc);
    if (rc) return rc;
    unsigned long long *d_counts = reinterpret_cast<unsigned long long *>(ctx->d_theo);
    float *d_min = reinterpret_cast<float *>(ctx->d_theo + up(cbytes));
    float *d_w = reinterpret_cast<float *>(ctx->d_theo + up(cbytes) + up(sizeof(float) * nc));
    float4 *d_scale = reinterpret_cast<float4 *>(ctx->d_theo + up(cbytes) + 2 * up(sizeof(float) * nc));
    CK(cudaMemcpyAsync(d_min, min_score, sizeof(float) * nc, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_w, width, sizeof(float) * nc, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemsetAsync(d_counts, 0, cbytes, ctx->stream));
    if (tc) {
        CK(cudaMemcpyAsync(d_scale, scale.data(), sizeof(float4) * nc, cudaMemcpyHostToDevice, ctx->stream));
        HistTcParams p{};
        p.seq2 = ctx->d_seq2;
        p.zmask = ctx->d_zmask;
        p.n = n;
        p.run_start = ctx->d_runs;
        p.nruns = nruns;
        p.P = ctx->d_P;
        p.p_rows = ctx->p_rows;
        p.ncols = ctx->ncols;
        p.lmax = ctx->lmax;
        p.col_len = ctx->d_len;
        p.min_score = d_min;
        p.width = d_w;
        p.scale = d_scale;
        p.nbins = nbins;
        p.counts = d_counts;
        p.status = reinterpret_cast<int *>(d_counts + nc * nbins);
        p.wait_limit = ctx->wait_limit;
        const int tiles = (ctx->ncols + kHistCols - 1) / kHistCols;
        p.cols = (ctx->ncols + tiles - 1) / tiles;
        // (more than 116 KB, so that two blocks, which each allocate all of TMEM, never share an SM)
        const uint32_t smem = std::max<uint32_t>(hist_tc_layout(ctx->lmax, nbins).total, 116 * 1024);
        const int64_t blocks = (n + kHistBlock - 1) / kHistBlock;
        const int64_t per = std::max<int64_t>(1, (int64_t)ctx->sm_count * (tiles > 8 ? 4 : 1) / tiles);
        CK(cudaFuncSetAttribute(hist_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem));
        hist_tc_kernel<<<dim3((unsigned)std::min(blocks, per), (unsigned)tiles), kHistThreads, smem, ctx->stream>>>(p);
        CK(cudaGetLastError());
    } else {
        PlainParams p{};
        p.seq2 = ctx->d_seq2;
        p.zmask = ctx->d_zmask;
        p.n = n;
        p.run_start = ctx->d_runs;
        p.nruns = nruns;
        p.P = ctx->d_P;
        p.p_rows = ctx->p_rows;
        p.ncols = ctx->ncols;
        p.lmax = ctx->lmax;
        p.col_len = ctx->d_len;
        p.min_score = d_min;
        p.width = d_w;
        p.nbins = nbins;
        p.counts = d_counts;
        p.shared_bins = plain_smem_bytes(4, p.lmax, nbins) <= (size_t)ctx->max_smem ? 1 : 0;
        if ((rc = launch_plain<true>(ctx, p))) return rc;
    }
    std::vector<unsigned long long> host(nc * nbins + 1);
    CK(cudaMemcpyAsync(host.data(), d_counts, cbytes, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (host[nc * nbins]) return fail(ctx, BLAMM_ERR_TIMEOUT, "histogram kernel: a device wait timed out");
    for (size_t i = 0; i < nc * (size_t)nbins; ++i) counts[i] += host[i];
    return BLAMM_OK;
}

int blamm_score_histograms(blamm_ctx *ctx, const char *bases, int64_t n, const int64_t *run_start,
                           int64_t nruns, const float *min_score, const float *width, int nbins,
                           uint64_t *counts)
{
    const NvtxRange nvtx_range("blamm_score_histograms");
    if (!ctx || n < 0 || nbins <= 0 || !min_score || !width || !counts) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "no motif bank");
    if (n == 0) return BLAMM_OK;
    if (!bases || !run_start || nruns <= 0) return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    int rc = ensure(ctx, &ctx->d_bases, &ctx->cap_bases, (size_t)n);
    if (rc) return rc;
    CK(cudaMemcpyAsync(ctx->d_bases, bases, (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    return score_histograms_on(ctx, ctx->d_bases, n, run_start, nruns, min_score, width, nbins, counts);
}

int blamm_score_histograms_stream(blamm_ctx *ctx, int64_t begin, int64_t n, const int64_t *run_start,
                                  int64_t nruns, const float *min_score, const float *width, int nbins,
                                  uint64_t *counts)
{
    const NvtxRange nvtx_range("blamm_score_histograms_stream");
    if (!ctx || n < 0 || begin < 0 || nbins <= 0 || !min_score || !width || !counts) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "no motif bank");
    if (begin > ctx->stream_n || n > ctx->stream_n - begin)
        return fail(ctx, BLAMM_ERR_ARG, "positions [%lld, %lld) outside the resident stream of %lld bases",
                    (long long)begin, (long long)(begin + n), (long long)ctx->stream_n);
    if (n == 0) return BLAMM_OK;
    if (!run_start || nruns <= 0) return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    if (run_start[0] != 0) return fail(ctx, BLAMM_ERR_ARG, "run_start[0] must be 0");
    for (int64_t r = 1; r < nruns; ++r)
        if (run_start[r] <= run_start[r - 1] || run_start[r] >= n)
            return fail(ctx, BLAMM_ERR_ARG, "run_start must ascend strictly inside [0, n)");
    CK(cudaSetDevice(ctx->device));
    return score_histograms_on(ctx, ctx->d_stream + begin, n, run_start, nruns, min_score, width, nbins, counts);
}

int blamm_debug_stall(blamm_ctx *ctx, int enable, long long wait_limit_cycles)
{
    if (!ctx || wait_limit_cycles < 0) return BLAMM_ERR_ARG;
    const int role = enable & 255;
    ctx->debug_stall = enable > 0 && role > kStallIssuers && role < kStallEnd ? enable : enable ? kStallIssuers : 0;
    ctx->wait_limit = wait_limit_cycles > 0 ? wait_limit_cycles : 4000000000LL;
    return BLAMM_OK;
}

int blamm_debug_profile(blamm_ctx *ctx, int enable)
{
    if (!ctx) return BLAMM_ERR_ARG;
    ctx->prof_on = enable != 0;
    return BLAMM_OK;
}

int blamm_debug_profile_read(const blamm_ctx *ctx, int64_t *out, int max_ctas, int *nctas)
{
    if (!ctx || !nctas) return BLAMM_ERR_ARG;
    *nctas = ctx->prof_ctas;
    if (out)
        for (int i = 0; i < 32 * std::min(max_ctas, ctx->prof_ctas); ++i) out[i] = ctx->prof[(size_t)i];
    return BLAMM_OK;
}

int blamm_ctx_stream(const blamm_ctx *ctx, void **stream)
{
    if (!ctx || !stream) return BLAMM_ERR_ARG;
    *stream = (void *)ctx->stream;
    return BLAMM_OK;
}

int blamm_last_stats(const blamm_ctx *ctx, blamm_stats *out)
{
    if (!ctx || !out) return BLAMM_ERR_ARG;
    *out = ctx->stats;
    return BLAMM_OK;
}

int blamm_guard_band(const blamm_ctx *ctx, float *out)
{
    if (!ctx || !out) return BLAMM_ERR_ARG;
    blamm_ctx *c = const_cast<blamm_ctx *>(ctx);
    if (c->mode == BLAMM_MODE_FP32) {
        std::fill(out, out + c->ncols, 0.0f);
        return BLAMM_OK;
    }
    int rc = ensure_plan(c);
    if (rc) return rc;
    for (int i = 0; i < c->ncols; ++i) out[i] = 0.0f;  // (columns that are not scanned)
    for (int i = 0; i < scanned_columns(c); ++i) {
        const int col = c->active.empty() ? i : (int)c->active[i];
        out[col] = (float)c->colq_guard[col];
    }
    return BLAMM_OK;
}

int blamm_debug_scores(blamm_ctx *ctx, const char *bases, int64_t n, int64_t p0, int64_t npos, float *out)
{
    if (!ctx || !bases || !out || n <= 0 || p0 < 0 || npos <= 0 || p0 + npos > n) return BLAMM_ERR_ARG;
    if (ctx->mode == BLAMM_MODE_FP32) return fail(ctx, BLAMM_ERR_STATE, "debug scores need a tcgen05 mode");
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "no motif bank");
    CK(cudaSetDevice(ctx->device));
    int rc = ensure(ctx, &ctx->d_bases, &ctx->cap_bases, (size_t)n);
    if (rc) return rc;
    CK(cudaMemcpyAsync(ctx->d_bases, bases, (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
    int64_t runs0 = 0;
    rc = ensure(ctx, &ctx->d_runs, &ctx->cap_runs, 1);
    if (rc) return rc;
    CK(cudaMemcpyAsync(ctx->d_runs, &runs0, sizeof runs0, cudaMemcpyHostToDevice, ctx->stream));
    float *d_dump = nullptr;
    CK(cudaMalloc(&d_dump, sizeof(float) * (size_t)npos * ctx->ncols));
    CK(cudaMemsetAsync(d_dump, 0, sizeof(float) * (size_t)npos * ctx->ncols, ctx->stream));
    int64_t nh = 0;
    rc = scan_core(ctx, ctx->d_bases, n, ctx->d_runs, 1, nullptr, 0, &nh, ScanDump{d_dump, p0, npos});
    if (rc == BLAMM_ERR_OVERFLOW && nh > 0) rc = BLAMM_OK;  // (no room for hits was given)
    if (rc == BLAMM_OK) {
        cudaError_t e = cudaMemcpyAsync(out, d_dump, sizeof(float) * (size_t)npos * ctx->ncols,
                                        cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) rc = fail(ctx, BLAMM_ERR_CUDA, "%s", cudaGetErrorString(e));
        // the E4M3 form's accumulator is scaled by 2^k (exact: a power of two)
        for (int64_t i = 0; rc == BLAMM_OK && ctx->plan_terms == kE4M3 && i < npos; ++i)
            for (int c = 0; c < ctx->ncols; ++c) {
                float &v = out[i * ctx->ncols + c];
                v = (float)std::ldexp((double)v, -ctx->colq_k[c]);
            }
    }
    cudaFree(d_dump);
    return rc;
}

}  // extern "C"

// ------------------------------------------------------------------ allocation-free scan
//
// blamm_scan_device_static keeps every per-call buffer of a scan (the packed
// stream, the candidate list, the counters and the status word) in one
// file-scope __device__ array instead of the context's cudaMalloc'd buffers,
// so the call itself allocates no device or host memory.  The array is part of
// this library's device image: each device gets its own copy when the module
// is loaded there.  Its device address is looked up once per device with
// cudaGetSymbolAddress (the host-side name of a __device__ array is not a
// device address) with that device current.

namespace {

constexpr int64_t kStaticMaxBases = int64_t(4) << 20;  // positions per call
constexpr int64_t kStaticWords32 = (kStaticMaxBases + kStreamPad + 31) / 32;
constexpr int64_t kStaticCandCap = int64_t(2) << 20;   // tensor-core candidate record slots per call
constexpr size_t round256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kStaticSeq2Off = 0;
constexpr size_t kStaticZmaskOff = round256(kStaticSeq2Off + sizeof(uint32_t) * 2 * kStaticWords32);
constexpr size_t kStaticE16Off = round256(kStaticZmaskOff + sizeof(uint32_t) * kStaticWords32);
constexpr size_t kStaticCandOff = round256(kStaticE16Off + sizeof(uint4) * (kStaticMaxBases + kStreamPad));
constexpr size_t kStaticCountOff = round256(kStaticCandOff + sizeof(uint4) * (kStaticCandCap + kRecBlock));
constexpr size_t kStaticBytes = round256(kStaticCountOff + sizeof(unsigned long long) * 4);  // about 97 MiB

constexpr int kStaticMaxDevices = 64;

}  // namespace

static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

static std::mutex g_static_mu;
static unsigned char *g_static_ptr[kStaticMaxDevices] = {};

// Device address of this device's scratch copy; the first call on a device
// looks it up (the current device must be ctx->device).
static int static_scratch(blamm_ctx *ctx, unsigned char **out)
{
    if (ctx->device < 0 || ctx->device >= kStaticMaxDevices)
        return fail(ctx, BLAMM_ERR_UNSUPPORTED, "device %d: no static scratch slot", ctx->device);
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[ctx->device]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return fail(ctx, BLAMM_ERR_CUDA, "cudaGetSymbolAddress(static scratch): %s", cudaGetErrorString(e));
        g_static_ptr[ctx->device] = static_cast<unsigned char *>(p);
    }
    *out = g_static_ptr[ctx->device];
    return BLAMM_OK;
}

extern "C" {

int blamm_scan_device_static(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_run_start,
                             int64_t nruns, blamm_hit *d_hits, int64_t hit_cap, int64_t *n_hits)
{
    const NvtxRange nvtx_range("blamm_scan_device_static");
    if (!ctx || !n_hits || n < 0 || hit_cap < 0) return BLAMM_ERR_ARG;
    *n_hits = 0;
    if (n > kStaticMaxBases)
        return fail(ctx, BLAMM_ERR_ARG, "blamm_scan_device_static: %lld positions > the static limit %lld",
                    (long long)n, (long long)kStaticMaxBases);
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    const bool tc = ctx->mode != BLAMM_MODE_FP32;
    const int terms = mode_terms(ctx);
    if (tc && !(ctx->plan_valid && ctx->plan_terms == terms))
        return fail(ctx, BLAMM_ERR_STATE,
                    "blamm_scan_device_static: no tensor-core plan for this bank, mode and thresholds "
                    "(one blamm_scan or blamm_scan_device call builds it)");
    if (n == 0) return BLAMM_OK;
    if (!d_bases || !d_run_start || nruns <= 0 || (hit_cap > 0 && !d_hits))
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    unsigned char *base = nullptr;
    int rc = static_scratch(ctx, &base);
    if (rc) return rc;
    uint32_t *seq2 = reinterpret_cast<uint32_t *>(base + kStaticSeq2Off);
    uint32_t *zmask = reinterpret_cast<uint32_t *>(base + kStaticZmaskOff);
    uint4 *e16 = reinterpret_cast<uint4 *>(base + kStaticE16Off);
    uint4 *cand = reinterpret_cast<uint4 *>(base + kStaticCandOff);
    unsigned long long *counters = reinterpret_cast<unsigned long long *>(base + kStaticCountOff);

    ctx->stats = blamm_stats{};
    ctx->stats.positions = n;
    ctx->stats.columns = scanned_columns(ctx);
    int launches = 0;
    // (the preparation sets the counters and the status word to zero)
    const PrepParams a = prep_params(ctx, d_bases, n, seq2, zmask, counters, 15u);
    if (!tc) {
        CK(launch_prep(a, 0, ctx->stream));
        PlainParams p = plain_params(ctx, seq2, zmask, n, d_run_start, nruns, d_hits, hit_cap, counters + 1);
        if ((rc = launch_plain<false>(ctx, p))) return rc;
        launches = 2;
    } else {
        TcParams p = tc_params(ctx, n);
        p.cand = cand;
        p.cand_count = counters;
        p.cand_cap = kStaticCandCap;
        p.status = reinterpret_cast<int *>(counters + 2);
        int grid = 0;
        if ((rc = launch_tc_windows(ctx, p, a, e16, false, &launches, &grid))) return rc;
        const RescoreParams r = rescore_params(ctx, cand, counters, kStaticCandCap, seq2, zmask, n, d_run_start, nruns,
                                               d_hits, counters + 1, hit_cap, counters + 3);
        if ((rc = launch_rescore(ctx, r, n, grid))) return rc;
        ++launches;
    }
    unsigned long long cnt[4] = {0, 0, 0, 0};  // record slots, hits, status, candidates
    CK(cudaMemcpyAsync(cnt, counters, sizeof cnt, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if ((int)cnt[2]) return fail(ctx, BLAMM_ERR_TIMEOUT, "scan kernel: a device wait timed out");
    if (tc && (int64_t)cnt[0] > kStaticCandCap)
        return fail(ctx, BLAMM_ERR_OVERFLOW,
                    "blamm_scan_device_static: %llu candidate record slots > the static limit %lld (scan "
                    "fewer positions per call)", cnt[0], (long long)kStaticCandCap);
    const unsigned long long nh = cnt[1];
    if (tc) ctx->stats.candidates = (int64_t)cnt[3];
    ctx->stats.hits = (int64_t)nh;
    ctx->stats.tiles = (int32_t)(tc ? ctx->ntiles : 0);
    ctx->stats.launches = launches;
    *n_hits = (int64_t)nh;
    return (int64_t)nh > hit_cap ? fail(ctx, BLAMM_ERR_OVERFLOW, "%lld hits > capacity %lld", (long long)nh,
                                        (long long)hit_cap)
                                 : BLAMM_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ enqueued scans, graphs, autotuning

extern "C" {

int blamm_reserve(blamm_ctx *ctx, int64_t max_positions, int64_t max_candidates)
{
    const NvtxRange nvtx_range("blamm_reserve");
    if (!ctx || max_positions < 0 || max_candidates < 0) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    CK(cudaSetDevice(ctx->device));
    int rc = ensure_packed(ctx, max_positions, ctx->mode != BLAMM_MODE_FP32);
    if (rc) return rc;
    if (ctx->mode != BLAMM_MODE_FP32) {
        if ((rc = ensure_plan(ctx))) return rc;
        // record slots: at most one record per candidate, plus the blocks the warps reserve
        const int64_t slots = std::min(max_candidates + record_slots_reserved(ctx->sm_count), kMaxRecordSlots);
        if ((rc = ensure_cand(ctx, slots, spare_slots(ctx)))) return rc;
    }
    CK(cudaStreamSynchronize(ctx->stream));
    return BLAMM_OK;
}

int blamm_scan_enqueue(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_run_start, int64_t nruns,
                       blamm_hit *d_hits, int64_t hit_cap, uint64_t *d_counts)
{
    const NvtxRange nvtx_range("blamm_scan_enqueue");
    if (!ctx || !d_counts || n < 0 || hit_cap < 0) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    const int64_t nwords32 = (n + kStreamPad + 31) / 32;
    if ((size_t)(2 * nwords32) > ctx->cap_words32 || (size_t)nwords32 > ctx->cap_zmask)
        return fail(ctx, BLAMM_ERR_STATE, "blamm_scan_enqueue: %lld positions exceed the reservation",
                    (long long)n);
    const bool tc = ctx->mode != BLAMM_MODE_FP32;
    const int terms = mode_terms(ctx);
    if (tc && (!(ctx->plan_valid && ctx->plan_terms == terms) || ctx->cand_cap <= 0 ||
               (size_t)e16_entries(ctx, n) > ctx->cap_e16))
        return fail(ctx, BLAMM_ERR_STATE, "blamm_scan_enqueue: call blamm_reserve after changing the bank, "
                                          "columns, thresholds or mode");
    if (n > 0 && (!d_bases || !d_run_start || nruns <= 0 || (hit_cap > 0 && !d_hits)))
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    if (n == 0) {
        CK(cudaMemsetAsync(d_counts, 0, 4 * sizeof(uint64_t), ctx->stream));
        return BLAMM_OK;
    }
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(d_counts);
    const PrepParams a = prep_params(ctx, d_bases, n, ctx->d_seq2, ctx->d_zmask, cnt, 15u);
    if (!tc) {
        CK(launch_prep(a, 0, ctx->stream));
        PlainParams p = plain_params(ctx, ctx->d_seq2, ctx->d_zmask, n, d_run_start, nruns, d_hits, hit_cap, cnt + 1);
        return launch_plain<false>(ctx, p);
    }
    if (int rc = check_jobs(ctx, n)) return rc;
    TcParams p = tc_params(ctx, n);
    p.cand = ctx->d_cand;
    p.cand_count = cnt;
    p.cand_cap = ctx->cand_cap;
    p.ncand = ctx->cand_spare >= spare_slots(ctx) ? cnt + 3 : nullptr;  // (room that blamm_reserve makes)
    p.status = reinterpret_cast<int *>(cnt + 2);
    int grid = 0;
    if (int rc = launch_tc_windows(ctx, p, a, ctx->d_e16, false, nullptr, &grid)) return rc;
    return launch_rescore(ctx, rescore_params(ctx, ctx->d_cand, cnt, ctx->cand_cap, ctx->d_seq2, ctx->d_zmask, n,
                                              d_run_start, nruns, d_hits, cnt + 1, hit_cap, cnt + 3), n, grid);
}

int blamm_scan_graph_create(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_run_start,
                            int64_t nruns, blamm_hit *d_hits, int64_t hit_cap, uint64_t *d_counts, void **graph)
{
    if (!ctx || !graph) return BLAMM_ERR_ARG;
    *graph = nullptr;
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = blamm_scan_enqueue(ctx, d_bases, n, d_run_start, nruns, d_hits, hit_cap, d_counts);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) return fail(ctx, BLAMM_ERR_CUDA, "stream capture: %s", cudaGetErrorString(e));
    cudaGraphExec_t ge = nullptr;
    const cudaError_t e2 = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (e2 != cudaSuccess) return fail(ctx, BLAMM_ERR_CUDA, "graph instantiation: %s", cudaGetErrorString(e2));
    *graph = ge;
    return BLAMM_OK;
}

int blamm_scan_graph_launch(blamm_ctx *ctx, void *graph)
{
    const NvtxRange nvtx_range("blamm_scan_graph_launch");
    if (!ctx || !graph) return BLAMM_ERR_ARG;
    CK(cudaSetDevice(ctx->device));
    CK(cudaGraphLaunch(static_cast<cudaGraphExec_t>(graph), ctx->stream));
    return BLAMM_OK;
}

void blamm_scan_graph_destroy(void *graph)
{
    if (graph) cudaGraphExecDestroy(static_cast<cudaGraphExec_t>(graph));
}

int blamm_set_plan_options(blamm_ctx *ctx, int max_tile_columns, float job_cost)
{
    if (!ctx || max_tile_columns < 32 || max_tile_columns > 256 || !(job_cost >= 0.0f)) return BLAMM_ERR_ARG;
    ctx->plan_nmax = max_tile_columns;
    ctx->plan_job_cost = job_cost;
    ctx->plan_valid = false;
    return BLAMM_OK;
}

int blamm_get_terms(const blamm_ctx *ctx)
{
    if (!ctx) return 0;
    return ctx->mode == BLAMM_MODE_FP32 ? 0 : mode_terms(ctx);
}

int blamm_get_plan_options(const blamm_ctx *ctx, int *max_tile_columns, float *job_cost)
{
    if (!ctx || !max_tile_columns || !job_cost) return BLAMM_ERR_ARG;
    *max_tile_columns = ctx->plan_nmax;
    *job_cost = (float)ctx->plan_job_cost;
    return BLAMM_OK;
}

int blamm_autotune(blamm_ctx *ctx, const char *d_bases, int64_t n, const int64_t *d_run_start, int64_t nruns,
                   float *best_ms)
{
    const NvtxRange nvtx_range("blamm_autotune");
    if (!ctx || n < 0) return BLAMM_ERR_ARG;
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    if (best_ms) *best_ms = 0.0f;
    if (ctx->mode == BLAMM_MODE_FP32 || n == 0) return BLAMM_OK;
    if (!d_bases || !d_run_start || nruns <= 0) return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    // a sample of up to 16 Mi positions (the runs that start inside it)
    const int64_t ns = std::min<int64_t>(n, int64_t(16) << 20);
    std::vector<int64_t> runs((size_t)nruns);
    CK(cudaMemcpy(runs.data(), d_run_start, sizeof(int64_t) * nruns, cudaMemcpyDeviceToHost));
    const int64_t nrs = std::max<int64_t>(1, std::lower_bound(runs.begin(), runs.end(), ns) - runs.begin());
    size_t hc = (size_t)ctx->hits_cap;
    int rc = ensure(ctx, &ctx->d_hits, &hc, (size_t)1 << 20);
    if (rc) return rc;
    ctx->hits_cap = (int64_t)hc;
    const int keep_terms = ctx->auto_terms;
    // BLAMM_MODE_AUTO also chooses the form: one BF16 term halves the MMAs of two and
    // widens the guard band (more candidates to rescore), one E4M3 term (motifs up to 64
    // positions) halves them again with a still wider band, so the whole call's kernel
    // time (packing, scan, rescoring) decides
    int lmax_sel = 1;
    if (ctx->active.empty())
        for (int c = 0; c < ctx->ncols; ++c) lmax_sel = std::max(lmax_sel, ctx->len[c]);
    else
        for (const int c : ctx->active) lmax_sel = std::max(lmax_sel, ctx->len[c]);
    int term_opts[3] = {1, 2, kE4M3};
    const int nterm_opts = ctx->mode == BLAMM_MODE_AUTO ? (lmax_sel <= kMaxE4M3Len ? 3 : 2) : 1;
    float best = std::numeric_limits<float>::infinity();
    int bt = keep_terms;
    for (int ti = 0; ti < nterm_opts; ++ti) {
        if (ctx->mode == BLAMM_MODE_AUTO) ctx->auto_terms = term_opts[ti];
        ctx->plan_valid = false;
        float t[5];
        for (float &ms : t) {
            int64_t nh = 0;
            rc = scan_core(ctx, d_bases, ns, d_run_start, nrs, ctx->d_hits, ctx->hits_cap, &nh);
            if (rc && rc != BLAMM_ERR_OVERFLOW) {
                ctx->auto_terms = keep_terms;
                ctx->plan_valid = false;
                return rc;
            }
            ms = ctx->stats.kernel_ms;
        }
        std::sort(t, t + 5);
        // (a form is taken over the ones before it only if it is faster by more than such
        // medians differ from run to run, about 2 %: otherwise the choice would be a toss-up)
        if (t[2] < 0.97f * best) {
            best = t[2];
            bt = ctx->auto_terms;
        }
    }
    ctx->auto_terms = bt;
    ctx->plan_valid = false;
    if ((rc = ensure_plan(ctx))) return rc;
    if (best_ms) *best_ms = best;
    return BLAMM_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ theoretical histograms, thresholds

extern "C" {

int blamm_theoretical_hist(blamm_ctx *ctx, const float *P, int p_rows, int ncols, const int32_t *col_len,
                           const int32_t *hist_of, const float bg_prob[4], int nbins, uint64_t max_length,
                           int fp64_dp, const float *pvalues, int npv, float *thr, uint64_t *counts)
{
    const NvtxRange nvtx_range("blamm_theoretical_hist");
    if (!ctx || !P || !col_len || !bg_prob || ncols <= 0 || p_rows <= 0 || nbins < 1 || nbins > 4096 ||
        npv < 0 || (npv > 0 && (!pvalues || !thr)))
        return BLAMM_ERR_ARG;
    for (int c = 0; c < ncols; ++c) {
        const int h = hist_of ? hist_of[c] : c;
        if (h < 0 || h >= ncols) return fail(ctx, BLAMM_ERR_ARG, "hist_of[%d] = %d is not a column", c, h);
        if (col_len[h] <= 0 || col_len[h] > kMaxMotifLen || 4 * col_len[h] > p_rows)
            return fail(ctx, BLAMM_ERR_ARG, "column %d: bad length %d", h, col_len[h]);
    }
    CK(cudaSetDevice(ctx->device));
    // the distinct distributions, and the columns that have each
    std::vector<int32_t> slot(ncols, -1), dist, tab;
    int lmax = 1;
    for (int c = 0; c < ncols; ++c) {
        const int h = hist_of ? hist_of[c] : c;
        if (slot[h] < 0) {
            slot[h] = (int32_t)dist.size();
            dist.push_back(h);
            lmax = std::max(lmax, (int)col_len[h]);
        }
    }
    const int nd = (int)dist.size();
    std::vector<int32_t> user0(nd + 1, 0), users(ncols), fill;
    for (int c = 0; c < ncols; ++c) ++user0[slot[hist_of ? hist_of[c] : c] + 1];
    for (int i = 0; i < nd; ++i) user0[i + 1] += user0[i];
    fill.assign(user0.begin(), user0.end() - 1);
    for (int c = 0; c < ncols; ++c) users[fill[slot[hist_of ? hist_of[c] : c]]++] = c;
    // one table of 32-bit words: lengths, distributions, users, their offsets, p-values, status
    tab.assign(col_len, col_len + ncols);
    tab.insert(tab.end(), dist.begin(), dist.end());
    tab.insert(tab.end(), users.begin(), users.end());
    tab.insert(tab.end(), user0.begin(), user0.end());
    const size_t pv_at = tab.size(), status_at = pv_at + (size_t)npv;
    tab.resize(status_at + 1, 0);
    if (npv > 0) std::memcpy(&tab[pv_at], pvalues, sizeof(float) * (size_t)npv);
    const size_t pbytes = sizeof(float) * (size_t)p_rows * ncols, tbytes = sizeof(int32_t) * tab.size();
    const size_t thr_bytes = sizeof(float) * (size_t)npv * ncols;
    const size_t cnt_bytes = counts ? sizeof(unsigned long long) * (size_t)ncols * nbins : 0;
    auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
    int rc = ensure(ctx, &ctx->d_theo, &ctx->cap_theo, up(cnt_bytes) + up(pbytes) + up(tbytes) + up(thr_bytes));
    if (rc) return rc;
    uint8_t *at = ctx->d_theo;
    auto take = [&](size_t bytes) {
        uint8_t *r = at;
        at += up(bytes);
        return r;
    };
    unsigned long long *d_counts = reinterpret_cast<unsigned long long *>(take(cnt_bytes));
    float *d_P = reinterpret_cast<float *>(take(pbytes));
    int32_t *d_tab = reinterpret_cast<int32_t *>(take(tbytes));
    float *d_thr = reinterpret_cast<float *>(take(thr_bytes));
    CK(cudaMemcpyAsync(d_P, P, pbytes, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_tab, tab.data(), tbytes, cudaMemcpyHostToDevice, ctx->stream));
    TheoHistParams p{};
    p.P = d_P;
    p.p_rows = p_rows;
    p.ncols = ncols;
    p.col_len = d_tab;
    p.dist = d_tab + ncols;
    p.users = p.dist + nd;
    p.user0 = p.users + ncols;
    for (int k = 0; k < 4; ++k) p.bg[k] = bg_prob[k];
    p.nbins = nbins;
    p.max_length = max_length;
    p.lmax = lmax;
    p.pvalues = reinterpret_cast<const float *>(d_tab + pv_at);
    p.npv = npv;
    p.thr = npv > 0 ? d_thr : nullptr;
    p.counts = counts ? d_counts : nullptr;
    p.status = d_tab + status_at;
    // Key ranges are about nbins + L, up to a few times that where the rows' minima differ: 2048
    // keys leave room for several CTAs per SM, and what exceeds them is run again with 8192.
    for (const int kmax : {2048, 8192}) {
        if (kmax == 2048 && nbins > 1024) continue;
        p.kmax = kmax;
        const size_t smem = theo_smem_bytes(kmax, nbins, lmax, fp64_dp);
        if (smem > (size_t)ctx->max_smem) return fail(ctx, BLAMM_ERR_UNSUPPORTED, "histogram does not fit");
        const auto kernel = fp64_dp ? theoretical_hist64_kernel : theoretical_hist_kernel;
        CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<nd, kTheoThreads, smem, ctx->stream>>>(p);
        CK(cudaGetLastError());
        // Results up to 16 MB come back through pinned staging: a caller's fresh pages are then
        // touched by the CPU only (8 MB straight into pages that are unmapped soon after took
        // 0.2 ms or 7, depending on the process; this way 0.3).
        const bool stage = cnt_bytes + thr_bytes <= (size_t(16) << 20);
        uint8_t *to_thr = reinterpret_cast<uint8_t *>(thr), *to_counts = reinterpret_cast<uint8_t *>(counts);
        if (stage) {
            if ((rc = ensure_stage(ctx, cnt_bytes + thr_bytes))) return rc;
            to_counts = ctx->h_stage;
            to_thr = ctx->h_stage + cnt_bytes;
        }
        if (npv > 0) CK(cudaMemcpyAsync(to_thr, d_thr, thr_bytes, cudaMemcpyDeviceToHost, ctx->stream));
        if (counts) CK(cudaMemcpyAsync(to_counts, d_counts, cnt_bytes, cudaMemcpyDeviceToHost, ctx->stream));
        int status = 0;
        CK(cudaMemcpyAsync(&status, p.status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        if (!status) {
            if (stage && npv > 0) std::memcpy(thr, to_thr, thr_bytes);
            if (stage && counts) copy_out(counts, to_counts, cnt_bytes);
            return BLAMM_OK;
        }
        CK(cudaMemsetAsync(p.status, 0, sizeof(int), ctx->stream));
    }
    return fail(ctx, BLAMM_ERR_UNSUPPORTED, "a score range exceeds %d keys (fewer bins)", p.kmax);
}

}  // extern "C"

// ------------------------------------------------------------------ FASTA ingest on the GPU

// FASTA text on the device -> filtered stream, run table and header offsets.  Outputs go
// to the caller's buffers, or (resident: the caller's pointers are null) into the
// context's resident-stream buffers, sized once the counts are known.
static int fasta_parse(blamm_ctx *ctx, const char *d_raw, int64_t nraw, bool resident, char *d_bases,
                       int64_t *d_run_start, int64_t *d_run_seq, int64_t *d_run_seqpos, int64_t *d_header_pos,
                       int64_t *n_bases, int64_t *nruns, int64_t *nseqs, uint64_t *nucl_counts)
{
    cudaStream_t st = ctx->stream;
    const int64_t ntiles = (nraw + kIngTile - 1) / kIngTile;
    if (ntiles > 0x7fffffff) return fail(ctx, BLAMM_ERR_UNSUPPORTED, "%lld bytes of text in one call", (long long)nraw);
    const int vec = (reinterpret_cast<uintptr_t>(d_raw) & 15u) == 0 ? 1 : 0;  // 16-byte loads
    int rc = ensure(ctx, &ctx->d_ing_tiles, &ctx->cap_ing_tiles, (size_t)(kIngTileWords * ntiles));
    if (!rc) rc = ensure(ctx, &ctx->d_ing_prefix, &ctx->cap_ing_prefix, (size_t)ntiles);
    if (!rc) rc = ensure(ctx, &ctx->d_ing_totals, &ctx->cap_ing_totals, (size_t)kIngTotals);
    if (rc) return rc;
    IngTile tiles{};  // (the arrays of 16-byte words first)
    tiles.e = ctx->d_ing_tiles;
    tiles.warps = tiles.e + 2 * ntiles;
    tiles.bases = reinterpret_cast<uint64_t *>(tiles.warps + 2 * kIngWarps * ntiles);
    tiles.info = reinterpret_cast<uint32_t *>(tiles.bases + kIngThreads * ntiles);
    tiles.count = (int)ntiles;
    ingest_tiles_kernel<<<(unsigned)ntiles, kIngThreads, 0, st>>>(d_raw, nraw, vec, tiles);
    CK(cudaGetLastError());
    ingest_scan_kernel<<<1, kIngScanThreads, 0, st>>>(tiles, ctx->d_ing_prefix, ctx->d_ing_totals);
    CK(cudaGetLastError());
    auto emit = [&]() -> int {
        ingest_emit_kernel<<<(unsigned)(ntiles * (kIngThreads / kIngEmit)), kIngEmit, 0, st>>>(d_raw, nraw, vec, tiles, ctx->d_ing_prefix, ctx->d_ing_totals,
                                                                     d_bases, d_run_start, d_run_seq, d_run_seqpos,
                                                                     d_header_pos);
        CK(cudaGetLastError());
        return BLAMM_OK;
    };
    if (!resident && (rc = emit())) return rc;
    unsigned long long tot[kIngTotals];
    CK(cudaMemcpyAsync(tot, ctx->d_ing_totals, sizeof tot, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (tot[3]) return fail(ctx, BLAMM_ERR_ARG, "Input file does not appear to be in fasta format");
    const int64_t nb = (int64_t)tot[0], nr = (int64_t)tot[1], ns = (int64_t)tot[2];
    if (resident) {
        // (the writes are ordered on the context's stream like everything that reads them)
        rc = ensure(ctx, &ctx->d_shdr, &ctx->cap_shdr, (size_t)std::max<int64_t>(ns, 1));
        if (!rc) rc = ensure(ctx, &ctx->d_stream, &ctx->cap_stream, (size_t)std::max<int64_t>(nb, 1));
        for (int k = 0; k < 3 && !rc; ++k)
            rc = ensure(ctx, &ctx->d_srun[k], &ctx->cap_srun[k], (size_t)std::max<int64_t>(nr, 1));
        if (rc) return rc;
        d_header_pos = ctx->d_shdr;
        d_bases = ctx->d_stream;
        d_run_start = ctx->d_srun[0];
        d_run_seq = ctx->d_srun[1];
        d_run_seqpos = ctx->d_srun[2];
        if ((rc = emit())) return rc;
    }
    *n_bases = nb;
    *nruns = nr;
    *nseqs = ns;
    if (nucl_counts)
        for (int b = 0; b < 4; ++b) nucl_counts[b] = tot[4 + b];
    return BLAMM_OK;
}

extern "C" {

int blamm_fasta_parse_device(blamm_ctx *ctx, const char *d_raw, int64_t nraw, char *d_bases, int64_t *n_bases,
                             int64_t *d_run_start, int64_t *d_run_seq, int64_t *d_run_seqpos, int64_t *nruns,
                             int64_t *d_header_pos, int64_t *nseqs, uint64_t *nucl_counts)
{
    const NvtxRange nvtx_range("blamm_fasta_parse_device");
    if (!ctx || nraw < 0 || !n_bases || !nruns || !nseqs) return BLAMM_ERR_ARG;
    *n_bases = *nruns = *nseqs = 0;
    if (nucl_counts)
        for (int b = 0; b < 4; ++b) nucl_counts[b] = 0;
    if (nraw == 0) return BLAMM_OK;
    if (!d_raw || !d_bases || !d_run_start || !d_run_seq || !d_run_seqpos || !d_header_pos)
        return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    CK(cudaSetDevice(ctx->device));
    return fasta_parse(ctx, d_raw, nraw, false, d_bases, d_run_start, d_run_seq, d_run_seqpos, d_header_pos,
                       n_bases, nruns, nseqs, nucl_counts);
}

int blamm_stream_load_fasta(blamm_ctx *ctx, const char *raw, int64_t nraw, int64_t *n_bases, int64_t *nruns,
                            int64_t *nseqs, uint64_t *nucl_counts)
{
    const NvtxRange nvtx_range("blamm_stream_load_fasta");
    if (!ctx || nraw < 0 || !n_bases || !nruns || !nseqs || (nraw > 0 && !raw)) return BLAMM_ERR_ARG;
    *n_bases = *nruns = *nseqs = 0;
    if (nucl_counts)
        for (int b = 0; b < 4; ++b) nucl_counts[b] = 0;
    ctx->stream_n = ctx->stream_nruns = ctx->stream_nseqs = 0;
    if (nraw == 0) return BLAMM_OK;
    CK(cudaSetDevice(ctx->device));
    int rc = ensure(ctx, &ctx->d_raw, &ctx->cap_raw, (size_t)nraw);
    if (rc) return rc;
    CK(cudaMemcpyAsync(ctx->d_raw, raw, (size_t)nraw, cudaMemcpyHostToDevice, ctx->stream));
    rc = fasta_parse(ctx, ctx->d_raw, nraw, true, nullptr, nullptr, nullptr, nullptr, nullptr, n_bases, nruns,
                     nseqs, nucl_counts);
    if (rc) return rc;
    ctx->stream_n = *n_bases;
    ctx->stream_nruns = *nruns;
    ctx->stream_nseqs = *nseqs;
    return BLAMM_OK;
}

int blamm_stream_tables(blamm_ctx *ctx, int64_t *run_start, int64_t *run_seq, int64_t *run_seqpos,
                        int64_t *header_pos)
{
    if (!ctx) return BLAMM_ERR_ARG;
    CK(cudaSetDevice(ctx->device));
    int64_t *dst[4] = {run_start, run_seq, run_seqpos, header_pos};
    const int64_t *src[4] = {ctx->d_srun[0], ctx->d_srun[1], ctx->d_srun[2], ctx->d_shdr};
    const int64_t cnt[4] = {ctx->stream_nruns, ctx->stream_nruns, ctx->stream_nruns, ctx->stream_nseqs};
    for (int k = 0; k < 4; ++k)
        if (dst[k] && cnt[k] > 0)
            CK(cudaMemcpyAsync(dst[k], src[k], 8 * (size_t)cnt[k], cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    return BLAMM_OK;
}

int blamm_scan_stream(blamm_ctx *ctx, int64_t begin, int64_t n, const int64_t *run_start, int64_t nruns,
                      blamm_hit *hits, int64_t hit_cap, int64_t *n_hits)
{
    const NvtxRange nvtx_range("blamm_scan_stream");
    if (!ctx || !n_hits || n < 0 || hit_cap < 0 || begin < 0) return BLAMM_ERR_ARG;
    *n_hits = 0;
    if (begin > ctx->stream_n || n > ctx->stream_n - begin)
        return fail(ctx, BLAMM_ERR_ARG, "positions [%lld, %lld) outside the resident stream of %lld bases",
                    (long long)begin, (long long)(begin + n), (long long)ctx->stream_n);
    if (n == 0) return BLAMM_OK;
    if (!run_start || nruns <= 0 || (hit_cap > 0 && !hits)) return fail(ctx, BLAMM_ERR_ARG, "null buffer");
    if (run_start[0] != 0) return fail(ctx, BLAMM_ERR_ARG, "run_start[0] must be 0");
    for (int64_t r = 1; r < nruns; ++r)
        if (run_start[r] <= run_start[r - 1] || run_start[r] >= n)
            return fail(ctx, BLAMM_ERR_ARG, "run_start must ascend strictly inside [0, n)");
    CK(cudaSetDevice(ctx->device));
    if (ctx->ncols == 0) return fail(ctx, BLAMM_ERR_STATE, "blamm_set_motifs was not called");
    return scan_host_once(ctx, nullptr, ctx->d_stream + begin, n, run_start, nruns, hits, hit_cap, n_hits);
}

}  // extern "C"
