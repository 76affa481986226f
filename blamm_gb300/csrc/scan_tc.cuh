// scan_tc.cuh -- the fused tensor-core PWM scan (tcgen05 + TMA bulk + TMEM),
// one persistent CTA per SM.
//
// Score of motif column c at position p:  sum_j P(4j + base(p+j), c).
// prep_kernel packs the stream and writes one 16-byte entry per position of a
// window of at most 16 Mi positions (the scan runs once per window, so the entry
// array stays 256 MB whatever the stream length),
// E[i] = onehot(base i) ++ onehot(base i+1) (2 bases x 4 channels x bf16).
// The contraction is D = A B^T with the motifs as rows: A is a tile of 128 motif
// columns (UMMA M = 128, one TMEM lane per motif), B the overlapping one-hot
// windows of a block of 256 positions (UMMA N = 256, one TMEM column per
// position).  A bulk copy brings the block's 256 + 4g entries into shared memory;
// read with row stride 16 B, 8-row group stride (SBO) 128 B and K-core stride
// (LBO) 32 B, the entries starting at E[4g] form exactly the B operand of motif
// bases 4g..4g+3 for all 256 positions -- the overlapping one-hot windows of the
// reference's S matrix (src/sequence.cpp:299-340) without materialising them:
// each k-step is a shifted descriptor over the same ~300 entries.
//
// Why motifs are the rows.  A lane holds one motif, so the threshold is one
// register per lane: the drain compares the maximum that its TMEM load returns
// with it, and no MMA is spent on a bias.  A tile is 128 columns of similar length
// instead of up to 256, so less zero padding is multiplied (genome_100mbp's bank:
// 41 MMAs of 128x256x16 per 256 positions against 48 with the motifs as 256-wide
// columns and a bias; 22 against 32 in the E4M3 form).  And a tile takes only 4 KB
// of shared memory per k-step, so a whole bank of about 1000 columns is resident
// and a block's entries are read once for all its tiles instead of once per tile.
//
// Arithmetic.  Column c's P enters as fixed-point BF16 terms: hi on the grid
// 2^-k, lo on 2^-(k+8), k = 7 - ceil(log2 max|P_c|), so |hi| <= 128 * 2^-k.
// Every partial sum is then an integer multiple of u = 2^-(k+8) below 2^24 u in
// magnitude (motifs up to 256 long), i.e. exactly representable in FP32, so an
// accumulation that keeps 24 significant bits holds sum(q) exactly (the
// raw-score dump instance compares the accumulator with the exact sum on
// every position and column of a test bank).  A position is a candidate iff
// sum(q) >= T, T a lower bound of sum(q) over the windows that are hits of the
// column, the reference's own FP32 rounding included, rounded down to the grid
// (plan_kernels.cuh), so every reference hit is a candidate; candidates are
// rescored in exact sequential FP32.
//
// The E4M3 form (kTerms = kE4M3, kind::f8f6f4, motifs up to 64 positions): entries hold
// four bases as 16 E4M3 bytes, so an MMA covers 8 positions; P enters as P x 2^s_c rounded
// to E4M3, s_c such that max|P| 2^s_c lies in (32, 64].  Every product is then a multiple of
// 2^-9 and every partial sum below 2^13, exact in FP32.  Its T is scaled by 2^s_c too.
//
// Roles (640 threads, warp w on SM sub-partition w % 4): warps 0-15 drain TMEM
// (lane quarter = warp % 4, two of the block's eight 32-position chunks each) and
// test for candidates; warp 16 reserves the drain warps' record blocks; warps 19 and 18
// issue the MMAs of the even and the odd jobs (a job is one tile on one block; the
// whole warp runs the loop, one elected lane issues), so that one issuer's waits,
// commits and loop overhead overlap the other's MMAs; warp 17 (one lane) loads A
// tiles and E windows with TMA bulk copies up to kEStages blocks ahead; warp 19 also
// allocates TMEM.
//
// What bounds it.  A job's accumulator is half of TMEM, so only two jobs are in
// flight, and the time per job is the larger of its MMAs (128 cycles each; 5.1 a job
// with one BF16 term, 2.75 with E4M3 on genome_100mbp's bank) and half of MMAs +
// hand-off: commit -> drain warps awake (~250 cycles) -> their TMEM loads (~180) ->
// all 16 have handed back -> the issuer issues (~120).  A drain warp that met a
// candidate is late for the next job, and one of the 16 nearly always has, so the
// rare path's latency counts in full: masks in eight short chains, predicated stores,
// record blocks reserved by a warp of their own, no shared memory in the issuers' loop.
// The hand-back is a hardware barrier because 16 arrivals on a shared-memory mbarrier
// queue behind the tensor cores' operand reads.  16 Mi positions x 1024 columns, ms, scan
// kernel alone (BF16, E4M3, two BF16 terms): 1.31, 1.11, 2.34, the tensor pipe busy for
// 87, 56 and 97 % of it.  With the motifs as columns of 256-wide tiles and bias MMAs the scan took
// 2.0, 2.0, 2.8 with the entries' kernel in it.
// Slower: accumulators of 128 columns (an MMA of N = 128 takes 1.1-1.2 times its share and
// every barrier is met twice as often), TMEM loads of 16 or 64 columns, the rare values
// through a shared-memory queue, one issuer.
//
// A drain warp hands its accumulator back right after its two TMEM loads; a chunk
// holds a candidate iff the maximum that the load returns reaches the lane's
// threshold, and only then (rare) are the masks built and one 16-byte record
// (chunk, slot, mask) per lane with candidates written to global memory, into a
// block of record slots (kRecBlock slots per atomic; slot 0 of a block counts its
// records).  Warp 16 keeps the next block ready for every drain warp, so that none of
// them has an atomic in flight.  The rescoring kernel expands the masks.
//
// Work: the tiles are cut into groups of `tg` consecutive tiles whose A fits in
// shared memory; a unit is (group, block of 256 positions), and units are dealt to
// the CTAs group by group.  Within a unit the tiles follow one another on the same
// E window.  Where the blocks are fewer than the CTAs, each CTA takes a contiguous
// range of units instead, so that it keeps its group.  At a group change both
// issuers commit their MMAs to a tile-done barrier, the loader then copies the new
// A, and both wait for it.  A tile too long for shared memory (two BF16 terms
// beyond about 90 positions) is streamed: instance kStream, one issuer, A in
// chunks of kChunkBlocks k-steps through a ring of kChunks.
// Every mbarrier wait is bounded (the issuers poll with test_wait, the drain warps wait
// with try_wait without a suspend hint, the loader's try_wait sleeps): on a timeout the
// CTA raises an abort flag, every role stops, copies and MMAs in flight are drained,
// TMEM is freed and the status word tells the host.  The hardware barriers have no
// timeout and count arrivals, not jobs, so their rule is exact: every drain warp arrives
// once for each job that was issued, in order, and only after it was (job_ready).  A drain
// warp whose wait gave up therefore goes on arriving, without looking at the values, until
// the issuers have left; these leave at their next mbarrier wait that is not yet complete,
// at most kEStages units later, because the loader stops at the abort.
#pragma once
#include <cstdint>

#include "blamm_gpu.h"
#include "ptx_sm100.cuh"
#include "scan_kernels.cuh"

namespace blamm {

constexpr int kTileCols = 128;   // motif columns per tile (= UMMA M, TMEM lanes)
constexpr int kBlockPos = 256;   // positions per block (= UMMA N, TMEM columns)
constexpr int kMaxTcLen = BLAMM_MAX_TC_MOTIF_LEN;  // longest motif on the tensor-core path
constexpr int kEpiWarps = 16;    // TMEM drain warps (4 per lane quarter)
constexpr int kBlockWarp = 16;   // reserves record blocks for the drain warps
constexpr int kLoadWarp = 17;    // TMA bulk copies of A tiles and E windows
constexpr int kMmaWarp2 = 18;    // issuer of the odd jobs
constexpr int kMmaWarp = 19;     // issuer of the even jobs; TMEM allocation
constexpr int kRecBlock = kRecBlockSlots;  // candidate record slots a drain warp reserves at a time
constexpr uint32_t kBlockTries = 1u << 24;  // looks for the next record block before a drain warp gives up (about 0.3 s)
constexpr uint32_t kNoBlock = 0xFFFFFFFFu;  // no slot index: the capacity is below 2^31
constexpr int kTcThreads = 640;  // 20 warps (registers are allocated per 4 warps)
constexpr int kEStages = 6;      // E windows in flight
constexpr int kE4M3 = 8;         // kTerms of the E4M3 form (one term, K = 32 per MMA)
constexpr int kMaxE4M3Len = 64;  // longest motif of the E4M3 form
constexpr int kAcc = 2;          // TMEM accumulator stages (256 columns each: the whole TMEM)
constexpr int kStepBytes = kTileCols * 32;  // A bytes of one k-step of one term (both forms)
constexpr uint32_t kBarEmpty = 1;        // hardware barriers 1, 2: accumulator drained
constexpr uint32_t kEmptyThreads = 32 * (kEpiWarps + 1);  // the drain warps and its issuer
constexpr int kChunkBlocks = 8;  // streamed A: k-steps per chunk
constexpr int kChunks = 4;       // streamed A: chunks in the ring

// Test hook (blamm_debug_stall): the issuers before their first job; and, in the raw-score
// instance only, at a CTA's unit number u (the value is role | u << 8): all drain warps, one
// of them, the loader, one issuer, the loader between a unit's entries and its streamed A.
enum { kStallIssuers = 1, kStallDrains, kStallDrain, kStallLoader, kStallIssuer, kStallChunks, kStallEnd };

// Per-tile description (host-built, read through the read-only path).
struct TileDesc {
    int32_t g;    // k-steps per term: ceil(longest motif in the tile / 4 (BF16) or 8 (E4M3))
    int32_t off;  // first k-step of the tile in the A buffer (kStepBytes each, terms one after another)
};

struct TcParams {
    const uint4 *e16;    // one-hot entries of this launch's window (16 B per position, padded)
    int64_t n;           // stream positions
    int32_t nblocks;     // blocks of kBlockPos positions of this launch's window
    uint32_t chunk0;     // the window's first 32-position chunk in the stream
    const TileDesc *tiles;  // ntiles + 1: the last one holds the end offset; longest motifs first
    int32_t ntiles;
    int32_t tg;          // tiles per group
    int32_t contiguous;  // 1: each CTA takes consecutive units
    int32_t turn;        // 1 (two BF16 terms only): every other unit takes its tiles in reverse
    int32_t terms;       // 1 (hi) or 2 (hi + lo) or kE4M3
    const uint8_t *abuf; // A tiles
    const int32_t *slot_col;  // per slot (tile * 128 + row): motif column, -1 for padding
    const float *slot_thr;    // per slot: T on the accumulator's scale, +inf for padding
    int32_t erows;       // E entries per stage
    uint32_t a_bytes;    // shared memory for A
    uint4 *cand;                      // candidate record slots: blocks of kRecBlock
    unsigned long long *cand_count;   // record slots reserved
    int64_t cand_cap;                 // record slots available (a multiple of kRecBlock); behind them: one spare
                                      // block, or (ncand: kCount) two per drain warp, whose candidates
    unsigned long long *ncand;        // are added to *ncand (the rescoring adds the others)
    unsigned long long *times;  // may be null
    int *status;         // bit 0: a device wait timed out
    long long wait_limit;  // clock64 cycles a wait may last
    int32_t debug_stall;   // test hook: who waits on a barrier nobody completes (kStall*)
    // debug dump of the accumulator (positions [dump_p0, dump_p0+dump_npos))
    float *dump;
    int64_t dump_p0, dump_npos;
    int32_t dump_ncols;
    // optional per-CTA role timing (32 counters per CTA, clock64 cycles): see tc_prof_fields
    long long *prof;
};

// tc_prof_fields: 0/1 issuers' waits for a drained accumulator, 2 issuers' waits for A
// tiles, 3 MMA loop, 4 loader waits for free E stages, 5 loader waits at group changes,
// 7 drain warp 0's accumulator waits, 8 its loop, 9 its drain (full accumulator -> hand-back),
// 10 tiles x 128-position half blocks, 11 issuers' waits for E, 12 drain warp 0's rounds with
// a candidate, 13 its record block changes, 15 its candidate test and record writing

struct TcSmem {
    // byte offsets into dynamic shared memory
    uint32_t a, e0, bars, ctl, total;
};

// control words in shared memory
enum {
    CTL_ABORT = 0,     // set by the first wait that times out
    CTL_TMEM = 1,      // TMEM base address
    CTL_DONE = 2,      // drain warps that have finished
    CTL_LEFT = 3,      // per accumulator: its issuer has left its loop
    CTL_BLOCK = 5,     // per drain warp: its next record block (kNoBlock: none yet)
    CTL_WORDS = CTL_BLOCK + kEpiWarps
};

__host__ __device__ inline TcSmem tc_smem_layout(uint32_t a_bytes, int erows)
{
    TcSmem L;
    uint32_t o = 0;
    auto take = [&](uint32_t bytes, uint32_t align) {
        o = (o + align - 1) / align * align;
        uint32_t r = o;
        o += bytes;
        return r;
    };
    L.a = take(a_bytes, 1024);
    L.e0 = take((uint32_t)kEStages * erows * 16, 128);  // kEStages stages of erows entries
    L.bars = take(32 * 8, 8);  // BAR_COUNT <= 32
    L.ctl = take(CTL_WORDS * 4, 16);
    L.total = take(0, 1024) + 1024;  // + slack for aligning the runtime base
    return L;
}

enum {
    BAR_EFULL = 0,                       // E window landed       (kEStages)
    BAR_EEMPTY = BAR_EFULL + kEStages,   // E window consumed     (kEStages)
    BAR_AFULL = BAR_EEMPTY + kEStages,   // accumulator ready     (kAcc)
    BAR_BFULL = BAR_AFULL + kAcc,       // A tiles of a group landed
    BAR_TILE = BAR_BFULL + 1,            // both issuers done with the old group
    BAR_CFULL = BAR_TILE + 1,            // streamed A chunk landed   (kChunks)
    BAR_CEMPTY = BAR_CFULL + kChunks,    // streamed A chunk consumed (kChunks)
    BAR_DRAIN = BAR_CEMPTY + kChunks,    // an issuer's MMAs drained (2)
    BAR_NEVER = BAR_DRAIN + 2,           // never completed (the stall test hook)
    BAR_COUNT = BAR_NEVER + 1
};
static_assert(BAR_COUNT <= 32, "the barrier area holds 32 mbarriers");

// Bit i set <=> value i >= thr (nt: -thr twice).  The difference has the sign of the
// comparison (an FP32 difference of unequal values never rounds to zero): 16 packed
// subtractions and one funnel shift per value ((m << 1) | sign), in eight chains of four.
__device__ __forceinline__ uint32_t ge_mask(const uint32_t (&v)[32], uint64_t nt)
{
    uint32_t m[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) m[c] = 0u;
#pragma unroll
    for (int i = 2; i >= 0; i -= 2) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            uint32_t lo, hi;
            ptx::unpack2(ptx::add_f32x2(ptx::pack2(v[4 * c + i], v[4 * c + i + 1]), nt), lo, hi);
            m[c] = __funnelshift_l(hi, m[c], 1);
            m[c] = __funnelshift_l(lo, m[c], 1);
        }
    }
#pragma unroll
    for (int c = 0; c < 8; c += 2) m[c] += m[c + 1] << 4;
    m[0] += m[2] << 8;
    m[4] += m[6] << 8;
    return ~(m[0] + (m[4] << 16));
}

// One block of record slots.  The capacity is a multiple of kRecBlock below 2^31; a block
// reserved beyond it becomes a spare block behind the buffer, which the rescoring does not read.
__device__ __forceinline__ uint32_t reserve_block(const TcParams &p)
{
    const unsigned long long b = atomicAdd(p.cand_count, (unsigned long long)kRecBlock);
    return b < (unsigned long long)p.cand_cap ? (uint32_t)b : (uint32_t)p.cand_cap;
}

// Spare block k (0, 1) of a drain warp.
__device__ __forceinline__ uint32_t spare_block(const TcParams &p, int warp, int k)
{
    return (uint32_t)p.cand_cap + (((uint32_t)blockIdx.x * kEpiWarps + warp) * 2u + k) * kRecBlock;
}

// Adds the candidates of closed spare blocks to *ncand; block: per lane (kNoBlock or below the
// capacity: none).  A whole warp.
__device__ __noinline__ void count_spare(const TcParams &p, uint32_t block)
{
    const int lane = threadIdx.x & 31;
    __threadfence_block();
    for (uint32_t m = __ballot_sync(0xffffffffu, block != kNoBlock && block >= (uint32_t)p.cand_cap); m; m &= m - 1u) {
        const uint4 *b = p.cand + __shfl_sync(0xffffffffu, block, __ffs(m) - 1);
        const uint32_t n = __ldcg(&b->x);
        uint32_t c = 0;
        for (uint32_t k = 1u + lane; k <= n; k += 32) {
            const uint4 r = __ldcg(b + k);
            c += (uint32_t)__popc(r.z & valid_positions(p.n, r.x));
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(p.ncand, (unsigned long long)c);
    }
}

// The units of one CTA: unit u = group * nblocks + block, advanced without divisions after
// the first.  Indices are 32-bit (the host launches at most 2^31 - 1 jobs).
struct UnitIter {
    int u, end, stride;
    int group, block;
    __device__ __forceinline__ void init(const TcParams &p, int ngroups)
    {
        const int units = ngroups * p.nblocks;
        if (p.contiguous) {
            u = (int)((long long)blockIdx.x * units / gridDim.x);
            end = (int)((long long)(blockIdx.x + 1) * units / gridDim.x);
            stride = 1;
        } else {
            u = blockIdx.x;
            end = units;
            stride = gridDim.x;
        }
        group = u / p.nblocks;
        block = u - group * p.nblocks;
    }
    __device__ __forceinline__ void next(int nblocks)
    {
        u += stride;
        block += stride;
        while (block >= nblocks) {
            block -= nblocks;
            ++group;
        }
    }
};

// For a drain warp after an abort: waits until the job's accumulator is ready (true: the warp
// arrives for it) or its issuer has left (false: nobody will wait for this accumulator again).
// Every other wait of the CTA ends at the abort flag, so one of the two comes soon; should an MMA
// never complete, the wait ends after limit_cycles, with the issuer at the barrier for this job.
__device__ __noinline__ bool job_ready(uint32_t bar, uint32_t parity, volatile int *left, long long limit_cycles)
{
    const long long t0 = clock64();
    for (;;) {
        if (__all_sync(0xffffffffu, ptx::mbar_try_wait_nohint(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *left != 0)) return false;
        if (__any_sync(0xffffffffu, clock64() - t0 > limit_cycles)) return true;
    }
}

template <bool kProf>
__device__ __forceinline__ long long tick()
{
    if constexpr (kProf) return clock64();
    else return 0;
}

// kDump: also write the raw accumulator of some positions (test hook);
// kProf: role timing into p.prof; kTerms: p.terms (1 or 2 BF16 terms, or kE4M3,
// one E4M3 term); kStream: A in chunks through a ring (tg == 1); kCount: candidates of
// records that do not fit are counted (p.ncand).  The scan itself is <false, false,
// p.terms, *, *>.  The issuing threads run once per MMA and per
// job, so every branch taken out of their loops at compile time shows in the
// scan time (runtime mode switches cost 2-4 %).
template <bool kDump, bool kProf, int kTerms, bool kStream, bool kCount>
__global__ void __launch_bounds__(kTcThreads, 1) scan_tc_kernel(TcParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024 - (ptx::smem_addr(smem_raw) & 1023)) & 1023);
    const TcSmem L = tc_smem_layout(p.a_bytes, p.erows);
    const uint32_t sbase = ptx::smem_addr(smem);
    const uint32_t bars = sbase + L.bars;
    volatile int *ctl = reinterpret_cast<volatile int *>(smem + L.ctl);
    volatile int *s_abort = ctl + CTL_ABORT;

    // (by a shuffle: the compiler then knows that roles and descriptors are warp-uniform)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    // ---- set-up
    if (threadIdx.x < CTL_WORDS && threadIdx.x != CTL_TMEM) ctl[threadIdx.x] = threadIdx.x >= CTL_BLOCK ? (int)kNoBlock : 0;
    if (threadIdx.x == 0) {
        if (p.times && blockIdx.x == 0) p.times[2] = ptx::global_ns();
        for (int s = 0; s < kEStages; ++s) {
            ptx::mbar_init(bars + 8 * (BAR_EFULL + s), 1);
            ptx::mbar_init(bars + 8 * (BAR_EEMPTY + s), kStream ? 1 : 2);
        }
        for (int s = 0; s < kAcc; ++s) {
            ptx::mbar_init(bars + 8 * (BAR_AFULL + s), 1);
        }
        ptx::mbar_init(bars + 8 * BAR_BFULL, 1);
        ptx::mbar_init(bars + 8 * BAR_TILE, 2);
        for (int s = 0; s < kChunks; ++s) {
            ptx::mbar_init(bars + 8 * (BAR_CFULL + s), 1);
            ptx::mbar_init(bars + 8 * (BAR_CEMPTY + s), 1);
        }
        ptx::mbar_init(bars + 8 * (BAR_DRAIN + 0), 1);
        ptx::mbar_init(bars + 8 * (BAR_DRAIN + 1), 1);
        ptx::mbar_init(bars + 8 * BAR_NEVER, 1);
        ptx::fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        ptx::tmem_alloc(sbase + L.ctl + 4 * CTL_TMEM, kAcc * kBlockPos);
        ptx::tmem_relinquish();
        ptx::tc_fence_before();
    }
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = (uint32_t)ctl[CTL_TMEM];
    const int ngroups = (p.ntiles + p.tg - 1) / p.tg;
    constexpr uint32_t kStepPos = kTerms == kE4M3 ? 8u : 4u;  // positions (= 16 B entries) per k-step
    constexpr uint32_t kNTerm = kTerms == 2 ? 2u : 1u;
    constexpr uint32_t kStep16 = kStepBytes / 16;  // one k-step of A in 16 B units
    UnitIter it;
    it.init(p, ngroups);
    const bool turn = kTerms == 2 && !kStream && p.turn != 0;
    int unit = 0;  // (test hook) this CTA's units so far
    auto stalls = [&](int role) { return kDump && p.debug_stall == (role | unit << 8); };
    auto never = [&]() { return ptx::mbar_wait(bars + 8 * BAR_NEVER, 0, s_abort, p.wait_limit); };

    if (warp == kMmaWarp || warp == kMmaWarp2) {
        // ============ MMA issuers: warp 19 the even jobs, warp 18 the odd ones ============
        // Both walk every job of the CTA.  The whole warp runs the loop (warp-uniform
        // descriptors, one vote per wait); one elected lane issues each MMA and commit.
        const uint32_t mine = warp == kMmaWarp ? 0u : 1u;
        int cur_group = -1, t0 = 0, t1 = 0;
        uint32_t bphase = 0, es = 0, eph = 0, jc = 0, cs = 0, cph = 0;
        long long t_acc = 0, t_w = 0, t_b = 0, t_jobs = 0;
        const long long t_start = tick<kProf>();
        // A: 8-row groups 128 B apart, K cores 2048 B apart; a k-step is kStepBytes further
        uint64_t adesc_g = 0;
        const uint64_t adesc0 = ptx::smem_desc(sbase + L.a, 2048u, 128u);
        // B: K cores 2 (BF16) or 4 (E4M3) entries apart, k-steps 4 or 8
        const uint64_t bdesc_e = ptx::smem_desc(sbase + L.e0, 8u * kStepPos, 128u);
        constexpr uint32_t idesc = kTerms == kE4M3 ? ptx::idesc_e4m3_f32(kTileCols, kBlockPos)
                                                   : ptx::idesc_bf16_f32(kTileCols, kBlockPos);
        auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
            if constexpr (kTerms == kE4M3) ptx::mma_e4m3_elect(d, a, b, idesc, acc);
            else ptx::mma_bf16_elect(d, a, b, idesc, acc);
        };
        const uint32_t e_step = (uint32_t)p.erows;  // one E stage in 16 B units
        bool ok = true, down = false;
        if (p.debug_stall == kStallIssuers) ok = never();
        ok = __all_sync(0xffffffffu, ok);
        if (kStream && mine == 1u) ok = false;  // one issuer walks the ring
        for (; it.u < it.end && ok; it.next(p.nblocks), ++unit) {
            if (stalls(kStallIssuer) && mine == (kStream ? 0u : 1u)) {
                ok = __all_sync(0xffffffffu, never());
                if (!ok) break;
            }
            if (it.group != cur_group) {
                const long long tb = tick<kProf>();
                if (!kStream) {
                    // this issuer is done with the old group once its MMAs so far are complete
                    if (cur_group >= 0) ptx::mma_commit_elect(bars + 8 * BAR_TILE);
                    ok = __all_sync(0xffffffffu, ptx::mbar_wait(bars + 8 * BAR_BFULL, bphase, s_abort, p.wait_limit));
                    bphase ^= 1;
                    if (!ok) break;
                    ptx::tc_fence_after();
                }
                cur_group = it.group;
                t0 = cur_group * p.tg;
                t1 = min(t0 + p.tg, p.ntiles);
                adesc_g = adesc0 - (uint64_t)__ldg(&p.tiles[t0].off) * kStep16;
                if (kProf) t_b += tick<kProf>() - tb;
            }
            const long long te = tick<kProf>();
            ok = __all_sync(0xffffffffu, ptx::mbar_wait_spin(bars + 8 * (BAR_EFULL + es), eph, s_abort, p.wait_limit));
            if (kProf) t_w += tick<kProf>() - te;
            if (!ok) break;
            const uint64_t bdesc = bdesc_e + es * e_step;
            int2 td = __ldg(reinterpret_cast<const int2 *>(p.tiles) + (down ? t1 - 1 : t0));
            for (int t = t0; t < t1; ++t, ++jc) {  // (down: tile t0 + t1 - 1 - t)
                const int2 tn = __ldg(reinterpret_cast<const int2 *>(p.tiles) + (down ? max(t0 + t1 - 2 - t, 0) : t + 1));
                if (kProf)
                    t_jobs += 2 - (((int64_t)p.chunk0 + it.block * 8 + 4) * 32 >= p.n ? 1 : 0);
                if (kStream || (jc & 1u) == mine) {
                    const uint32_t s = jc & 1u;  // accumulator
                    const long long ta = tick<kProf>();
                    // (returns after an abort too: the drain warps still arrive for every job issued)
                    if (jc >= 2u) ptx::named_sync(kBarEmpty + s, kEmptyThreads);
                    if (kProf) t_acc += tick<kProf>() - ta;
                    ptx::tc_fence_after();
                    const uint32_t d_tmem = tmem_base + s * kBlockPos, g = (uint32_t)td.x;
                    if constexpr (kStream) {
                        const uint32_t nb = g * kNTerm;
                        uint32_t kk = 0;  // k-step within the term
                        for (uint32_t b0 = 0; b0 < nb && ok; b0 += kChunkBlocks) {
                            ok = __all_sync(0xffffffffu, ptx::mbar_wait_spin(bars + 8 * (BAR_CFULL + cs), cph, s_abort,
                                                                            p.wait_limit));
                            if (!ok) break;
                            ptx::tc_fence_after();
                            const uint64_t ad = adesc0 + cs * (kChunkBlocks * kStep16);
                            const uint32_t m = min((uint32_t)kChunkBlocks, nb - b0);
                            for (uint32_t i = 0; i < m; ++i) {
                                mma(d_tmem, ad + i * kStep16, bdesc + kStepPos * kk, b0 + i != 0u);
                                if (++kk == g) kk = 0;
                            }
                            ptx::mma_commit_elect(bars + 8 * (BAR_CEMPTY + cs));
                            if (++cs == (uint32_t)kChunks) {
                                cs = 0;
                                cph ^= 1u;
                            }
                        }
                        if (!ok) break;
                    } else {
                        const uint64_t ad = adesc_g + (uint64_t)((uint32_t)td.y * kStep16);
                        for (uint32_t k = 0; k < g; ++k) {
                            mma(d_tmem, ad + k * kStep16, bdesc + kStepPos * k, k != 0u);
                            if (kTerms == 2) mma(d_tmem, ad + (g + k) * kStep16, bdesc + kStepPos * k, 1u);
                        }
                    }
                    ptx::mma_commit_elect(bars + 8 * (BAR_AFULL + s));
                }
                td = tn;
            }
            if (!ok) break;
            down = turn && !down;
            ptx::mma_commit_elect(bars + 8 * (BAR_EEMPTY + es));
            if (++es == (uint32_t)kEStages) {
                es = 0;
                eph ^= 1u;
            }
        }
        // the drain warps need not wait for jobs of this issuer any more
        if (lane == 0 && (!kStream || mine == 0u)) {
            ctl[CTL_LEFT + mine] = 1;
            if (kStream) ctl[CTL_LEFT + 1] = 1;
        }
        // drain: nothing may still write TMEM or shared memory when they are freed
        ptx::mma_commit_elect(bars + 8 * (BAR_DRAIN + mine));
        if (!ptx::mbar_wait_drain(bars + 8 * (BAR_DRAIN + mine), 0, p.wait_limit)) *s_abort = 1;
        if (kProf && lane == 0) {
            long long *pr = p.prof + 32 * blockIdx.x;
            pr[mine] += t_acc;
            if (mine == 0) {
                pr[2] += t_b;
                pr[3] += tick<kProf>() - t_start;
                pr[10] += t_jobs;
                pr[11] += t_w;
            }
        }
    } else if (warp == kLoadWarp && lane == 0) {
        // ============ loader: A tiles at group changes, E windows kEStages blocks ahead ============
        int cur_group = -1;
        uint32_t tphase = 0, bphase = 0, es = 0, eph = 0, cs = 0, cph = 0, e_bytes = 0;
        uint32_t issued[kEStages], cissued[kChunks];  // per stage: 1 + the phase of its last copy, 0 = none
        for (int k = 0; k < kEStages; ++k) issued[k] = 0;
        for (int k = 0; k < kChunks; ++k) cissued[k] = 0;
        bool a_pending = false, ok = true;
        long long t_we = 0, t_tile = 0;
        const uint8_t *a_src = nullptr;
        uint32_t a_len = 0;
        for (; it.u < it.end && ok; it.next(p.nblocks), ++unit) {
            if (*s_abort) break;  // (the issuers then run out of entries)
            if (stalls(kStallLoader) && !never()) break;
            if (it.group != cur_group) {
                const int t0 = it.group * p.tg, t1 = min(t0 + p.tg, p.ntiles);
                a_src = p.abuf + (int64_t)p.tiles[t0].off * kStepBytes;
                a_len = (uint32_t)(p.tiles[t1].off - p.tiles[t0].off) * (uint32_t)kStepBytes;
                // entries of a block: its positions and the reach of the group's longest motif
                e_bytes = 16u * ((uint32_t)kBlockPos + kStepPos * (uint32_t)p.tiles[t0].g);
                if (!kStream) {
                    if (cur_group >= 0) {  // both issuers' MMAs on the old A are complete
                        const long long tt = tick<kProf>();
                        ok = ptx::mbar_wait(bars + 8 * BAR_TILE, tphase, s_abort, p.wait_limit);
                        tphase ^= 1;
                        if (kProf) t_tile += tick<kProf>() - tt;
                        if (!ok) break;
                        // the previous A copy has landed (both issuers waited for it)
                    }
                    ptx::mbar_arrive_expect_tx(bars + 8 * BAR_BFULL, a_len);
                    ptx::bulk_g2s(sbase + L.a, a_src, a_len, bars + 8 * BAR_BFULL);
                    a_pending = true;
                    bphase ^= 1;
                }
                cur_group = it.group;
            }
            const long long tw = tick<kProf>();
            ok = ptx::mbar_wait(bars + 8 * (BAR_EEMPTY + es), eph ^ 1u, s_abort, p.wait_limit);
            if (kProf) t_we += tick<kProf>() - tw;
            if (!ok) break;
            ptx::mbar_arrive_expect_tx(bars + 8 * (BAR_EFULL + es), e_bytes);
            ptx::bulk_g2s(sbase + L.e0 + es * (uint32_t)p.erows * 16u, p.e16 + (int64_t)it.block * kBlockPos, e_bytes,
                          bars + 8 * (BAR_EFULL + es));
            issued[es] = 1u + eph;
            if (++es == (uint32_t)kEStages) {
                es = 0;
                eph ^= 1u;
            }
            if constexpr (kStream) {
                for (uint32_t o = 0; o < a_len; o += kChunkBlocks * kStepBytes) {
                    if (stalls(kStallChunks)) ok = never();
                    else ok = ptx::mbar_wait(bars + 8 * (BAR_CEMPTY + cs), cph ^ 1u, s_abort, p.wait_limit);
                    if (!ok) break;
                    const uint32_t len = min((uint32_t)(kChunkBlocks * kStepBytes), a_len - o);
                    ptx::mbar_arrive_expect_tx(bars + 8 * (BAR_CFULL + cs), len);
                    ptx::bulk_g2s(sbase + L.a + cs * (uint32_t)(kChunkBlocks * kStepBytes), a_src + o, len,
                                  bars + 8 * (BAR_CFULL + cs));
                    cissued[cs] = 1u + cph;
                    if (++cs == (uint32_t)kChunks) {
                        cs = 0;
                        cph ^= 1u;
                    }
                }
            }
        }
        // on an abort, copies still in flight must land before the CTA frees its memory
        if (*s_abort) {
            for (int k = 0; k < kEStages; ++k)
                if (issued[k]) ptx::mbar_wait_drain(bars + 8 * (BAR_EFULL + k), issued[k] - 1u, p.wait_limit);
            for (int k = 0; k < kChunks; ++k)
                if (cissued[k]) ptx::mbar_wait_drain(bars + 8 * (BAR_CFULL + k), cissued[k] - 1u, p.wait_limit);
            if (a_pending) ptx::mbar_wait_drain(bars + 8 * BAR_BFULL, bphase ^ 1u, p.wait_limit);
        }
        if (kProf) {
            long long *pr = p.prof + 32 * blockIdx.x;
            pr[4] += t_we;
            pr[5] += t_tile;
        }
    } else if (warp == kBlockWarp) {
        // ============ record blocks: one ahead for every drain warp ============
        // Lane k serves drain warp k.  That the block handed last was taken says that the one before
        // it is closed: if it is a spare block, its candidates are counted, and it can be handed again.
        // (One load and one vote a look: the loop shares its issue slots with four drain warps.)
        const int word = lane < kEpiWarps ? CTL_BLOCK + lane : lane == kEpiWarps ? CTL_DONE : CTL_ABORT;
        long long gone = 0;  // when the abort was seen
        uint32_t last = kNoBlock, before = kNoBlock;
        int which = 0;
        for (bool done = false; !done;) {
            const int v = ctl[word];
            if (!__any_sync(0xffffffffu, lane < kEpiWarps ? v == (int)kNoBlock : lane == kEpiWarps ? v == kEpiWarps : v != 0)) {
                __nanosleep(500);
                continue;
            }
            done = ctl[CTL_DONE] == kEpiWarps;  // (read before the blocks: none is taken after that)
            if (*s_abort) {  // (the drain warps' waits end too; should they not, this one does)
                if (gone == 0) gone = clock64();
                done = done || clock64() - gone > 64 * p.wait_limit;
            }
            done = __any_sync(0xffffffffu, done);
            const uint32_t b = lane < kEpiWarps ? (uint32_t)ctl[CTL_BLOCK + lane] : 0u;
            const bool taken = b == kNoBlock;
            if (kCount) {
                count_spare(p, taken || done ? before : kNoBlock);
                if (done) count_spare(p, taken ? last : kNoBlock);
            }
            if (done) {  // every reserved block states its count
                if (lane < kEpiWarps && !taken) p.cand[b] = make_uint4(0u, 0u, 0u, 0u);
            } else if (taken) {
                uint32_t next = reserve_block(p);
                if (kCount && next >= (uint32_t)p.cand_cap) next = spare_block(p, lane, which ^= 1);
                before = last;
                last = next;
                ctl[CTL_BLOCK + lane] = (int)next;
            }
            __syncwarp();
        }
    } else if (warp < kEpiWarps) {
        // ===================== epilogue (warps 0-15) ======================
        const int q = warp & 3;     // TMEM lanes (motif rows) 32q .. 32q+31
        const int grp = warp >> 2;  // the block's 32-position chunks 2 grp and 2 grp + 1
        const uint32_t lt = (1u << lane) - 1u;
        const uint32_t row = (uint32_t)(q * 32 + lane);  // this lane's motif row in a tile
        // The current record block (slot indices).  The next one is usually waiting in shared
        // memory: an atomic's answer takes a microsecond, and even a warp that does not look
        // at it is held up by its next load.
        uint32_t rec = 0, left = 0;  // the current block's next record, how many still fit
        bool have = false;           // there is a current block
        auto close_block = [&]() {   // slot 0 of a block: its number of records
            const uint32_t n = (uint32_t)(kRecBlock - 1) - left;
            if (have && lane == 0) p.cand[rec - n - 1u] = make_uint4(n, 0u, 0u, 0u);
            have = true;
        };
        auto next_block = [&]() {
            close_block();
            uint32_t b = 0;
            if constexpr (kCount) {  // every block comes from warp 16, which counts the spare ones
                __threadfence_block();
                __syncwarp();
                if (lane == 0) {
                    for (uint32_t k = 0; (b = (uint32_t)ctl[CTL_BLOCK + warp]) == kNoBlock; ++k)
                        if (k == kBlockTries) {
                            *s_abort = 1;
                            b = (uint32_t)p.cand_cap;  // (the spare area)
                            break;
                        }
                    ctl[CTL_BLOCK + warp] = (int)kNoBlock;
                }
            } else {
                b = (uint32_t)ctl[CTL_BLOCK + warp];
                __syncwarp();
                if (lane == 0) {
                    if (b == kNoBlock) b = reserve_block(p);
                    else ctl[CTL_BLOCK + warp] = (int)kNoBlock;
                }
            }
            rec = __shfl_sync(0xffffffffu, b, 0) + 1u;
            left = (uint32_t)(kRecBlock - 1);
        };
        long long t_af = 0, t_dr = 0, n_rare = 0, t_red = 0, t_full = 0;
        const long long t_start = tick<kProf>();
        const uint32_t taddr0 = tmem_base + ((uint32_t)(q * 32) << 16) + 64u * grp;
        uint32_t s = 0, ph = 0;  // accumulator stage and its phase
        const float *lane_thr = p.slot_thr + row;
        int cur_group = -1, t0 = 0, t1 = 0;
        float thr_next = 0.f;
        bool ok = true, down = false;
        for (; it.u < it.end && ok; it.next(p.nblocks), ++unit, down = turn && !down) {
            if (it.group != cur_group) {
                cur_group = it.group;
                t0 = cur_group * p.tg;
                t1 = min(t0 + p.tg, p.ntiles);
                thr_next = __ldg(lane_thr + (down ? t1 - 1 : t0) * kTileCols);
            }
            const uint32_t chunk = p.chunk0 + (uint32_t)it.block * 8u + 2u * grp;
            for (int t = t0; t < t1; ++t) {
                // this job's threshold; the next one's arrives during this job
                const float thr = thr_next;
                const int tile = down ? t0 + t1 - 1 - t : t;
                // (turning, a unit begins with the tile that the one before it ended with)
                const int tile_next = t + 1 < t1 ? (down ? tile - 1 : t + 1) : turn ? tile : t0;
                thr_next = __ldg(lane_thr + tile_next * kTileCols);
                const uint32_t slot = (uint32_t)tile * kTileCols + row;
                const long long ta = tick<kProf>();
                if (t == t0 && (stalls(kStallDrains) || (stalls(kStallDrain) && warp == 5))) ok = never();
                else ok = ptx::mbar_wait_warp(bars + 8 * (BAR_AFULL + s), ph, s_abort, p.wait_limit);
                if (!ok) {  // aborted: the jobs already issued, or about to be, are still handed back
                    for (uint32_t gone = 0; it.u < it.end && gone != 3u; it.next(p.nblocks), t = 0) {
                        t0 = it.group * p.tg;
                        t1 = min(t0 + p.tg, p.ntiles);
                        for (t = t < t0 ? t0 : t; t < t1; ++t) {
                            if (!((gone >> s) & 1u)) {
                                if (job_ready(bars + 8 * (BAR_AFULL + s), ph, ctl + CTL_LEFT + s, 4 * p.wait_limit))
                                    ptx::named_arrive(kBarEmpty + s, kEmptyThreads);
                                else gone |= 1u << s;
                            }
                            s ^= 1u;
                            ph ^= s ^ 1u;
                        }
                    }
                    break;
                }
                const long long tb = tick<kProf>();
                if (kProf) t_af += tb - ta;
                ptx::tc_fence_after();
                // Two TMEM loads that also return each lane's maximum over the chunk, after which
                // the accumulator is handed back at once; the candidate test on the maxima and the
                // rare mask building run on the registers.
                const uint32_t taddr = taddr0 + s * kBlockPos;
                uint32_t va[32], vb[32];
                float ma, mb;
                ptx::tmem_ld_max_32x32b_x32(taddr, va, ma);
                ptx::tmem_ld_max_32x32b_x32(taddr + 32, vb, mb);
                ptx::tmem_wait_ld();
                ptx::reg_fence(va);
                ptx::reg_fence(vb);
                asm volatile("" : "+f"(ma), "+f"(mb));  // the same fence for the maxima
                ptx::tc_fence_before();
                // (the wait is warp-collective: every lane's loads are complete)
                ptx::named_arrive(kBarEmpty + s, kEmptyThreads);
                s ^= 1u;
                ph ^= s ^ 1u;
                if (kProf) t_dr += tick<kProf>() - tb;
                const long long tr0 = tick<kProf>();
                const uint32_t ba = __ballot_sync(0xffffffffu, ma >= thr), bb = __ballot_sync(0xffffffffu, mb >= thr);
                if (ba | bb) {  // rare: publish records
                    ++n_rare;
                    const uint32_t na = (uint32_t)__popc(ba), cnt = na + (uint32_t)__popc(bb);
                    if (cnt > left) {
                        const long long tw = tick<kProf>();
                        next_block();
                        if (kProf) t_full += tick<kProf>() - tw;
                    }
                    const uint32_t nt1 = __float_as_uint(__fsub_rn(0.f, thr));  // thr = 0: +0, so that -0.0 passes too
                    const uint64_t nt = ptx::pack2(nt1, nt1);
                    // record: 32-position chunk, tile slot, mask over the chunk's positions
                    if (ba) ptx::st_global_v4_if(ma >= thr, p.cand + (rec + __popc(ba & lt)), chunk, slot, ge_mask(va, nt), 0u);
                    if (bb) ptx::st_global_v4_if(mb >= thr, p.cand + (rec + na + __popc(bb & lt)), chunk + 1u, slot, ge_mask(vb, nt), 0u);
                    rec += cnt;
                    left -= cnt;
                }
                if (kDump) {  // debug instantiation only: raw accumulator of some positions
                    const int col = __ldg(p.slot_col + slot);
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int64_t pa = (int64_t)chunk * 32 + i - p.dump_p0, pb = pa + 32;
                        if (col >= 0 && pa >= 0 && pa < p.dump_npos)
                            p.dump[pa * p.dump_ncols + col] = __uint_as_float(va[i]);
                        if (col >= 0 && pb >= 0 && pb < p.dump_npos)
                            p.dump[pb * p.dump_ncols + col] = __uint_as_float(vb[i]);
                    }
                }
                if (kProf) t_red += tick<kProf>() - tr0;
            }
        }
        close_block();
        __threadfence_block();
        __syncwarp();
        if (lane == 0) {
            atomicAdd(const_cast<int *>(ctl) + CTL_DONE, 1);
        }
        if (kProf && lane == 0 && warp == 0) {
            long long *pr = p.prof + 32 * blockIdx.x;
            pr[7] += t_af;
            pr[8] += tick<kProf>() - t_start;
            pr[9] += t_dr;
            pr[12] += n_rare;
            pr[13] += t_full;
            pr[15] += t_red;
        }
    }

    // ---- teardown
    __syncthreads();
    if (threadIdx.x == 0 && *s_abort) atomicOr(p.status, 1);
    if (warp == kMmaWarp) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, kAcc * kBlockPos);
    }
}

}  // namespace blamm
