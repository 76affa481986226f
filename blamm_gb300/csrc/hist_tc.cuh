// hist_tc.cuh -- empirical score histograms on the tensor cores (tcgen05 + TMEM).
//
// The counts of plain_scores_kernel<true>, window for window: a contraction gives every score
// to within a known error, which settles its bin unless the score lies that near a bin
// boundary; then the sequential FP32 sum is formed and binned as there.
//
// D = A B^T like the scan's, motifs as rows, but a tile has 64 columns and uses the 128 TMEM
// lanes twice: row r holds column r, row 64 + r the same column one position later, and B has
// every second position (an entry is the one-hot codes of bases 2i and 2i + 1, 16 bytes; row
// stride, K-core stride 16 B, k-step 32 B).  An accumulator of 256 TMEM columns then holds 512
// positions of 64 columns, and all lanes work.  Column c's P enters as hi + lo on the grids 1
// and 2^-8 after a scaling by 2^k (max|P| 2^k in (64, 128]), so sums of up to 256 positions are
// exact in FP32 and off by at most L 2^-9 from P's, in scaled units.
//
// Roles (576 threads): warps 0-15 bin what the accumulator holds (lane quarter warp % 4, 64 of
// its columns each), warp 16 makes the entries from the packed stream, warp 17 issues the MMAs
// and owns TMEM.  The counts stay in shared memory (32 bits) until the block ends.
//
// What bounds it: the issue of the binning, 19 instructions a score in all (the queue and the
// exact sums of the unsettled included: 0.8 % of the scores at 8 Mbp x 64 columns of 6-20
// positions and 250 bins), one of them a shared-memory atomic.  That case: kernel 0.39 ms under
// the profiler, call 0.51; the plain form, which is bound by one shared-memory wavefront per
// addition, 1.09 and 1.17.  With the counts column by column (the lanes' bins in random banks,
// 4.5 wavefronts an atomic) and a branch around each atomic 22 instructions, 0.49 ms.
#pragma once
#include <cstdint>

#include "ptx_sm100.cuh"
#include "scan_kernels.cuh"

namespace blamm {

constexpr int kHistCols = 64;    // columns of a tile
constexpr int kHistBlock = 512;  // positions of an accumulator
constexpr int kHistWarps = 16;   // warps that bin
constexpr int kHistThreads = 32 * (kHistWarps + 2);
constexpr int kHistStages = 3;   // blocks of entries in flight
constexpr int kHistQueue = 64;   // windows per warp waiting for their exact sums
constexpr int kHistStep = 4096;  // bytes of A per k-step and term

struct HistTcParams {
    const uint32_t *seq2, *zmask;
    int64_t n;
    const int64_t *run_start;
    int64_t nruns;
    const float *P;
    int32_t p_rows, ncols, lmax;
    const int32_t *col_len;
    const float *min_score, *width;
    const float4 *scale;  // per column: {2^k, factor and offset from scaled score to bin - 1/2, how far from it settles a bin}
    int32_t nbins, cols;  // cols: columns per tile, at most kHistCols
    unsigned long long *counts;
    int *status;
    long long wait_limit;
};

struct HistTcSmem {
    uint32_t a, e, rows, counts, queue, bars, total;
    int32_t ksteps, entries, prow;
};

// ksteps: of the shifted rows; prow: FP32 rows per column.  Counts are bin by bin, 64 columns
// each: a lane's column is its bank, whatever the bins.
__host__ __device__ inline HistTcSmem hist_tc_layout(int lmax, int nbins)
{
    HistTcSmem s;
    s.ksteps = (lmax + 1 + 3) / 4;
    s.entries = kHistBlock / 2 + 2 * s.ksteps;
    s.prow = (lmax + 3) / 4 * 4;
    uint32_t o = 0;
    auto take = [&](uint32_t bytes) {
        const uint32_t r = o;
        o += (bytes + 127) / 128 * 128;
        return r;
    };
    s.a = take((uint32_t)s.ksteps * 2 * kHistStep);
    s.e = take((uint32_t)kHistStages * s.entries * 16);
    s.rows = take((uint32_t)kHistCols * s.prow * 16);
    s.counts = take((uint32_t)kHistCols * nbins * 4);
    s.queue = take((uint32_t)kHistWarps * kHistQueue * 8);
    s.bars = take(256);
    s.total = o + 1024;
    return s;
}

// Sequential FP32 score of a window from rows in shared memory (window_score's sum: the rows
// beyond the length add +0).  row: the shared-memory address of the first row.
__device__ __forceinline__ float staged_score(const uint32_t *seq2, const uint32_t *zmask, uint32_t row, int64_t pos, int L)
{
    float s = 0.0f;
    const uint32_t *w = seq2 + (pos >> 4), *z = zmask + (pos >> 5);
    const uint32_t ws = 2u * ((uint32_t)pos & 15u), zs = (uint32_t)pos & 31u;
    for (int j = 0; j < L; j += 32, w += 2, ++z, row += 32 * 16) {
        const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
        const uint32_t use = ~__funnelshift_r(__ldg(z), __ldg(z + 1), zs);
        const uint32_t c[2] = {__funnelshift_r(w0, w1, ws), __funnelshift_r(w1, w2, ws)};
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            if (j + 4 * h >= L) break;
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = 4 * h + k, sh = 2 * (i & 15) - 2;  // (row addresses have 4 zero bits)
                const uint32_t x = sh < 0 ? c[i >> 4] << 2 : c[i >> 4] >> sh;
                v[k] = ptx::ld_shared_f32(((x & 12u) | row) + 16u * i);
                if (!((use >> i) & 1u)) v[k] = 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) s = __fadd_rn(s, v[k]);
        }
    }
    return s;
}

__global__ void __launch_bounds__(kHistThreads, 1) hist_tc_kernel(HistTcParams p)
{
    extern __shared__ uint8_t hist_raw[];
    enum { EFULL = 0, EEMPTY = EFULL + kHistStages, AFULL = EEMPTY + kHistStages, AEMPTY = AFULL + 2, DRAIN = AEMPTY + 2, BARS };
    uint8_t *smem = hist_raw + ((1024 - (ptx::smem_addr(hist_raw) & 1023)) & 1023);
    const HistTcSmem S = hist_tc_layout(p.lmax, p.nbins);
    const uint32_t sbase = ptx::smem_addr(smem), bars = sbase + S.bars;
    volatile int *ctl = reinterpret_cast<volatile int *>(smem + S.bars + 8 * BARS);  // abort flag, TMEM base
    volatile int *s_abort = ctl;
    uint32_t *H = reinterpret_cast<uint32_t *>(smem + S.counts);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int c0 = (int)blockIdx.y * p.cols, nc = min(p.cols, p.ncols - c0);
    const int64_t nblocks = (p.n + kHistBlock - 1) / kHistBlock;

    // ---- set-up: barriers, TMEM, A, the FP32 rows, counts
    if (threadIdx.x == 0) {
        ctl[0] = 0;
        for (int s = 0; s < kHistStages; ++s) {
            ptx::mbar_init(bars + 8 * (EFULL + s), 1);
            ptx::mbar_init(bars + 8 * (EEMPTY + s), 1);
        }
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(bars + 8 * (AFULL + s), 1);
            ptx::mbar_init(bars + 8 * (AEMPTY + s), kHistWarps);
        }
        ptx::mbar_init(bars + 8 * DRAIN, 1);
        ptx::fence_mbar_init();
    }
    if (warp == kHistWarps + 1) {
        ptx::tmem_alloc(sbase + S.bars + 8 * BARS + 4, 512);
        ptx::tmem_relinquish();
        ptx::tc_fence_before();
    }
    for (int i = threadIdx.x; i < kHistCols * p.nbins; i += kHistThreads) H[i] = 0u;
    for (int i = threadIdx.x; i < kHistCols * S.prow * 4; i += kHistThreads) {
        const int c = i / (S.prow * 4), r = i - c * (S.prow * 4);
        reinterpret_cast<float *>(smem + S.rows)[i] = c < nc && r < 4 * p.col_len[c0 + c] ? p.P[(size_t)(c0 + c) * p.p_rows + r] : 0.f;
    }
    // (one 4-base position of one row and both terms at a time)
    for (int i = threadIdx.x; i < S.ksteps * 4 * 128; i += kHistThreads) {
        const int row = i & 127, pos = i >> 7, c = row & 63, j = pos - (row >> 6);
        uint2 hi = make_uint2(0u, 0u), lo = hi;
        if (c < nc && j >= 0 && j < p.col_len[c0 + c]) {
            const float scale = p.scale[c0 + c].x;
            uint32_t h[4], l[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float x = p.P[(size_t)(c0 + c) * p.p_rows + 4 * j + b] * scale, q = rintf(x);
                h[b] = __float_as_uint(q) >> 16;                                  // whole numbers up to 128: exact in BF16
                l[b] = __float_as_uint(rintf((x - q) * 256.0f) * 0x1p-8f) >> 16;  // (x - q is exact)
            }
            hi = make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
            lo = make_uint2(l[0] | l[1] << 16, l[2] | l[3] << 16);
        }
        uint8_t *at = smem + S.a + (pos >> 2) * kHistStep + (16 * ((pos >> 1) & 1) + row / 8) * 128 + (row % 8) * 16 + 8 * (pos & 1);
        *reinterpret_cast<uint2 *>(at) = hi;
        *reinterpret_cast<uint2 *>(at + S.ksteps * kHistStep) = lo;
    }
    ptx::fence_proxy_async_smem();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = (uint32_t)ctl[1];

    if (warp == kHistWarps + 1) {
        // ============ MMAs ============
        const uint64_t adesc = ptx::smem_desc(sbase + S.a, 2048u, 128u);
        const uint64_t bdesc = ptx::smem_desc(sbase + S.e, 16u, 128u);
        constexpr uint32_t idesc = ptx::idesc_bf16_f32(128, 256);
        constexpr uint32_t kStep16 = kHistStep / 16;
        uint32_t es = 0, eph = 0, job = 0;
        bool ok = true;
        for (int64_t b = blockIdx.x; b < nblocks && ok; b += gridDim.x, ++job) {
            const uint32_t s = job & 1u;
            if (job >= 2u) ok = ptx::mbar_wait(bars + 8 * (AEMPTY + s), ((job >> 1) - 1u) & 1u, s_abort, p.wait_limit);
            ok = ok && ptx::mbar_wait(bars + 8 * (EFULL + es), eph, s_abort, p.wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t d = tmem + 256u * s;
            const uint64_t bd = bdesc + es * (uint32_t)S.entries;
            for (uint32_t k = 0; k < (uint32_t)S.ksteps; ++k) {
                ptx::mma_bf16_elect(d, adesc + k * kStep16, bd + 2u * k, idesc, k != 0u);
                ptx::mma_bf16_elect(d, adesc + (S.ksteps + k) * kStep16, bd + 2u * k, idesc, 1u);
            }
            ptx::mma_commit_elect(bars + 8 * (EEMPTY + es));
            ptx::mma_commit_elect(bars + 8 * (AFULL + s));
            if (++es == (uint32_t)kHistStages) {
                es = 0;
                eph ^= 1u;
            }
        }
        // nothing may still read shared memory or write TMEM when they are freed
        ptx::mma_commit_elect(bars + 8 * DRAIN);
        if (!ptx::mbar_wait_drain(bars + 8 * DRAIN, 0, p.wait_limit)) *s_abort = 1;
    } else if (warp == kHistWarps) {
        // ============ one-hot entries of a block ============
        uint32_t es = 0, eph = 0;
        for (int64_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
            const bool ok = ptx::mbar_wait(bars + 8 * (EEMPTY + es), eph ^ 1u, s_abort, p.wait_limit);
            if (!__all_sync(0xffffffffu, ok)) break;
            const int64_t i0 = b * (kHistBlock / 2);  // first entry: a multiple of 256
            uint4 *e = reinterpret_cast<uint4 *>(smem + S.e) + es * S.entries;
            for (int i = lane; i < S.entries; i += 32) {
                const uint32_t c = __ldg(p.seq2 + ((i0 + i) >> 3)) >> (4 * (i & 7));
                const uint32_t z = __ldg(p.zmask + ((i0 + i) >> 4)) >> (2 * (i & 15));
                const uint2 x = onehot_bf16(c & 3u, z & 1u), y = onehot_bf16((c >> 2) & 3u, z & 2u);
                e[i] = make_uint4(x.x, x.y, y.x, y.y);
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bars + 8 * (EFULL + es));
            if (++es == (uint32_t)kHistStages) {
                es = 0;
                eph ^= 1u;
            }
        }
    } else {
        // ============ bins ============
        const int q = warp & 3, grp = warp >> 2, row = 32 * q + lane, c = row & 63, shift = row >> 6;
        const bool act = c < nc;
        const bool warp_act = __any_sync(0xffffffffu, act);
        const int col = c0 + (act ? c : 0);
        const int L = p.col_len[col];
        const float4 sc = p.scale[col];
        const float mn = p.min_score[col], wd = p.width[col], rcp = __frcp_rn(wd);
        const uint64_t fac = ptx::pack2(__float_as_uint(sc.y), __float_as_uint(sc.y));
        const uint64_t off = ptx::pack2(__float_as_uint(sc.z), __float_as_uint(sc.z));
        constexpr uint32_t kMagic = 0x4B400000u;  // 1.5 2^23: adding it rounds to a whole number
        const uint64_t magic = ptx::pack2(kMagic, kMagic), nmagic = ptx::pack2(kMagic | 0x80000000u, kMagic | 0x80000000u);
        const uint64_t minus1 = ptx::pack2(0xBF800000u, 0xBF800000u);
        const float lim = sc.w;
        const int top = p.nbins - 1;
        uint32_t *Hc = H + c;
        const uint32_t lt = (1u << lane) - 1u;
        uint2 *queue = reinterpret_cast<uint2 *>(smem + S.queue) + warp * kHistQueue;
        const uint32_t rows = sbase + S.rows;
        int nq = 0;
        // the first n (at most 32) windows of the queue: their sums as the plain form makes them
        auto exact = [&](int n) {
            __syncwarp();
            const uint2 e = queue[lane < n ? lane : 0];
            const int qc = (int)(e.y >> 1);  // (the warp's columns: their values are other lanes')
            const int from = qc & 31;
            const int ql = __shfl_sync(0xffffffffu, L, from);
            const float qm = __shfl_sync(0xffffffffu, mn, from), qw = __shfl_sync(0xffffffffu, wd, from);
            const float qr = __shfl_sync(0xffffffffu, rcp, from);
            if (lane < n) {
                const int64_t pos = 2 * (int64_t)e.x + (e.y & 1u);
                const float s = staged_score(p.seq2, p.zmask, rows + (uint32_t)(qc * S.prow * 16), pos, ql);
                const int b = max(0, min(p.nbins - 1, bin_of(__fsub_rn(s, qm), qw, qr)));
                atomicAdd(&H[b * kHistCols + qc], 1u);
            }
            __syncwarp();
        };
        // 32 scores of a lane: windows at 2 (i0 + i) + shift; rem: bases to the run's end for i = lane
        auto bin = [&](const uint32_t (&v)[32], uint32_t i0, bool all, int rem) {
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                // t: bin - 1/2; u: t rounded to the bin; f: the distance from the bin's middle
                const uint64_t t = ptx::fma_f32x2(ptx::pack2(v[i], v[i + 1]), fac, off), uu = ptx::add_f32x2(t, magic);
                uint32_t u[2], f[2];
                ptx::unpack2(uu, u[0], u[1]);
                ptx::unpack2(ptx::fma_f32x2(ptx::add_f32x2(uu, nmagic), minus1, t), f[0], f[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const bool in = all || L <= __shfl_sync(0xffffffffu, rem, i + h);
                    const bool settled = fabsf(__uint_as_float(f[h])) < lim;
                    // (no branch: what does not count here adds 0)
                    atomicAdd(Hc + kHistCols * __vimin_s32_relu((int)(u[h] - kMagic), top), act && in && settled ? 1u : 0u);
                    if (in && !settled) m |= 1u << (i + h);
                }
            }
            if (!act) m = 0;
            for (uint32_t b; (b = __ballot_sync(0xffffffffu, m != 0u)) != 0u;) {
                if (m) queue[nq + __popc(b & lt)] = make_uint2(i0 + (uint32_t)(__ffs(m) - 1), (uint32_t)(2 * c + shift));
                m &= m - 1u;
                nq += __popc(b);
                if (nq >= 32) {
                    exact(32);
                    nq -= 32;
                    const uint2 e = queue[32 + lane];
                    __syncwarp();
                    if (lane < nq) queue[lane] = e;
                    __syncwarp();
                }
            }
        };
        int64_t end = blockIdx.x < nblocks ? run_end_of(p.run_start, p.nruns, p.n, blockIdx.x * (int64_t)kHistBlock) : 0;
        uint32_t job = 0;
        for (int64_t b = blockIdx.x; b < nblocks; b += gridDim.x, ++job) {
            const uint32_t s = job & 1u;
            const int64_t i0 = b * (kHistBlock / 2) + 64 * grp, p0 = b * kHistBlock;
            const bool all = p0 + kHistBlock - 1 + p.lmax <= end;  // every window of the block is inside its run
            const int64_t next = p0 + (int64_t)gridDim.x * kHistBlock;
            if (next < p.n) end = run_end_of(p.run_start, p.nruns, p.n, next);
            const bool ok = ptx::mbar_wait_nohint(bars + 8 * (AFULL + s), (job >> 1) & 1u, s_abort, p.wait_limit);
            if (!__all_sync(0xffffffffu, ok)) break;
            ptx::tc_fence_after();
            const uint32_t taddr = tmem + 256u * s + ((uint32_t)(32 * q) << 16) + 64u * grp;
            uint32_t v[32];
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                if (warp_act) {
                    ptx::tmem_ld_32x32b_x32(taddr + 32u * half, v);
                    ptx::tmem_wait_ld();
                    ptx::reg_fence(v);
                }
                if (half == 1) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(bars + 8 * (AEMPTY + s));
                }
                if (!warp_act) continue;
                if (all) {
                    bin(v, (uint32_t)(i0 + 32 * half), true, 0);
                } else {
                    const int64_t pos = 2 * (i0 + 32 * half + lane) + shift;
                    const int64_t left = pos < p.n ? run_end_of(p.run_start, p.nruns, p.n, pos) - pos : 0;
                    bin(v, (uint32_t)(i0 + 32 * half), false, (int)min(left, (int64_t)kMaxMotifLen));
                }
            }
        }
        if (nq) exact(nq);
    }

    // ---- teardown
    ptx::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *s_abort) atomicOr(p.status, 1);
    for (int i = threadIdx.x; i < nc * p.nbins; i += kHistThreads) {
        const int c = i / p.nbins, b = i - c * p.nbins;
        const uint32_t x = H[b * kHistCols + c];
        if (x) atomicAdd(&p.counts[(size_t)(c0 + c) * p.nbins + b], (unsigned long long)x);
    }
    if (warp == kHistWarps + 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
}

}  // namespace blamm
