// scan_kernels.cuh -- SIMT device code of the GB300 PWM scan: stream packing,
// the plain FP32 scan, empirical histograms, candidate rescoring and the
// reference-compatible threshold filter.  The tensor-core scan is scan_tc.cuh.
//
// Data layout in HBM (one species' filtered base stream of n positions):
//   seq2[]  : 2-bit base codes, 16 per uint32 (A=0 C=1 G=2 T=3), base i at
//             bits 2*(i%16) of word i/16;
//   zmask[] : 1 bit per base, bit i%32 of word i/32 set when the base adds
//             nothing to a score (lowercase, or past the end of the stream);
//   both padded by kStreamPad bases so that tile loads need no bounds checks.
// Motif bank: the reference's column-major FP32 P (4*Lmax rows), per-column
// lengths and thresholds.
#pragma once
#include <cstdint>
#include <type_traits>

#include "blamm_gpu.h"

#include "ptx_sm100.cuh"

namespace blamm {

constexpr int kStreamPad = 2048;   // padding bases after the stream end
constexpr int kMaxMotifLen = BLAMM_MAX_MOTIF_LEN;  // the plain kernel reads up to 255 + L bases past a block
constexpr int kColBits = 20;       // a bank has fewer than 2^20 columns

// ------------------------------------------------------------------------
// helpers
// ------------------------------------------------------------------------
// Sequential FP32 score of the window at pos (motif position order, __fadd_rn: the
// reference's sum), zero-masked bases adding nothing (adding +0 changes no sum that starts
// at +0).  The 2-bit codes and mask bits of 16 positions come from two words of each array
// (the padded stream covers the reads); the P values of 8 positions are loaded together, so
// their latencies overlap (2.9 M candidates over 16 Mi positions and 1024 columns: 0.167 ms
// with one load at a time, each behind the last one's branch, 0.149 with 8 together).
__device__ __forceinline__ float window_score(const uint32_t *seq2, const uint32_t *zmask, const float *pc,
                                              int64_t pos, int L)
{
    float s = 0.0f;
    for (int j = 0; j < L; j += 16) {
        const int64_t q = pos + j;
        const int64_t w = q >> 4, wz = q >> 5;
        const uint64_t cw = (uint64_t)__ldg(seq2 + w) | ((uint64_t)__ldg(seq2 + w + 1) << 32);
        const uint64_t zw = (uint64_t)__ldg(zmask + wz) | ((uint64_t)__ldg(zmask + wz + 1) << 32);
        uint32_t codes = (uint32_t)(cw >> (2 * (q & 15)));
        uint32_t use = ~(uint32_t)(zw >> (q & 31));
        if (L - j < 16) use &= (1u << (L - j)) - 1u;
        const float *pj = pc + 4 * j;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && L - j <= 8) break;
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                v[k] = (use >> (8 * h + k)) & 1u ? __ldg(pj + 4 * (8 * h + k) + ((codes >> (2 * (8 * h + k))) & 3u)) : 0.0f;
#pragma unroll
            for (int k = 0; k < 8; ++k) s = __fadd_rn(s, v[k]);
        }
    }
    return s;
}

// end (exclusive) of the run that contains position p
__device__ __forceinline__ int64_t run_end_of(const int64_t *run_start, int64_t nruns, int64_t n,
                                              int64_t p)
{
    int64_t lo = 0, hi = nruns;  // first run_start > p
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (__ldg(run_start + mid) <= p) lo = mid + 1;
        else hi = mid;
    }
    return lo < nruns ? __ldg(run_start + lo) : n;
}

// Times of a synchronous scan's kernels, in ns of the device's clock, each noted by one thread of a
// kernel as it begins: [0] the first preparation, [1] the scan kernels' times added up (a scan lasts
// until the next kernel begins), [2] the current scan kernel, [3] the rescoring.  (An event between
// two kernels costs a short call 2 to 7 us; these cost nothing.)
__device__ __forceinline__ void note_scan_end(unsigned long long *times)
{
    times[1] += ptx::global_ns() - times[2];
}

// ------------------------------------------------------------------------
// 1. prepare: filtered ASCII bases -> 2-bit codes + zero mask, and the one-hot entries of a
//    scan window
// ------------------------------------------------------------------------
// One-hot entries for the tensor-core scan: E[i] = onehot(base i) ++ onehot(base i+1),
// 4 bf16 channels per base (1.0 = 0x3F80 in channel code, zeros for a zero-masked base).
__device__ __forceinline__ uint2 onehot_bf16(uint32_t code, uint32_t zero)
{
    const uint32_t h = zero ? 0u : (0x3F80u << ((code & 1u) << 4));
    return make_uint2((code & 2u) ? 0u : h, (code & 2u) ? h : 0u);
}

// E4M3 one-hot of one base: byte `code` of the 4 is 1.0 (0x38), zeros for a zero-masked base.
__device__ __forceinline__ uint32_t onehot_e4m3(uint32_t code, uint32_t zero)
{
    return zero ? 0u : 0x38u << (8 * code);
}

// 0x80 in every byte of x that is zero (exact, no borrow between bytes)
__device__ __forceinline__ uint32_t zero_bytes(uint32_t x)
{
    return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
}

// 0x80 in every byte that is one of ACGTacgt: bits 1-2 of a base name the only letter it can be
__device__ __forceinline__ uint32_t base_bytes(uint32_t x)
{
    const uint32_t c = (x >> 1) & 0x03030303u;      // A 0, C 1, T 2, G 3
    const uint32_t t = (c | c >> 4) & 0x00ff00ffu;  // two nibbles per 16 bits
    return zero_bytes((x & 0xDFDFDFDFu) ^ __byte_perm(0x47544341u, 0u, t | t >> 8));
}

struct PrepParams {
    const char *bases;
    int64_t n;           // stream positions (beyond them: zero-masked)
    int64_t base;        // the window's first position (a multiple of 32)
    int64_t pack_end;    // positions [base, pack_end) are packed (a multiple of 32)
    uint32_t *seq2, *zmask;
    int64_t ne;          // entries of positions base .. base + ne - 1
    uint4 *e;
    int32_t lower_scores;
    uint32_t zero;       // bit i: counts[i] = 0
    unsigned long long *counts;
    unsigned long long *times;  // may be null
    int32_t first;       // the scan's first window
};

constexpr int kPrepThreads = 256;
constexpr int kPrepTile = 16 * kPrepThreads;  // positions per block, 16 per thread

// The packed form of 16 bases from position p on: 2-bit codes, zero mask (16 bits).
__device__ __forceinline__ uint2 prep_pack16(const PrepParams &a, int64_t p)
{
    uint32_t w[4];
    if (p + 16 <= a.n) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(a.bases + p);
        if ((at & 15u) == 0) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(at));
            w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        } else {  // aligned words that hold these bytes (the last one only where it does)
            const uint32_t *q = reinterpret_cast<const uint32_t *>(at & ~(uintptr_t)3);
            const uint32_t s = 8u * (uint32_t)(at & 3u);
            uint32_t x[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) x[k] = k < 4 || s ? __ldg(q + k) : 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(x[k], x[k + 1], s);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[k] = 0u;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (p + 4 * k + b < a.n) w[k] |= (uint32_t)(unsigned char)a.bases[p + 4 * k + b] << (8 * b);
        }
    }
    uint32_t codes = 0, zero = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t x = w[k];
        // A/a=0 C/c=1 G/g=2 T/t=3, four bytes to eight bits by a dot product with 1, 4, 16, 64
        codes |= __dp4a(((x >> 1) ^ (x >> 2)) & 0x03030303u, 0x40100401u, 0u) << (8 * k);
        uint32_t z = ~base_bytes(x) & 0x80808080u;
        if (!a.lower_scores) z |= (x << 2) & 0x80808080u;  // lowercase
        zero |= (__dp4a(z, 0x08040201u, 0u) >> 7) << (4 * k);
    }
    return make_uint2(codes, zero);
}

// kForm: 0 packs only; 1 also writes BF16 entries (E[i] = bases i, i + 1), 8 E4M3 entries
// (bases i .. i + 3).  A thread packs 16 positions from one 16-byte load; the entries are then
// written from the block's codes in shared memory, consecutive threads consecutive entries.
// Bound by the 17.4 bytes per position that move: 100 Mbp in 16 Mi windows 0.26 ms; separate
// passes (bytes one by one to codes, codes to entries) took 0.54.
template <int kForm>
__global__ void __launch_bounds__(kPrepThreads) prep_kernel(PrepParams a)
{
    __shared__ uint32_t s_code[kPrepThreads + 1], s_zero[kPrepThreads + 1];
    if (blockIdx.x == 0 && threadIdx.x < 4 && ((a.zero >> threadIdx.x) & 1u)) a.counts[threadIdx.x] = 0ull;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.times) {
        if (a.first) {
            a.times[0] = ptx::global_ns();
            a.times[1] = 0ull;
        } else {
            note_scan_end(a.times);
        }
    }
    const int64_t tile = a.base + (int64_t)blockIdx.x * kPrepTile;
    const int64_t p = tile + threadIdx.x * 16;
    const uint2 v = prep_pack16(a, p);
    const uint32_t next = __shfl_down_sync(0xffffffffu, v.y, 1);
    if (p < a.pack_end) {
        a.seq2[p >> 4] = v.x;
        if (!(threadIdx.x & 1)) a.zmask[p >> 5] = v.y | next << 16;
    }
    if (kForm == 0) return;
    s_code[threadIdx.x] = v.x;
    s_zero[threadIdx.x] = v.y;
    if (threadIdx.x == 0) {  // the bases after the block
        const uint2 h = prep_pack16(a, tile + kPrepTile);
        s_code[kPrepThreads] = h.x;
        s_zero[kPrepThreads] = h.y;
    }
    __syncthreads();
    uint4 *e = a.e + (tile - a.base);
    const int64_t left = a.ne - (tile - a.base);
#pragma unroll 4
    for (int k = 0; k < 16; ++k) {
        const int i = k * kPrepThreads + threadIdx.x, w = i >> 4;
        if (i >= left) break;
        const uint32_t c = __funnelshift_r(s_code[w], s_code[w + 1], 2 * (i & 15));
        const uint32_t z = (s_zero[w] | s_zero[w + 1] << 16) >> (i & 15);
        if (kForm == 8) {
            e[i] = make_uint4(onehot_e4m3(c & 3u, z & 1u), onehot_e4m3((c >> 2) & 3u, z & 2u),
                              onehot_e4m3((c >> 4) & 3u, z & 4u), onehot_e4m3((c >> 6) & 3u, z & 8u));
        } else {
            const uint2 x = onehot_bf16(c & 3u, z & 1u), y = onehot_bf16((c >> 2) & 3u, z & 2u);
            e[i] = make_uint4(x.x, x.y, y.x, y.y);
        }
    }
}

// ------------------------------------------------------------------------
// 2. plain FP32 scores: one thread per position, sequential FP32 sums
//    (the straightforward GPU form of PWMScan::scanThreadBLAS + extractOccurrences),
//    ending in hits (2a) or in empirical score histograms (2b: Histogram::histThread /
//    extractObsScore, hist.cpp:70-140)
// ------------------------------------------------------------------------
// A block keeps some columns' P in shared memory, four columns side by side, and walks over
// tiles of 256 positions.  A thread turns the 32 bases from its position on into byte
// offsets once and uses them for all the columns: a motif position of four columns is one
// 16-byte load at (offset, column group) and four additions.  The lanes of a warp read at
// most five different rows of one motif position, which shared memory serves as a broadcast.
// Row 4 is zero (masked bases), and so are the rows beyond a column's length: adding +0
// changes no sum that starts at +0.
// What bounds it: shared memory, which delivers 128 bytes a cycle and SM whatever the lanes
// share (a 16-byte load of a warp is four cycles): 32 additions a cycle and SM.  2 Mbp x 256
// columns: 1.02 ms, 0.93 at that rate (one 4-byte load at a byte-coded address, a branch and an
// addition per motif position: 2.91); 8 Mbp x 64 columns with 250 bins: 1.09 (2.57 with a
// division per score).  Banks of some dozen columns on longer streams are binned by hist_tc_kernel.
// Motif positions from 32 on take their codes from two words per 32 bases, for each column group
// anew (10 Mbp x 4 columns of 100-130 positions 0.65 ms; with two loads per position 1.30; with
// byte codes in shared memory 1.22), and a group of one or two columns loads 4 or 8 bytes (10 Mbp x
// 1 column of 12: 0.110 ms, 0.149 with 16, 0.123 in the byte-coded form; that is still ahead for one
// column of more than 32 positions, 0.20 against 0.18 ms with 40-60).
constexpr int kPlainThreads = 256;
constexpr int kPlainReg = 32;  // motif positions whose offsets are kept in registers
constexpr int kPlainRow = 5 * 16;  // bytes of one motif position of four columns

struct PlainParams {
    const uint32_t *seq2;
    const uint32_t *zmask;
    int64_t n;
    const int64_t *run_start;
    int64_t nruns;
    const float *P;
    int32_t p_rows;
    int32_t ncols;
    int32_t cols_per_block;  // a multiple of 4
    int32_t lmax;
    const int32_t *col_len;
    const int32_t *cols;  // the ncols bank columns to scan (nullptr: columns 0 .. ncols-1)
    // hits
    const float *thr;
    void *hits;  // blamm_hit*
    unsigned long long *hit_count;
    int64_t hit_cap;
    int64_t keep_below;  // hits at positions >= keep_below are dropped (0: none are)
    int64_t pos_base;    // added to the positions written
    // histograms
    const float *min_score;
    const float *width;
    int32_t nbins;
    int32_t shared_bins;         // 1: the block's counts are in shared memory until it ends
    unsigned long long *counts;  // ncols x nbins
};

// The 32 bases from a position on: codes and zero mask; row16: 16 times the row of one of them.
struct PlainCodes {
    uint32_t code[2], zero;
    __device__ __forceinline__ uint32_t row16(int i) const
    {
        const int sh = 2 * (i & 15) - 4;
        const uint32_t c = (sh < 0 ? code[i >> 4] << -sh : code[i >> 4] >> sh) & 0x30u;
        return (zero >> i) & 1u ? 0x40u : c;
    }
};
__device__ __forceinline__ PlainCodes plain_codes(const uint32_t *seq2, const uint32_t *zmask, int64_t pos)
{
    const int64_t w = pos >> 4, wz = pos >> 5;
    const uint32_t s = 2 * (uint32_t)(pos & 15);
    const uint32_t w0 = __ldg(seq2 + w), w1 = __ldg(seq2 + w + 1), w2 = __ldg(seq2 + w + 2);
    PlainCodes c;
    c.code[0] = __funnelshift_r(w0, w1, s);
    c.code[1] = __funnelshift_r(w1, w2, s);
    c.zero = __funnelshift_r(__ldg(zmask + wz), __ldg(zmask + wz + 1), (uint32_t)(pos & 31));
    return c;
}

struct alignas(16) HitRec {
    int64_t pos;
    int32_t col;
    float score;
};

__device__ __forceinline__ void emit_hits_warp(bool hit, int64_t pos, int32_t col, float score,
                                               HitRec *hits, unsigned long long *count,
                                               int64_t cap)
{
    unsigned m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    if (hit) {
        unsigned long long idx = base + __popc(m & ((1u << lane) - 1u));
        if ((int64_t)idx < cap) {
            HitRec h;
            h.pos = pos;
            h.col = col;
            h.score = score;
            hits[idx] = h;
        }
    }
}

// Shared memory of a block: P, then per column its length and three values (threshold; or least
// score, bin width and its reciprocal), then the counts of a histogram.
__host__ __device__ inline size_t plain_smem_bytes(int cols, int lmax, int bins)
{
    return (size_t)(cols / 4) * lmax * kPlainRow + (size_t)cols * 16 + (size_t)cols * bins * 4;
}

// (int)(x / w) with the division rounded to nearest, as the reference bins a score: from the
// product with the reciprocal (r) unless that is so near an integer that the two could fall on
// different sides (relative error of product and quotient below 2^-22 together; r is NaN
// where the reciprocal would not be that accurate, and then the division decides).
__device__ __forceinline__ int bin_of(float x, float w, float r)
{
    const float f = __fmul_rn(x, r);
    const float near = fabsf(__fsub_rn(f, rintf(f)));
    int b = (int)f;
    if (!(near > fabsf(f) * 0x1p-21f)) b = (int)__fdiv_rn(x, w);
    return b;
}

template <bool kHist>
__global__ void __launch_bounds__(kPlainThreads, 4) plain_scores_kernel(PlainParams p)
{
    extern __shared__ __align__(16) uint8_t smem_plain[];
    const int cpb = p.cols_per_block, ngrp = cpb / 4, lmax = p.lmax;
    float *sP = reinterpret_cast<float *>(smem_plain);
    int32_t *sLen = reinterpret_cast<int32_t *>(smem_plain + (size_t)ngrp * lmax * kPlainRow);
    float *sA = reinterpret_cast<float *>(sLen + cpb), *sB = sA + cpb, *sR = sB + cpb;
    uint32_t *sH = reinterpret_cast<uint32_t *>(sR + cpb);
    const int c0 = blockIdx.y * cpb;
    const int nc = min(cpb, p.ncols - c0);
    auto bank = [&](int i) { return p.cols ? p.cols[c0 + i] : c0 + i; };
    for (int i = threadIdx.x; i < cpb; i += kPlainThreads) {
        const int col = i < nc ? bank(i) : -1;
        sLen[i] = col < 0 ? 0 : p.col_len[col];
        sA[i] = col < 0 ? 0.f : kHist ? p.min_score[col] : p.thr[col];
        if (kHist) {
            const float w = sB[i] = col < 0 ? 1.f : p.width[col];
            sR[i] = fabsf(w) > 0x1p-100f && fabsf(w) < 0x1p100f ? __frcp_rn(w) : __int_as_float(0x7fffffff);
        }
    }
    if (kHist && p.shared_bins)
        for (int i = threadIdx.x; i < cpb * p.nbins; i += kPlainThreads) sH[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < cpb * lmax * 5; i += kPlainThreads) {
        const int c = i / (lmax * 5), r = i - c * (lmax * 5), j = r / 5, b = r - j * 5;
        const float v = b < 4 && j < sLen[c] ? p.P[(size_t)bank(c) * p.p_rows + 4 * j + b] : 0.f;
        sP[((size_t)(c / 4) * lmax + j) * 20 + b * 4 + (c & 3)] = v;
    }
    __syncthreads();
    const uint32_t base = ptx::smem_addr(smem_plain);
    const int64_t ntiles = (p.n + kPlainThreads - 1) / kPlainThreads;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t pos = tile * kPlainThreads + threadIdx.x;
        const int64_t end = pos < p.n ? run_end_of(p.run_start, p.nruns, p.n, pos) : pos;
        const int rem = (int)min(end - pos, (int64_t)kMaxMotifLen);  // bases from here to the run's end
        // offsets of the 32 bases from pos on (the padded stream covers the reads)
        uint32_t off[kPlainReg];
        {
            const PlainCodes c = plain_codes(p.seq2, p.zmask, pos);
#pragma unroll
            for (int j = 0; j < kPlainReg; ++j) {
                if ((j & 3) == 0 && j >= lmax) break;
                off[j] = base + (uint32_t)(j * kPlainRow) + c.row16(j);
            }
        }
        for (int g = 0; g < ngrp; ++g) {
            const int4 len = reinterpret_cast<const int4 *>(sLen)[g];
            const int L = max(max(len.x, len.y), max(len.z, len.w));
            const uint32_t at = (uint32_t)(g * lmax * kPlainRow);
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            // (W: the group's columns that exist, 1, 2 or more; less is loaded for fewer)
            auto scores = [&](auto W) {
                auto add = [&](uint32_t a) {
                    if constexpr (decltype(W)::value == 1) {
                        s.x = __fadd_rn(s.x, ptx::ld_shared_f32(a));
                    } else if constexpr (decltype(W)::value == 2) {
                        const float2 v = ptx::ld_shared_v2(a);
                        s.x = __fadd_rn(s.x, v.x);
                        s.y = __fadd_rn(s.y, v.y);
                    } else {
                        const float4 v = ptx::ld_shared_v4(a);
                        s.x = __fadd_rn(s.x, v.x);
                        s.y = __fadd_rn(s.y, v.y);
                        s.z = __fadd_rn(s.z, v.z);
                        s.w = __fadd_rn(s.w, v.w);
                    }
                };
#pragma unroll
                for (int j = 0; j < kPlainReg; j += 4) {
                    if (j >= L) break;
                    add(off[j] + at);
                    if (j + 1 < L) add(off[j + 1] + at);
                    if (j + 2 < L) add(off[j + 2] + at);
                    if (j + 3 < L) add(off[j + 3] + at);
                }
                // longer motifs: 32 bases at a time, offsets made for this group
                for (int j0 = kPlainReg; j0 < L; j0 += 32) {
                    const PlainCodes c = plain_codes(p.seq2, p.zmask, pos + j0);
                    const uint32_t row = base + at + (uint32_t)(j0 * kPlainRow);
                    const int left = L - j0;
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        if (i >= left) break;
                        add(row + (uint32_t)(i * kPlainRow) + c.row16(i));
                        if (i + 1 < left) add(row + (uint32_t)((i + 1) * kPlainRow) + c.row16(i + 1));
                        if (i + 2 < left) add(row + (uint32_t)((i + 2) * kPlainRow) + c.row16(i + 2));
                        if (i + 3 < left) add(row + (uint32_t)((i + 3) * kPlainRow) + c.row16(i + 3));
                    }
                }
            };
            const int width = nc - 4 * g;
            if (width > 2) scores(std::integral_constant<int, 4>());
            else if (width == 2) scores(std::integral_constant<int, 2>());
            else scores(std::integral_constant<int, 1>());
            const float sc[4] = {s.x, s.y, s.z, s.w};
            const int ln[4] = {len.x, len.y, len.z, len.w};
            if (kHist) {
                const float4 lo = reinterpret_cast<const float4 *>(sA)[g], wd = reinterpret_cast<const float4 *>(sB)[g];
                const float4 rc = reinterpret_cast<const float4 *>(sR)[g];
                const float ls[4] = {lo.x, lo.y, lo.z, lo.w}, ws[4] = {wd.x, wd.y, wd.z, wd.w};
                const float rs[4] = {rc.x, rc.y, rc.z, rc.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (ln[k] == 0 || ln[k] > rem) continue;
                    const int b = max(0, min(p.nbins - 1, bin_of(__fsub_rn(sc[k], ls[k]), ws[k], rs[k])));
                    if (p.shared_bins) atomicAdd(&sH[(4 * g + k) * p.nbins + b], 1u);
                    else atomicAdd(&p.counts[(size_t)(c0 + 4 * g + k) * p.nbins + b], 1ull);
                }
            } else {
                const float4 th = reinterpret_cast<const float4 *>(sA)[g];
                const float ts[4] = {th.x, th.y, th.z, th.w};
                const bool keep = p.keep_below == 0 || pos < p.keep_below;
                bool hit[4], any = false;
#pragma unroll
                for (int k = 0; k < 4; ++k) any |= hit[k] = ln[k] > 0 && ln[k] <= rem && sc[k] >= ts[k] && keep;
                if (__any_sync(0xffffffffu, any)) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        emit_hits_warp(hit[k], pos + p.pos_base, 4 * g + k < nc ? bank(4 * g + k) : 0, sc[k],
                                       reinterpret_cast<HitRec *>(p.hits), p.hit_count, p.hit_cap);
                }
            }
        }
    }
    if (kHist && p.shared_bins) {
        __syncthreads();
        for (int i = threadIdx.x; i < nc * p.nbins; i += kPlainThreads)
            if (sH[i]) atomicAdd(&p.counts[(size_t)c0 * p.nbins + i], (unsigned long long)sH[i]);
    }
}

// ------------------------------------------------------------------------
// 3. rescoring of tensor-core candidates: run check + exact FP32 score
// ------------------------------------------------------------------------
// Candidates come as 16-byte records {chunk, slot, mask, 0}: bit i of mask = position
// 32 chunk + i is a candidate of the tile slot's motif column.  The scan writes them in
// blocks of kRecBlockSlots slots; slot 0 of a block holds the number of records that follow
// it (the rest of the block is unused).
constexpr int kRecBlockSlots = 128;

// A chunk's positions before the end of the stream (those behind it are no candidates).
__device__ __forceinline__ uint32_t valid_positions(int64_t n, uint32_t chunk)
{
    const int64_t room = n - (int64_t)chunk * 32;
    return room >= 32 ? 0xffffffffu : room > 0 ? (1u << room) - 1u : 0u;
}

struct RescoreParams {
    const uint4 *cand;                // record slots
    const int32_t *slot_col;          // tile slot -> motif column
    const unsigned long long *cand_count;  // record slots reserved
    int64_t cand_cap;                 // record slots available
    const uint32_t *seq2;
    const uint32_t *zmask;
    int64_t n;
    const int64_t *run_start;
    int64_t nruns;
    const float *P;
    int32_t p_rows;
    const int32_t *col_len;
    const float *thr;
    void *hits;
    unsigned long long *hit_count;
    unsigned long long *ncand;  // candidates (set mask bits), added up (the scan adds those of records that did not fit)
    int64_t hit_cap;
    int64_t keep_below;  // hits at positions >= keep_below are dropped (0: none are)
    int64_t pos_base;    // added to the positions written
    unsigned long long *times;  // may be null
};

// One thread per record slot; the candidates of a warp's 32 records are then shared out
// over its lanes (a prefix sum of the masks' bit counts), 32 at a time, so that a record
// with several candidates does not leave the other lanes idle.  A warp gathers its hits in
// shared memory and reserves room for about a hundred of them with one atomic: the atomics
// on the one counter are serial, about 1.1 ns each.
constexpr int kRescoreThreads = 256;
constexpr int kRescoreBuf = 128;  // hits a warp gathers (flushed before a round could overflow it)

__global__ void __launch_bounds__(kRescoreThreads) rescore_kernel(RescoreParams p)
{
    unsigned long long ns = *p.cand_count;
    if ((int64_t)ns > p.cand_cap) ns = (unsigned long long)p.cand_cap;
    __shared__ HitRec s_hits[kRescoreThreads / 32][kRescoreBuf];
    __shared__ unsigned int s_cand;
    if (threadIdx.x == 0) s_cand = 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.times) {
        note_scan_end(p.times);
        p.times[3] = ptx::global_ns();
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    HitRec *buf = s_hits[threadIdx.x >> 5];
    int nbuf = 0;
    auto flush = [&]() {
        __syncwarp();
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(p.hit_count, (unsigned long long)nbuf);
        at = __shfl_sync(0xffffffffu, at, 0);
        const uint4 *from = reinterpret_cast<const uint4 *>(buf);
        uint4 *to = reinterpret_cast<uint4 *>(p.hits);
        for (int k = lane; k < nbuf; k += 32)
            if ((int64_t)(at + k) < p.hit_cap) to[at + k] = from[k];
        __syncwarp();
        nbuf = 0;
    };
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned int my_cand = 0;
    for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < ns; base += stride) {
        const unsigned long long i = base + threadIdx.x;
        uint32_t mask = 0u, chunk = 0u, slot = 0u;
        const unsigned long long b = i & ~(unsigned long long)(kRecBlockSlots - 1);
        const uint32_t k = (uint32_t)(i & (kRecBlockSlots - 1));
        if (i < ns && k != 0u && k <= __ldg(&p.cand[b].x)) {
            const uint4 r = p.cand[i];
            chunk = r.x;
            slot = r.y;
            mask = r.z;
            mask &= valid_positions(p.n, chunk);
        }
        const int c = __popc(mask);
        my_cand += (unsigned int)c;
        int incl = c;  // inclusive prefix sum of the lanes' candidate counts
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int t0 = 0; t0 < total; t0 += 32) {
            const int t = t0 + lane;
            // the lane r whose record holds candidate t: the first with incl[r] > t
            int r = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int v = __shfl_sync(0xffffffffu, incl, r + step - 1);
                if (v <= t) r += step;
            }
            uint32_t rmask = __shfl_sync(0xffffffffu, mask, r);
            const uint32_t rchunk = __shfl_sync(0xffffffffu, chunk, r);
            const uint32_t rslot = __shfl_sync(0xffffffffu, slot, r);
            const int before = __shfl_sync(0xffffffffu, incl, r) - __shfl_sync(0xffffffffu, c, r);
            bool hit = false;
            int64_t pos = 0;
            int32_t col = 0;
            float s = 0.0f;
            if (t < total) {
                for (int d = t - before; d > 0; --d) rmask &= rmask - 1u;  // (mostly one bit a mask)
                pos = (int64_t)rchunk * 32 + (__ffs(rmask) - 1);
                col = __ldg(p.slot_col + rslot);
                const int L = __ldg(p.col_len + col);
                // Windows that reach beyond the stream are dropped unscored: the masked bases there add 0,
                // so every one of a column with a negative threshold is a candidate, a thousand to a warp
                // (50 kbp x 64 columns of 250 positions, 14.4 k candidates, 10.5 k of them such: 0.272 ms
                // with them scored, 0.036 without).
                if (pos + L <= p.n) {
                    s = window_score(p.seq2, p.zmask, p.P + (size_t)col * p.p_rows, pos, L);
                    // the run is looked up for what reaches the threshold only
                    hit = s >= __ldg(p.thr + col) && (p.keep_below == 0 || pos < p.keep_below) &&
                          pos + L <= run_end_of(p.run_start, p.nruns, p.n, pos);
                }
            }
            const uint32_t hm = __ballot_sync(0xffffffffu, hit);
            if (hit) {
                HitRec h;
                h.pos = pos + p.pos_base;
                h.col = col;
                h.score = s;
                buf[nbuf + __popc(hm & ((1u << lane) - 1u))] = h;
            }
            nbuf += __popc(hm);
            if (nbuf > kRescoreBuf - 32) flush();
        }
    }
    if (nbuf) flush();
    my_cand = __reduce_add_sync(0xffffffffu, my_cand);
    if (lane == 0 && my_cand) atomicAdd(&s_cand, my_cand);
    __syncthreads();
    if (threadIdx.x == 0 && s_cand) atomicAdd(p.ncand, (unsigned long long)s_cand);
}

// ------------------------------------------------------------------------
// 4. the reference's filterScore (kernel.cu:21-34), for the drop-in entry point
// ------------------------------------------------------------------------
__global__ void filter_score_kernel(const float *R, int m, int n, const float *threshold,
                                    int *occIdx, float *occScore, int *nOcc)
{
    const long long total = (long long)m * n;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x; base < total; base += stride) {
        long long idx = base + threadIdx.x;
        bool hit = false;
        float v = 0.0f;
        if (idx < total) {
            int j = (int)(idx / m);
            v = R[idx];
            hit = v >= threshold[j];
        }
        unsigned msk = __ballot_sync(0xffffffffu, hit);
        if (!msk) continue;
        int lane = threadIdx.x & 31, leader = __ffs(msk) - 1;
        int b = 0;
        if (lane == leader) b = atomicAdd(nOcc, __popc(msk));
        b = __shfl_sync(0xffffffffu, b, leader);
        if (hit) {
            int slot = b + __popc(msk & ((1u << lane) - 1u));
            occScore[slot] = v;
            occIdx[slot] = (int)idx;
        }
    }
}

}  // namespace blamm
