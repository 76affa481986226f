// ingest_kernels.cuh -- FASTA text -> filtered base stream + run table on the GPU.
//
// The same stream and markers the host's FastaStream builds (FastaBatch,
// src/sequence.cpp:142-293): lines split at '\n'; a line starting with '>'
// opens a sequence; every other character of a sequence line (including 'N',
// '\r' and other non-bases) advances the position in the sequence; the
// stream holds the A/C/G/T/a/c/g/t characters; a run (SeqBlock marker,
// src/sequence.cpp:35-50) starts where the stream position and the sequence
// position stop advancing together.
//
// Data-parallel form: a thread reads 64 bytes as bit masks (newlines, header starts, bases)
// and sums them up as one IngState; states of consecutive pieces of text compose
// (ing_compose, associative).  Whether a piece starts inside a header line is the one thing
// its own bytes may not tell, so ingest_tiles_kernel sums each 16 KB tile up for both
// answers; ingest_scan_kernel (one block) resolves the answers and composes the tiles;
// ingest_emit_kernel reads the text again and writes the bases, header offsets and runs,
// each at the place that its prefix gives.
//
// What bounds it: the instructions that turn bytes into masks and back; memory is touched
// three times (text twice, bases once).  100 Mbp of text, 60 bases a line: 66 + 39 + 96 us
// (a copy of the same bytes takes 45).  The first form -- one int64 per byte and array, prefix
// scans in place, 56 bytes of temporaries per byte of text allocated per call -- took 6.6 ms
// of kernels in a call of 18.8 ms; the call now takes 0.25 ms.
#pragma once
#include <cstdint>

#include "scan_kernels.cuh"

namespace blamm {

constexpr int kIngThreads = 256;
constexpr int kIngBytes = 64;                           // bytes per thread: one bit of a 64-bit mask each
constexpr int kIngTile = kIngThreads * kIngBytes;       // bytes per tile (counts fit 16 bits)
constexpr int kIngScanThreads = 1024;

// What a piece of text does to the parser: header lines, bases, run starts other than a run
// start at its first base, sequence characters since its last header (or its start).
template <class T>
struct IngState {
    T nh, nb, nr, sc;
    uint32_t fl;
};
// flags; a break is a header start or a sequence character that is no base
constexpr uint32_t kIngFirstBrk = 1;  // a break before the first base (or at all, without bases)
constexpr uint32_t kIngTailBrk = 2;   // a break after the last base (or at all)
constexpr uint32_t kIngBare = 4;      // sequence characters before the first header

// A tile: its two states (h = 0, 1: it starts inside a header line or not), the type of its
// last line, its A/C/G/T counts for both.
struct IngTile {
    IngState<uint16_t> e[2];
    uint32_t line;  // 0: no line starts in the tile, 2: the last line that does is no header, 3: it is
    uint16_t acgt[2][4];
};
// The parser before a tile.
struct IngPrefix {
    IngState<int64_t> s;
    uint32_t h;
};
// Totals: bases, runs, sequences, a flag for sequence data before the first header, A/C/G/T counts.
constexpr int kIngTotals = 8;

template <class T, class U>
__device__ __forceinline__ IngState<T> ing_compose(const IngState<T> &a, const IngState<U> &b)
{
    IngState<T> r;
    r.nh = (T)(a.nh + b.nh);
    r.nb = (T)(a.nb + b.nb);
    r.sc = (T)(b.nh ? b.sc : a.sc + b.sc);
    const uint32_t first = a.nb ? a.fl & kIngFirstBrk : ((a.fl >> 1) | b.fl) & kIngFirstBrk;
    const uint32_t tail = b.nb ? b.fl & kIngTailBrk : (a.fl | b.fl) & kIngTailBrk;
    const uint32_t bare = a.nh ? a.fl & kIngBare : (a.fl | b.fl) & kIngBare;
    r.fl = first | tail | bare;
    r.nr = (T)(a.nr + b.nr + (a.nb && b.nb && ((a.fl & kIngTailBrk) || (b.fl & kIngFirstBrk)) ? 1 : 0));
    return r;
}

// The masks of one thread's 64 bytes (bytes past the end of the text count as newlines).
struct IngMasks {
    uint64_t nl, base;
    uint64_t b1, b2;  // bits 1 and 2 of the characters: A 0 0, C 1 0, G 1 1, T 0 1
};

// The 0x80 bits of two words' bytes as 8 mask bits at bit 7 (dot products with the bits' weights)
__device__ __forceinline__ uint32_t ing_bits(uint32_t lo, uint32_t hi)
{
    return __dp4a(hi, 0x80402010u, __dp4a(lo, 0x08040201u, 0u));
}

__device__ __forceinline__ void ing_load(const char *raw, int64_t n, int64_t at, bool vec, uint32_t (&w)[16])
{
    if (vec && at + kIngBytes <= n) {
        const uint4 *p = reinterpret_cast<const uint4 *>(raw + at);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint4 v = __ldg(p + k);
            w[4 * k] = v.x;
            w[4 * k + 1] = v.y;
            w[4 * k + 2] = v.z;
            w[4 * k + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            w[k] = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int64_t i = at + 4 * k + b;
                w[k] |= (i < n ? (uint32_t)(unsigned char)raw[i] : (uint32_t)'\n') << (8 * b);
            }
        }
    }
}

template <bool kCodes>
__device__ __forceinline__ IngMasks ing_masks(const uint32_t (&w)[16])
{
    uint32_t nl[2], base[2], b1[2] = {0, 0}, b2[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        nl[h] = base[h] = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t x = w[8 * h + 2 * k], y = w[8 * h + 2 * k + 1];
            nl[h] |= (ing_bits(zero_bytes(x ^ 0x0A0A0A0Au), zero_bytes(y ^ 0x0A0A0A0Au)) >> 7) << (8 * k);
            base[h] |= (ing_bits(base_bytes(x), base_bytes(y)) >> 7) << (8 * k);
            if (kCodes) {
                b1[h] |= (ing_bits((x << 6) & 0x80808080u, (y << 6) & 0x80808080u) >> 7) << (8 * k);
                b2[h] |= (ing_bits((x << 5) & 0x80808080u, (y << 5) & 0x80808080u) >> 7) << (8 * k);
            }
        }
    }
    return IngMasks{nl[0] | (uint64_t)nl[1] << 32, base[0] | (uint64_t)base[1] << 32, b1[0] | (uint64_t)b1[1] << 32,
                    b2[0] | (uint64_t)b2[1] << 32};
}

// The thread's characters once it is known whether it starts inside a header line.
struct IngChars {
    uint64_t head, seq, base;  // header starts, sequence characters, bases
    __device__ __forceinline__ uint64_t brk() const { return head | (seq & ~base); }
};

__device__ __forceinline__ IngChars ing_chars(const IngMasks &m, uint64_t ls, uint64_t head, bool in_header)
{
    IngChars c;
    c.head = head;
    // header text: a start added to the mask of non-newlines carries up to the line's end
    const uint64_t text = ~m.nl;
    const uint64_t s = c.head | (in_header && !((ls | m.nl) & 1u) ? 1u : 0u);
    const uint64_t in = text & ~(text + s);
    c.seq = text & ~in;
    c.base = c.seq & m.base;
    return c;
}

// Bases that start a run: the next event (base or break) after a break, or after the piece's
// start with brk_in (a break added to the mask of non-events carries up to the next event).
__device__ __forceinline__ uint64_t ing_run_starts(const IngChars &c, bool brk_in)
{
    const uint64_t b = c.brk(), gap = ~(c.base | b);
    return c.base & ~gap & (gap + ((b << 1) | (brk_in ? 1u : 0u)));
}

__device__ __forceinline__ IngState<uint16_t> ing_state(const IngChars &c)
{
    IngState<uint16_t> e;
    const uint64_t b = c.brk();
    const uint64_t first = c.base & (0 - c.base);
    e.nh = (uint16_t)__popcll(c.head);
    e.nb = (uint16_t)__popcll(c.base);
    e.nr = (uint16_t)__popcll(ing_run_starts(c, false) & ~first);
    // (2 << k) - 1 with k = 63 wraps to all ones, as it should
    const uint64_t upto_head = c.head ? ((uint64_t)2 << (63 - __clzll((long long)c.head))) - 1u : 0u;
    e.sc = (uint16_t)__popcll(c.seq & ~upto_head);
    const uint64_t upto_base = c.base ? ((uint64_t)2 << (63 - __clzll((long long)c.base))) - 1u : 0u;
    const uint64_t below_base = c.base ? first - 1u : ~(uint64_t)0;
    const uint64_t below_head = c.head ? (c.head & (0 - c.head)) - 1u : ~(uint64_t)0;
    e.fl = ((b & below_base) ? kIngFirstBrk : 0u) | ((b & ~upto_base) ? kIngTailBrk : 0u) |
           ((c.seq & below_head) ? kIngBare : 0u);
    return e;
}

__device__ __forceinline__ IngState<uint16_t> ing_shfl(const IngState<uint16_t> &e, int src)
{
    const uint32_t a = __shfl_sync(0xffffffffu, (uint32_t)e.nh | (uint32_t)e.nb << 16, src);
    const uint32_t b = __shfl_sync(0xffffffffu, (uint32_t)e.nr | (uint32_t)e.sc << 16, src);
    IngState<uint16_t> r;
    r.nh = (uint16_t)a;
    r.nb = (uint16_t)(a >> 16);
    r.nr = (uint16_t)b;
    r.sc = (uint16_t)(b >> 16);
    r.fl = __shfl_sync(0xffffffffu, e.fl, src);
    return r;
}

// Inclusive composition over the warp's lanes.
__device__ __forceinline__ IngState<uint16_t> ing_warp_scan(IngState<uint16_t> e, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const IngState<uint16_t> p = ing_shfl(e, lane >= o ? lane - o : lane);
        if (lane >= o) e = ing_compose(p, e);
    }
    return e;
}

// The type of the last line that starts before this thread in the block (as IngTile::line;
// 0: none does), and the block's in *all.  line: this thread's.
__device__ __forceinline__ uint32_t ing_line_before(uint32_t line, uint32_t *s_line, uint32_t *all)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t any = __ballot_sync(0xffffffffu, line != 0u), head = __ballot_sync(0xffffffffu, line == 3u);
    auto last = [&](uint32_t among) {  // of the lanes `among`
        const uint32_t a = any & among;
        return a ? 2u + ((head >> (31 - __clz((int)a))) & 1u) : 0u;
    };
    if (lane == 0) s_line[warp] = last(0xffffffffu);
    __syncthreads();
    uint32_t r = last((1u << lane) - 1u), t = 0;
#pragma unroll
    for (int w = 0; w < kIngThreads / 32; ++w) {
        if (w == warp && r == 0u) r = t;
        if (s_line[w]) t = s_line[w];
    }
    *all = t;
    return r;
}

// The line starts among the thread's bytes, and (looked up one by one: a line or two in 64
// bytes) which of them start a header.
__device__ __forceinline__ uint64_t ing_line_starts(const char *raw, int64_t n, int64_t at, uint64_t nl, uint64_t *head)
{
    const bool start = at == 0 || (at < n && raw[at - 1] == '\n');
    const uint64_t ls = nl << 1 | (start ? 1u : 0u);
    uint64_t h = 0;
    for (uint64_t r = ls & ~nl; r; r &= r - 1u)
        if (raw[at + __ffsll((long long)r) - 1] == '>') h |= r & (0 - r);
    *head = h;
    return ls;
}

__device__ __forceinline__ uint32_t ing_last_line(uint64_t ls, uint64_t head)
{
    return ls ? 2u + (uint32_t)((head >> (63 - __clzll((long long)ls))) & 1u) : 0u;
}

// Sums one tile up for both answers to "does it start inside a header line".
__global__ void __launch_bounds__(kIngThreads) ingest_tiles_kernel(const char *raw, int64_t n, int vec, IngTile *tiles)
{
    __shared__ uint32_t s_line[kIngThreads / 32];
    __shared__ IngState<uint16_t> s_e[2][kIngThreads / 32];
    __shared__ uint32_t s_acgt[2][4], s_wacgt[kIngThreads / 32][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 8) s_acgt[threadIdx.x >> 2][threadIdx.x & 3] = 0u;
    const int64_t at = (int64_t)blockIdx.x * kIngTile + threadIdx.x * kIngBytes;
    uint32_t w[16];
    ing_load(raw, n, at, vec != 0, w);
    const IngMasks m = ing_masks<true>(w);
    uint64_t head;
    const uint64_t ls = ing_line_starts(raw, n, at, m.nl, &head);
    uint32_t all;
    const uint32_t before = ing_line_before(ing_last_line(ls, head), s_line, &all);
    const bool open = __any_sync(0xffffffffu, before == 0u);  // the answer matters to this warp
    for (int h = 0; h < 2; ++h) {
        if (h == 1 && !open) {  // the same as for the other answer
            if (lane == 31) s_e[1][warp] = s_e[0][warp];
            if (lane < 4) atomicAdd(&s_acgt[1][lane], s_wacgt[warp][lane]);
            break;
        }
        const IngChars c = ing_chars(m, ls, head, before ? before == 3u : h == 1);
        const IngState<uint16_t> e = ing_warp_scan(ing_state(c), lane);
        if (lane == 31) s_e[h][warp] = e;
        // 16-bit counts (at most 2048 a warp)
        uint32_t ca = (uint32_t)__popcll(c.base & ~m.b1 & ~m.b2) | (uint32_t)__popcll(c.base & m.b1 & ~m.b2) << 16;
        uint32_t gt = (uint32_t)__popcll(c.base & m.b1 & m.b2) | (uint32_t)__popcll(c.base & ~m.b1 & m.b2) << 16;
        ca = __reduce_add_sync(0xffffffffu, ca);
        gt = __reduce_add_sync(0xffffffffu, gt);
        if (lane < 4) {
            const uint32_t v = ((lane < 2 ? ca : gt) >> (16 * (lane & 1))) & 0xffffu;
            atomicAdd(&s_acgt[h][lane], v);
            s_wacgt[warp][lane] = v;
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        IngState<uint16_t> e = s_e[threadIdx.x][0];
        for (int k = 1; k < kIngThreads / 32; ++k) e = ing_compose(e, s_e[threadIdx.x][k]);
        IngTile &t = tiles[blockIdx.x];
        t.e[threadIdx.x] = e;
        for (int k = 0; k < 4; ++k) t.acgt[threadIdx.x][k] = (uint16_t)s_acgt[threadIdx.x][k];
        if (threadIdx.x == 0) t.line = all;
    }
}

__device__ __forceinline__ IngState<int32_t> ing_shfl(const IngState<int32_t> &e, int src)
{
    IngState<int32_t> r;
    r.nh = __shfl_sync(0xffffffffu, e.nh, src);
    r.nb = __shfl_sync(0xffffffffu, e.nb, src);
    r.nr = __shfl_sync(0xffffffffu, e.nr, src);
    r.sc = __shfl_sync(0xffffffffu, e.sc, src);
    r.fl = __shfl_sync(0xffffffffu, e.fl, src);
    return r;
}

// One block: the parser's state before every tile, and the totals.  4096 tiles (64 MB of
// text: 32-bit counts) at a time, four per thread (the scans over the block are what this
// kernel's time goes into); 64-bit totals are carried from batch to batch.
constexpr int kIngPer = 4;

__global__ void __launch_bounds__(kIngScanThreads) ingest_scan_kernel(const IngTile *tiles, int ntiles, IngPrefix *prefix,
                                                                      unsigned long long *totals)
{
    constexpr int kWarps = kIngScanThreads / 32;
    __shared__ uint32_t s_line[kWarps];
    __shared__ IngState<int32_t> s_e[kWarps];
    __shared__ unsigned long long s_acgt[4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t < 4) s_acgt[t] = 0ull;
    IngState<int64_t> carry{0, 0, 0, 0, 0u};
    uint32_t carry_h = 0;             // the text starts outside any header line
    uint32_t acgt[4] = {0, 0, 0, 0};  // below 2^32: at most ntiles / 1024 x 2^14 each
    for (int64_t b0 = 0; b0 < ntiles; b0 += kIngScanThreads * kIngPer) {
        const int k0 = (int)b0 + t * kIngPer;
        uint32_t lines[kIngPer], line = 0;
#pragma unroll
        for (int j = 0; j < kIngPer; ++j) {
            lines[j] = k0 + j < ntiles ? tiles[k0 + j].line : 0u;
            if (lines[j]) line = lines[j];
        }
        // the type of the last line that starts in an earlier tile
        const uint32_t any = __ballot_sync(0xffffffffu, line != 0u), head = __ballot_sync(0xffffffffu, line == 3u);
        auto last = [&](uint32_t among) {
            const uint32_t a = any & among;
            return a ? 2u + ((head >> (31 - __clz((int)a))) & 1u) : 0u;
        };
        __syncthreads();  // the last batch's s_line and s_e have been read
        if (lane == 0) s_line[warp] = last(0xffffffffu);
        __syncthreads();
        const uint32_t lw = s_line[lane];  // (32 warps: one word a lane)
        const uint32_t wany = __ballot_sync(0xffffffffu, lw != 0u), whead = __ballot_sync(0xffffffffu, lw == 3u);
        const uint32_t wbefore = wany & ((1u << warp) - 1u);
        uint32_t before = last((1u << lane) - 1u);
        if (before == 0u && wbefore) before = 2u + ((whead >> (31 - __clz((int)wbefore))) & 1u);
        const uint32_t h0 = before ? (before == 3u) : carry_h;
        if (wany) carry_h = (whead >> (31 - __clz((int)wany))) & 1u;
        // the states: over the thread's tiles, the warp, the warps
        IngState<uint16_t> own[kIngPer];
        IngState<int32_t> e{0, 0, 0, 0, 0u};
        uint32_t h = h0;
#pragma unroll
        for (int j = 0; j < kIngPer; ++j) {
            own[j] = IngState<uint16_t>{0, 0, 0, 0, 0u};
            if (k0 + j < ntiles) {
                const IngTile &tile = tiles[k0 + j];
                own[j] = tile.e[h];
#pragma unroll
                for (int b = 0; b < 4; ++b) acgt[b] += tile.acgt[h][b];
            }
            e = ing_compose(e, own[j]);
            if (lines[j]) h = lines[j] == 3u;
        }
        auto scan = [&](IngState<int32_t> v) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const IngState<int32_t> p = ing_shfl(v, lane >= o ? lane - o : lane);
                if (lane >= o) v = ing_compose(p, v);
            }
            return v;
        };
        e = scan(e);
        if (lane == 31) s_e[warp] = e;
        __syncthreads();
        const IngState<int32_t> w = scan(s_e[lane]);
        const IngState<int32_t> up = ing_shfl(e, lane ? lane - 1 : 0), wup = ing_shfl(w, warp ? warp - 1 : 0);
        IngState<int32_t> in{0, 0, 0, 0, 0u};  // before this thread in the batch
        if (warp) in = wup;
        if (lane) in = ing_compose(in, up);
        h = h0;
#pragma unroll
        for (int j = 0; j < kIngPer; ++j) {
            if (k0 + j < ntiles) {
                prefix[k0 + j].s = ing_compose(carry, in);
                prefix[k0 + j].h = h;
            }
            in = ing_compose(in, own[j]);
            if (lines[j]) h = lines[j] == 3u;
        }
        carry = ing_compose(carry, ing_shfl(w, 31));
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const unsigned long long lo = __reduce_add_sync(0xffffffffu, acgt[b] & 0xffffu);
        const unsigned long long hi = __reduce_add_sync(0xffffffffu, acgt[b] >> 16);
        if (lane == 0) atomicAdd(&s_acgt[b], lo + (hi << 16));
    }
    __syncthreads();
    if (t == 0) {
        totals[0] = (unsigned long long)carry.nb;
        totals[1] = (unsigned long long)(carry.nb ? carry.nr + 1 : 0);
        totals[2] = (unsigned long long)carry.nh;
        totals[3] = (carry.fl & kIngBare) ? 1ull : 0ull;
        for (int b = 0; b < 4; ++b) totals[4 + b] = s_acgt[b];
    }
}

// Writes one tile's bases, header offsets and runs; nothing where the text was refused.
__global__ void __launch_bounds__(kIngThreads) ingest_emit_kernel(const char *raw, int64_t n, int vec, const IngPrefix *prefix,
                                                                  const unsigned long long *totals, char *bases,
                                                                  int64_t *run_start, int64_t *run_seq, int64_t *run_seqpos,
                                                                  int64_t *header_pos)
{
    __shared__ uint32_t s_line[kIngThreads / 32];
    __shared__ IngState<uint16_t> s_e[kIngThreads / 32];
    __shared__ __align__(16) unsigned char s_out[kIngTile + 16];
    __shared__ uint32_t s_pack[16];  // by nibble: __byte_perm selector of the set bits' bytes, their number
    if (totals[3]) return;
    if (threadIdx.x < 16) {
        uint32_t sel = 0x4444u, j = 0;  // (4: a zero byte)
        for (uint32_t i = 0; i < 4; ++i)
            if ((threadIdx.x >> i) & 1u) {
                sel = (sel & ~(15u << (4 * j))) | i << (4 * j);
                ++j;
            }
        s_pack[threadIdx.x] = sel | j << 16;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = (int64_t)blockIdx.x * kIngTile + threadIdx.x * kIngBytes;
    uint32_t w[16];
    ing_load(raw, n, at, vec != 0, w);
    const IngMasks m = ing_masks<false>(w);
    uint64_t head;
    const uint64_t ls = ing_line_starts(raw, n, at, m.nl, &head);
    uint32_t all;
    const uint32_t before = ing_line_before(ing_last_line(ls, head), s_line, &all);
    const IngPrefix pre = prefix[blockIdx.x];
    const IngChars c = ing_chars(m, ls, head, before ? before == 3u : pre.h != 0u);
    IngState<uint16_t> e = ing_warp_scan(ing_state(c), lane);
    if (lane == 31) s_e[warp] = e;
    __syncthreads();
    IngState<uint16_t> x{0, 0, 0, 0, 0u};  // before this thread in the tile
    for (int k = 0; k < warp; ++k) x = ing_compose(x, s_e[k]);
    int nb = x.nb;
    for (int k = warp; k < kIngThreads / 32; ++k) nb += s_e[k].nb;  // the tile's bases
    e = ing_shfl(e, lane ? lane - 1 : 0);
    if (lane) x = ing_compose(x, e);

    // the bases, compacted in shared memory at the destination's alignment
    char *dst = bases + pre.s.nb;
    const int mis = (int)(reinterpret_cast<uintptr_t>(dst) & 15u);
    {
        // A word at a time: its bases packed (byte selectors by the nibble of the mask), shifted
        // behind the bytes kept back, whole words stored.  The first and last words are shared
        // with the neighbours: byte by byte.
        const int o = mis + x.nb;
        unsigned char *const out0 = s_out + (o & ~3);
        unsigned char *out = out0;
        uint32_t have = (uint32_t)o & 3u;  // bytes in acc (at first: those before this thread's)
        uint32_t acc = 0, first = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const uint32_t sel = s_pack[(uint32_t)(c.base >> (4 * k)) & 15u];
            const uint32_t v = __byte_perm(w[k], 0u, sel);
            acc |= v << (8u * have);
            const uint32_t over = __funnelshift_l(v, 0u, 8u * have);
            have += sel >> 16;
            if (have >= 4u) {
                if (out == out0) first = acc;
                else *reinterpret_cast<uint32_t *>(out) = acc;
                out += 4;
                acc = over;
                have -= 4u;
            }
        }
        const bool one = out == out0;  // less than a word in all: acc is the first word
        if (one) first = acc;
        for (uint32_t i = (uint32_t)o & 3u; i < (one ? have : 4u); ++i) out0[i] = (unsigned char)(first >> (8u * i));
        if (!one)
            for (uint32_t i = 0; i < have; ++i) out[i] = (unsigned char)(acc >> (8u * i));
    }
    const IngState<int64_t> g = ing_compose(pre.s, x);  // before this thread in the text
    // headers and runs: rare
    for (uint64_t r = c.head; r; r &= r - 1u) {
        const int i = __ffsll((long long)r) - 1;
        header_pos[g.nh + __popcll(c.head & (((uint64_t)1 << i) - 1u))] = at + i;
    }
    const uint64_t rs = ing_run_starts(c, g.nb == 0 || (g.fl & kIngTailBrk));
    int64_t run = g.nr + (g.nb ? 1 : 0);
    for (uint64_t r = rs; r; r &= r - 1u, ++run) {
        const uint64_t below = (r & (0 - r)) - 1u;
        const uint64_t heads = c.head & below;
        const uint64_t since = heads ? ~(((uint64_t)2 << (63 - __clzll((long long)heads))) - 1u) : ~(uint64_t)0;
        run_start[run] = g.nb + __popcll(c.base & below);
        run_seq[run] = g.nh + __popcll(heads) - 1;
        run_seqpos[run] = (heads ? 0 : g.sc) + __popcll(c.seq & below & since);
    }
    __syncthreads();
    const int end = mis + nb;
    char *d0 = dst - mis;
    for (int k = threadIdx.x; 16 * k < end; k += kIngThreads) {
        if (16 * k >= mis && 16 * k + 16 <= end) {
            reinterpret_cast<uint4 *>(d0)[k] = reinterpret_cast<const uint4 *>(s_out)[k];
        } else {
            for (int i = max(mis, 16 * k); i < min(end, 16 * k + 16); ++i) d0[i] = (char)s_out[i];
        }
    }
}

}  // namespace blamm
