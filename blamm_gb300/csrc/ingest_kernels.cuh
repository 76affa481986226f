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
// Data-parallel form: a thread reads 64 bytes as bit masks (newlines, header starts, bases), a
// warp sums its 2 KB up as one IngState with votes on its lanes' masks; states of consecutive
// pieces of text compose (ing_compose, associative).  Whether a piece starts inside a header
// line is the one thing its own bytes may not tell, so ingest_tiles_kernel sums each 32 KB tile
// up for both answers; ingest_scan_kernel (one block) resolves the answers and composes the
// tiles; ingest_emit_kernel reads the text and the first kernel's base masks and warp sums and
// writes the bases, each at the place that its prefix gives; only warps with a header or run
// start take their text apart again.
//
// What bounds it: the instructions that turn bytes into masks and back; memory is touched
// three times (text twice, bases once).  100 Mbp of text, 60 bases a line: 52 + 16 + 57 us
// (a copy of the same bytes takes 45), 0.17 ms a call.  Composing states lane by lane in both
// passes and making all masks twice, 16 KB a tile, took 66 + 39 + 96 us and 0.25 ms; one int64
// per byte and array, prefix scans in place, 56 bytes of temporaries per byte of text allocated
// per call, 6.6 ms of kernels in a call of 18.8 ms.
#pragma once
#include <cstdint>

#include "scan_kernels.cuh"

namespace blamm {

constexpr int kIngThreads = 512;
constexpr int kIngWarps = kIngThreads / 32;
constexpr int kIngEmit = 256;                           // threads that write a part of a tile
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

// A tile: its two states (h = 0, 1: it starts inside a header line or not), each in 16 bytes
// with its A/C/G/T counts, and a word of their flags and the type of the tile's last line.
struct IngTile {
    uint4 *e;        // [h * count + tile]: {nh | nb << 16, nr | sc << 16, a | c << 16, g | t << 16}
    uint32_t *info;  // fl of h = 0 | fl of h = 1 << 8 | line << 16
    // what ingest_emit_kernel takes over: [(h * count + tile) * kIngWarps + warp]:
    // {nh | nb << 16, nr | sc << 16, fl, kIngW*}; [64-byte piece]: its bases (for h = 0)
    uint4 *warps;
    uint64_t *bases;
    int count;
};
// a warp's last event (0: none, 2: a base, 3: a break), and flags
constexpr uint32_t kIngWLast = 3;
constexpr uint32_t kIngWFirst = 4;    // its first event is a base
constexpr uint32_t kIngWRare = 8;     // a header start, or a run start whatever came before
constexpr uint32_t kIngWHeader = 16;  // it starts inside a header line
constexpr uint32_t kIngWOpen = 32;    // its sums depend on h
// line: 0: no line starts in the tile, 2: the last line that does is no header, 3: it is
// 16-byte words of the arrays, per tile
constexpr int kIngTileWords = 2 + 2 * kIngWarps + kIngThreads / 2 + 1;
// The parser before a tile.
struct __align__(16) IngPrefix {
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

// *head: the line starts that start a header; the line starts are returned.  Called by whole
// warps.  What is no base is mostly a newline or two in 64 bytes, which are then looked at one by
// one; where a lane has more, the newline mask is made like the base mask.
template <bool kCodes>
__device__ __forceinline__ uint64_t ing_masks(const char *raw, int64_t n, int64_t at, const uint32_t (&w)[16], IngMasks &m,
                                              uint64_t *head)
{
    uint32_t base[2], b1[2] = {0, 0}, b2[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        base[h] = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t x = w[8 * h + 2 * k], y = w[8 * h + 2 * k + 1];
            base[h] |= (ing_bits(base_bytes(x), base_bytes(y)) >> 7) << (8 * k);
            if (kCodes) {
                b1[h] |= (ing_bits((x << 6) & 0x80808080u, (y << 6) & 0x80808080u) >> 7) << (8 * k);
                b2[h] |= (ing_bits((x << 5) & 0x80808080u, (y << 5) & 0x80808080u) >> 7) << (8 * k);
            }
        }
    }
    m.base = base[0] | (uint64_t)base[1] << 32;
    m.b1 = b1[0] | (uint64_t)b1[1] << 32;
    m.b2 = b2[0] | (uint64_t)b2[1] << 32;
    const uint64_t start = at == 0 || (at < n && raw[at - 1] == '\n') ? 1u : 0u;
    uint64_t hd = 0, nl = 0;
    if (__all_sync(0xffffffffu, __popcll(~m.base) <= 4 && at + kIngBytes <= n)) {
        for (uint64_t r = ~m.base; r; r &= r - 1u) {
            const uint64_t bit = r & (0 - r);
            const char c = raw[at + __ffsll((long long)r) - 1];
            if (c == '\n') nl |= bit;
            if (c == '>' && ((nl << 1 | start) & bit)) hd |= bit;
        }
    } else {
        uint32_t l[2] = {0u, 0u};
#pragma unroll
        for (int k = 0; k < 8; ++k)
            l[k >> 2] |= (ing_bits(zero_bytes(w[2 * k] ^ 0x0A0A0A0Au), zero_bytes(w[2 * k + 1] ^ 0x0A0A0A0Au)) >> 7) << (8 * (k & 3));
        nl = l[0] | (uint64_t)l[1] << 32;
        for (uint64_t r = (nl << 1 | start) & ~nl; r; r &= r - 1u)
            if (raw[at + __ffsll((long long)r) - 1] == '>') hd |= r & (0 - r);
    }
    m.nl = nl;
    *head = hd;
    return nl << 1 | start;
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

// Sums a warp's 2 KB up (every lane gets the sums): votes on which lanes have events (bases and
// breaks), of which kind the last one is, and where the first and the last bases and headers are.
// *prev: the lane's last event before its bytes in the warp (0: none, 2: a base, 3: a break);
// *last: the warp's.
__device__ __forceinline__ IngState<uint16_t> ing_warp_state(const IngChars &c, int lane, uint32_t *prev, uint32_t *last)
{
    const uint64_t b = c.brk(), first = c.base & (0 - c.base);
    const uint32_t bases = __ballot_sync(0xffffffffu, c.base != 0), brks = __ballot_sync(0xffffffffu, b != 0);
    const uint32_t any = bases | brks, ends_brk = __ballot_sync(0xffffffffu, b > c.base);  // (disjoint masks)
    auto last_of = [&](uint32_t among) {
        const uint32_t a = any & among;
        return a ? 2u + ((ends_brk >> (31 - __clz((int)a))) & 1u) : 0u;
    };
    *prev = last_of((1u << lane) - 1u);
    *last = last_of(0xffffffffu);
    const int f = bases ? __ffs((int)bases) - 1 : 32, l = 31 - __clz((int)bases);  // first and last lane with a base
    uint64_t rs = ing_run_starts(c, *prev == 3u);
    if (lane == f) rs &= ~first;
    const uint32_t sum = __reduce_add_sync(0xffffffffu, (uint32_t)__popcll(c.base) | (uint32_t)__popcll(rs) << 16);
    const uint32_t heads = __ballot_sync(0xffffffffu, c.head != 0);
    uint32_t nh = 0, sc = (uint32_t)__popcll(c.seq), bare = 0;
    if (heads) {
        nh = __reduce_add_sync(0xffffffffu, (uint32_t)__popcll(c.head));
        const int lh = 31 - __clz((int)heads), fh = __ffs((int)heads) - 1;
        const uint64_t below = c.head ? (c.head & (0 - c.head)) - 1u : ~(uint64_t)0;
        bare = __ballot_sync(0xffffffffu, (c.seq & below) != 0) & ((2u << fh) - 1u);
        // ((2 << k) - 1 with k = 63 wraps to all ones, as it should)
        if (lane == lh) sc = (uint32_t)__popcll(c.seq & ~(((uint64_t)2 << (63 - __clzll((long long)c.head))) - 1u));
        else if (lane < lh) sc = 0;
    }
    sc = __reduce_add_sync(0xffffffffu, sc);
    if (!heads) bare = sc;
    const uint32_t early = __ballot_sync(0xffffffffu, (b & (first - 1u)) != 0);  // a break before the lane's first base
    IngState<uint16_t> e;
    e.nh = (uint16_t)nh;
    e.nb = (uint16_t)sum;
    e.nr = (uint16_t)(sum >> 16);
    e.sc = (uint16_t)sc;
    const bool fb = bases ? (early & ((2u << f) - 1u)) != 0u : brks != 0u;
    const bool tb = bases ? ((ends_brk >> l) & 1u) != 0u || (brks & ~((2u << l) - 1u)) != 0u : brks != 0u;
    e.fl = (fb ? kIngFirstBrk : 0u) | (tb ? kIngTailBrk : 0u) | (bare ? kIngBare : 0u);
    return e;
}

// w: lane k has warp k's word (0, 2 or 3).  The word of the last warp before `warp` that is not
// 0 (0: none), and the block's last in *all.
__device__ __forceinline__ uint32_t ing_last_before(uint32_t w, int warp, uint32_t *all)
{
    const uint32_t any = __ballot_sync(0xffffffffu, w != 0u), odd = __ballot_sync(0xffffffffu, (w & 1u) != 0u);
    const uint32_t a = any & ((1u << warp) - 1u);
    *all = any ? 2u + ((odd >> (31 - __clz((int)any))) & 1u) : 0u;
    return a ? 2u + ((odd >> (31 - __clz((int)a))) & 1u) : 0u;
}

// The type of the last line that starts in an earlier lane (0: none does, 2: no header, 3: a
// header), and the warp's in *all.  line: this lane's.
__device__ __forceinline__ uint32_t ing_line_before(uint32_t line, int lane, uint32_t *all)
{
    const uint32_t any = __ballot_sync(0xffffffffu, line != 0u), head = __ballot_sync(0xffffffffu, line == 3u);
    auto last = [&](uint32_t among) {  // of the lanes `among`
        const uint32_t a = any & among;
        return a ? 2u + ((head >> (31 - __clz((int)a))) & 1u) : 0u;
    };
    *all = last(0xffffffffu);
    return last((1u << lane) - 1u);
}

__device__ __forceinline__ uint32_t ing_last_line(uint64_t ls, uint64_t head)
{
    return ls ? 2u + (uint32_t)((head >> (63 - __clzll((long long)ls))) & 1u) : 0u;
}

// Sums one tile up for both answers to "does it start inside a header line".
__global__ void __launch_bounds__(kIngThreads, 3) ingest_tiles_kernel(const char *raw, int64_t n, int vec, IngTile tiles)
{
    __shared__ uint32_t s_line[kIngWarps];
    __shared__ IngState<uint16_t> s_e[2][kIngWarps];
    __shared__ uint32_t s_acgt[2][2];  // packed pairs: a, c and g, t (at most 32768 each)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 4) s_acgt[threadIdx.x >> 1][threadIdx.x & 1] = 0u;
    const int64_t at = (int64_t)blockIdx.x * kIngTile + threadIdx.x * kIngBytes;
    uint32_t w[16];
    ing_load(raw, n, at, vec != 0, w);
    IngMasks m;
    uint64_t head;
    const uint64_t ls = ing_masks<true>(raw, n, at, w, m, &head);
    uint32_t wline, all;
    uint32_t before = ing_line_before(ing_last_line(ls, head), lane, &wline);
    if (lane == 0) s_line[warp] = wline;
    __syncthreads();
    const uint32_t start = ing_last_before(lane < kIngWarps ? s_line[lane] : 0u, warp, &all);  // the line that the warp starts in
    if (before == 0u) before = start;
    const bool open = __any_sync(0xffffffffu, before == 0u);  // the answer matters to this warp
    IngState<uint16_t> e{0, 0, 0, 0, 0u};
    uint32_t ac = 0, gt = 0, info = 0;
    for (int h = 0; h < 2; ++h) {
        if (h == 0 || open) {
            const IngChars c = ing_chars(m, ls, head, before ? before == 3u : h == 1);
            uint32_t prev, last;
            e = ing_warp_state(c, lane, &prev, &last);
            info = last | (last && !(e.fl & kIngFirstBrk) ? kIngWFirst : 0u) |
                   (e.nh || e.nr || (e.nb && (e.fl & kIngFirstBrk)) ? kIngWRare : 0u) |
                   ((start ? start == 3u : h == 1) ? kIngWHeader : 0u) | (open ? kIngWOpen : 0u);
            if (h == 0 && at < n) tiles.bases[at / kIngBytes] = c.base;
            // bit 1 of a base: C and G, bit 2: G and T
            const uint32_t cg = (uint32_t)__popcll(c.base & m.b1), g = (uint32_t)__popcll(c.base & m.b1 & m.b2);
            const uint32_t gt1 = (uint32_t)__popcll(c.base & m.b2);
            const uint32_t x = __reduce_add_sync(0xffffffffu, cg | gt1 << 16), y = __reduce_add_sync(0xffffffffu, g);
            const uint32_t cgs = x & 0xffffu, gts = x >> 16;
            ac = (e.nb - cgs - gts + y) | (cgs - y) << 16;
            gt = y | (gts - y) << 16;
        }
        if (lane == 0) {
            s_e[h][warp] = e;
            tiles.warps[((size_t)h * tiles.count + blockIdx.x) * kIngWarps + warp] =
                make_uint4((uint32_t)e.nh | (uint32_t)e.nb << 16, (uint32_t)e.nr | (uint32_t)e.sc << 16, e.fl, info);
            atomicAdd(&s_acgt[h][0], ac);
            atomicAdd(&s_acgt[h][1], gt);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    // lanes 0-15: the warps' states for h = 0, 16-31: for h = 1
    static_assert(kIngWarps == 16, "two states a warp");
    e = s_e[lane >> 4][lane & 15];
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const IngState<uint16_t> b = ing_shfl(e, lane + o);
        if ((lane & (2 * o - 1)) == 0) e = ing_compose(e, b);
    }
    const uint32_t fl1 = __shfl_sync(0xffffffffu, e.fl, 16);
    if ((lane & 15) == 0) {
        const uint32_t *a = s_acgt[lane >> 4];
        tiles.e[(size_t)(lane >> 4) * tiles.count + blockIdx.x] = make_uint4((uint32_t)e.nh | (uint32_t)e.nb << 16, (uint32_t)e.nr | (uint32_t)e.sc << 16, a[0], a[1]);
        if (lane == 0) tiles.info[blockIdx.x] = e.fl | fl1 << 8 | all << 16;
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

// One block: the parser's state before every tile, and the totals.  4096 tiles (128 MB of
// text: 32-bit counts) at a time, four per thread (the scans over the block are what this
// kernel's time goes into); 64-bit totals are carried from batch to batch.
constexpr int kIngPer = 4;

__global__ void __launch_bounds__(kIngScanThreads) ingest_scan_kernel(IngTile tiles, IngPrefix *prefix,
                                                                      unsigned long long *totals)
{
    constexpr int kWarps = kIngScanThreads / 32;
    const int ntiles = tiles.count;
    __shared__ uint32_t s_line[kWarps];
    __shared__ IngState<int32_t> s_e[kWarps];
    __shared__ unsigned long long s_acgt[4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t < 4) s_acgt[t] = 0ull;
    IngState<int64_t> carry{0, 0, 0, 0, 0u};
    uint32_t carry_h = 0;             // the text starts outside any header line
    uint32_t acgt[4] = {0, 0, 0, 0};  // below 2^32: at most ntiles / 1024 x 2^15 each
    for (int64_t b0 = 0; b0 < ntiles; b0 += kIngScanThreads * kIngPer) {
        const int k0 = (int)b0 + t * kIngPer;
        uint32_t info[kIngPer], lines[kIngPer], line = 0;
#pragma unroll
        for (int j = 0; j < kIngPer; ++j) {
            info[j] = k0 + j < ntiles ? tiles.info[k0 + j] : 0u;
            lines[j] = info[j] >> 16;
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
                const uint4 v = tiles.e[(size_t)h * tiles.count + k0 + j];
                own[j] = IngState<uint16_t>{(uint16_t)v.x, (uint16_t)(v.x >> 16), (uint16_t)v.y, (uint16_t)(v.y >> 16),
                                            (info[j] >> (8 * h)) & 255u};
                acgt[0] += v.z & 0xffffu;
                acgt[1] += v.z >> 16;
                acgt[2] += v.w & 0xffffu;
                acgt[3] += v.w >> 16;
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

// Headers and runs of one warp's text (called by whole warps): the pieces are taken apart again.
// xs: lane k has warp k's state of the tile; prev: the last event before the warp in the tile.
// The bases of the thread's piece.
__device__ __noinline__ uint64_t ing_emit_rare(const char *raw, int64_t n, int64_t at, bool vec, int warp, uint4 xs,
                                               bool header, uint32_t prev_event, const IngPrefix &pre, int64_t *run_start,
                                               int64_t *run_seq, int64_t *run_seqpos, int64_t *header_pos)
{
    const int lane = threadIdx.x & 31;
    uint32_t w[16];
    ing_load(raw, n, at, vec, w);
    IngMasks m;
    uint64_t head;
    const uint64_t ls = ing_masks<false>(raw, n, at, w, m, &head);
    uint32_t all, prev, last;
    const uint32_t before = ing_line_before(ing_last_line(ls, head), lane, &all);
    const IngChars c = ing_chars(m, ls, head, before ? before == 3u : header);
    ing_warp_state(c, lane, &prev, &last);
    // runs: after a break, or the text's first base
    const uint64_t rs = ing_run_starts(c, prev         ? prev == 3u
                                          : prev_event ? prev_event == 3u
                                                       : pre.s.nb == 0 || (pre.s.fl & kIngTailBrk));
    IngState<uint16_t> x{0, 0, 0, 0, 0u};  // before this thread in the tile
    for (int k = 0; k < warp; ++k) {
        const uint32_t a = __shfl_sync(0xffffffffu, xs.x, k), b = __shfl_sync(0xffffffffu, xs.y, k);
        x = ing_compose(x, IngState<uint16_t>{(uint16_t)a, (uint16_t)(a >> 16), (uint16_t)b, (uint16_t)(b >> 16),
                                              __shfl_sync(0xffffffffu, xs.z, k)});
    }
    const IngState<uint16_t> e = ing_shfl(ing_warp_scan(ing_state(c), lane), lane ? lane - 1 : 0);
    if (lane) x = ing_compose(x, e);
    const IngState<int64_t> g = ing_compose(pre.s, x);  // before this thread in the text
    for (uint64_t r = c.head; r; r &= r - 1u) {
        const int i = __ffsll((long long)r) - 1;
        header_pos[g.nh + __popcll(c.head & (((uint64_t)1 << i) - 1u))] = at + i;
    }
    int64_t run = g.nr + (g.nb ? 1 : 0);
    for (uint64_t r = rs; r; r &= r - 1u, ++run) {
        const uint64_t below = (r & (0 - r)) - 1u;
        const uint64_t heads = c.head & below;
        const uint64_t since = heads ? ~(((uint64_t)2 << (63 - __clzll((long long)heads))) - 1u) : ~(uint64_t)0;
        run_start[run] = g.nb + __popcll(c.base & below);
        run_seq[run] = g.nh + __popcll(heads) - 1;
        run_seqpos[run] = (heads ? 0 : g.sc) + __popcll(c.seq & below & since);
    }
    return c.base;
}

// Writes a part of a tile: bases, header offsets and runs; nothing where the text was refused.
__global__ void __launch_bounds__(kIngEmit) ingest_emit_kernel(const char *raw, int64_t n, int vec, IngTile tiles,
                                                                  const IngPrefix *prefix, const unsigned long long *totals,
                                                                  char *bases, int64_t *run_start, int64_t *run_seq,
                                                                  int64_t *run_seqpos, int64_t *header_pos)
{
    __shared__ __align__(16) unsigned char s_out[kIngEmit * kIngBytes + 16];
    __shared__ uint32_t s_pack[16];  // by nibble: __byte_perm selector of the set bits' bytes, their number
    // (all loads first: what they wait for, not their bytes, is what a block's time goes into)
    constexpr int kParts = kIngThreads / kIngEmit, kPartWarps = kIngWarps / kParts;
    const int tile = blockIdx.x / kParts, part = blockIdx.x % kParts;
    const int lane = threadIdx.x & 31, warp = part * kPartWarps + (threadIdx.x >> 5);  // in the tile
    const int64_t at = (int64_t)blockIdx.x * (kIngEmit * kIngBytes) + threadIdx.x * kIngBytes;
    uint32_t w[16];
    ing_load(raw, n, at, vec != 0, w);
    uint64_t base = at < n ? tiles.bases[at / kIngBytes] : 0;
    uint4 xs = make_uint4(0u, 0u, 0u, 0u), xs1 = xs;
    if (lane < kIngWarps) {
        xs = tiles.warps[(size_t)tile * kIngWarps + lane];
        xs1 = tiles.warps[((size_t)tiles.count + tile) * kIngWarps + lane];
    }
    const IngPrefix &pre = prefix[tile];
    const uint32_t h = pre.h, pre_fl = pre.s.fl;
    const int64_t pre_nb = pre.s.nb;
    if (totals[3]) return;
    if (h) xs = xs1;
    if (threadIdx.x < 16) {
        uint32_t sel = 0x4444u, j = 0;  // (4: a zero byte)
        for (uint32_t i = 0; i < 4; ++i)
            if ((threadIdx.x >> i) & 1u) {
                sel = (sel & ~(15u << (4 * j))) | i << (4 * j);
                ++j;
            }
        s_pack[threadIdx.x] = sel | j << 16;
    }
    __syncthreads();  // s_pack
    uint32_t tile_last;
    const uint32_t prev = ing_last_before(xs.w & kIngWLast, warp, &tile_last), own = __shfl_sync(0xffffffffu, xs.w, warp);
    const bool starts = (own & kIngWFirst) && (prev ? prev == 3u : pre_nb == 0 || (pre_fl & kIngTailBrk));
    if (starts || (own & (kIngWRare | (h ? kIngWOpen : 0u))))
        base = ing_emit_rare(raw, n, at, vec != 0, warp, xs, (own & kIngWHeader) != 0u, prev, pre, run_start, run_seq, run_seqpos,
                             header_pos);
    const uint32_t wnb = xs.x >> 16;
    const int before = (int)__reduce_add_sync(0xffffffffu, lane < part * kPartWarps ? wnb : 0u);  // the parts before
    const int nb = (int)__reduce_add_sync(0xffffffffu, lane / kPartWarps == part ? wnb : 0u);     // this part
    uint32_t upto = (uint32_t)__popcll(base);  // bases up to this thread in the warp
    const uint32_t mine = upto;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    // before this thread in the part
    const int xnb = (int)(__reduce_add_sync(0xffffffffu, lane < warp ? wnb : 0u) + upto - mine) - before;

    // the bases, compacted in shared memory at the destination's alignment
    char *dst = bases + pre_nb + before;
    const int mis = (int)(reinterpret_cast<uintptr_t>(dst) & 15u);
    {
        // A word at a time: its bases packed (byte selectors by the nibble of the mask), shifted
        // behind the bytes kept back, whole words stored.  The first and last words are shared
        // with the neighbours: byte by byte.
        const int o = mis + xnb;
        unsigned char *const out0 = s_out + (o & ~3);
        unsigned char *out = out0;
        uint32_t have = (uint32_t)o & 3u;  // bytes in acc (at first: those before this thread's)
        uint32_t acc = 0, first = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const uint32_t sel = s_pack[(uint32_t)(base >> (4 * k)) & 15u];
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
    __syncthreads();
    const int end = mis + nb;
    char *d0 = dst - mis;
    for (int k = threadIdx.x; 16 * k < end; k += kIngEmit) {
        if (16 * k >= mis && 16 * k + 16 <= end) {
            reinterpret_cast<uint4 *>(d0)[k] = reinterpret_cast<const uint4 *>(s_out)[k];
        } else {
            for (int i = max(mis, 16 * k); i < min(end, 16 * k + 16); ++i) d0[i] = (char)s_out[i];
        }
    }
}

}  // namespace blamm
