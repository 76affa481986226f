// plan_kernels.cuh -- the tensor-core plan of a set of columns, built on the device from the
// quantised bank: thresholds on the accumulator's scale, and the A tiles.
//
// Threshold.  A window is a candidate iff its quantised sum reaches T, so T may be any lower
// bound of sum(q) over the windows that are hits: T = thr - (worst sum(P - q)) is one, but the
// worst case takes, at every position, the base whose quantisation lost most -- mostly a base
// with a large negative score, which no hit can have many of.  Of all base choices, only those
// with sum(P) >= thr' matter (thr' = thr minus the bound on the reference's own FP32
// rounding), and for every lambda >= 0
//     min { sum(q) : sum(P) >= thr' } >= lambda thr' + sum_j min_b (q_jb - lambda P_jb)
// (Lagrangian bound; a masked base is a fifth choice with q = P = 0).  lambda = 1 is the worst
// case above; the best lambda is usually a few thousandths (BF16) or hundredths (E4M3) more.
// A warp compares 64 values of lambda in FP32 and then forms the bound of the best one in 64-bit
// fixed point (the FP64 units are slow here: a plan of 4000 columns takes 58 us in FP32 alone, 83
// with the bound in FP64, 62 so), or takes the worst case (FP64) where that is larger.  (Which lambda it is decides how tight the bound is,
// not whether it holds.)  Candidates per hit, 512 motifs x 16 Mi positions at p = 1e-4, by the worst
// case and so: E4M3 2.03, 1.17; one BF16 term 1.25, 1.11.
#pragma once
#include <cstdint>

#include "scan_kernels.cuh"
#include "scan_tc.cuh"

namespace blamm {

struct PlanParams {
    const TileDesc *tiles;    // ntiles + 1
    int32_t ntiles;
    const int32_t *slot_col;  // per slot: motif column, -1 for padding
    float *slot_thr;
    uint8_t *abuf;
    int32_t nsteps;
    int32_t terms;            // 1, 2 or kE4M3
    // the bank and its quantised terms: column c's values start at entry off[c] (4 per position)
    const float *P;
    int32_t p_rows;
    const int32_t *col_len;
    const float *thr;
    const uint32_t *off;
    const uint16_t *hi, *lo;  // BF16
    const uint8_t *e8;        // E4M3 codes of P x 2^k
    const int32_t *k;         // exponents: grid 2^-k (BF16), scale 2^k (E4M3)
    const double *guard;      // worst case of sum(P - q), with the reference's own rounding
};

// An E4M3 code in units of 2^-9.
__device__ __forceinline__ float e4m3_units_f(uint32_t code)
{
    const int e = (int)(code >> 3) & 15, m = (int)code & 7;
    const float a = e == 0 ? (float)m : ldexpf((float)(8 + m), e - 1);
    return code & 0x80u ? -a : a;
}

// Entry i of a column in units of 2^-s: the quantised value (a whole number below 2^16) and P.
struct PlanEntry {
    float q, x;
};
__device__ __forceinline__ PlanEntry plan_entry(const PlanParams &p, const float *P, uint32_t o, int s, int i)
{
    PlanEntry e;
    e.x = ldexpf(__ldg(P + i), s);
    if (p.terms == kE4M3) {
        e.q = e4m3_units_f(__ldg(p.e8 + o + i));
    } else {
        e.q = ldexpf(__uint_as_float((uint32_t)__ldg(p.hi + o + i) << 16), s);
        if (p.terms == 2) e.q += ldexpf(__uint_as_float((uint32_t)__ldg(p.lo + o + i) << 16), s);  // exact
    }
    return e;
}

__device__ __forceinline__ long long warp_sum(long long v)
{
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// One warp per slot: its threshold.
__global__ void __launch_bounds__(256) plan_thr_kernel(PlanParams p)
{
    const int slot = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (slot >= p.ntiles * kTileCols) return;
    const int c = p.slot_col[slot];
    if (c < 0) {
        if (lane == 0) p.slot_thr[slot] = __int_as_float(0x7f800000);
        return;
    }
    const bool e8 = p.terms == kE4M3;
    const int L = p.col_len[c], s = p.k[c] + (e8 ? 9 : 8);  // everything below in units of 2^-s
    const float *P = p.P + (size_t)c * p.p_rows;
    const uint32_t o = p.off[c];
    // lambda: 0, 1 - d for 14 values of d from 1/2 down to 2^-12.4, 1, 1 + d for 48 from 2^-14 up to 3.9
    float lam[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;  // 0..63
        lam[h] = i == 0    ? 0.0f
                 : i == 1  ? 1.0f
                 : i < 16  ? 1.0f - exp2f(-1.0f - 0.875f * (float)(i - 2))
                           : 1.0f + exp2f(-14.0f + 0.34f * (float)(i - 16));
    }
    // each lane's two lambdas, in FP32: which one is best
    float sum[2] = {0.f, 0.f};
    for (int j = 0; j < L; ++j) {
        PlanEntry e[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) e[b] = plan_entry(p, P, o, s, 4 * j + b);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float m = 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b) m = fminf(m, fmaf(-lam[h], e[b].x, e[b].q));
            sum[h] += m;
        }
    }
    const float thr32 = ldexpf(p.thr[c], s);
    const float v0 = fmaf(lam[0], thr32, sum[0]), v1 = fmaf(lam[1], thr32, sum[1]);
    float best = v1 > v0 ? v1 : v0, l32 = v1 > v0 ? lam[1] : lam[0];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, d), ol = __shfl_xor_sync(0xffffffffu, l32, d);
        if (ob > best || (ob == best && ol < l32) || best != best) best = ob, l32 = ol;
    }
    // Its bound in whole numbers, motif positions over the lanes: lambda = l 2^-20, P = X 2^-15 to
    // within 2^-16, so the sum is one of multiples of 2^-35 and off by at most L lambda 2^-16; |q|,
    // |P| <= 2^15 and L <= 256 keep it below 2^62.
    const int l = __float2int_rn(__shfl_sync(0xffffffffu, l32, 0) * 0x1p20f);
    long long sum64 = 0, maxabs = 0;
    bool fits = true;
    for (int j = lane; j < L; j += 32) {
        long long m = 0;
        int mx = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const PlanEntry e = plan_entry(p, P, o, s, 4 * j + b);
            fits = fits && fabsf(e.x) <= 32768.0f;
            const int X = __float2int_rn(e.x * 0x1p15f);
            m = min(m, ((long long)__float2int_rn(e.q) << 35) - (long long)l * X);
            mx = max(mx, abs(X));
        }
        sum64 += m;
        maxabs += mx;
    }
    sum64 = warp_sum(sum64);
    maxabs = warp_sum(maxabs);
    fits = __all_sync(0xffffffffu, fits);
    if (lane != 0) return;
    const double lambda = (double)l * 0x1p-20;
    // the reference's own rounding: |fl(sum) - sum| <= (L - 1) 2^-24 sum |P| (1 + 2^-14)
    const double thr = ldexp((double)p.thr[c], s) - (double)L * 0x1p-24 * ((double)maxabs * 0x1p-15 + 1.0);
    double bound = lambda * thr + (double)sum64 * 0x1p-35;
    bound -= (double)L * lambda * 0x1p-16 + 0x1p-48 * (lambda * fabs(thr) + fabs((double)sum64) * 0x1p-35);  // (FP64's own rounding)
    // down to the grid, kept within the scores a window can reach (2^23 units; 64 L scaled):
    // below them every window is a candidate, above them none is
    const double worst = ((double)p.thr[c] - p.guard[c]) * exp2((double)s);
    const double lim = e8 ? (double)(64 * L + 1) * 512.0 : 8388608.0;
    double t = worst;
    if (fits && bound > t) t = bound;  // (NaN: not taken)
    const double units = isnan(t) ? lim : floor(fmax(-lim, fmin(lim, t)));
    p.slot_thr[slot] = ldexpf((float)units, e8 ? -9 : -s);  // exact: |units| <= 2^23
}

// One block per k-step of a term: 256 units of 16 bytes, unit u = K core u / 128, row u % 128
// (at (16 core + row / 8) * 128 + (row % 8) * 16 of the step).  A core holds 2 (BF16) or 4 (E4M3)
// motif positions; rows without a column and positions beyond a column's length are zero.
__global__ void __launch_bounds__(256) plan_fill_kernel(PlanParams p)
{
    const int step = blockIdx.x;
    int t = 0, hi = p.ntiles;  // the tile: the last one that starts at or before the step
    while (hi - t > 1) {
        const int mid = (t + hi) >> 1;
        if (p.tiles[mid].off <= step) t = mid;
        else hi = mid;
    }
    const TileDesc td = p.tiles[t];
    const int within = step - td.off, term = within / td.g, k = within - term * td.g;
    const int core = threadIdx.x >> 7, row = threadIdx.x & 127;
    const int c = p.slot_col[t * kTileCols + row];
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c >= 0) {
        const int L = p.col_len[c];
        const uint32_t o = p.off[c];
        if (p.terms == kE4M3) {
            const int j = 8 * k + 4 * core;
            const uint32_t *src = reinterpret_cast<const uint32_t *>(p.e8 + o);
            if (j < L) v.x = src[j];
            if (j + 1 < L) v.y = src[j + 1];
            if (j + 2 < L) v.z = src[j + 2];
            if (j + 3 < L) v.w = src[j + 3];
        } else {
            const int j = 4 * k + 2 * core;
            const uint2 *src = reinterpret_cast<const uint2 *>((term ? p.lo : p.hi) + o);
            if (j < L) {
                const uint2 w = src[j];
                v.x = w.x, v.y = w.y;
            }
            if (j + 1 < L) {
                const uint2 w = src[j + 1];
                v.z = w.x, v.w = w.y;
            }
        }
    }
    reinterpret_cast<uint4 *>(p.abuf + (size_t)step * kStepBytes)[threadIdx.x] = v;
}

}  // namespace blamm
