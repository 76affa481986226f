// hist_kernels.cuh -- the hist module's theoretical score distributions and
// their p-value inversion on the GPU (one CTA per distinct distribution).
//
// Follows, operation for operation in FP32 (no contraction: __fmul_rn /
// __fadd_rn), the reference's
//   Motif::computeTheoreticalSpectrum  src/motif.cpp:151-192
//     a = nbins / (max - min), b = -a*min / L, q = round(a*PWM + b),
//     DP over positions with std::map<int, float> (a key exists once touched;
//     each key's float sum takes its terms in ascending source key, then base);
//   Histogram::generateTheoreticalHist src/hist.cpp:162-175
//     spectrum map<float, float>: score = (key - L*b) / a, insert keeps the
//     first of equal scores; setNumObservations overwrites the bin with
//     (size_t)(maxLength * probability) (src/motif.h:109-115);
//   ScoreHistogram::getScoreCutoff src/motif.cpp:47-69, in FP64.
// so thresholds equal the host's (and the reference's) bit for bit.  With
// fp64_dp the DP runs in FP64 instead (a more accurate distribution; not the
// reference's numbers).
//
// What bounds it: latency, the chain of positions (one barrier each) and what
// surrounds it.  A column's keys sit in shared memory, a step touches only the keys
// that its prefix can reach, and everything after the DP is done by all threads: which
// key of equal scores is the first is seen from its predecessor, which of a bin's keys
// is the last by a maximum, and the cutoff's running subtraction is exact while the
// counts add up to less than 2^53, so a suffix sum finds the same bin (above that one
// thread walks the bins as the reference does).  Columns that share a distribution
// (reverse complements) share the CTA.  4000 columns of 2000 motifs, 3 p-values, 250
// bins: 0.063 ms; with one CTA per column and the spectrum and the inversion walked by one
// thread 1.22 ms.
#pragma once
#include <cstdint>

namespace blamm {

constexpr int kTheoThreads = 256;

struct TheoHistParams {
    const float *P;         // column-major, p_rows x ncols
    int32_t p_rows;
    int32_t ncols;
    const int32_t *col_len;
    const int32_t *dist;    // per CTA: the column whose PWM gives the distribution
    const int32_t *users;   // the columns that have distribution i: users[user0[i]] .. users[user0[i + 1] - 1]
    const int32_t *user0;
    float bg[4];
    int32_t nbins;
    uint64_t max_length;
    int32_t kmax;            // capacity of the key arrays (entries)
    int32_t lmax;            // capacity in motif positions
    const float *pvalues;
    int32_t npv;
    float *thr;              // npv x ncols (or nullptr)
    unsigned long long *counts;  // ncols x nbins (or nullptr)
    int *status;             // set to 1 when a column's key range exceeds kmax
};

// Shared memory: two value arrays of kmax (float or double), nbins counts and winners, per
// motif position 4 quantised values, their order, the row's extremes and the prefix's key
// range.
__host__ __device__ inline size_t theo_smem_bytes(int kmax, int nbins, int lmax, int fp64)
{
    return 2 * (size_t)kmax * (fp64 ? 8 : 4) + 12 * (size_t)nbins + 36 * (size_t)lmax + 64;
}

template <typename T>
__device__ __forceinline__ T theo_mul(T a, T b);
template <>
__device__ __forceinline__ float theo_mul<float>(float a, float b) { return __fmul_rn(a, b); }
template <>
__device__ __forceinline__ double theo_mul<double>(double a, double b) { return __dmul_rn(a, b); }
template <typename T>
__device__ __forceinline__ T theo_add(T a, T b);
template <>
__device__ __forceinline__ float theo_add<float>(float a, float b) { return __fadd_rn(a, b); }
template <>
__device__ __forceinline__ double theo_add<double>(double a, double b) { return __dadd_rn(a, b); }

// A key that does not exist: a NaN that no arithmetic returns.
template <typename T>
__device__ __forceinline__ T theo_absent();
template <>
__device__ __forceinline__ float theo_absent<float>() { return __uint_as_float(0xFFABCDEFu); }
template <>
__device__ __forceinline__ double theo_absent<double>() { return __longlong_as_double((long long)0xFFFABCDEF0123456ull); }
__device__ __forceinline__ bool theo_exists(float v) { return __float_as_uint(v) != 0xFFABCDEFu; }
__device__ __forceinline__ bool theo_exists(double v) { return (unsigned long long)__double_as_longlong(v) != 0xFFFABCDEF0123456ull; }

template <typename T>
__device__ void theo_column(const TheoHistParams &p, uint8_t *smem)
{
    const int h = p.dist[blockIdx.x];
    const int L = p.col_len[h];
    const float *pwm = p.P + (size_t)h * p.p_rows;
    T *cur = reinterpret_cast<T *>(smem);
    T *nxt = cur + p.kmax;
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(nxt + p.kmax);
    int *win = reinterpret_cast<int *>(cnt + p.nbins);      // per bin: its last key
    int *q = win + p.nbins;                                 // 4 per position
    float *ext = reinterpret_cast<float *>(q + 4 * p.lmax); // per position: smallest and largest entry
    int *rng = reinterpret_cast<int *>(ext + 2 * p.lmax);   // per position: the prefix's first and last key
    uchar4 *ord = reinterpret_cast<uchar4 *>(rng + 2 * p.lmax);
    __shared__ float s_min, s_max, s_a, s_b;
    __shared__ int s_base, s_w;
    __shared__ unsigned long long s_part[kTheoThreads / 32], s_before[kTheoThreads / 32];
    __shared__ int s_found, s_serial;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const float *r = pwm + 4 * j;
        ext[2 * j] = fminf(fminf(r[0], r[1]), fminf(r[2], r[3]));
        ext[2 * j + 1] = fmaxf(fmaxf(r[0], r[1]), fmaxf(r[2], r[3]));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // Motif::getMinScore / getMaxScore: sequential float sums of the row extremes
        float mn = 0.0f, mx = 0.0f;
        for (int j = 0; j < L; ++j) {
            mn = __fadd_rn(mn, ext[2 * j]);
            mx = __fadd_rn(mx, ext[2 * j + 1]);
        }
        const float range = __fadd_rn(mx, -mn);
        const float a = __fdiv_rn((float)p.nbins, range);
        s_min = mn;
        s_max = mx;
        s_a = a;
        s_b = __fdiv_rn(__fmul_rn(-a, mn), (float)L);
    }
    __syncthreads();
    const float a = s_a, b = s_b;
    // per position: the quantised values, their extremes, and the order in which a key's
    // terms arrive: ascending source key = descending q, ties by base
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        int v[4];
        for (int k = 0; k < 4; ++k) q[4 * j + k] = v[k] = (int)roundf(__fadd_rn(__fmul_rn(a, pwm[4 * j + k]), b));
        rng[2 * j] = min(min(v[0], v[1]), min(v[2], v[3]));
        rng[2 * j + 1] = max(max(v[0], v[1]), max(v[2], v[3]));
        unsigned char o[4];
        for (int k = 0; k < 4; ++k) {
            int rank = 0;
            for (int m = 0; m < 4; ++m) rank += v[m] > v[k] || (v[m] == v[k] && m < k);
            o[rank] = (unsigned char)k;
        }
        ord[j] = make_uchar4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // the prefixes' key ranges, relative to the smallest key of any
        long long plo = 0, phi = 0, qmin = 0, qmax = 0;
        for (int j = 0; j < L; ++j) {
            plo += rng[2 * j];
            phi += rng[2 * j + 1];
            if (j == 0 || plo < qmin) qmin = plo;
            if (j == 0 || phi > qmax) qmax = phi;
        }
        const long long w = qmax - qmin + 1;
        s_base = (int)qmin;
        s_w = w > p.kmax ? -1 : (int)w;
        if (w <= p.kmax) {
            plo = phi = -qmin;
            for (int j = 0; j < L; ++j) {
                rng[2 * j] = (int)(plo += rng[2 * j]);
                rng[2 * j + 1] = (int)(phi += rng[2 * j + 1]);
            }
        }
    }
    __syncthreads();
    const int base = s_base;
    if (s_w < 0) {
        if (threadIdx.x == 0) atomicOr(p.status, 1);
        return;
    }
    // the DP; a step's keys outside its prefix's range do not exist (and are not touched)
    int lo = rng[0], hi = rng[1];
    for (int t = lo + threadIdx.x; t <= hi; t += blockDim.x) {  // position 0, bases in order
        T s = T(0);
        bool any = false;
        for (int k = 0; k < 4; ++k)
            if (q[k] - base == t) {
                s = theo_add<T>(s, (T)p.bg[k]);
                any = true;
            }
        cur[t] = any ? s : theo_absent<T>();
    }
    __syncthreads();
    for (int j = 1; j < L; ++j) {
        const int lo1 = rng[2 * j], hi1 = rng[2 * j + 1];
        const uchar4 o = ord[j];
        const int k0 = o.x, k1 = o.y, k2 = o.z, k3 = o.w;
        const int d[4] = {q[4 * j + k0], q[4 * j + k1], q[4 * j + k2], q[4 * j + k3]};
        const T g[4] = {(T)p.bg[k0], (T)p.bg[k1], (T)p.bg[k2], (T)p.bg[k3]};
        for (int t = lo1 + threadIdx.x; t <= hi1; t += blockDim.x) {
            T s = T(0);
            bool any = false;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int src = t - d[x];
                if (src >= lo && src <= hi) {
                    const T v = cur[src];
                    if (theo_exists(v)) {
                        s = theo_add<T>(s, theo_mul<T>(v, g[x]));
                        any = true;
                    }
                }
            }
            nxt[t] = any ? s : theo_absent<T>();
        }
        __syncthreads();
        T *const sw = cur;
        cur = nxt;
        nxt = sw;
        lo = lo1;
        hi = hi1;
    }
    // the histogram: of equal scores the first key is kept, of a bin's keys the last
    const float mn = s_min, mx = s_max;
    const float width = __fdiv_rn(__fadd_rn(mx, -mn), (float)p.nbins);
    const float lb = __fmul_rn((float)L, b);
    const float maxlen = (float)p.max_length;
    for (int i = threadIdx.x; i < p.nbins; i += blockDim.x) win[i] = -1;
    __syncthreads();
    auto score_of = [&](int t) { return __fdiv_rn(__fadd_rn((float)(t + base), -lb), a); };
    for (int t = lo + threadIdx.x; t <= hi; t += blockDim.x) {
        if (!theo_exists(cur[t])) continue;
        const float score = score_of(t);
        int u = t - 1;
        while (u >= lo && !theo_exists(cur[u])) --u;
        if (u >= lo && score == score_of(u)) continue;  // map::insert keeps the first
        int bin = (int)__fdiv_rn(__fadd_rn(score, -mn), width);
        bin = max(0, min(p.nbins - 1, bin));
        atomicMax(&win[bin], t);
    }
    __syncthreads();
    unsigned long long mine = 0;
    bool big = false;  // a count, or their sum, may exceed 2^53
    for (int i = threadIdx.x; i < p.nbins; i += blockDim.x) {
        unsigned long long n = 0;
        if (win[i] >= 0) {
            const T v = cur[win[i]];
            if (sizeof(T) == 4) n = (unsigned long long)__fmul_rn(maxlen, (float)v);
            else n = (unsigned long long)__dmul_rn((double)p.max_length, (double)v);
        }
        cnt[i] = n;
        big = big || n > (1ull << 40);  // (at most 4096 bins)
    }
    if (threadIdx.x == 0) s_serial = 0;
    __syncthreads();
    if (big) s_serial = 1;
    __syncthreads();
    for (int i = p.user0[blockIdx.x]; i < p.user0[blockIdx.x + 1]; ++i)
        if (p.counts)
            for (int k = threadIdx.x; k < p.nbins; k += blockDim.x)
                p.counts[(size_t)p.users[i] * p.nbins + k] = cnt[k];
    if (!p.thr) return;
    auto publish = [&](int v, float cut) {  // one thread
        for (int i = p.user0[blockIdx.x]; i < p.user0[blockIdx.x + 1]; ++i)
            p.thr[(size_t)v * p.ncols + p.users[i]] = cut;
    };
    auto cutoff = [&](double curr, int i) {  // inside bin i, curr left of its count
        const double frac = __ddiv_rn(curr, (double)cnt[i]);
        const float c = (float)__dadd_rn(__dmul_rn(frac, (double)i), __dmul_rn(__dadd_rn(1.0, -frac), (double)(i + 1)));
        return __fadd_rn(__fmul_rn(c, width), mn);
    };
    if (s_serial) {
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int i = 0; i < p.nbins; ++i) tot = __dadd_rn(tot, (double)cnt[i]);
            for (int v = 0; v < p.npv; ++v) {
                double curr = __dmul_rn((double)p.pvalues[v], tot);
                float cut = mx;
                for (int i = p.nbins - 1; i >= 0; --i) {
                    if (!((double)cnt[i] < curr)) {
                        cut = cutoff(curr, i);
                        break;
                    }
                    curr = __dadd_rn(curr, -(double)cnt[i]);
                }
                publish(v, cut);
            }
        }
        return;
    }
    // thread i's contiguous bins (from the top), the sum of the bins above them
    const int per = (p.nbins + blockDim.x - 1) / blockDim.x;
    const int i1 = p.nbins - 1 - (int)threadIdx.x * per, i0 = max(0, i1 - per + 1);  // empty if i1 < 0
    for (int i = i1; i >= i0; --i) mine += cnt[i];
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    if (threadIdx.x < kTheoThreads / 32) {
        unsigned long long v = 0;
        for (int k = 0; k < (int)threadIdx.x; ++k) v += s_part[k];
        s_before[threadIdx.x] = v;
    }
    __syncthreads();
    const unsigned long long above = s_before[warp] + incl - mine;
    const unsigned long long total = s_before[kTheoThreads / 32 - 1] + s_part[kTheoThreads / 32 - 1];
    for (int v = 0; v < p.npv; ++v) {
        const double x = __dmul_rn((double)p.pvalues[v], (double)total);
        // the first bin from the top whose count is not less than what is left: every sum is
        // an integer below 2^53 and every difference exact
        if (threadIdx.x == 0) s_found = 0;
        __syncthreads();
        unsigned long long sum = above;
        if (!((double)(above + mine) < x) && (threadIdx.x == 0 || (double)above < x))
            for (int i = i1; i >= i0; --i) {
                if (!((double)(sum + cnt[i]) < x)) {
                    publish(v, cutoff(__dadd_rn(x, -(double)sum), i));
                    s_found = 1;
                    break;
                }
                sum += cnt[i];
            }
        __syncthreads();
        if (threadIdx.x == 0 && !s_found) publish(v, mx);
    }
}

__global__ void __launch_bounds__(kTheoThreads) theoretical_hist_kernel(TheoHistParams p)
{
    extern __shared__ __align__(16) uint8_t smem_theo[];
    theo_column<float>(p, smem_theo);
}

__global__ void __launch_bounds__(kTheoThreads) theoretical_hist64_kernel(TheoHistParams p)
{
    extern __shared__ __align__(16) uint8_t smem_theo[];
    theo_column<double>(p, smem_theo);
}

}  // namespace blamm
