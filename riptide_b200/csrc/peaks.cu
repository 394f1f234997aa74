// Peak detection on the device (peak_detection.py:38-240 of the reference): the per-segment
// S/N statistics that the dynamic threshold is fitted to, and the selection of the
// periodogram points above that threshold, for every (trial, width) of a batch of
// periodograms at once. The threshold fit itself (a degree-2 polynomial in log f over a few
// hundred control points) and the clustering of the selected points run on the host, in the
// reference's own numpy calls (riptide_b200/peaks.py).
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace rt {

constexpr int kSegMaxPoints = 16384;  // points per segment

// numpy's linear interpolation between two order statistics (numpy _lerp) of float64
// values: the reference takes the percentiles of each width's S/N after casting them to
// float64 (peak_detection.py:205), so the difference b - a is a float64 one.
__device__ __forceinline__ double np_lerp(double a, double b, double t)
{
    const double d = __dsub_rn(b, a);
    return (t >= 0.5) ? __dsub_rn(b, __dmul_rn(d, __dsub_rn(1.0, t))) : __dadd_rn(a, __dmul_rn(d, t));
}


struct SegTrial {
    unsigned long long row0;  // first periodogram row of the trial
    int seg0, m, p, pad;      // first global segment, segments, points per segment
};

// ------------------------------------------------------------------------------------
// Segment statistics (segment_stats, peak_detection.py:38-86): for every segment and width,
// sc = median + nstd * IQR / 1.349 of the segment's S/N, and the segment's median frequency fc.
//
// What is asked for is three percentiles, six order statistics, of some thousand values; a warp
// selects them without sorting. It histograms its column over 1,024 equal spans of the keys
// (integers in the order of the values) between the column's least and largest, finds the spans
// of the ranks by a scan, and gathers the few values in them, which are ranked against one
// another. A span with more than kSelList values is divided again, until it holds one key.
// The CTA holds its columns in shared memory, one read of the periodogram. Bound: the warps'
// instructions, six to ten a value and pass. 1,048 segments of 1,174 points by 10 widths: 750 us
// by bitonic sorts of columns padded to 2,048; by selection 80 us.
// ------------------------------------------------------------------------------------
constexpr int kSelSpans = 1024;  // 32 per lane
constexpr int kSelList = 128;    // 4 values per lane
constexpr int kKeys = 8;         // keys a lane holds at a time
constexpr int kSegWarps = 16;    // most warps of a CTA
constexpr size_t kSegSmem = 110 * 1024;  // two CTAs per SM

struct SelWarp {
    unsigned hist[kSelSpans + 32];  // a lane's 32 spans are 33 words from the next one's
    union {
        unsigned k32[3][kSelList];
        unsigned long long k64[kSelList];
    } list;
    unsigned long long found[2];
};

// Values of the keys (order_key).
__device__ __forceinline__ float key_value(unsigned k)
{
    return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu));
}
__device__ __forceinline__ double key_value(unsigned long long k)
{
    return __longlong_as_double((long long)(k ^ ((k >> 63) ? 1ull << 63 : ~0ull)));
}

__device__ __forceinline__ int key_bits(unsigned k) { return 32 - __clz((int)k); }
__device__ __forceinline__ int key_bits(unsigned long long k) { return 64 - __clzll((long long)k); }

// A warp's selection among the n keys key(0..n-1) that lie in [lo, hi].
template <typename K, typename Read>
struct Selection {
    SelWarp& w;
    Read key;
    int n, lane;
    K lo, hi;
    int shift;
    unsigned base, sum;  // keys in the spans before the lane's 32, and in them

    // f(k, valid) of the keys, the warp together, kKeys loads in flight
    template <typename F>
    __device__ __forceinline__ void each(F f) const
    {
        int i = lane;
#pragma unroll 1
        for (; i - lane + 32 * kKeys <= n; i += 32 * kKeys) {
            K k[kKeys];
#pragma unroll
            for (int u = 0; u < kKeys; ++u) k[u] = key(i + 32 * u);
#pragma unroll
            for (int u = 0; u < kKeys; ++u) f(k[u], true);
        }
#pragma unroll 1
        for (; i - lane < n; i += 32) f(i < n ? key(i) : K(0), i < n);
    }

    // appends k to the list where `in`; `count` keys are in it
    __device__ __forceinline__ void append(K* list, unsigned& count, K k, bool in) const
    {
        const unsigned m = __ballot_sync(~0u, in);
        if (m == 0) return;
        if (in) list[count + __popc(m & ((1u << lane) - 1))] = k;
        count += __popc(m);
    }

    __device__ void range()  // [lo, hi] of all keys
    {
        K a = ~K(0), b = 0;
        each([&](K k, bool valid) {
            a = min(a, valid ? k : ~K(0));
            b = max(b, k);
        });
        lo = a;
        hi = b;
        for (int d = 16; d > 0; d >>= 1) {
            lo = min(lo, __shfl_xor_sync(~0u, lo, d));
            hi = max(hi, __shfl_xor_sync(~0u, hi, d));
        }
    }

    template <bool kAll>  // kAll: every key is in [lo, hi]
    __device__ __forceinline__ void histogram()
    {
        shift = max(0, key_bits(hi - lo) - 10);
        __syncwarp();
        for (int i = lane; i < kSelSpans + 32; i += 32) w.hist[i] = 0;
        __syncwarp();
        const K span = hi - lo;
        each([&](K k, bool valid) {
            const K d = k - lo;
            const unsigned s = (unsigned)(d >> shift);
            if (kAll ? valid : valid && d <= span) atomicAdd(&w.hist[s + (s >> 5)], 1u);
        });
        __syncwarp();
        sum = 0;
        for (int j = 0; j < 32; ++j) sum += w.hist[lane * 33 + j];
        base = sum;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(~0u, base, d);
            if (lane >= d) base += o;
        }
        base -= sum;
    }

    // the span of rank r among the keys in [lo, hi]: its number, the keys below it, its keys
    __device__ void find(unsigned r, unsigned& span, unsigned& below, unsigned& in) const
    {
        const int L = __ffs(__ballot_sync(~0u, r >= base && r < base + sum)) - 1;
        const unsigned b0 = __shfl_sync(~0u, base, L);
        const unsigned c = w.hist[L * 33 + lane];
        unsigned incl = c;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(~0u, incl, d);
            if (lane >= d) incl += o;
        }
        const int j = __ffs(__ballot_sync(~0u, b0 + incl > r)) - 1;
        in = __shfl_sync(~0u, c, j);
        below = b0 + __shfl_sync(~0u, incl, j) - in;
        span = 32u * L + j;
    }

    // last offset from lo of span s
    __device__ K span_end(unsigned s) const
    {
        const K e = (K(s + 1) << shift) - 1;
        return min(e, K(hi - lo));
    }

    // the values of ranks r0 and r1 among the c listed keys
    __device__ __noinline__ void rank(const K* list, unsigned c, unsigned r0, unsigned r1, K& v0, K& v1)
    {
        K* found = reinterpret_cast<K*>(w.found);
        __syncwarp();
        for (unsigned i = lane; i < c; i += 32) {
            const K x = list[i];
            unsigned r = 0;
            for (unsigned j = 0; j < c; ++j) {
                const K y = list[j];
                r += y < x || (y == x && j < i);
            }
            if (r == r0) found[0] = x;
            if (r == r1) found[1] = x;
        }
        __syncwarp();
        v0 = found[0];
        v1 = found[1];
        __syncwarp();
    }

    // the values of ranks r0 and r1 (r0 or r0 + 1) among the keys in [lo, hi]
    __device__ __noinline__ void pair(unsigned r0, unsigned r1, K* list, K& v0, K& v1)
    {
        for (;;) {
            histogram<false>();
            unsigned s0, b0, c0, s1, b1, c1;
            find(r0, s0, b0, c0);
            find(r1, s1, b1, c1);
            const unsigned c = b1 + c1 - b0;
            const K first = lo + (K(s0) << shift), end0 = lo + span_end(s0);
            if (c <= kSelList) {
                const K span = lo + span_end(s1) - first;
                unsigned count = 0;
                each([&](K k, bool valid) { append(list, count, k, valid && k - first <= span); });
                rank(list, c, r0 - b0, r1 - b0, v0, v1);
                return;
            }
            if (s0 != s1) {  // the last one of its span and the first one of another
                const K first1 = lo + (K(s1) << shift);
                K a = 0, b = ~K(0);
                each([&](K k, bool valid) {
                    if (valid && k <= end0) a = max(a, k);
                    if (valid && k >= first1) b = min(b, k);
                });
                v0 = a;
                v1 = b;
                for (int d = 16; d > 0; d >>= 1) {
                    v0 = max(v0, __shfl_xor_sync(~0u, v0, d));
                    v1 = min(v1, __shfl_xor_sync(~0u, v1, d));
                }
                return;
            }
            if (shift == 0) {
                v0 = v1 = first;
                return;
            }
            lo = first;
            hi = end0;
            r0 -= b0;
            r1 -= b0;
        }
    }
};

template <typename K, typename Read>
__device__ __forceinline__ Selection<K, Read> selection(SelWarp& w, Read key, int n)
{
    return Selection<K, Read>{w, key, n, (int)(threadIdx.x & 31), 0, 0, 0, 0, 0};
}

// sc of one column of n keys in shared memory
__device__ double column_threshold(SelWarp& w, const unsigned* col, int n, double nstd)
{
    auto S = selection<unsigned>(w, [col](int i) { return col[i]; }, n);
    const int lane = S.lane;
    S.range();
    S.histogram<true>();
    // np.percentile(x, q), method 'linear', of float32 S/N cast to float64: their order is the
    // same either way
    const double qs[3] = {0.25, 0.5, 0.75};
    double frac[3];
    unsigned r0[3], r1[3], below[3], c[3], first[3], span[3], last[3];
    bool listed = true;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double v = __dmul_rn((double)(n - 1), qs[q]);
        const double prev = floor(v);
        frac[q] = __dsub_rn(v, prev);
        r0[q] = (unsigned)prev;
        r1[q] = min(r0[q] + 1, (unsigned)n - 1);
        unsigned s0, s1, c0, b1, c1;
        S.find(r0[q], s0, below[q], c0);
        s1 = s0;
        b1 = below[q];
        c1 = c0;
        if (r1[q] >= b1 + c1) S.find(r1[q], s1, b1, c1);
        c[q] = b1 + c1 - below[q];
        first[q] = S.lo + (s0 << S.shift);
        last[q] = S.lo + S.span_end(s1);
        span[q] = last[q] - first[q];
        listed = listed && c[q] <= kSelList;
    }
    unsigned v0[3], v1[3];
    if (listed) {
        unsigned count[3] = {0, 0, 0};
        S.each([&](unsigned k, bool valid) {
            const bool in0 = k - first[0] <= span[0], in1 = k - first[1] <= span[1],
                       in2 = k - first[2] <= span[2];
            if (!__any_sync(~0u, valid && (in0 || in1 || in2))) return;
            S.append(w.list.k32[0], count[0], k, valid && in0);
            S.append(w.list.k32[1], count[1], k, valid && in1);
            S.append(w.list.k32[2], count[2], k, valid && in2);
        });
#pragma unroll
        for (int q = 0; q < 3; ++q)
            S.rank(w.list.k32[q], c[q], r0[q] - below[q], r1[q] - below[q], v0[q], v1[q]);
    } else {
#pragma unroll 1
        for (int q = 0; q < 3; ++q) {
            S.lo = first[q];
            S.hi = last[q];
            S.pair(r0[q] - below[q], r1[q] - below[q], w.list.k32[0], v0[q], v1[q]);
        }
    }
    double s[3];
#pragma unroll
    for (int q = 0; q < 3; ++q)
        s[q] = np_lerp((double)key_value(v0[q]), (double)key_value(v1[q]), frac[q]);
    const double sstd = __ddiv_rn(__dsub_rn(s[2], s[0]), 1.349);
    return __dadd_rn(s[1], __dmul_rn(nstd, sstd));
}

// np.median of the frequencies 1/period: the middle value, or the mean of the middle two. The
// reciprocal of positive periods falls as they rise, so the middle ones are found among the
// periods and two reciprocals taken. Those of a search rise but for overlaps at its changes of
// bins: the ones in the middle are checked first, by counting. (Other periods, none of a search,
// are selected by their reciprocals.)
struct PeriodKey {
    const double* periods;
    __device__ __forceinline__ unsigned long long operator()(int i) const
    {
        return order_key(__ldg(periods + i));
    }
};
struct ReciprocalKey {
    const double* periods;
    __device__ __noinline__ unsigned long long operator()(int i) const
    {
        return order_key(__ddiv_rn(1.0, __ldg(periods + i)));
    }
};

__device__ __noinline__ double median_frequency(SelWarp& w, const double* __restrict__ periods, int n)
{
    typedef unsigned long long K;
    const int mid = n / 2, mid0 = (n & 1) ? mid : mid - 1;  // ranks of the middle frequencies
    auto P = selection<K>(w, PeriodKey{periods}, n);
    // ranks of the periods
    const unsigned r0 = n - 1 - mid, r1 = n - 1 - mid0;
    K v0 = P.key(r0), v1 = P.key(r1);
    const K zero = order_key(0.0), inf = order_key((double)INFINITY);
    unsigned below0 = 0, upto0 = 0, below1 = 0, upto1 = 0, bad = 0;
    P.each([&](K k, bool valid) {
        below0 += valid && k < v0;
        upto0 += valid && k <= v0;
        below1 += valid && k < v1;
        upto1 += valid && k <= v1;
        bad += valid && !(k > zero && k <= inf);
    });
    below0 = __reduce_add_sync(~0u, below0);
    upto0 = __reduce_add_sync(~0u, upto0);
    below1 = __reduce_add_sync(~0u, below1);
    upto1 = __reduce_add_sync(~0u, upto1);
    double f0, f1;
    if (__any_sync(~0u, bad)) {
        auto F = selection<K>(w, ReciprocalKey{periods}, n);
        F.range();
        F.pair(mid0, mid, w.list.k64, v0, v1);
        f0 = key_value(v0);
        f1 = key_value(v1);
    } else {
        if (!(below0 <= r0 && r0 < upto0 && below1 <= r1 && r1 < upto1)) {
            P.range();
            P.pair(r0, r1, w.list.k64, v0, v1);
        }
        f0 = __ddiv_rn(1.0, key_value(v1));
        f1 = __ddiv_rn(1.0, key_value(v0));
    }
    return (n & 1) ? f1 : __ddiv_rn(__dadd_rn(f0, f1), 2.0);
}

// words from one column of n keys to the next: the columns of a row fall into different banks
__host__ __device__ __forceinline__ int seg_pitch(int n) { return ((n + 27) & ~31) + 4; }

// CTA (segment, group of `gw` widths): one warp per column; the first group has the frequencies.
__global__ void __launch_bounds__(32 * kSegWarps, 2)
    k_peak_segments(const double* __restrict__ periods, const float* __restrict__ snrs, int nw,
                    int gw, const SegTrial* __restrict__ trials, int ntrials, double nstd,
                    double* __restrict__ fc, double* __restrict__ sc)
{
    extern __shared__ __align__(16) char seg_smem[];
    const int seg = blockIdx.x, col0 = blockIdx.y * gw, cols = min(gw, nw - col0);
    int lo = 0, hi = ntrials - 1;  // trial of this segment
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (trials[mid].seg0 <= seg) lo = mid;
        else hi = mid - 1;
    }
    const SegTrial T = trials[lo];
    const int p = T.p, pitch = seg_pitch(p), warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const size_t r0 = T.row0 + (size_t)(seg - T.seg0) * p;
    SelWarp& w = reinterpret_cast<SelWarp*>(seg_smem)[warp];
    unsigned* keys = reinterpret_cast<unsigned*>(seg_smem + warps * sizeof(SelWarp));
    if (warp == warps - 1) {  // the frequencies, while the others load the columns
        if (blockIdx.y == 0) {
            const double f = median_frequency(w, periods + r0, p);
            if ((threadIdx.x & 31) == 0) fc[seg] = f;
        }
    } else {
        // a thread keeps to one column: as many whole rows at a time as there are threads for
        const int di = (blockDim.x - 32) / cols, i0 = threadIdx.x / cols, c = threadIdx.x - i0 * cols;
        const float* from = snrs + (r0 + i0) * nw + col0 + c;
        unsigned* to = keys + c * pitch;
        for (int i = i0 < di ? i0 : p; i < p; i += 8 * di, from += 8 * (size_t)di * nw) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i + u * di < p) v[u] = __ldg(from + (size_t)(u * di) * nw);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i + u * di < p) to[i + u * di] = order_key(v[u]);
        }
    }
    __syncthreads();
    for (int t = warp; t < cols; t += warps) {
        const double v = column_threshold(w, keys + t * pitch, p, nstd);
        if ((threadIdx.x & 31) == 0) sc[(size_t)seg * nw + col0 + t] = v;
    }
}

// First and last period of every trial's periodogram (the segment layout's frequency span).
__global__ void k_period_ends(const double* __restrict__ periods,
                              const unsigned long long* __restrict__ row_offsets, int ntrials,
                              double* __restrict__ ends)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntrials) return;
    ends[2 * t] = periods[row_offsets[t]];
    ends[2 * t + 1] = periods[row_offsets[t + 1] - 1];
}

// Points above the dynamic threshold poly(log f) and above smin (find_peaks_single,
// peak_detection.py:112-146), as (row * nw + iw), in any order.
__global__ void k_peak_select(const double* __restrict__ periods, const float* __restrict__ snrs,
                              int nw, const unsigned long long* __restrict__ row_trial_end,
                              int ntrials, const double* __restrict__ coef, int ncoef,
                              double smin, unsigned long long rows,
                              unsigned long long* __restrict__ sel, unsigned long long cap,
                              unsigned long long* __restrict__ count)
{
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x, n = rows * nw;
    for (unsigned long long e0 = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; e0 < n;
         e0 += 8 * step) {
        float v[8];  // eight loads in flight
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (e0 + u * step < n) v[u] = __ldg(snrs + e0 + u * step);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const unsigned long long e = e0 + u * step;
            // nearly all points end here: the row and width of the others only
            if (e >= n || !((double)v[u] > smin)) continue;
            const double s = (double)v[u];
            const unsigned long long r = e / nw;
            const int iw = (int)(e - r * nw);
            int lo = 0, hi = ntrials - 1;  // first trial whose end is beyond r
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (row_trial_end[mid] > r) hi = mid;
                else lo = mid + 1;
            }
            const double x = log(__ddiv_rn(1.0, periods[r]));
            const double* c = coef + ((size_t)lo * nw + iw) * ncoef;
            double y = 0.0;  // np.polyval: y = y * x + c_k, no fused multiply-add
            for (int k = 0; k < ncoef; ++k) y = __dadd_rn(__dmul_rn(y, x), c[k]);
            if (s > y) {
                const unsigned long long slot = atomicAdd(count, 1ull);
                if (slot < cap) sel[slot] = e;
            }
        }
    }
}

}  // namespace rt

using namespace rt;

extern "C" int rt_peak_segments(const double* d_periods, const float* d_snrs, size_t num_widths,
                                const uint64_t* h_row_offsets, size_t ntrials,
                                const double* h_tobs, double segwidth, double nstd,
                                uint64_t* h_seg_offsets, double* d_fc, double* d_sc, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (!d_periods || !h_row_offsets || !h_tobs || !h_seg_offsets)
        return set_error(RT_EINVAL, "null argument");
    if (num_widths == 0 || num_widths > 65535) return set_error(RT_EINVAL, "bad number of widths");
    // segment layout of every trial: m = ceil(|f[-1] - f[0]| / w), p = rows // m; the first
    // and last period of every trial gathered on the device and copied back at once
    if (ntrials == 0) return set_error(RT_EINVAL, "no periodograms");
    for (size_t t = 0; t < ntrials; ++t)
        if (h_row_offsets[t + 1] <= h_row_offsets[t])
            return set_error(RT_EINVAL, "periodogram %zu is empty", t);
    std::vector<double> ends(2 * ntrials);
    {
        unsigned long long* d_ro = nullptr;
        double* d_ends = nullptr;
        const size_t ro_bytes = (ntrials + 1) * sizeof(uint64_t);
        const size_t ro_room = (ro_bytes + 15) & ~size_t(15);
        RT_TRY_CUDA(scratch_malloc((void**)&d_ro, ro_room + 2 * ntrials * sizeof(double), st));
        d_ends = reinterpret_cast<double*>(reinterpret_cast<char*>(d_ro) + ro_room);
        cudaError_t e = cudaMemcpyAsync(d_ro, h_row_offsets, ro_bytes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            k_period_ends<<<(unsigned)((ntrials + 255) / 256), 256, 0, st>>>(d_periods, d_ro,
                                                                            (int)ntrials, d_ends);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(ends.data(), d_ends, 2 * ntrials * sizeof(double),
                                cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaFreeAsync(d_ro, st);
        if (e != cudaSuccess) return check_cuda(e, "peak_segments layout");
    }
    std::vector<SegTrial> tr(ntrials);
    uint64_t seg = 0, pmax = 1;
    h_seg_offsets[0] = 0;
    for (size_t t = 0; t < ntrials; ++t) {
        const double w = segwidth / h_tobs[t];
        const double span = std::fabs(1.0 / ends[2 * t + 1] - 1.0 / ends[2 * t]);
        const double mf = std::ceil(span / w);
        if (!(mf >= 1.0) || !std::isfinite(mf))
            return set_error(RT_EINVAL, "periodogram %zu spans no frequency segment", t);
        const uint64_t rows = h_row_offsets[t + 1] - h_row_offsets[t];
        const uint64_t m = (uint64_t)mf;
        const uint64_t p = rows / m;
        if (p == 0) return set_error(RT_EINVAL, "periodogram %zu has fewer rows than segments", t);
        if (p > (uint64_t)kSegMaxPoints)
            return set_error(RT_EINVAL, "segments of %llu points exceed the device limit (%d)",
                             (unsigned long long)p, kSegMaxPoints);
        pmax = std::max(pmax, p);
        tr[t].row0 = h_row_offsets[t];
        tr[t].seg0 = (int)seg;
        tr[t].m = (int)m;
        tr[t].p = (int)p;
        tr[t].pad = 0;
        seg += m;
        h_seg_offsets[t + 1] = seg;
    }
    if (!d_fc || !d_sc) return RT_OK;  // layout only
    if (!d_snrs) return set_error(RT_EINVAL, "null argument");
    if (seg >= (1ull << 31)) return set_error(RT_EINVAL, "too many segments");
    SegTrial* d_tr = nullptr;
    RT_TRY_CUDA(scratch_malloc((void**)&d_tr, ntrials * sizeof(SegTrial), st));
    int s = check_cuda(cudaMemcpyAsync(d_tr, tr.data(), ntrials * sizeof(SegTrial),
                                       cudaMemcpyHostToDevice, st), "peak_segments");
    // the fewest groups of widths whose columns leave room for two CTAs per SM and
    // have a loading thread each; a group of one
    // always does (16,384 points: 64 KiB)
    const int nw = (int)num_widths;
    auto warps_of = [](int gw) { return std::min(gw + 1, kSegWarps); };
    auto smem_of = [&](int gw) {
        return warps_of(gw) * sizeof(SelWarp) + (size_t)gw * seg_pitch((int)pmax) * sizeof(unsigned);
    };
    int groups = 1, gw = nw;
    while (gw > 32 * (kSegWarps - 1) || (gw > 1 && smem_of(gw) > kSegSmem)) {
        ++groups;
        gw = (nw + groups - 1) / groups;
    }
    groups = (nw + gw - 1) / gw;
    if (s == RT_OK)
        s = check_cuda(cudaFuncSetAttribute(k_peak_segments,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kSegSmem),
                       "peak_segments");
    if (s == RT_OK && seg > 0) {
        k_peak_segments<<<dim3((unsigned)seg, (unsigned)groups), 32 * warps_of(gw), smem_of(gw),
                          st>>>(d_periods, d_snrs, nw, gw, d_tr, (int)ntrials, nstd, d_fc, d_sc);
        s = check_cuda(cudaGetLastError(), "peak_segments");
    }
    cudaFreeAsync(d_tr, st);
    return s;
}

extern "C" int rt_peak_select(const double* d_periods, const float* d_snrs, size_t num_widths,
                              const uint64_t* h_row_offsets, size_t ntrials, const double* d_coef,
                              size_t num_coef, double smin, uint64_t* d_sel, size_t capacity,
                              size_t* h_count, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (!d_periods || !d_snrs || !h_row_offsets || !d_coef || !d_sel || !h_count)
        return set_error(RT_EINVAL, "null argument");
    if (num_coef == 0 || num_widths == 0) return set_error(RT_EINVAL, "bad coefficient count");
    const uint64_t rows = h_row_offsets[ntrials];
    unsigned long long* d_aux = nullptr;  // [ntrials] trial row ends, then the counter
    RT_TRY_CUDA(scratch_malloc((void**)&d_aux, (ntrials + 1) * sizeof(unsigned long long), st));
    int s = check_cuda(cudaMemcpyAsync(d_aux, h_row_offsets + 1, ntrials * sizeof(uint64_t),
                                       cudaMemcpyHostToDevice, st), "peak_select");
    if (s == RT_OK)
        s = check_cuda(cudaMemsetAsync(d_aux + ntrials, 0, sizeof(unsigned long long), st), "peak_select");
    if (s == RT_OK && rows > 0) {
        const size_t work = (size_t)rows * num_widths;
        const int grid = (int)std::min<size_t>((work + 255) / 256, 148 * 8);
        k_peak_select<<<grid, 256, 0, st>>>(d_periods, d_snrs, (int)num_widths, d_aux,
                                            (int)ntrials, d_coef, (int)num_coef, smin, rows,
                                            (unsigned long long*)d_sel, capacity, d_aux + ntrials);
        s = check_cuda(cudaGetLastError(), "peak_select");
    }
    unsigned long long count = 0;
    if (s == RT_OK)
        s = check_cuda(cudaMemcpyAsync(&count, d_aux + ntrials, sizeof(count),
                                       cudaMemcpyDeviceToHost, st), "peak_select");
    if (s == RT_OK) s = check_cuda(cudaStreamSynchronize(st), "peak_select");
    cudaFreeAsync(d_aux, st);
    if (s != RT_OK) return s;
    *h_count = (size_t)count;
    if (count > capacity)
        return set_error(RT_EINVAL, "%llu points pass the threshold (capacity %zu)", count, capacity);
    return RT_OK;
}
