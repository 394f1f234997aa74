// Adjoints (transposed Jacobians) of the search steps, for gradients of a loss of the
// periodogram with respect to the searched series. The reference's search is not
// differentiable; these follow its forward arithmetic (snr.hpp:37-65, transforms.hpp:13-61,
// downsample.hpp:44-82, time_series.py:67-93) so that the gradient is the one of the function
// the forward computes.
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "snr_core.cuh"

namespace rt {

// ------------------------------------------------------------------------------------
// Boxcar S/N: S/N_w = ((h+b) dmax_w - b sum) / sigma, dmax_w = max_i C[i+w] - C[i] with C the
// circular prefix sum. d S/N_w / d x_q = (h+b)/sigma on the w phases after the first
// maximising i, minus b/sigma on every phase.
// ------------------------------------------------------------------------------------
constexpr int kSnrBwdMaxWidths = 64;

__global__ void k_snr2_backward(const float* __restrict__ x, int rows, int b,
                                const int* __restrict__ widths, int nw, float stdnoise,
                                const float* __restrict__ gsnr, float* __restrict__ gx, int wmax)
{
    extern __shared__ float sC[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    float* C = sC + (size_t)wib * (b + wmax + 1);
    __shared__ int s_best[32][kSnrBwdMaxWidths];
    for (int r = blockIdx.x * wpb + wib; r < rows; r += gridDim.x * wpb) {
        const float* xr = x + (size_t)r * b;
        // circular prefix: float of the double running sum (kernels.hpp:73-101), as the
        // forward stores it; the wrap-around part as cr[j] + float(sum)
        double carry = 0.0;
        for (int c0 = 0; c0 < b; c0 += 32) {
            const int c = c0 + lane;
            const double v = (c < b) ? (double)xr[c] : 0.0;
            double incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (c < b) C[c] = (float)(carry + incl);
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        const float sumx = (float)carry;
        for (int j = lane; j < wmax; j += 32) C[b + j] = __fadd_rn(C[j], sumx);
        __syncwarp();
        // first maximising phase per width
        for (int k = 0; k < nw; ++k) {
            const int w = widths[k];
            float best = -INFINITY;
            int bi = b;
            for (int i = lane; i < b; i += 32) {
                const float d = __fsub_rn(C[i + w], C[i]);
                if (d > best) {
                    best = d;
                    bi = i;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            if (lane == 0) s_best[wib][k] = bi;
        }
        __syncwarp();
        // gradient of the row
        const float* g = gsnr + (size_t)r * nw;
        double base = 0.0;
        for (int k = 0; k < nw; ++k) {
            float hb, be;
            boxcar_coefs(b, widths[k], &hb, &be);
            base -= (double)g[k] * (double)be / (double)stdnoise;
        }
        for (int q = lane; q < b; q += 32) {
            double acc = base;
            for (int k = 0; k < nw; ++k) {
                const int w = widths[k];
                int off = q - s_best[wib][k] - 1;  // position of q in the window
                off += (off < 0) ? b : 0;
                if (off < w) {
                    float hb, be;
                    boxcar_coefs(b, w, &hb, &be);
                    acc += (double)g[k] * (double)hb / (double)stdnoise;
                }
            }
            gx[(size_t)r * b + q] = (float)acc;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------
// FFA transpose. The forward merges node (row0, n) from its head (rows row0 + [0, n/2)) and
// tail (the rest): out[s] = head[h(s)] + roll(tail[t(s)], -(s - t(s))). The transpose, level by
// level from the root: a head row j gathers the rows s with h(s) = j; a tail row j gathers the
// rows s with t(s) = j, rolled back by s - t(s). Rows of nodes that no longer split are copied.
// ------------------------------------------------------------------------------------
struct TRow {
    int row0, n, kind, j;  // parent node; kind 0 copy, 1 head row j, 2 tail row j
};

// first s in [0, n) with merge_row(k, s) >= v (merge_row is non-decreasing in s)
__device__ __forceinline__ int first_at_least(float k, int n, int v)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (merge_row(k, mid) >= v) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

__global__ void k_ffa_transpose_level(const float* __restrict__ gp, float* __restrict__ gc,
                                      const TRow* __restrict__ tab, int m, int b)
{
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < m;
         r += (gridDim.x * blockDim.x) >> 5) {
        const TRow e = tab[r];
        float* out = gc + (size_t)r * b;
        if (e.kind == 0) {
            for (int c = lane; c < b; c += 32) out[c] = gp[(size_t)r * b + c];
            continue;
        }
        const MergeCoef mc = merge_coef(e.n);
        const float k = (e.kind == 1) ? mc.kh : mc.kt;
        const int s0 = first_at_least(k, e.n, e.j), s1 = first_at_least(k, e.n, e.j + 1);
        for (int c = lane; c < b; c += 32) {
            float acc = 0.0f;
            for (int s = s0; s < s1; ++s) {
                const float* src = gp + (size_t)(e.row0 + s) * b;
                if (e.kind == 1) {
                    acc = __fadd_rn(acc, src[c]);
                } else {
                    const int t = merge_row(mc.kt, s);
                    int idx = c - (s - t) % b;
                    idx += (idx < 0) ? b : 0;
                    acc = __fadd_rn(acc, src[idx]);
                }
            }
            out[c] = acc;
        }
    }
}

// Transition tables, root level first: tab[l][r] maps row r of level l + 1 to level l.
static int ffa_transpose_tables(int m, std::vector<TRow>& tabs, int* nlevels)
{
    std::vector<int2> nodes{make_int2(0, m)};
    tabs.clear();
    int L = 0;
    while (true) {
        bool split = false;
        for (const int2& nd : nodes) split |= nd.y >= 2;
        if (!split) break;
        std::vector<int2> next;
        const size_t base = tabs.size();
        tabs.resize(base + (size_t)m);
        for (const int2& nd : nodes) {
            if (nd.y < 2) {
                tabs[base + nd.x] = TRow{nd.x, 1, 0, 0};
                next.push_back(nd);
                continue;
            }
            const int nh = nd.y >> 1;
            for (int j = 0; j < nh; ++j) tabs[base + nd.x + j] = TRow{nd.x, nd.y, 1, j};
            for (int j = 0; j < nd.y - nh; ++j)
                tabs[base + nd.x + nh + j] = TRow{nd.x, nd.y, 2, j};
            next.push_back(make_int2(nd.x, nh));
            next.push_back(make_int2(nd.x + nh, nd.y - nh));
        }
        nodes.swap(next);
        ++L;
        if (L > 64) return set_error(RT_EINTERNAL, "FFA transpose: too many levels");
    }
    *nlevels = L;
    return RT_OK;
}

// ------------------------------------------------------------------------------------
// Downsampling adjoint: out[k] = wmin x[imin] + sum_{imin < i < imax} x[i] + wmax x[imax]
// (written as a prefix difference, so imax == imin gives (wmin + wmax - 1) x[imin]).
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double ds_coef(size_t k, double f, size_t N, size_t i)
{
    const double start = (double)k * f;
    const double end = start + f;
    const size_t imin = (size_t)floor(start);
    const double fe = floor(end);
    const size_t imax = (size_t)(fe < (double)N - 1.0 ? fe : (double)N - 1.0);
    const float wmin = __double2float_rn((double)(imin + 1) - start);
    const float wmax = __double2float_rn(end - (double)imax);
    double c = 0.0;
    if (i == imin) c += (double)wmin;
    if (i == imax) c += (double)wmax;
    if (i > imin && i < imax) c += 1.0;
    if (imax == imin && i == imin) c -= 1.0;
    return c;
}

__global__ void k_downsample_adjoint(const float* __restrict__ gout, size_t N, double f,
                                     size_t n, float* __restrict__ gin)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
         i += (size_t)gridDim.x * blockDim.x) {
        const double q = floor((double)i / f);
        const size_t k0 = q >= 1.0 ? (size_t)q - 1 : 0;
        const size_t k1 = std::min(n, (size_t)floor((double)(i + 1) / f) + 2);
        double acc = 0.0;
        for (size_t k = k0; k < k1; ++k) {
            const double c = ds_coef(k, f, N, i);
            if (c != 0.0) acc += c * (double)gout[k];
        }
        if (acc != 0.0) gin[i] = __fadd_rn(gin[i], (float)acc);
    }
}

// ------------------------------------------------------------------------------------
// Normalisation adjoint (population statistics)
// ------------------------------------------------------------------------------------
constexpr int kNormBwdThreads = 256;

// Packed series of a batch (all arrays on the device).
struct AdjBatch {
    const size_t *len, *off;        // [ntrials] lengths, offsets into the packed series
    const size_t *lo_len, *lo_off;  // [ntrials] the same of the scrunched series
    const double* inv_std;          // [ntrials]
};

__global__ void __launch_bounds__(kNormBwdThreads)
    k_norm_adj_sums(const float* __restrict__ g, const float* __restrict__ z, AdjBatch B,
                    double2* __restrict__ part)
{
    const int trial = blockIdx.y;
    const size_t N = B.len[trial], off = B.off[trial];
    double s1 = 0.0, s2 = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
         i += (size_t)gridDim.x * blockDim.x) {
        const double gv = (double)g[off + i];
        s1 += gv;
        s2 += gv * (double)z[off + i];
    }
    __shared__ double r1[kNormBwdThreads], r2[kNormBwdThreads];
    r1[threadIdx.x] = s1;
    r2[threadIdx.x] = s2;
    __syncthreads();
    for (int o = kNormBwdThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            r1[threadIdx.x] += r1[threadIdx.x + o];
            r2[threadIdx.x] += r2[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[(size_t)trial * gridDim.x + blockIdx.x] = make_double2(r1[0], r2[0]);
}

// (Every CTA adds up its series' partial sums first, a warp at a time: by one thread that took
// 20 of 26 us.)
__global__ void __launch_bounds__(kNormBwdThreads)
    k_norm_adj_apply(const float* __restrict__ g, const float* __restrict__ z, AdjBatch B,
                     const double2* __restrict__ part, float* __restrict__ gy)
{
    __shared__ double s_m1, s_m2;
    const int trial = blockIdx.y;
    const size_t N = B.len[trial], off = B.off[trial];
    if (threadIdx.x < 32) {
        const double2* p = part + (size_t)trial * gridDim.x;
        double a = 0.0, c = 0.0;
        for (unsigned k = threadIdx.x; k < gridDim.x; k += 32) {
            a += p[k].x;
            c += p[k].y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if (threadIdx.x == 0) {
            s_m1 = a / (double)N;
            s_m2 = c / (double)N;
        }
    }
    __syncthreads();
    const double m1 = s_m1, m2 = s_m2, inv_std = B.inv_std[trial];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
         i += (size_t)gridDim.x * blockDim.x)
        gy[off + i] = (float)(((double)g[off + i] - m1 - (double)z[off + i] * m2) * inv_std);
}

// ------------------------------------------------------------------------------------
// Deredden adjoint: y = x - r(x) with r = np.interp of the running median of the mean-scrunched
// series (running_medians.py:49-85), so gx = gy - r^T gy: through the interpolation (each point
// gathers from the samples around it), the median (to the element it selects) and the mean.
// All in float64; every sum is a gather, so the result does not depend on scheduling.
// ------------------------------------------------------------------------------------
// Scrunched means, and the interpolation's transpose of g at every point j: with a = the
// sample's position past point j over k, sum g (1 - a) over the samples from point j to j + 1
// and g a over those from j - 1 to j; samples outside the points go to the end points. A warp
// per point. k == 1: the samples themselves.
__global__ void __launch_bounds__(256)
    k_dered_adj_points(const float* __restrict__ x, const float* __restrict__ g, AdjBatch B, int k,
                       double* __restrict__ lores, double* __restrict__ glo)
{
    const int trial = blockIdx.y, lane = threadIdx.x & 31;
    const size_t N = B.len[trial], nl = B.lo_len[trial];
    const float *xr = x + B.off[trial], *gr = g + B.off[trial];
    double *lo = lores + B.lo_off[trial], *go = glo + B.lo_off[trial];
    const double rk = 1.0 / (double)k;
    for (size_t j = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5; j < nl;
         j += ((size_t)gridDim.x * blockDim.x) >> 5) {
        if (k == 1) {
            if (lane == 0) {
                lo[j] = (double)xr[j];
                go[j] = (double)gr[j];
            }
            continue;
        }
        double s = 0.0, c = 0.0;
        for (int i = lane; i < k; i += 32) s += (double)xr[j * k + i];
        const size_t at = j * k + k / 2;  // first sample at or past point j
        const size_t lo_i = j == 0 ? 0 : at - k;
        const size_t hi_i = j + 1 == nl ? N : at + k;
        for (size_t i = lo_i + lane; i < hi_i; i += 32) {
            // 2 (i - point j), an exact integer
            const double d = (double)(2LL * ((long long)i - (long long)(j * k)) - (k - 1)) * 0.5;
            double w = 1.0;
            if (i < at) w = j == 0 ? 1.0 : 1.0 + d * rk;
            else if (j + 1 < nl) w = 1.0 - d * rk;
            c += w * (double)gr[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if (lane == 0) {
            lo[j] = s * rk;
            go[j] = c;
        }
    }
}

// Index of the element that the running median selects at every point: the tile's values ranked
// by (value, position) as in k_running_median_sorted, compared by their order_key.
constexpr int kAdjTile = 128;
constexpr int kAdjMaxWidth = 257;
constexpr int kAdjSpan = kAdjTile + kAdjMaxWidth - 1;

__global__ void __launch_bounds__(kAdjTile)
    k_dered_adj_select(const double* __restrict__ lores, AdjBatch B, int width,
                       unsigned* __restrict__ sel)
{
    __shared__ unsigned long long sk[kAdjSpan];
    __shared__ unsigned short sp[kAdjSpan];
    const int trial = blockIdx.y;
    const size_t nl = B.lo_len[trial], t0 = (size_t)blockIdx.x * kAdjTile;
    if (t0 >= nl) return;
    const double* lo = lores + B.lo_off[trial];
    const int half = width / 2, span = kAdjTile + width - 1;
    auto clamped = [&](long long i) { return i < 0 ? 0LL : i >= (long long)nl ? (long long)nl - 1 : i; };
    for (int i = threadIdx.x; i < span; i += kAdjTile) {
        // (+ 0.0: a zero's sign is left out)
        sk[i] = order_key(__dadd_rn(lo[clamped((long long)t0 + i - half)], 0.0));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < span; i += kAdjTile) {
        const unsigned long long v = sk[i];
        int c = 0;
        for (int j = 0; j < span; ++j) c += (sk[j] < v || (sk[j] == v && j < i)) ? 1 : 0;
        sp[c] = (unsigned short)i;
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t0 + t >= nl) return;
    int left = half, at = t + half;
    for (int q = 0; q < span; ++q) {
        const unsigned p = sp[q];
        if (p - (unsigned)t < (unsigned)width && left-- == 0) {
            at = (int)p;
            break;
        }
    }
    sel[B.lo_off[trial] + t0 + t] = (unsigned)clamped((long long)t0 + at - half);
}

// gradient of the scrunched series: element e gathers the points whose window selected it
__global__ void k_dered_adj_gather(const double* __restrict__ glo, const unsigned* __restrict__ sel,
                                   AdjBatch B, int width, int k, float* __restrict__ gsel)
{
    const int trial = blockIdx.y;
    const size_t nl = B.lo_len[trial], lo = B.lo_off[trial];
    const int half = width / 2;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < nl;
         e += (size_t)gridDim.x * blockDim.x) {
        const size_t a = e >= (size_t)half ? e - half : 0, z = min(nl, e + half + 1);
        double s = 0.0;
        for (size_t t = a; t < z; ++t)
            if (sel[lo + t] == (unsigned)e) s += glo[lo + t];
        gsel[lo + e] = (float)(s / (double)k);
    }
}

__global__ void k_dered_adj_apply(const float* __restrict__ gsel, AdjBatch B, int k,
                                  float* __restrict__ gx)
{
    const int trial = blockIdx.y;
    const size_t nl = B.lo_len[trial];
    const float* s = gsel + B.lo_off[trial];
    float* g = gx + B.off[trial];
    // a CTA takes whole points, so that no thread divides
    for (size_t j = blockIdx.x; j < nl; j += gridDim.x) {
        const float v = s[j];
        for (int i = threadIdx.x; i < k; i += blockDim.x) g[j * k + i] = __fsub_rn(g[j * k + i], v);
    }
}

__global__ void k_dered_adj_apply1(const float* __restrict__ gsel, AdjBatch B, float* __restrict__ gx)
{
    const int trial = blockIdx.y;
    const size_t nl = B.lo_len[trial], off = B.off[trial], lo = B.lo_off[trial];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nl;
         i += (size_t)gridDim.x * blockDim.x)
        gx[off + i] = __fsub_rn(gx[off + i], gsel[lo + i]);
}

}  // namespace rt

using namespace rt;

extern "C" int rt_snr2_backward(const float* d_in, size_t rows, size_t cols,
                                const uint64_t* h_widths, size_t num_widths, float stdnoise,
                                const float* d_gsnr, float* d_gin, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (rows == 0) return RT_OK;
    if (!d_in || !d_gin || !d_gsnr || (!h_widths && num_widths))
        return set_error(RT_EINVAL, "null argument");
    if (num_widths > (size_t)kSnrBwdMaxWidths)
        return set_error(RT_EINVAL, "at most %d trial widths are supported", kSnrBwdMaxWidths);
    std::vector<int> w(num_widths);
    int wmax = 1;
    for (size_t k = 0; k < num_widths; ++k) {
        if (!(h_widths[k] > 0 && h_widths[k] < cols))  // snr.hpp:21-31
            return set_error(RT_EINVAL, "trial widths must be all > 0 and < columns");
        w[k] = (int)h_widths[k];
        wmax = std::max(wmax, w[k]);
    }
    if (!(stdnoise > 0.0f)) return set_error(RT_EINVAL, "stdnoise must be > 0");
    const size_t per_warp = (cols + wmax + 1) * sizeof(float);
    int wpb = (int)std::min<size_t>(8, (160 * 1024) / per_warp);
    if (wpb < 1) return set_error(RT_EINVAL, "profiles of %zu bins are too long", cols);
    int* d_w = nullptr;
    RT_TRY_CUDA(scratch_malloc((void**)&d_w, std::max<size_t>(num_widths, 1) * sizeof(int), st));
    int s = check_cuda(cudaMemcpyAsync(d_w, w.data(), num_widths * sizeof(int),
                                       cudaMemcpyHostToDevice, st), "snr2_backward");
    const size_t smem = (size_t)wpb * per_warp;
    if (s == RT_OK && smem > 48 * 1024)
        s = check_cuda(cudaFuncSetAttribute(k_snr2_backward,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                       "snr2_backward");
    if (s == RT_OK) {
        const int grid = (int)std::min<size_t>((rows + wpb - 1) / wpb, 148 * 16);
        k_snr2_backward<<<grid, 32 * wpb, smem, st>>>(d_in, (int)rows, (int)cols, d_w,
                                                     (int)num_widths, stdnoise, d_gsnr, d_gin, wmax);
        s = check_cuda(cudaGetLastError(), "snr2_backward");
    }
    cudaFreeAsync(d_w, st);
    return s;
}

extern "C" int rt_ffa2_transpose(const float* d_gout, size_t rows, size_t cols, float* d_gin,
                                 void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (rows == 0 || cols == 0) return RT_OK;
    if (!d_gout || !d_gin) return set_error(RT_EINVAL, "null argument");
    if (rows >= (1u << 24) || cols >= (1u << 24))
        return set_error(RT_EINVAL, "a %zu x %zu block is too large", rows, cols);
    const int m = (int)rows, b = (int)cols;
    std::vector<TRow> tabs;
    int L = 0;
    RT_TRY(ffa_transpose_tables(m, tabs, &L));
    if (L == 0)
        return check_cuda(cudaMemcpyAsync(d_gin, d_gout, rows * cols * sizeof(float),
                                          cudaMemcpyDeviceToDevice, st), "ffa2_transpose");
    TRow* d_tab = nullptr;
    float* tmp = nullptr;
    RT_TRY_CUDA(scratch_malloc((void**)&d_tab, tabs.size() * sizeof(TRow), st));
    int s = check_cuda(scratch_malloc((void**)&tmp, rows * cols * sizeof(float), st), "ffa2_transpose");
    if (s == RT_OK)
        s = check_cuda(cudaMemcpyAsync(d_tab, tabs.data(), tabs.size() * sizeof(TRow),
                                       cudaMemcpyHostToDevice, st), "ffa2_transpose");
    // ping-pong so that the last level lands in d_gin
    const float* src = d_gout;
    for (int l = 0; l < L && s == RT_OK; ++l) {
        float* dst = ((L - 1 - l) % 2 == 0) ? d_gin : tmp;
        const int grid = (int)std::min<size_t>(((size_t)m * 32 + 255) / 256, 148 * 8);
        k_ffa_transpose_level<<<grid, 256, 0, st>>>(src, dst, d_tab + (size_t)l * m, m, b);
        s = check_cuda(cudaGetLastError(), "ffa2_transpose");
        src = dst;
    }
    cudaFreeAsync(tmp, st);
    cudaFreeAsync(d_tab, st);
    return s;
}

extern "C" int rt_downsample_adjoint(const float* d_gout, size_t size, double f, float* d_gin,
                                     void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (!((f > 1.0) && (f <= (double)size)))  // downsample.hpp:11-16
        return set_error(RT_EINVAL, "Downsampling factor must verify: 1 < f <= size");
    if (!d_gout || !d_gin) return set_error(RT_EINVAL, "null argument");
    const size_t n = downsampled_size(size, f);
    const int grid = (int)std::min<size_t>((size + 255) / 256, 148 * 16);
    k_downsample_adjoint<<<grid, 256, 0, st>>>(d_gout, size, f, n, d_gin);
    return check_cuda(cudaGetLastError(), "downsample_adjoint");
}

// Lengths and offsets of a batch on the device, with 1 / std of each series.
static int adj_batch(const uint64_t* h_lengths, size_t ntrials, const double* h_std, size_t k,
                     AdjBatch* B, void** blob, size_t* total, size_t* lo_total, size_t* max_len,
                     cudaStream_t st)
{
    std::vector<size_t> h(5 * ntrials);
    size_t off = 0, lo = 0, most = 0;
    for (size_t t = 0; t < ntrials; ++t) {
        h[t] = h_lengths[t];
        h[ntrials + t] = off;
        h[2 * ntrials + t] = h_lengths[t] / k;
        h[3 * ntrials + t] = lo;
        const double inv = h_std ? 1.0 / h_std[t] : 1.0;
        memcpy(&h[4 * ntrials + t], &inv, sizeof(double));
        off += h_lengths[t];
        lo += h_lengths[t] / k;
        most = std::max(most, (size_t)h_lengths[t]);
    }
    static_assert(sizeof(size_t) == sizeof(double), "one array for both");
    RT_TRY_CUDA(scratch_malloc(blob, h.size() * sizeof(size_t), st));
    // (pageable memory: the copy has read it when the call returns)
    const cudaError_t e = cudaMemcpyAsync(*blob, h.data(), h.size() * sizeof(size_t),
                                          cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) {
        cudaFreeAsync(*blob, st);
        return check_cuda(e, "adjoint");
    }
    const size_t* d = static_cast<const size_t*>(*blob);
    *B = AdjBatch{d, d + ntrials, d + 2 * ntrials, d + 3 * ntrials,
                  reinterpret_cast<const double*>(d + 4 * ntrials)};
    *total = off;
    *lo_total = lo;
    *max_len = most;
    return RT_OK;
}

// gy = (g - mean g - z mean(g z)) / std of every series of the batch.
static int normalise_adjoint(const float* d_g, const float* d_z, const AdjBatch& B, size_t ntrials,
                             size_t max_len, float* d_gy, cudaStream_t st)
{
    const size_t most = std::max<size_t>(8, 148 * 16 / ntrials);
    const unsigned blocks =
        (unsigned)std::max<size_t>(1, std::min((max_len + kNormBwdThreads - 1) / kNormBwdThreads, most));
    double2* part = nullptr;
    RT_TRY_CUDA(scratch_malloc((void**)&part, blocks * ntrials * sizeof(double2), st));
    const dim3 grid(blocks, (unsigned)ntrials);
    k_norm_adj_sums<<<grid, kNormBwdThreads, 0, st>>>(d_g, d_z, B, part);
    int s = check_cuda(cudaGetLastError(), "normalise_adjoint");
    if (s == RT_OK) {
        k_norm_adj_apply<<<grid, kNormBwdThreads, 0, st>>>(d_g, d_z, B, part, d_gy);
        s = check_cuda(cudaGetLastError(), "normalise_adjoint");
    }
    cudaFreeAsync(part, st);
    return s;
}

extern "C" int rt_normalise_adjoint(const float* d_g, const float* d_z, size_t size,
                                    double std_, float* d_gy, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (size == 0) return RT_OK;
    if (!d_g || !d_z || !d_gy) return set_error(RT_EINVAL, "null argument");
    if (!(std_ > 0.0)) return set_error(RT_EINVAL, "std must be > 0");
    AdjBatch B;
    void* blob = nullptr;
    size_t total, lo, most;
    const uint64_t len = size;
    RT_TRY(adj_batch(&len, 1, &std_, 1, &B, &blob, &total, &lo, &most, st));
    const int s = normalise_adjoint(d_g, d_z, B, 1, size, d_gy, st);
    cudaFreeAsync(blob, st);
    return s;
}

extern "C" int rt_front_adjoint(const float* d_x, const float* d_z, const float* d_gz,
                                const uint64_t* h_lengths, size_t ntrials, const double* h_std,
                                size_t width_samples, size_t min_points, float* d_gx, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (!d_x || !d_gz || !d_gx || !h_lengths || (h_std && !d_z))
        return set_error(RT_EINVAL, "null argument");
    if (ntrials == 0) return RT_OK;
    if (ntrials > 65535) return set_error(RT_EINVAL, "at most 65535 series per call");
    size_t k = 1, width = 0;
    if (min_points) {
        // running_medians.py:72-80
        if (!(min_points % 2)) return set_error(RT_EINVAL, "min_points must be an odd number");
        k = (size_t)std::max(1.0, (double)width_samples / (double)min_points);
        width = k == 1 ? width_samples : min_points;
        if (!(width % 2)) return set_error(RT_EINVAL, "width must be an odd number");
        if (width > (size_t)kAdjMaxWidth || k > (1u << 30))
            return set_error(RT_EINVAL, "a running median of %zu points is too wide", width);
    }
    for (size_t t = 0; t < ntrials; ++t) {
        if (h_lengths[t] == 0) return set_error(RT_EINVAL, "series %zu is empty", t);
        if (min_points && !(width < h_lengths[t] / k))
            return set_error(RT_EINVAL, "width must be < size");
        if (min_points && h_lengths[t] / k >= (1ull << 32))
            return set_error(RT_EINVAL, "series %zu is too long", t);
        if (h_std && !(h_std[t] > 0.0)) return set_error(RT_EINVAL, "std must be > 0");
    }
    AdjBatch B;
    void* blob = nullptr;
    size_t total, lo_total, max_len;
    RT_TRY(adj_batch(h_lengths, ntrials, h_std, k, &B, &blob, &total, &lo_total, &max_len, st));
    int s = RT_OK;
    if (h_std)
        s = normalise_adjoint(d_gz, d_z, B, ntrials, max_len, d_gx, st);
    else if (d_gx != d_gz)
        s = check_cuda(cudaMemcpyAsync(d_gx, d_gz, total * sizeof(float), cudaMemcpyDeviceToDevice, st),
                       "front_adjoint");
    unsigned char* buf = nullptr;
    if (s == RT_OK && min_points)
        s = check_cuda(scratch_malloc((void**)&buf, lo_total * (2 * sizeof(double) + 8), st), "front_adjoint");
    if (s == RT_OK && min_points) {
        double* lores = reinterpret_cast<double*>(buf);
        double* glo = lores + lo_total;
        unsigned* sel = reinterpret_cast<unsigned*>(glo + lo_total);
        float* gsel = reinterpret_cast<float*>(sel + lo_total);
        const size_t max_lo = max_len / k;
        const unsigned T = (unsigned)ntrials;
        auto blocks = [](size_t n, size_t per) {
            return (unsigned)std::max<size_t>(1, std::min<size_t>((n + per - 1) / per, 1 << 20));
        };
        k_dered_adj_points<<<dim3(blocks(max_lo, 8), T), 256, 0, st>>>(d_x, d_gx, B, (int)k, lores, glo);
        k_dered_adj_select<<<dim3((unsigned)((max_lo + kAdjTile - 1) / kAdjTile), T), kAdjTile, 0, st>>>(
            lores, B, (int)width, sel);
        k_dered_adj_gather<<<dim3(blocks(max_lo, 128), T), 128, 0, st>>>(glo, sel, B, (int)width,
                                                                        (int)k, gsel);
        if (k == 1)
            k_dered_adj_apply1<<<dim3(blocks(max_lo, 1024), T), 256, 0, st>>>(gsel, B, d_gx);
        else
            k_dered_adj_apply<<<dim3(blocks(max_lo, 1), T), 256, 0, st>>>(gsel, B, (int)k, d_gx);
        s = check_cuda(cudaGetLastError(), "front_adjoint");
    }
    if (buf) cudaFreeAsync(buf, st);
    cudaFreeAsync(blob, st);
    return s;
}
