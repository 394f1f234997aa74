// Folding of a time series at trial periods (TimeSeries.fold / folding.py:21-85 of the
// reference), for one period or a batch of candidates of the same series.
//
// The reference downsamples the series by tbin / tsamp (tbin = period / bins), reshapes the
// first m * bins samples to (m, bins), multiplies by (m * factor)^-1/2 in float32, and either
// sums the rows (subints = 1, or m = 1), returns the rows (subints = None or m), or downsamples
// each phase column by m / subints (downsample_vertical, folding.py:6-18). Here the downsampled
// samples are formed straight from the raw series (FP64 sum of the window, rounded once, as
// rt_downsample forms them) and scaled, by as many lanes per window as it has samples for
// (k_fold_windows); then the folded block is summed or column-downsampled in the reference's
// order (k_fold_reduce), unless its rows are the result.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace rt {

// Folded values held in scratch memory at a time (128 MiB); a larger block is never written.
constexpr size_t kFoldBlock = size_t(1) << 25;

enum FoldMode : int { kFoldSum = 0, kFoldRows = 1, kFoldColumns = 2 };

struct FoldJob {
    double f;          // time downsampling factor tbin / tsamp
    double vf;         // column downsampling factor m / subints (kFoldColumns)
    size_t out_off;    // first output value
    int bins, m;       // phase bins, rows of the folded block
    int rows;          // output rows (1 for kFoldSum)
    int mode;
    float scale;       // float32((m * factor) ** -0.5)
    int lanes;         // log2 of the lanes per window
    size_t block_off;  // the folded block in the scratch memory (of d_out for kFoldRows)
    size_t tile0;      // first tile of windows of the fold
    int tile;          // windows per tile
    int pad;
};

struct FoldShape {
    int mode;
    size_t m, rows;
    double f, vf;
    float scale;
};

// Sample k of the series downsampled by f (downsample.hpp:44-82): the window sum in FP64,
// rounded once to float32.
__device__ __forceinline__ float ds_value(const float* __restrict__ x, size_t N, double f, size_t k)
{
    const double start = (double)k * f;
    const double end = start + f;
    const size_t imin = (size_t)floor(start);
    const double fe = floor(end);
    const size_t imax = (size_t)(fe < (double)N - 1.0 ? fe : (double)N - 1.0);
    double acc = 0.0;
    for (size_t i = imin + 1; i < imax; ++i) acc += (double)__ldg(x + i);
    const float wmin = __double2float_rn((double)(imin + 1) - start);
    const float wmax = __double2float_rn(end - (double)imax);
    return __double2float_rn((double)wmin * __ldg(x + imin) + acc + (double)wmax * __ldg(x + imax));
}

// Folded value (row i, phase j): downsampled sample i * bins + j times the float32 scale.
__device__ __forceinline__ float folded(const float* x, size_t N, const FoldJob& J, size_t i, int j)
{
    return __fmul_rn(ds_value(x, N, J.f, i * (size_t)J.bins + j), J.scale);
}

// ------------------------------------------------------------------------------------
// The folded blocks of a batch of folds, in tiles of some ten thousand samples. 2^lanes
// neighbouring lanes sum a window (about six samples a lane, so that the loads of a warp cover
// few lines and the per-window arithmetic stays small), and the next window is the next lanes'.
// Bound: instructions (81% of the issue slots), most of them a window's own, and conversions to
// float64 (57% of their rate). 48 folds of 2^22 samples into 256 bins, 32 sub-integrations: 385 us
// with a thread per output value; 180 us for both kernels.
// ------------------------------------------------------------------------------------
constexpr int kFoldThreads = 256;

// The windows [k0, k1) of fold J, 2^LANES lanes each.
template <int LANES>
__device__ __forceinline__ void fold_windows(const float* __restrict__ x, size_t N,
                                             const FoldJob& J, size_t k0, size_t k1, float* dst)
{
    constexpr int G = 1 << LANES;
    const int g = threadIdx.x & (G - 1);
    const double n1 = (double)N - 1.0;
    // whole warps take part in the sums of a window
    for (size_t kw = k0 + ((threadIdx.x & ~31) >> LANES); kw < k1; kw += kFoldThreads >> LANES) {
        const size_t k = kw + ((threadIdx.x & 31) >> LANES);
        const bool live = k < k1;
        const double start = __dmul_rn(whole_double(k), J.f);
        const double end = __dadd_rn(start, J.f);
        size_t imin, imax;
        const double first = floor_index(start, imin);
        double last = floor_index(end, imax);
        if (!(last < n1)) {
            last = n1;
            imax = N - 1;
        }
        const double wmin = (double)__double2float_rn((first + 1.0) - start);
        const double wmax = (double)__double2float_rn(end - last);
        double acc = 0.0;
        // the lane's samples of imin..imax, those at the ends weighted: `left` samples to imax
        const float* v = x + imin + g;
        int left = live ? (int)(imax - imin) - g : -1;
        if (left > 0 || (left == 0 && g == 0)) acc = (g == 0 ? wmin : 1.0) * (double)__ldg(v);
        if (left > 0) {
            left -= G;
            v += G;
        }
        for (; left > 0; left -= 4 * G, v += 4 * G) {
            float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (left > u * G) w[u] = __ldg(v + u * G);
#pragma unroll
            for (int u = 0; u < 4; ++u) acc += (double)w[u];
            if (left < 4 * G && (left & (G - 1)) == 0) {  // imax is the lane's next sample
                v += left;
                left = 0;
                break;
            }
        }
        if (left == 0) acc += wmax * (double)__ldg(v);
#pragma unroll
        for (int d = G >> 1; d > 0; d >>= 1) acc += __shfl_xor_sync(~0u, acc, d);
        if (live && g == 0) dst[k] = __fmul_rn(__double2float_rn(acc), J.scale);
    }
}

__global__ void __launch_bounds__(kFoldThreads)
    k_fold_windows(const float* __restrict__ x, size_t N, const FoldJob* __restrict__ jobs,
                   int njobs, size_t tiles, float* __restrict__ blocks, float* __restrict__ out)
{
    for (size_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int lo = 0, hi = njobs - 1;  // fold of this tile
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].tile0 <= tile) lo = mid;
            else hi = mid - 1;
        }
        const FoldJob J = jobs[lo];
        const size_t k0 = (tile - J.tile0) * J.tile;
        const size_t k1 = min((size_t)J.m * J.bins, k0 + J.tile);
        float* dst = J.mode == kFoldRows ? out + J.out_off : blocks + J.block_off;
        switch (J.lanes) {
            case 0: fold_windows<0>(x, N, J, k0, k1, dst); break;
            case 1: fold_windows<1>(x, N, J, k0, k1, dst); break;
            case 2: fold_windows<2>(x, N, J, k0, k1, dst); break;
            case 3: fold_windows<3>(x, N, J, k0, k1, dst); break;
            case 4: fold_windows<4>(x, N, J, k0, k1, dst); break;
            default: fold_windows<5>(x, N, J, k0, k1, dst); break;
        }
    }
}

// Sums the rows of the folded blocks (kFoldSum: a tile of rows and 32 columns at a time in shared
// memory, one lane adds up a column) or downsamples their columns (kFoldColumns: a thread per
// output value; neighbouring threads read neighbouring columns).
__global__ void __launch_bounds__(kFoldThreads)
    k_fold_reduce(const FoldJob* __restrict__ jobs, const float* __restrict__ blocks,
                  float* __restrict__ out)
{
    constexpr int kRows = 128;
    __shared__ float tile[kRows][32];
    const FoldJob J = jobs[blockIdx.y];
    const float* y = blocks + J.block_off;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (J.mode == kFoldSum) {
        for (int j0 = blockIdx.x * 32; j0 < J.bins; j0 += gridDim.x * 32) {
            const int j = j0 + lane;
            float v = 0.0f;
            for (int i0 = 0; i0 < J.m; i0 += kRows) {
                __syncthreads();
#pragma unroll
                for (int r = warp; r < kRows; r += kFoldThreads / 32)
                    if (i0 + r < J.m && j < J.bins) tile[r][lane] = y[(size_t)(i0 + r) * J.bins + j];
                __syncthreads();
                if (warp == 0 && j < J.bins) {
                    // numpy's sum over axis 0: the rows accumulated in order in float32
                    const int n = min(kRows, J.m - i0);
                    int r = 0;
                    if (i0 == 0) v = tile[r++][lane];
#pragma unroll 8
                    for (; r < n; ++r) v = __fadd_rn(v, tile[r][lane]);
                }
            }
            if (warp == 0 && j < J.bins) out[J.out_off + j] = v;
        }
    } else if (J.mode == kFoldColumns) {
        const size_t total = (size_t)J.rows * J.bins;
        for (size_t o = (size_t)blockIdx.x * kFoldThreads + threadIdx.x; o < total;
             o += (size_t)gridDim.x * kFoldThreads) {
            const int j = (int)(o % J.bins);
            const size_t r = o / J.bins;
            const float* col = y + j;
            // column j downsampled by vf (downsample_vertical): window sum in FP64, rounded once
            const double start = (double)r * J.vf;
            const double end = start + J.vf;
            const size_t imin = (size_t)floor(start);
            const double fe = floor(end);
            const size_t imax = (size_t)(fe < (double)J.m - 1.0 ? fe : (double)J.m - 1.0);
            double acc = 0.0;
#pragma unroll 8
            for (size_t i = imin + 1; i < imax; ++i) acc += (double)col[i * J.bins];
            const float wmin = __double2float_rn((double)(imin + 1) - start);
            const float wmax = __double2float_rn(end - (double)imax);
            out[J.out_off + o] = __double2float_rn((double)wmin * col[imin * J.bins] + acc +
                                                   (double)wmax * col[imax * J.bins]);
        }
    }
}

// A thread per output value, for folded blocks beyond kFoldBlock (no scratch memory) and windows
// of 2^30 samples and more.
__global__ void k_fold(const float* __restrict__ x, size_t N, const FoldJob* __restrict__ jobs,
                       float* __restrict__ out)
{
    const FoldJob J = jobs[blockIdx.y];
    const size_t total = (size_t)J.rows * J.bins;
    for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
         o += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(o % J.bins);
        const size_t r = o / J.bins;
        float v;
        if (J.mode == kFoldRows) {
            v = folded(x, N, J, r, j);
        } else if (J.mode == kFoldSum) {
            // numpy's sum over axis 0: the rows accumulated in order in float32
            v = J.m > 0 ? folded(x, N, J, 0, j) : 0.0f;
            for (int i = 1; i < J.m; ++i) v = __fadd_rn(v, folded(x, N, J, i, j));
        } else {
            // column j downsampled by vf (downsample_vertical): window sum in FP64, rounded once
            const double start = (double)r * J.vf;
            const double end = start + J.vf;
            const size_t imin = (size_t)floor(start);
            const double fe = floor(end);
            const size_t imax = (size_t)(fe < (double)J.m - 1.0 ? fe : (double)J.m - 1.0);
            double acc = 0.0;
            for (size_t i = imin + 1; i < imax; ++i) acc += (double)folded(x, N, J, i, j);
            const float wmin = __double2float_rn((double)(imin + 1) - start);
            const float wmax = __double2float_rn(end - (double)imax);
            v = __double2float_rn((double)wmin * folded(x, N, J, imin, j) + acc +
                                  (double)wmax * folded(x, N, J, imax, j));
        }
        out[J.out_off + o] = v;
    }
}

// The reference's argument checks and output shape (folding.py:21-85; TimeSeries.downsample
// checks the factor, downsample.hpp:11-19; downsample_vertical checks its factor, :7-14).
// subints < 0 stands for None.
static int fold_shape(size_t size, double tsamp, double period, size_t bins, long long subints,
                      FoldShape& s)
{
    if (!(tsamp > 0)) return set_error(RT_EINVAL, "tsamp must be > 0");
    if (bins < 1) return set_error(RT_EINVAL, "bins must be >= 1");
    const double length = (double)size * tsamp;
    if (period > length) return set_error(RT_EINVAL, "Period exceeds data length");
    const double tbin = period / (double)bins;
    if (!(tbin > tsamp)) return set_error(RT_EINVAL, "Bin width is shorter than sampling time");
    if (subints == 0) return set_error(RT_EINVAL, "subints must be >= 1 or None");
    if (subints > 0) {
        const double full_periods = length / period;
        if ((double)subints > full_periods)
            return set_error(RT_EINVAL,
                             "subints (%lld) exceeds the number of signal periods that fit in the data (%g)",
                             subints, full_periods);
    }
    const double f = tbin / tsamp;
    if (!(f > 1.0) || f > (double)size)
        return set_error(RT_EINVAL, "Downsampling factor must be > 1 and <= input size");
    const size_t n = downsampled_size(size, f);
    const size_t m = n / bins;
    if (m == 0) return set_error(RT_EINVAL, "the downsampled series holds no full period");
    s.f = f;
    s.m = m;
    s.vf = 0.0;
    s.scale = (float)std::pow((double)m * f, -0.5);
    if (subints == 1 || m == 1) {
        s.mode = kFoldSum;
        s.rows = 1;
    } else if (subints < 0 || (size_t)subints == m) {
        s.mode = kFoldRows;
        s.rows = m;
    } else {
        const double vf = (double)m / (double)subints;
        if (!(vf > 1.0)) return set_error(RT_EINVAL, "factor must be > 1");
        if (!(vf < (double)m))
            return set_error(RT_EINVAL, "factor must be strictly smaller than the number of input lines");
        s.mode = kFoldColumns;
        s.vf = vf;
        s.rows = downsampled_size(m, vf);
    }
    if (m > (size_t)INT32_MAX || bins > (size_t)INT32_MAX)
        return set_error(RT_EINVAL, "fold too large");
    return RT_OK;
}

}  // namespace rt

using namespace rt;

extern "C" int rt_fold_shape(size_t size, double tsamp, double period, size_t bins,
                             long long subints, size_t* rows, int* ndim)
{
    FoldShape s;
    RT_TRY(fold_shape(size, tsamp, period, bins, subints, s));
    if (rows) *rows = s.rows;
    if (ndim) *ndim = s.mode == kFoldSum ? 1 : 2;
    return RT_OK;
}

extern "C" int rt_fold_batched(const float* d_in, size_t size, double tsamp,
                               const double* h_periods, const size_t* h_bins,
                               const long long* h_subints, size_t count,
                               const uint64_t* h_out_offsets, float* d_out, void* stream_)
{
    cudaStream_t stream = (cudaStream_t)stream_;
    if (count == 0) return RT_OK;
    if (!d_in || !d_out || !h_periods || !h_bins || !h_subints || !h_out_offsets)
        return set_error(RT_EINVAL, "null argument");
    if (count > 65535) return set_error(RT_EINVAL, "at most 65535 folds per call");
    // Batches of folds whose blocks fit the scratch memory; a block that alone does not is folded
    // by itself. Folds into rows take none.
    struct Batch {
        size_t first, end, block, tiles, most;
        bool direct;
    };
    std::vector<FoldJob> jobs(count);
    std::vector<Batch> batches;
    size_t block = 0;
    for (size_t c = 0; c < count; ++c) {
        FoldShape s;
        RT_TRY(fold_shape(size, tsamp, h_periods[c], h_bins[c], h_subints[c], s));
        FoldJob& J = jobs[c];
        J.f = s.f;
        J.vf = s.vf;
        J.out_off = h_out_offsets[c];
        J.bins = (int)h_bins[c];
        J.m = (int)s.m;
        J.rows = (int)s.rows;
        J.mode = s.mode;
        J.scale = s.scale;
        J.pad = 0;
        // about six samples a lane: 2^22 samples at 12 a window took 2 lanes, at 1,831 all 32
        J.lanes = 0;
        while (J.lanes < 5 && (double)(9 << J.lanes) <= s.f) ++J.lanes;
        J.tile = kFoldThreads >> J.lanes;
        while (J.tile < 1024 && J.tile * s.f < 8192.0) J.tile *= 2;
        const size_t windows = s.m * h_bins[c];
        const size_t need = s.mode == kFoldRows ? 0 : windows;
        // (windows of 2^30 samples and more: beyond the 32-bit counts of k_fold_windows)
        const bool direct = need > kFoldBlock || s.f >= 1073741824.0;
        if (batches.empty() || direct || batches.back().direct ||
            batches.back().block + need > kFoldBlock)
            batches.push_back(Batch{c, c, 0, 0, 0, direct});
        Batch& B = batches.back();
        J.block_off = B.block;
        J.tile0 = B.tiles;
        if (!direct) B.block += need;
        B.tiles += (windows + J.tile - 1) / J.tile;
        if (s.mode != kFoldRows || direct) B.most = std::max(B.most, s.rows * h_bins[c]);
        B.end = c + 1;
        block = std::max(block, B.block);
    }
    const size_t job_bytes = (count * sizeof(FoldJob) + 255) & ~size_t(255);
    char* scratch = nullptr;
    bool no_block = false;
    cudaError_t room = scratch_malloc((void**)&scratch, job_bytes + block * sizeof(float), stream);
    if (room == cudaErrorMemoryAllocation && block > 0) {  // no room for blocks: none is written
        cudaGetLastError();
        no_block = true;
        room = scratch_malloc((void**)&scratch, job_bytes, stream);
    }
    if (room != cudaSuccess) return check_cuda(room, "fold scratch memory");
    FoldJob* d_jobs = reinterpret_cast<FoldJob*>(scratch);
    float* d_blocks = reinterpret_cast<float*>(scratch + job_bytes);
    cudaError_t e = cudaMemcpyAsync(d_jobs, jobs.data(), count * sizeof(FoldJob),
                                    cudaMemcpyHostToDevice, stream);
    for (const Batch& B : batches) {
        if (e != cudaSuccess) break;
        const unsigned n = (unsigned)(B.end - B.first);
        if (B.direct || (no_block && B.block > 0)) {
            const size_t bx = std::min<size_t>((B.most + 127) / 128, 4096);
            k_fold<<<dim3((unsigned)bx, n), 128, 0, stream>>>(d_in, size, d_jobs + B.first, d_out);
            e = cudaGetLastError();
            continue;
        }
        if (B.tiles > 0) {
            k_fold_windows<<<(unsigned)std::min<size_t>(B.tiles, 1 << 20), kFoldThreads, 0, stream>>>(
                d_in, size, d_jobs + B.first, (int)n, B.tiles, d_blocks, d_out);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess && B.most > 0) {
            const size_t bx = std::min<size_t>((B.most + kFoldThreads - 1) / kFoldThreads, 4096);
            // a sum over all rows takes a CTA per 32 columns
            const size_t by = std::max<size_t>(bx, std::min<size_t>((B.most + 31) / 32, 64));
            k_fold_reduce<<<dim3((unsigned)by, n), kFoldThreads, 0, stream>>>(d_jobs + B.first,
                                                                             d_blocks, d_out);
            e = cudaGetLastError();
        }
    }
    // a copy from pageable memory has read `jobs` when cudaMemcpyAsync returns
    cudaFreeAsync(scratch, stream);
    if (e != cudaSuccess) return check_cuda(e, "k_fold");
    return RT_OK;
}

extern "C" int rt_fold(const float* d_in, size_t size, double tsamp, double period, size_t bins,
                       long long subints, float* d_out, void* stream)
{
    const uint64_t off = 0;
    return rt_fold_batched(d_in, size, tsamp, &period, &bins, &subints, 1, &off, d_out, stream);
}
