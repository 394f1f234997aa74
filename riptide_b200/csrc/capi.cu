// C ABI entry points: drop-ins for the reference's riptide.libcpp functions
// (cpp/python_bindings.cpp) on device buffers.
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "snr_core.cuh"

using namespace rt;

extern "C" const char* rt_last_error(void) { return rt::last_error(); }
extern "C" int rt_version(void) { return 100; }

extern "C" int rt_release_scratch(void)
{
    rt::release_scratch();
    return RT_OK;
}

extern "C" int rt_inject_scratch_fault(int nth)
{
    if (nth < 0) return set_error(RT_EINVAL, "scratch allocations are numbered from 1");
    rt::inject_scratch_fault(nth);
    return RT_OK;
}

extern "C" int rt_rollback(const float* d_x, size_t size, size_t shift, float* d_out,
                           void* stream)
{
    return rt::rollback(d_x, size, shift, d_out, (cudaStream_t)stream);
}

extern "C" int rt_fused_rollback_add(const float* d_x, const float* d_y, size_t size,
                                     size_t shift, float* d_out, void* stream)
{
    return rt::fused_rollback_add(d_x, d_y, size, shift, d_out, (cudaStream_t)stream);
}

extern "C" int rt_circular_prefix_sum(const float* d_x, size_t size, size_t nsum, float* d_out,
                                      void* stream)
{
    return rt::circular_prefix_sum(d_x, size, nsum, d_out, (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------
// ffa2
// ------------------------------------------------------------------------------------
// d_status (or null) receives the status of the transform, in stream order. wait_polls, dep_bias:
// see ffa_transform_persistent.
static int ffa2(const float* d_in, size_t rows, size_t cols, float* d_out, int* d_status,
                long long wait_polls, int dep_bias, cudaStream_t st)
{
    if (d_status) RT_TRY_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), st));  // RT_OK
    if (rows == 0 || cols == 0) return RT_OK;
    if (rows >= (1u << 24) || cols > 4096)
        return set_error(RT_EINVAL, "ffa2 input of %zu x %zu is larger than supported", rows, cols);
    const int m = (int)rows, b = (int)cols;
    float* scratch = nullptr;
    if (const size_t bytes = ffa_persistent_bytes(m, b, m)) {
        void* room = nullptr;
        const cudaError_t e = scratch_malloc(&room, bytes, st);
        if (e == cudaSuccess) {
            const int s = ffa_transform_persistent(d_in, m, b, m, d_out, room, d_status, st,
                                                   wait_polls, dep_bias);
            cudaFreeAsync(room, st);
            return s;
        }
        if (e != cudaErrorMemoryAllocation) return check_cuda(e, "ffa2 scratch");
        cudaGetLastError();  // a launch per stage needs a little less
    }
    const size_t sf = ffa_scratch_floats(m, b);
    if (sf) {
        const cudaError_t e = scratch_malloc((void**)&scratch, sf * sizeof(float), st);
        if (e != cudaSuccess) return check_cuda(e, "ffa2 scratch");
    }
    // (the plan is checked on the host before any launch: no kernel waits for another here)
    const int s = ffa_transform(d_in, m, b, m, d_out, scratch, d_status, st);
    if (scratch) cudaFreeAsync(scratch, st);
    return s;
}

extern "C" int rt_ffa2(const float* d_in, size_t rows, size_t cols, float* d_out, void* stream)
{
    return ffa2(d_in, rows, cols, d_out, nullptr, 0, 0, (cudaStream_t)stream);
}

extern "C" int rt_ffa2_status(const float* d_in, size_t rows, size_t cols, float* d_out,
                              int32_t* d_status, long long wait_polls, int fault, void* stream)
{
    if (!d_status) return set_error(RT_EINVAL, "null argument");
    if (wait_polls < 0) return set_error(RT_EINVAL, "the wait limit must not be negative");
    if (fault != RT_FAULT_NONE && fault != RT_FAULT_STAGE_WAIT)
        return set_error(RT_EINVAL, "unknown fault kind %d", fault);
    return ffa2(d_in, rows, cols, d_out, d_status, wait_polls, fault == RT_FAULT_STAGE_WAIT ? 1 : 0,
                (cudaStream_t)stream);
}

extern "C" int rt_benchmark_ffa2(size_t rows, size_t cols, size_t loops, double* h_seconds)
{
    if (!h_seconds) return set_error(RT_EINVAL, "null argument");
    if (rows == 0 || cols == 0 || loops == 0) {
        *h_seconds = 0.0;
        return RT_OK;
    }
    const int m = (int)rows, b = (int)cols;
    float *in = nullptr, *out = nullptr;
    void* scratch = nullptr;
    int* d_err = nullptr;
    const size_t n = rows * cols, sf = ffa_scratch_floats(m, b);
    size_t persistent = ffa_persistent_bytes(m, b, m);  // as rt_ffa2, also where that finds no room
    cudaError_t e = cudaMalloc((void**)&in, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void**)&out, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void**)&d_err, sizeof(int));
    if (e == cudaSuccess && persistent) {
        e = scratch_malloc(&scratch, persistent, 0);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            persistent = 0;
            e = cudaSuccess;
        }
    }
    if (e == cudaSuccess && !persistent && sf) e = scratch_malloc(&scratch, sf * sizeof(float), 0);
    if (e == cudaSuccess) e = cudaMemset(in, 0, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(d_err, 0, sizeof(int));
    auto release = [&]() {
        cudaFree(in);
        cudaFree(out);
        cudaFree(d_err);
        if (scratch) cudaFreeAsync(scratch, 0);
    };
    if (e != cudaSuccess) {
        release();
        return check_cuda(e, "benchmark_ffa2");
    }
    auto transform = [&]() {
        return persistent ? ffa_transform_persistent(in, m, b, m, out, scratch, d_err, 0)
                          : ffa_transform(in, m, b, m, out, static_cast<float*>(scratch), d_err, 0);
    };
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int s = transform();  // warm-up
    cudaEventRecord(e0, 0);
    for (size_t i = 0; i < loops && s == RT_OK; ++i) s = transform();
    cudaEventRecord(e1, 0);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    release();
    if (s != RT_OK) return s;
    *h_seconds = (double)ms * 1e-3 / (double)loops;
    return RT_OK;
}

// ------------------------------------------------------------------------------------
// snr2
// ------------------------------------------------------------------------------------
static int check_widths(const uint64_t* w, size_t nw, size_t bins, std::vector<int>& out)
{
    out.clear();
    for (size_t i = 0; i < nw; ++i) {
        // snr.hpp:21-31
        if (!((w[i] > 0) & (w[i] < bins)))
            return set_error(RT_EINVAL, "trial widths must be all > 0 and < columns");
        out.push_back((int)w[i]);
    }
    if (nw > (size_t)kMaxWidths)
        return set_error(RT_EINVAL, "at most %d trial widths are supported", kMaxWidths);
    return RT_OK;
}

extern "C" int rt_snr2(const float* d_in, size_t rows, size_t cols, const uint64_t* h_widths,
                       size_t num_widths, float stdnoise, float* d_out, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (!(stdnoise > 0)) return set_error(RT_EINVAL, "stdnoise must be > 0");  // snr.hpp:14-18
    std::vector<int> w;
    RT_TRY(check_widths(h_widths, num_widths, cols, w));
    if (rows == 0 || num_widths == 0) return RT_OK;
    if (cols > 4096) return set_error(RT_EINVAL, "profiles longer than 4096 bins are not supported");
    return rt::snr2(d_in, rows, cols, w.data(), (int)w.size(), stdnoise, d_out, st);
}

// ------------------------------------------------------------------------------------
// downsample
// ------------------------------------------------------------------------------------
extern "C" size_t rt_downsampled_size(size_t size, double f) { return downsampled_size(size, f); }

static int downsample_one(const float* d_in, size_t size, double f, float* d_out, cudaStream_t st)
{
    DsJob job{};
    job.in = d_in;
    job.one_len = size;
    job.one_f = f;
    job.out = d_out;
    job.ncycles = 1;
    const int use_seg = ds_use_segments(f) ? 1 : 0, skip = 0;
    job.use_seg_host = &use_seg;
    job.f_host = &f;
    job.skip_host = &skip;
    return launch_downsample(job, 1, size, st);
}

extern "C" int rt_downsample(const float* d_in, size_t size, double f, float* d_out,
                             void* stream)
{
    // downsample.hpp:11-16
    if (!((f > 1.0) & (f <= (double)size)))
        return set_error(RT_EINVAL, "Downsampling factor must verify: 1 < f <= size");
    return downsample_one(d_in, size, f, d_out, (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------
// running median
// ------------------------------------------------------------------------------------
extern "C" int rt_running_median(const float* d_in, size_t size, size_t width, float* d_out,
                                 void* stream)
{
    // running_median.hpp:103-107
    if (!(width % 2)) return set_error(RT_EINVAL, "width must be an odd number");
    if (!(width < size)) return set_error(RT_EINVAL, "width must be < size");
    return launch_running_median(d_in, nullptr, nullptr, 1, size, (int)width, d_out,
                                 (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------
// periodogram
// ------------------------------------------------------------------------------------
extern "C" int rt_periodogram_length(size_t size, double tsamp, double period_min,
                                     double period_max, size_t bins_min, size_t bins_max,
                                     size_t* h_length)
{
    if (!h_length) return set_error(RT_EINVAL, "null argument");
    if (!(tsamp > 0)) return set_error(RT_EINVAL, "tsamp must be > 0");
    if (!(period_min > 0)) return set_error(RT_EINVAL, "period_min must be > 0");
    if (!(period_max > period_min)) return set_error(RT_EINVAL, "period_max must be > period_min");
    if (!(bins_min > 1)) return set_error(RT_EINVAL, "bins_min must be > 1");
    if (!(bins_max >= bins_min)) return set_error(RT_EINVAL, "bins_max must be >= bins_min");
    if (!(period_min >= tsamp * bins_min))
        return set_error(RT_EINVAL, "Must have: period_min >= tsamp * bins_min ");
    const double ds_ini = period_min / (tsamp * bins_min);
    const double ds_geo = (bins_max + 1.0) / bins_min;
    const size_t nds = (size_t)ceil(log(period_max / period_min) / log(ds_geo));
    size_t len = 0;
    for (size_t ids = 0; ids < nds; ++ids) {
        const double f = ds_ini * pow(ds_geo, (double)ids);
        const double tau = f * tsamp;
        const double pms = period_max / tau;
        const size_t n = downsampled_size(size, f);
        const size_t bstop = std::min({bins_max, n, (size_t)pms});
        for (size_t b = bins_min; b <= bstop; ++b) len += rows_to_evaluate(n / b, b, pms);
    }
    *h_length = len;
    return RT_OK;
}

extern "C" int rt_search_plan_create(const uint64_t*, size_t, const rt_search_config*,
                                     const uint64_t*, size_t, rt_search_plan**);
extern "C" int rt_search_run(rt_search_plan*, const float*, float*, double*, uint32_t*, float*,
                             void*);
extern "C" int rt_search_check(rt_search_plan*, void*);
extern "C" void rt_search_plan_destroy(rt_search_plan*);

// Plans of the single-series periodogram, cached by geometry (a series length and search
// parameters reused across calls is the common case: all DM trials of one observation).
namespace {
struct PgKey {
    size_t size;
    double tsamp, pmin, pmax;
    size_t bmin, bmax;
    std::vector<uint64_t> widths;
    bool operator<(const PgKey& o) const
    {
        return std::tie(size, tsamp, pmin, pmax, bmin, bmax, widths) <
               std::tie(o.size, o.tsamp, o.pmin, o.pmax, o.bmin, o.bmax, o.widths);
    }
};
std::mutex g_pg_mutex;
std::map<PgKey, rt_search_plan*> g_pg_cache;
}  // namespace

extern "C" int rt_periodogram(const float* d_data, size_t size, double tsamp,
                              const uint64_t* h_widths, size_t num_widths, double period_min,
                              double period_max, size_t bins_min, size_t bins_max,
                              double* d_periods, uint32_t* d_foldbins, float* d_snrs,
                              void* stream)
{
    size_t L = 0;
    RT_TRY(rt_periodogram_length(size, tsamp, period_min, period_max, bins_min, bins_max, &L));
    if (L == 0) return RT_OK;
    std::lock_guard<std::mutex> lock(g_pg_mutex);
    PgKey key{size, tsamp, period_min, period_max, bins_min, bins_max,
              std::vector<uint64_t>(h_widths, h_widths + num_widths)};
    rt_search_plan* plan = nullptr;
    auto it = g_pg_cache.find(key);
    if (it != g_pg_cache.end()) {
        plan = it->second;
    } else {
        rt_search_config cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.tsamp = tsamp;
        cfg.period_min = period_min;
        cfg.period_max = period_max;
        cfg.bins_min = bins_min;
        cfg.bins_max = bins_max;
        cfg.deredden = 0;
        cfg.already_normalised = 1;
        const uint64_t len = size;
        RT_TRY(rt_search_plan_create(&len, 1, &cfg, h_widths, num_widths, &plan));
        if (g_pg_cache.size() >= 8) {
            rt_search_plan_destroy(g_pg_cache.begin()->second);
            g_pg_cache.erase(g_pg_cache.begin());
        }
        g_pg_cache[key] = plan;
    }
    RT_TRY(rt_search_run(plan, d_data, nullptr, d_periods, d_foldbins, d_snrs, stream));
    return rt_search_check(plan, stream);
}

extern "C" int rt_periodogram_plain(const float* d_data, size_t size, double tsamp,
                                    const uint64_t* h_widths, size_t num_widths,
                                    double period_min, double period_max, size_t bins_min,
                                    size_t bins_max, double* d_periods, uint32_t* d_foldbins,
                                    float* d_snrs, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    size_t L = 0;
    RT_TRY(rt_periodogram_length(size, tsamp, period_min, period_max, bins_min, bins_max, &L));
    std::vector<int> w;
    RT_TRY(check_widths(h_widths, num_widths, bins_min, w));
    if (L == 0) return RT_OK;
    const double ds_ini = period_min / (tsamp * bins_min);
    const double ds_geo = (bins_max + 1.0) / bins_min;
    const size_t nds = (size_t)ceil(log(period_max / period_min) / log(ds_geo));
    const size_t bufsize = downsampled_size(size, ds_ini);
    float *input = nullptr, *ffaout = nullptr, *scratch = nullptr;
    int* d_err = nullptr;
    size_t scratch_floats = 0;
    for (size_t b = bins_min; b <= bins_max && b <= bufsize; ++b)
        scratch_floats = std::max(scratch_floats, ffa_scratch_floats((int)(bufsize / b), (int)b));
    RT_TRY_CUDA(scratch_malloc((void**)&input, std::max<size_t>(bufsize, 1) * sizeof(float), st));
    RT_TRY_CUDA(scratch_malloc((void**)&ffaout, std::max<size_t>(bufsize, 1) * sizeof(float), st));
    RT_TRY_CUDA(scratch_malloc((void**)&scratch, std::max<size_t>(scratch_floats, 1) * sizeof(float), st));
    RT_TRY_CUDA(scratch_malloc((void**)&d_err, sizeof(int), st));
    RT_TRY_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    int s = RT_OK;
    double* periods = d_periods;
    uint32_t* foldbins = d_foldbins;
    float* snr = d_snrs;
    for (size_t ids = 0; ids < nds && s == RT_OK; ++ids) {
        const double f = ds_ini * pow(ds_geo, (double)ids);
        const double tau = f * tsamp;
        const double pms = period_max / tau;
        const size_t n = downsampled_size(size, f);
        const float* in = d_data;
        if (f != 1) {
            if (!((f > 1.0) & (f <= (double)size))) {
                s = set_error(RT_EINVAL, "Downsampling factor must verify: 1 < f <= size");
                break;
            }
            s = downsample_one(d_data, size, f, input, st);
            in = input;
        }
        const size_t bstop = std::min({bins_max, n, (size_t)pms});
        for (size_t b = bins_min; b <= bstop && s == RT_OK; ++b) {
            const size_t rows = n / b;
            const float stdnoise = (float)sqrt((double)rows * downsampled_variance(size, f));
            const size_t re = rows_to_evaluate(rows, b, pms);
            if (re == 0) continue;
            s = ffa_transform(in, (int)rows, (int)b, (int)rows, ffaout, scratch, d_err, st);
            if (s != RT_OK) break;
            s = rt::snr2(ffaout, re, b, w.data(), (int)w.size(), stdnoise, snr, st);
            if (s != RT_OK) break;
            s = launch_periods(periods, foldbins, re, tau, (int)b, rows, st);
            snr += re * w.size();
            periods += re;
            foldbins += re;
        }
    }
    int herr = 0;
    cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(input, st);
    cudaFreeAsync(ffaout, st);
    cudaFreeAsync(scratch, st);
    cudaFreeAsync(d_err, st);
    if (s != RT_OK) return s;
    RT_TRY_CUDA(cudaStreamSynchronize(st));
    if (herr) return set_error(RT_EINTERNAL, "FFA device plan check failed (%d)", herr);
    return RT_OK;
}
