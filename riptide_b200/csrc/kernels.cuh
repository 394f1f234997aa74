// Declarations shared by the kernel files of riptide_b200.
#pragma once
#include "common.cuh"
#include "ffa_core.cuh"

namespace rt {

// Dynamic shared memory of the FFA / S/N kernels (one CTA per SM).
constexpr size_t kFfaSmemBytes = 226 * 1024;

size_t ffa_scratch_floats(int m, int b);
int detect_fast_widths(const int* w, int nw);
const char* last_error();

// Stream-ordered device scratch (freed with cudaFreeAsync) from a pool of this library, one per
// device, that keeps up to kScratchKept bytes over synchronisations: CUDA's default pool gives
// all its memory back at each one, and mapping it again cost the small entry points 100 to
// 400 us a call. release_scratch gives the kept memory of the current device back; a plan that
// runs out of device memory does so before it tries again.
constexpr size_t kScratchKept = size_t(512) << 20;
// inject_scratch_fault: the nth allocation of the calling thread from now on fails (0: none).
cudaError_t scratch_malloc(void** p, size_t bytes, cudaStream_t st);
void release_scratch();
void inject_scratch_fault(int nth);

// FFA transform of an m x b block (device pointers). rows_out <= m root rows are produced
// (the reference's ffa2 uses rows_out = m). `scratch` holds ffa_scratch_floats(m, b)
// floats. Errors of the device plan are reported through d_err and leave NaN in the rows concerned.
int ffa_transform(const float* in, int m, int b, int rows_out, float* out, float* scratch,
                  int* d_err, cudaStream_t st);

// The same by the persistent search kernel, with ffa_persistent_bytes(m, b, rows_out) bytes of
// 256-byte aligned scratch (0: not for this size). Its waits are bounded, by `wait_polls` polls
// (0: kSpinLimit): one that runs out leaves NaN in all of `out` and RT_ETIMEOUT in *d_err.
// `dep_bias` is added to what a later stage waits for (fault injection).
constexpr int kPersistentItems = 1000;
size_t ffa_persistent_bytes(int m, int b, int rows_out);
int ffa_transform_persistent(const float* in, int m, int b, int rows_out, float* out, void* scratch,
                             int* d_err, cudaStream_t st, long long wait_polls = 0,
                             int dep_bias = 0);

int snr2(const float* x, size_t rows, size_t cols, const int* h_widths, int nw, float stdnoise,
         float* out, cudaStream_t st);
int rollback(const float* x, size_t size, size_t shift, float* out, cudaStream_t st);
int fused_rollback_add(const float* x, const float* y, size_t size, size_t shift, float* out,
                       cudaStream_t st);
int circular_prefix_sum(const float* x, size_t size, size_t nsum, float* out, cudaStream_t st);
int launch_periods(double* periods, uint32_t* foldbins, size_t rows_eval, double tau, int bins,
                   size_t rows, cudaStream_t st);
// (d_lengths null: one series of max_len samples; dependent: by launch_dependent)
int launch_running_median(const float* x, const size_t* d_lengths, const size_t* d_offsets,
                          int ntrials, size_t max_len, int width, float* out, cudaStream_t st,
                          bool dependent = false);

// Downsampling of many series by many factors in one pass (device arrays).
constexpr int kDsStage = 8192;        // input samples staged per CTA (segment + halo)
constexpr int kDsHalo = 4096;         // largest halo: factors up to kDsHalo - 2
constexpr int kDsMaxCycles = 256;

struct DsJob {
    const float* in;            // packed input series
    const size_t* in_off;       // [ntrials] offset of each series
    const size_t* lengths;      // [ntrials]; null: one series of one_len samples and one factor
                                // one_f, the arrays in_off, f, use_seg and out_off are not read
    size_t one_len;
    double one_f;
    const double* mean;         // [ntrials] or null: values are normalised as (v - mean) / norm
    const double* norm;         // [ntrials] or null
    float* norm_out;            // packed normalised series (optional)
    const double* f;            // [ncycles] factors
    const int* use_seg;         // [ncycles] 1: segment kernel, 0: wide kernel
    float* out;                 // packed outputs
    const size_t* out_off;      // [ntrials * ncycles]
    int ncycles;
    int seg;                    // output ownership segment (input samples), set by the launcher
    // host copies for the launcher
    const double* f_host;       // [ncycles]
    const int* use_seg_host;
    const int* skip_host;       // [ncycles] cycles with nothing to produce (f == 1)

    __device__ size_t length(int t) const { return lengths ? lengths[t] : one_len; }
    __device__ size_t input(int t) const { return lengths ? in_off[t] : 0; }
    __device__ size_t output(int t, int c) const
    {
        return lengths ? out_off[(size_t)t * ncycles + c] : 0;
    }
    __device__ double factor(int c) const { return lengths ? f[c] : one_f; }
    __device__ bool segments(int c) const { return lengths ? use_seg[c] != 0 : true; }
};

int launch_downsample(const DsJob& job, int ntrials, size_t max_len, cudaStream_t st);

inline bool ds_use_segments(double f) { return f + 2.0 <= (double)kDsHalo; }

}  // namespace rt
