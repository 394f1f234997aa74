// Boxcar S/N of folded profiles held in shared memory (cpp/snr.hpp:37-65).
//
// Per profile x of b bins the reference computes the circular prefix sum
//     C[j] = float(sum_{i<=j} x[i])  (double accumulator),  C[b+j] = C[j] + float(total)
// (cpp/kernels.hpp:73-101) and, for every trial width w,
//     dmax = max_i (C[i+w] - C[i]),  h = sqrt((b-w)/(b*w)),  beta = w/(b-w)*h,
//     S/N = ((h + beta) * dmax - beta * C[b-1]) / stdnoise
// (snr.hpp:49-52; the reference build fuses the first product and the subtraction, which is
// reproduced with __fmaf_rn). Everything below follows that arithmetic exactly; the only
// change of order is the prefix sum: the TPR threads of a profile sum their segments, scan the
// segment totals and accumulate their running prefixes, all in double, which is identical to
// the reference's sequential double sum whenever the sums are exact (float inputs whose
// magnitudes within one profile span less than about 2^29).
//
// Work split: TPR threads share one profile; each builds its segment of C, then holds a
// window C[i .. i+SB+WMAX) in registers so that every width reads registers only. What bounds
// it is the number of instructions (about 21 per phase, of which 12.5 are the differences and
// maxima of the ten widths). A round of 60 profiles of 250 bins takes a CTA 6,800 cycles, of
// which 2,500 are the window and 1,000 the double-precision prefixes; the prefix in double-float
// pairs (eight float additions a value against one double addition and two conversions) and a
// guard on every load and store made it 8,000.
#pragma once
#include "common.cuh"
#include "ffa_core.cuh"

namespace rt {

// Trial widths generate_width_trials(bmin, ducy_max=0.2, wtsp=1.5) begin with these ten
// for every bmin >= 210 (ffautils.py:4-11). They get the register-window fast path.
struct FastWidths10 {
    static constexpr int NW = 10;
    static constexpr int WMAX = 42;
    __host__ __device__ static constexpr int w(int k)
    {
        return k == 0 ? 1 : k == 1 ? 2 : k == 2 ? 3 : k == 3 ? 4 : k == 4 ? 6 : k == 5 ? 9
             : k == 6 ? 13 : k == 7 ? 19 : k == 8 ? 28 : 42;
    }
};

constexpr int kMaxWidths = 64;

// Per-call width data, placed in shared memory by the caller.
struct SnrParams {
    int nw;                  // number of trial widths
    int nfast;               // leading widths handled by the register window (0 or 10)
    int wmax;                // largest width
    int b;                   // profile length the coefficients are for
    int w[kMaxWidths];
    float hb[kMaxWidths];    // h + beta (per width, for the current b)
    float beta[kMaxWidths];  // beta
};

// Boxcar coefficients for profile length b (snr.hpp:49-50).
__device__ __forceinline__ void boxcar_coefs(int b, int w, float* hb, float* beta)
{
    const float h = __fsqrt_rn(__fdiv_rn((float)(b - w), (float)((size_t)b * (size_t)w)));
    const float be = __fmul_rn(__fdiv_rn((float)w, (float)(b - w)), h);
    *hb = __fadd_rn(h, be);
    *beta = be;
}

__device__ inline void snr_params_fill(SnrParams& S, const int* widths, int nw, int nfast, int b)
{
    if (threadIdx.x == 0) {
        S.nw = nw;
        S.nfast = nfast;
        int wm = 0;
        for (int k = 0; k < nw; ++k) wm = widths[k] > wm ? widths[k] : wm;
        S.wmax = wm;
        S.b = b;
    }
    for (int k = threadIdx.x; k < nw; k += kThreads) {
        S.w[k] = widths[k];
        boxcar_coefs(b, widths[k], &S.hb[k], &S.beta[k]);
    }
    cta_sync();
}

// The widths alone, by one warp; the coefficients follow for each profile length.
__device__ inline void snr_widths_warp(SnrParams& S, const int* widths, int nw, int nfast)
{
    const int lane = threadIdx.x & 31;
    int wm = 0;
    for (int k = lane; k < nw; k += 32) {
        S.w[k] = widths[k];
        wm = max(wm, S.w[k]);
    }
    wm = __reduce_max_sync(0xffffffffu, wm);
    if (lane == 0) {
        S.nw = nw;
        S.nfast = nfast;
        S.wmax = wm;
        S.b = 0;
    }
    __syncwarp();
}

// The coefficients for profiles of b bins, by one warp (no CTA barrier).
__device__ inline void snr_coefs_warp(SnrParams& S, int b)
{
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < S.nw; k += 32) boxcar_coefs(b, S.w[k], &S.hb[k], &S.beta[k]);
    if (lane == 0) S.b = b;
    __syncwarp();
}

__device__ __forceinline__ float fmax3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Max over SB consecutive phases [start, start + SB) of C[i+w] - C[i], for the fast widths,
// from a register window (start + SB <= b, so every phase is a real phase of the profile).
// Threads of one profile may cover overlapping phases: a maximum does not mind duplicates.
template <class WS, int SB>
__device__ __forceinline__ void window_max(const float* cr, int start, float (&mx)[WS::NW])
{
    static_assert(SB % 2 == 0, "phase pairs");
    float win[SB + WS::WMAX];
#pragma unroll
    for (int j = 0; j < SB + WS::WMAX; ++j) win[j] = cr[start + j];
#pragma unroll
    for (int j = 0; j < SB; j += 2) {
#pragma unroll
        for (int k = 0; k < WS::NW; ++k) {
            if (WS::w(k) % 2 == 0) {
                // even width: both phases' differences in one packed subtraction (two
                // round-to-nearest float32 subtractions, as __fsub_rn)
                float d0, d1;
                asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
                    " sub.rn.f32x2 d, a, b;\n mov.b64 {%0, %1}, d;\n}"
                    : "=f"(d0), "=f"(d1)
                    : "f"(win[j + WS::w(k)]), "f"(win[j + 1 + WS::w(k)]), "f"(win[j]), "f"(win[j + 1]));
                mx[k] = fmax3(mx[k], d0, d1);
            } else {
                mx[k] = fmax3(mx[k], __fsub_rn(win[j + WS::w(k)], win[j]),
                              __fsub_rn(win[j + 1 + WS::w(k)], win[j + 1]));
            }
        }
    }
}

// Folds the N per-width maxima of TPR lanes by halves: at each step a lane keeps the maxima of
// one half of its widths (the middle one of an odd number goes to both sides) and sends the
// other half to its partner, until each lane holds the TPR-wide maxima of widths *k and up.
// 2 N + ... instead of N log2(TPR) shuffles. Returns how many a lane holds at the end.
template <int N, int OFF>
__device__ __forceinline__ void fold_maxima(float (&mx)[FastWidths10::NW], unsigned mask, int t, int* k)
{
    if constexpr (OFF > 0) {
        constexpr int KEEP = (N + 1) / 2, SKIP = N - KEEP;
        const bool up = t & OFF;
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const float send = up ? mx[i] : mx[i + SKIP];
            const float keep = up ? mx[i + SKIP] : mx[i];
            mx[i] = fmaxf(keep, __shfl_xor_sync(mask, send, OFF));
        }
        if (up) *k += SKIP;
        fold_maxima<KEEP, OFF / 2>(mx, mask, t, k);
    }
}
// Widths a lane holds after fold_maxima over TPR lanes.
constexpr int folded_widths(int n, int tpr) { return tpr > 1 ? folded_widths((n + 1) / 2, tpr / 2) : n; }

// Phases of a thread whose prefix passes are unrolled, the values held in registers: up to 264
// bins with 8 threads, 528 with 16. (An odd number: the threads of a profile hit distinct banks.)
constexpr int kSnrPhases = 33;
RT_HD int snr_phases(int b, int tpr)
{
    return b <= tpr * kSnrPhases ? kSnrPhases : ((b + tpr - 1) / tpr) | 1;
}

// Boxcar S/N of `nrows` folded profiles (rows of X, stride xs) straight from the FFA output:
// TPR threads per profile build its circular prefix sum (double accumulation, group scan) in
// the scratch rows C (stride cs), then take the width maxima from a register window. Only
// warp-level synchronisation: a profile's TPR threads are lanes of one warp. Writes
// out[r * out_stride + k]. `groups` profiles are processed at a time (C holds `groups` rows).
// kUnrolled: kSnrPhases phases per thread. kGuard: X must not be read past a row's end; without
// it all TPR * kSnrPhases values from the row's start are read (snr_overread floats past the last
// row, for which the caller has room): anything may be past bin b - 1, it only reaches prefix
// values past b - 1, which the wrap-around part replaces as far as they are read.
template <int TPR, int SB, bool kUnrolled, bool kGuard>
__device__ __forceinline__ void snr_rows_impl(const float* X, int xs, int nrows, int b,
                                              const SnrParams& S, float stdnoise,
                                              float* __restrict__ out, size_t out_stride, float* C,
                                              int cs, int groups)
{
    constexpr int PMAX = kUnrolled ? kSnrPhases : 1, PH = (kSnrPhases + 1) / 2;
    constexpr int NW = FastWidths10::NW;
    const int tid = threadIdx.x;
    const int g = tid / TPR, t = tid - g * TPR;
    const int ngroups = min(groups, kThreads / TPR);
    const int P = kUnrolled ? kSnrPhases : snr_phases(b, TPR);
    const int i0 = kGuard ? min(b, t * P) : t * P, i1 = min(b, t * P + P);
    const unsigned gmask = (TPR == 32) ? 0xffffffffu : (((1u << TPR) - 1u) << ((tid & 31) & ~(TPR - 1)));
    if (g >= ngroups) return;  // whole groups leave together
    float* cr = C + (size_t)g * cs;
    for (int r = g; r < nrows; r += ngroups) {
        const float* xr = X + (size_t)r * xs + i0;
        // prefix sums (kernels.hpp:73-101): the thread's segment total (two halves, so that the
        // additions form two chains), a scan of the totals, the running prefix of each half
        float v[PMAX];
        double s0 = 0.0, s1 = 0.0;
        if (kUnrolled) {
#pragma unroll
            for (int j = 0; j < PMAX; ++j) v[j] = (!kGuard || j < i1 - i0) ? xr[j] : 0.0f;
#pragma unroll
            for (int j = 0; j < PH; ++j) {
                s0 = __dadd_rn(s0, (double)v[j]);
                if (j + PH < PMAX) s1 = __dadd_rn(s1, (double)v[j + PH]);
            }
        } else {
            const int n = max(0, i1 - i0);
#pragma unroll 8
            for (int j = 0; j < n; ++j) s0 = __dadd_rn(s0, (double)xr[j]);
        }
        double incl = __dadd_rn(s0, s1);
#pragma unroll
        for (int o = 1; o < TPR; o <<= 1) {
            const double y = __shfl_up_sync(gmask, incl, o, TPR);
            if (t >= o) incl = __dadd_rn(y, incl);
        }
        double run = __shfl_up_sync(gmask, incl, 1, TPR);
        if (t == 0) run = 0.0;
        float* c0 = cr + i0;
        if (kUnrolled) {
            double run1 = __dadd_rn(run, s0);
#pragma unroll
            for (int j = 0; j < PH; ++j) {
                run = __dadd_rn(run, (double)v[j]);
                if (!kGuard || j < i1 - i0) c0[j] = __double2float_rn(run);
                if (j + PH < PMAX) {
                    run1 = __dadd_rn(run1, (double)v[j + PH]);
                    if (!kGuard || j + PH < i1 - i0) c0[j + PH] = __double2float_rn(run1);
                }
            }
        } else {
            const int n = max(0, i1 - i0);
#pragma unroll 8
            for (int j = 0; j < n; ++j) {
                run = __dadd_rn(run, (double)xr[j]);
                c0[j] = __double2float_rn(run);
            }
        }
        __syncwarp(gmask);
        const float sum = cr[b - 1];
        // the wrap-around part (it also replaces what unguarded tails left past bin b - 1)
        for (int j = t; j < S.wmax; j += TPR) cr[b + j] = __fadd_rn(cr[j], sum);
        __syncwarp(gmask);
        float* orow = out + (size_t)r * out_stride;
        if (S.nfast == NW) {
            float mx[NW];
#pragma unroll
            for (int k = 0; k < NW; ++k) mx[k] = -INFINITY;
            // (b > 42 >= SB: the fast widths end at 42)
            if (kUnrolled) {
                window_max<FastWidths10, SB>(cr, min(i0, b - SB), mx);
            } else {
#pragma unroll 1
                for (int i = i0; i < i1; i += SB) window_max<FastWidths10, SB>(cr, min(i, b - SB), mx);
            }
            int k0 = 0;
            fold_maxima<NW, TPR / 2>(mx, gmask, t, &k0);
#pragma unroll
            for (int q = 0; q < folded_widths(NW, TPR); ++q) {
                const int k = k0 + q;
                orow[k] = __fdiv_rn(__fmaf_rn(S.hb[k], mx[q], -__fmul_rn(S.beta[k], sum)), stdnoise);
            }
        }
        // remaining widths (63 and 94 for bins_min 480), two at a time straight from shared
        // memory: each phase's C[i] is loaded once for both widths, eight phases per step
        for (int k = S.nfast; k < S.nw; k += 2) {
            const bool two = k + 1 < S.nw;
            const int w1 = S.w[k], w2 = two ? S.w[k + 1] : w1;
            float m1 = -INFINITY, m2 = -INFINITY;
            int i = i0;
#pragma unroll 1
            for (; i + 8 <= i1; i += 8) {
                float a[8], p[8], q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    a[j] = cr[i + j];
                    p[j] = cr[i + j + w1];
                    q[j] = cr[i + j + w2];
                }
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    m1 = fmax3(m1, __fsub_rn(p[j], a[j]), __fsub_rn(p[j + 1], a[j + 1]));
                    m2 = fmax3(m2, __fsub_rn(q[j], a[j]), __fsub_rn(q[j + 1], a[j + 1]));
                }
            }
#pragma unroll 1
            for (; i < i1; ++i) {
                const float a = cr[i];
                m1 = fmaxf(m1, __fsub_rn(cr[i + w1], a));
                m2 = fmaxf(m2, __fsub_rn(cr[i + w2], a));
            }
#pragma unroll
            for (int o = TPR / 2; o > 0; o >>= 1) {
                m1 = fmaxf(m1, __shfl_xor_sync(gmask, m1, o, TPR));
                m2 = fmaxf(m2, __shfl_xor_sync(gmask, m2, o, TPR));
            }
            if (t == 0) {
                orow[k] = __fdiv_rn(__fmaf_rn(S.hb[k], m1, -__fmul_rn(S.beta[k], sum)), stdnoise);
                if (two)
                    orow[k + 1] =
                        __fdiv_rn(__fmaf_rn(S.hb[k + 1], m2, -__fmul_rn(S.beta[k + 1], sum)), stdnoise);
            }
        }
        __syncwarp(gmask);  // cr is rewritten for the next profile
    }
}

// Profiles in global memory.
template <int TPR, int SB>
__device__ __forceinline__ void snr_rows(const float* X, int xs, int nrows, int b,
                                         const SnrParams& S, float stdnoise,
                                         float* __restrict__ out, size_t out_stride, float* C,
                                         int cs, int groups)
{
    if (b <= TPR * kSnrPhases)
        snr_rows_impl<TPR, SB, true, true>(X, xs, nrows, b, S, stdnoise, out, out_stride, C, cs, groups);
    else
        snr_rows_impl<TPR, SB, false, true>(X, xs, nrows, b, S, stdnoise, out, out_stride, C, cs, groups);
}

// Row stride for prefix-sum rows: >= b + wmax and the whole segments of the TPR threads, and
// = TPR (mod 32), so that with an odd per-thread phase count the TPR threads of a profile and
// the 32/TPR profiles of a warp read distinct banks.
RT_HD int prefix_stride(int b, int wmax, int tpr)
{
    const int seg = tpr * snr_phases(b, tpr);
    int s = b + wmax > seg ? b + wmax : seg;
    s = (s + 31) & ~31;
    return s + tpr;
}

// Threads per profile: the fewest whose kSnrPhases phases each hold it, at least 4 (a window of
// 33 phases costs 75 reads, one of half the phases 58: fewer threads with long segments read
// and scan less), 32 beyond 1056 bins.
RT_HD int snr_tpr(int b)
{
    return b <= 4 * kSnrPhases ? 4 : b <= 8 * kSnrPhases ? 8 : b <= 16 * kSnrPhases ? 16 : 32;
}

// Floats past the end of a row of ffa_stride(b) floats that the S/N reads without its guard: up to
// 516 (529 bins, 32 threads) by the threads of snr_tpr, 508 by 16 threads for any b they hold.
RT_HD int snr_overread(int b, int tpr)
{
    const int past = tpr * kSnrPhases - ffa_stride(b);
    return b <= tpr * kSnrPhases && past > 0 ? past : 0;
}

// Kinds of S/N code a kernel instance may hold, one bit each: 4, 8, 16 or 32 threads a profile
// with the prefix passes unrolled, 32 threads with loops.
enum : int { kSnr4 = 1, kSnr8 = 2, kSnr16 = 4, kSnr32 = 8, kSnr32Loop = 16 };

RT_HD int snr_kind(int b, int tpr)
{
    return tpr < 32 ? tpr >> 2 : b <= 32 * kSnrPhases ? kSnr32 : kSnr32Loop;
}

}  // namespace rt
