// Batched FFA search engine: many DM trials of uneven length searched in one pass.
//
// Stream of work for one run (all stream-ordered, capturable in a CUDA graph):
//   1. deredden (time_series.py:95-124 / running_medians.py:40-85): mean-scrunch, exact
//      running median of the scrunched series, linear interpolation back, subtraction;
//   2. normalise (time_series.py:67-93): FP64 mean / variance per trial;
//   3. one pass over every series producing the downsampled copy for every octave cycle
//      (normalisation applied on the fly, cpp/periodogram.hpp:153-168);
//   4. one persistent kernel that walks a precomputed list of FFA jobs (ffa_core.cuh) for all
//      (trial, cycle, bins) transforms and writes the periodogram rows (S/N fused).
// Transforms too large for one CTA are split in stages; jobs of a stage wait for the previous
// stage through per-transform counters, and stage-0 jobs wait until their scratch slot is
// released. These waits, for other CTAs, are bounded and report RT_ETIMEOUT instead of hanging;
// inside a CTA, the compute warps wait for the scheduling warp, which always hands an item over.
#include <string.h>

#include <algorithm>
#include <deque>
#include <map>
#include <set>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "ffa_core.cuh"
#include "kernels.cuh"
#include "snr_core.cuh"

namespace rt {

struct XformRec {
    unsigned long long src_off;  // row 0 of the folded series (offset in its arena)
    unsigned long long out_row;  // first periodogram row of this transform
    double tau;                  // sampling time of the folded series
    int b, m, rows_eval;
    float stdnoise;
    int plan;                    // index into the stage-plan table
    int seq;                     // multi-stage sequence number, -1 for single-stage transforms
    int src_norm;                // 1: src is in the normalised series arena, 0: downsampled arena
    int tune;                    // rows per job (low 16 bits), S/N threads per profile (high)
};

struct WorkItem {
    int xform;
    int stage_job;       // stage << 24 | job
};

// Shared-memory layout of the persistent kernel: per item slot (static) a job tree and the
// boxcar coefficients; the dynamic part holds the row operations and two level buffers.
constexpr size_t kEngineTreeBytes = (sizeof(JobTree) + 255) & ~size_t(255);
constexpr size_t kEngineSnrBytes = (sizeof(SnrParams) + 255) & ~size_t(255);
constexpr size_t kEngineDynBytes = kFfaSmemBytes - 2 * (kEngineTreeBytes + kEngineSnrBytes);

constexpr int kSlots = 256;          // most scratch slots for multi-stage transforms
constexpr size_t kLagItems = 640;    // work items emitted between two stages of a transform
constexpr long long kSpinLimit = 20000000LL;  // default bound of the waits (about 2-20 s with backoff)

struct EngineArgs {
    const float* ds;         // downsampled series arena
    const float* norm;       // normalised series arena (cycles with f == 1)
    float* snrs;
    float* rows_out;         // kRowsOnly
    const XformRec* xforms;
    const WorkItem* items;
    long long nitems;
    const StagePlan* plans;
    const int* widths;
    int nw, nfast;
    float* scratch;          // slots * 2 * slot_floats
    size_t slot_floats;
    int* done;               // [nseq * kMaxStages]
    int* slot_release;       // [slots]: transform `seq` has slot seq & slot_mask, after
    int slot_mask, slot_shift;  // seq >> slot_shift others
    unsigned long long* ticket;
    int* error;              // RT_OK or an error code
    unsigned long long* phase_cycles;  // optional [kPhases] SM-cycle totals (thread 0 of each CTA)
    long long spin_limit;    // polls before a wait gives up with RT_ETIMEOUT
    int dep_bias;            // added to later-stage dependency targets (fault injection; 0)
    FfaLayout layout;        // operations and level buffers in dynamic shared memory
};

// Phases of one work item, for the optional in-kernel profile.
enum { kPhFetch = 0, kPhWait, kPhTree, kPhLevels, kPhSnr, kPhStore, kPhases = 8 };
// extra counters after the phases: blocked on a scratch slot, blocked on a previous stage,
// items claimed, scheduler polls that found nothing ready
constexpr int kCounters = 16;

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Boxcar S/N of a final-stage job's root rows (`root`); `work` is the other level buffer.
template <int TPR, bool kUnrolled>
__device__ __forceinline__ void final_stage_outputs(const JobTree& T, const XformRec& X, const EngineArgs& A,
                                    const SnrParams& S, const float* root, float* work,
                                    int fstride)
{
    const Node r = T.nodes[0];
    const int b = X.b;
    const int cs = prefix_stride(b, S.wmax, TPR);
    const int groups = A.layout.buf_floats / cs;
    snr_rows_impl<TPR, 34, kUnrolled, false>(root, fstride, r.hi - r.lo, b, S, X.stdnoise,
                                             A.snrs + ((size_t)X.out_row + r.lo) * S.nw, S.nw,
                                             work, cs, groups);
}

// Trial periods and fold bins of every transform (periodogram.hpp:190-194), a warp per
// transform. In the persistent kernel they were a tail of float64 divisions that two of the
// fifteen compute warps ran while the others waited: 0.3 of 9.5 ms for 16 trials of 2^22
// samples, against 15 us here.
__global__ void __launch_bounds__(256) k_search_periods(const XformRec* __restrict__ xforms, int n,
                                                        double* __restrict__ periods,
                                                        uint32_t* __restrict__ foldbins)
{
    after_previous_kernel();
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n;
         i += (gridDim.x * blockDim.x) >> 5) {
        const XformRec X = xforms[i];
        for (int s = lane; s < X.rows_eval; s += 32) {
            periods[X.out_row + s] = trial_period(X.tau, X.b, s, X.m);
            foldbins[X.out_row + s] = (uint32_t)X.b;
        }
    }
}

// The persistent kernel has kThreads compute threads and one scheduling warp. The scheduler
// claims the next ticket, loads its descriptors into one of two shared slots and waits for
// its dependencies while the compute threads work on the other slot. A slot is handed over by
// an mbarrier that every compute warp waits for by itself (a warp that is done with an item
// goes on to build the next one's operations), and handed back by a named barrier.
constexpr int kEngineThreads = kThreads + 32;
constexpr int kBarEmpty = 2;  // + slot
constexpr int kBarRead = 4;   // the previous item's root rows have left their level buffer

// A claimed work item. The scheduling warp keeps a pool of them: two handed to the compute
// threads, the others waiting for a dependency or decoded ahead.
struct ItemSlot {
    long long ticket;   // >= nitems: no more work
    int ok;             // 0: a wait failed, stop
    int done_ok;        // set by the compute threads: 0 if the item failed
    int root;           // set by the compute threads: level buffer (0, 1) of the root rows to
                        // store as a stage output, -1: nothing to store
    int stage, last, cap_rows, jobs_of_stage;
    int target;         // the item may start once *dep reaches this value
    const int* dep;     // (null: at once)
    JobSpec J;
    XformRec X;
};
constexpr int kParked = 4;            // items waiting for a dependency
constexpr int kPool = 2 + kParked + 1;  // at most 16: parked entries are numbered in 4 bits

__device__ __forceinline__ void named_sync(int id, int n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int n)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Per-slot count of compute warps done with the slot's item: each warp adds 1 with release
// semantics at CTA scope; the scheduling warp reads it with acquire semantics.
__device__ __forceinline__ void warp_done_release(unsigned* counter)
{
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(counter))
                 : "memory");
}
__device__ __forceinline__ unsigned warps_done_acquire(const unsigned* counter)
{
    unsigned v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(counter))
                 : "memory");
    return v;
}

// Completion of an item for the other CTAs: its stage counter and, after the last job of the
// last stage, the release of the transform's scratch slot. Called by one thread after every
// compute warp of the CTA has released the item (CTA scope) and its stage output is stored;
// the fence makes their global writes visible at GPU scope before the counters.
__device__ __forceinline__ void signal_item_done(const EngineArgs& A, const ItemSlot& P)
{
    if (P.X.seq < 0 || !P.done_ok) return;
    int* d = A.done + (size_t)P.X.seq * kMaxStages + P.stage;
    if (!P.last) {
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(d) : "memory");
        return;
    }
    __threadfence();
    const int prev = atomicAdd(d, 1);
    if (prev + 1 == P.jobs_of_stage) {
        __threadfence();
        atomicAdd(A.slot_release + (P.X.seq & A.slot_mask), 1);
    }
}

__device__ __forceinline__ bool sched_ready(const ItemSlot& L)
{
    return L.dep == nullptr || ld_acquire(L.dep) >= L.target;
}

__device__ __forceinline__ void sched_decode(const EngineArgs& A, long long t, ItemSlot& L)
{
    const WorkItem W = A.items[t];
    const XformRec X = A.xforms[W.xform];
    const StagePlan& P = A.plans[X.plan];
    const int stage = W.stage_job >> 24, job = W.stage_job & 0xffffff;
    const JobSpec J = stage_job(X.m, X.rows_eval, P, stage, job);
    L.ticket = t;
    L.ok = 1;
    L.X = X;
    L.J = J;
    L.stage = stage;
    L.last = stage == P.nstages - 1;
    L.jobs_of_stage = P.jobs[stage];
    L.cap_rows = X.tune & 0xffff;
    const int* dep = nullptr;
    int target = 0;
    if (J.hi > J.lo && X.seq >= 0) {
        const int seq = X.seq;
        if (stage == 0) {
            dep = A.slot_release + (seq & A.slot_mask);
            target = seq >> A.slot_shift;
        } else {
            dep = A.done + (size_t)seq * kMaxStages + stage - 1;
            target = P.jobs[stage - 1] + A.dep_bias;
        }
    }
    L.dep = dep;
    L.target = target;
}

// The level buffer that an item's source rows are staged in: the one that does not hold the
// root rows which the previous item leaves to be stored.
__device__ __forceinline__ int staging_buffer(int prev_root) { return prev_root < 0 ? 1 : 1 - prev_root; }

__device__ __forceinline__ float* level_buffer(unsigned char* smem, const EngineArgs& A, int i)
{
    return reinterpret_cast<float*>(smem + (size_t)A.layout.ops_units * 16) +
           (size_t)i * A.layout.buf_floats;
}

__device__ __forceinline__ float* stage_output(const EngineArgs& A, const XformRec& X, int stage)
{
    return A.scratch + ((size_t)(X.seq & A.slot_mask) * 2 + (stage & 1)) * A.slot_floats;
}

// Whether an item's source rows come by bulk copies (issued by the scheduling warp).
__device__ __forceinline__ bool staged_async(const ItemSlot& L, const JobTree& T)
{
    if (L.J.hi <= L.J.lo || T.error) return false;
    return L.stage == 0 ? !L.X.src_norm : T.pstaged != 0;
}

// Issues the bulk copies of an item's source rows into level buffer `buf` (one warp): for
// stage-0 jobs (whole subtrees) one contiguous block of the downsampled arena, in whole 16-byte
// units (the arena is padded); for later stages the blocks of the previous stage's output that
// the cone needs.
__device__ __forceinline__ void stage_item(const EngineArgs& A, const ItemSlot& L, const JobTree& T,
                                           float* buf, uint64_t* bar)
{
    if (!staged_async(L, T)) return;
    const int b = L.X.b;
    if (L.stage > 0)
        stage_source_rows_async(T, stage_output(A, L.X, L.stage - 1), ffa_stride(b), buf, bar);
    else if ((threadIdx.x & 31) == 0)
        stage_rows_async(buf, A.ds + L.X.src_off + (size_t)L.J.root_row0 * b,
                         (size_t)L.J.root_rows * b, bar);
}

// Issues the bulk store of a stage's root rows [lo, hi), one block in the level buffer and in
// the stage output (same stride, a multiple of 16 bytes). One thread; the writers of the rows
// have made them visible to the async proxy.
__device__ __forceinline__ void store_root_rows(const EngineArgs& A, const ItemSlot& L,
                                                const float* buf)
{
    const int fstride = ffa_stride(L.X.b);
    bulk_s2g(stage_output(A, L.X, L.stage) + (size_t)(L.J.root_row0 + L.J.lo) * fstride, buf,
             (size_t)(L.J.hi - L.J.lo) * fstride * sizeof(float));
}

// What the compute threads see of the scheduling warp.
struct Handover {
    ItemSlot pool[kPool + 1];    // the last entry: no more work
    int item[2];              // pool entry of each slot's item
    unsigned finished[2];     // compute warps done with the slot's item
    unsigned long long full[2];  // mbarriers: the slot's item is ready
    unsigned long long staged;   // mbarrier: the item's source rows have landed
};

// Hands the compute threads one ready item per slot. Items whose dependency is not met yet
// are parked (up to kParked) while later tickets are tried, so a waiting stage does not stall
// the CTA. Progress: the smallest unfinished ticket has all its dependencies finished (they
// have smaller tickets), so whichever scheduler holds it hands it over; every wait is bounded.
//
// The compute threads need an item every ten thousand cycles or so, and a claim with the loads
// behind it takes three to four thousand: the next ticket is claimed and decoded after an item
// is handed over, while the compute threads run the one before (not near the end of the list,
// where a ticket held ahead could have gone to an idle CTA).
__device__ void scheduler_warp(const EngineArgs& A, Handover& H, JobTree* trees, SnrParams* snr,
                               unsigned char* smem)
{
    const int lane = threadIdx.x & 31;
    uint64_t* bar = reinterpret_cast<uint64_t*>(&H.staged);
    // lane 0: free pool entries; parked entries in order of their tickets, 4 bits each
    unsigned free_mask = (1u << kPool) - 1, parked = 0;
    int nparked = 0, ahead = -1;
    bool exhausted = false;
    // items handed over whose completion is not signalled yet (lane 0), and whether their
    // stage output is on its way: signalled as soon as every compute warp has released them,
    // also while this warp waits for a dependency (an item it waits for may be the one here)
    bool pending[2] = {false, false}, stored[2] = {false, false};
    // signals an item that every compute warp has released
    auto settle = [&](int i, bool is_stored) {
        ItemSlot& L = H.pool[i];
        if (L.root >= 0) {
            if (!is_stored) store_root_rows(A, L, level_buffer(smem, A, L.root));
            bulk_s2g_wait_all();
        }
        signal_item_done(A, L);
    };
    auto claimed = [&](long long t) {  // a pool entry with item t, -1: no more
        if (t >= A.nitems) {
            exhausted = true;
            return -1;
        }
        const int i = __ffs(free_mask) - 1;
        free_mask &= ~(1u << i);
        sched_decode(A, t, H.pool[i]);
        if (A.phase_cycles) atomicAdd(A.phase_cycles + 10, 1ull);
        return i;
    };
    auto claim = [&]() { return claimed((long long)atomicAdd(A.ticket, 1ull)); };
    int k = 0;
    for (;; ++k) {
        const int s = k & 1;
        if (k >= 2) {
            named_sync(kBarEmpty + s, kEngineThreads);  // compute is done with item k-2
            // ... and starts item k-1: the stage output of item k-2 and the source rows of k-1
            const ItemSlot& P = H.pool[H.item[s]];
            if (lane == 0 && P.root >= 0 && !stored[s])
                store_root_rows(A, P, level_buffer(smem, A, P.root));
            stage_item(A, H.pool[H.item[s ^ 1]], trees[s ^ 1],
                       level_buffer(smem, A, staging_buffer(P.root)), bar);
            if (P.root >= 0) {
                if (lane == 0 && !stored[s]) bulk_s2g_wait_read();
                if (lane == 0) stored[s] = true;
                __syncwarp();
                named_arrive(kBarRead, kEngineThreads);
            }
        }
        int owed = -1;  // pool entry of item k-2 while it is not signalled
        if (lane == 0) {
            const long long w0 = clock64();
            if (k >= 2 && pending[s]) owed = H.item[s];
            else if (k >= 2) free_mask |= 1u << H.item[s];
            int chosen = -1;
            bool stop = false;
            unsigned ns = 32;
            for (long long spin = 0; chosen < 0 && !stop; ++spin) {
                for (int i = 0; i < nparked; ++i) {
                    const int c = (parked >> (4 * i)) & 15;
                    if (sched_ready(H.pool[c])) {
                        chosen = c;
                        const unsigned low = parked & ((1u << (4 * i)) - 1);
                        parked = low | ((parked >> (4 * i + 4)) << (4 * i));
                        --nparked;
                        break;
                    }
                }
                if (chosen >= 0) break;
                if (ahead < 0 && !exhausted && nparked < kParked) ahead = claim();
                if (ahead >= 0) {
                    if (sched_ready(H.pool[ahead])) {
                        chosen = ahead;
                        ahead = -1;
                        break;
                    }
                    if (nparked < kParked) {
                        if (A.phase_cycles)
                            atomicAdd(A.phase_cycles + (H.pool[ahead].stage == 0 ? 8 : 9), 1ull);
                        parked |= (unsigned)ahead << (4 * nparked++);
                        ahead = -1;
                        continue;
                    }
                }
                if (owed >= 0) {
                    settle(owed, stored[s]);
                    free_mask |= 1u << owed;
                    owed = -1;
                }
                if (pending[s ^ 1] && warps_done_acquire(H.finished + (s ^ 1)) >= (unsigned)kWarps) {
                    settle(H.item[s ^ 1], stored[s ^ 1]);  // item k-1
                    stored[s ^ 1] = true;
                    pending[s ^ 1] = false;
                }
                if (ld_acquire(A.error) != RT_OK) {
                    stop = true;
                } else if (exhausted && nparked == 0 && ahead < 0) {
                    stop = true;
                } else if (spin > A.spin_limit) {
                    atomicExch(A.error, RT_ETIMEOUT);
                    stop = true;
                } else if (exhausted || nparked == kParked) {
                    if (A.phase_cycles) atomicAdd(A.phase_cycles + 11, 1ull);
                    __nanosleep(ns);
                    if (ns < 1024) ns <<= 1;
                }
            }
            if (A.phase_cycles) atomicAdd(A.phase_cycles + 7, (unsigned long long)(clock64() - w0));
            if (stop) chosen = kPool;
            H.pool[chosen].done_ok = 1;
            H.pool[chosen].root = -1;
            H.item[s] = chosen;
            H.finished[s] = 0;
        }
        __syncwarp();
        const ItemSlot& L = H.pool[H.item[s]];
        const bool stop = !L.ok;
        // the previous stage's output was written before the counter that lane 0 acquired; it
        // is read by bulk copies
        asm volatile("fence.proxy.async.global;" ::: "memory");
        // the job tree and boxcar coefficients of the item, prepared while the compute threads
        // run the previous item
        if (!stop && L.J.hi > L.J.lo) {
            build_job_tree_warp(trees[s], L.J, L.X.b, L.cap_rows, A.layout.ops_units, L.stage == 0);
            const bool fill = L.last && snr[s].b != L.X.b;
            __syncwarp();
            if (fill) snr_coefs_warp(snr[s], L.X.b);
            if (k == 0) stage_item(A, L, trees[0], level_buffer(smem, A, staging_buffer(-1)), bar);
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(reinterpret_cast<uint64_t*>(H.full + s));
            const bool more = !stop && ahead < 0 && !exhausted &&
                              L.ticket + 8 * (long long)gridDim.x < A.nitems;
            long long t = 0;
            if (more) t = (long long)atomicAdd(A.ticket, 1ull);
            if (owed >= 0) {
                settle(owed, stored[s]);
                free_mask |= 1u << owed;
            }
            pending[s] = true;
            stored[s] = false;
            if (more) ahead = claimed(t);
        }
        if (stop) break;
    }
    // the compute threads still hand back the slot of item k-1
    if (k >= 1) {
        const int s = (k - 1) & 1;
        named_sync(kBarEmpty + s, kEngineThreads);
        if (lane == 0 && pending[s]) settle(H.item[s], stored[s]);
    }
}

constexpr int kRowsOnly = 0;

// The root rows of a job of a transform of its own, without halo, to A.rows_out: 16 bytes a
// thread where the rows allow.
__device__ __forceinline__ void store_rows_out(const EngineArgs& A, const ItemSlot& L,
                                               const float* rows, int stride)
{
    const int b = L.X.b, n = L.J.hi - L.J.lo, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* to = A.rows_out + (size_t)(L.J.root_row0 + L.J.lo) * b;
    if ((b & 3) == 0 && (reinterpret_cast<uintptr_t>(A.rows_out) & 15) == 0) {
        for (int r = warp; r < n; r += kWarps) {
            const float4* from = reinterpret_cast<const float4*>(rows + (size_t)r * stride);
            float4* row = reinterpret_cast<float4*>(to + (size_t)r * b);
            for (int c = lane; c < b >> 2; c += 32) row[c] = from[c];
        }
    } else {
        for (int r = warp; r < n; r += kWarps)
            for (int c = lane; c < b; c += 32) to[(size_t)r * b + c] = rows[(size_t)r * stride + c];
    }
}

// KINDS: the kinds of S/N code (snr_kind) the instance holds; kRowsOnly: none, the root rows of
// the last stage are the result. The host picks the instance (search_kernel_for).
template <int KINDS>
__global__ void __launch_bounds__(kEngineThreads, 1) k_search_persistent(EngineArgs A)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ Handover H;
    __shared__ JobTree trees[2];
    __shared__ SnrParams snr[2];

    after_previous_kernel();
    uint64_t* full = reinterpret_cast<uint64_t*>(H.full);
    uint64_t* staged = reinterpret_cast<uint64_t*>(&H.staged);
    if (threadIdx.x == 0) {
        mbar_init(staged, 1);
        mbar_init(full, 1);
        mbar_init(full + 1, 1);
        H.pool[kPool].ok = 0;
        H.pool[kPool].ticket = A.nitems;
    }
    __syncthreads();
    if (threadIdx.x >= kThreads) {
        // (read from memory for every profile length, they took longer than the node lists)
        snr_widths_warp(snr[0], A.widths, A.nw, A.nfast);
        snr_widths_warp(snr[1], A.widths, A.nw, A.nfast);
        scheduler_warp(A, H, trees, snr, smem);
        return;
    }
    uint4* ops = reinterpret_cast<uint4*>(smem);
    uint32_t bar_phase = 0;
    const bool prof = A.phase_cycles != nullptr;
    long long tprev = prof ? clock64() : 0;
    auto mark = [&](int phase) {
        if (prof && threadIdx.x == 0) {
            const long long t = clock64();
            atomicAdd(A.phase_cycles + phase, (unsigned long long)(t - tprev));
            tprev = t;
        }
    };
    int prev_root = -1;  // level buffer of the previous item's root rows while they are stored
    for (int k = 0;; ++k) {
        const int sl = k & 1;
        // the scheduling warp's own waits are bounded and it always hands a slot over: this
        // limit, hours, is only there so that the loop has one
        if (!mbar_wait(full + sl, (k >> 1) & 1, 1ll << 40)) break;
        mark(kPhWait);
        ItemSlot& L = H.pool[H.item[sl]];
        const JobTree& T = trees[sl];
        const SnrParams& S = snr[sl];
        if (!L.ok) break;
        const XformRec& X = L.X;
        const JobSpec& J = L.J;
        const int b = X.b;
        const int fstride = ffa_stride(b);
        const int buf = staging_buffer(prev_root);
        int root = -1;
        bool failed = false;
        if (J.hi > J.lo) {
            // The source rows are staged by the scheduling warp in the background of the
            // operations' build, except those of the normalised series (it may be the caller's
            // buffer, which bulk copies of whole 16-byte units could leave).
            float* sbuf = level_buffer(smem, A, buf);
            LevelIO io;
            io.phase = &bar_phase;
            if (L.stage == 0) {
                const float* from =
                    (X.src_norm ? A.norm : A.ds) + X.src_off + (size_t)J.root_row0 * b;
                int delta = 0;
                if (X.src_norm) {
                    cta_sync();  // every warp is done with the previous item's buffers
                    const int nraw = J.root_rows * b;
#pragma unroll 4
                    for (int i = threadIdx.x; i < nraw; i += kThreads) sbuf[i] = __ldg(from + i);
                } else {
                    delta = staged_delta(from);
                }
                io.staged = sbuf + delta - (ptrdiff_t)J.root_row0 * b;
            } else {
                io.src = stage_output(A, X, L.stage - 1);
                io.src_stride = fstride;  // stage outputs: level rows with halo
                io.staged_rows = true;
                if (T.pstaged) io.staged = sbuf;
            }
            if (staged_async(L, T)) io.bar = staged;
            failed = T.error != 0;
            mark(kPhTree);
            if (!failed) build_ops(T, b, ops);
            // the other level buffer is free once the previous item's root rows have left it
            if (prev_root >= 0) named_sync(kBarRead, kEngineThreads);
            else cta_sync();
            mark(kPhFetch);
            if (failed) {
                if (threadIdx.x == 0) atomicExch(A.error, RT_EINTERNAL);
            } else {
                if (prof && threadIdx.x == 0) {
                    unsigned long long rows = T.fused ? 2 * T.level_rows[T.depth] : 0;
                    for (int d = 0; d <= T.depth; ++d) rows += T.level_rows[d];
                    atomicAdd(A.phase_cycles + 12, rows * b);
                    atomicAdd(A.phase_cycles + 13, (unsigned long long)(J.G + 1));
                    atomicAdd(A.phase_cycles + 14, (unsigned long long)(J.hi - J.lo));
                    atomicAdd(A.phase_cycles + 15, (unsigned long long)(L.stage > 0));
                }
                bool ok = true;
                float* other = level_buffer(smem, A, buf ^ 1);
                float* rows = run_job_levels(T, b, sbuf, other, fstride, ops, io, &ok);
                if (!ok && threadIdx.x == 0) atomicExch(A.error, RT_ETIMEOUT);
                mark(kPhLevels);
                if (KINDS == kRowsOnly && L.last) {
                    store_rows_out(A, L, rows, fstride);
                    mark(kPhSnr);
                } else if (L.last) {
                    float* work = rows == sbuf ? other : sbuf;
                    constexpr bool one = (KINDS & (KINDS - 1)) == 0;
                    const int kind = one ? KINDS : snr_kind(b, X.tune >> 16);
                    if ((KINDS & kSnr4) && kind == kSnr4)
                        final_stage_outputs<4, true>(T, X, A, S, rows, work, fstride);
                    else if ((KINDS & kSnr8) && kind == kSnr8)
                        final_stage_outputs<8, true>(T, X, A, S, rows, work, fstride);
                    else if ((KINDS & kSnr16) && kind == kSnr16)
                        final_stage_outputs<16, true>(T, X, A, S, rows, work, fstride);
                    else if ((KINDS & kSnr32) && kind == kSnr32)
                        final_stage_outputs<32, true>(T, X, A, S, rows, work, fstride);
                    else if (KINDS & kSnr32Loop)
                        final_stage_outputs<32, false>(T, X, A, S, rows, work, fstride);
                    mark(kPhSnr);
                } else {
                    // the scheduling warp stores the root rows (bulk copy): make this thread's
                    // writes visible to the async proxy
                    root = rows == sbuf ? buf : buf ^ 1;
                    fence_proxy_async_smem();
                }
            }
        } else if (prev_root >= 0) {
            named_sync(kBarRead, kEngineThreads);
        }
        prev_root = root;
        // hand the item back: the scheduling warp signals its completion to the other CTAs
        // once every compute warp has released it
        if (threadIdx.x == 0) {
            L.root = root;
            if (failed) L.done_ok = 0;
        }
        __syncwarp();
        if ((threadIdx.x & 31) == 0) warp_done_release(H.finished + sl);
        mark(kPhStore);
        named_arrive(kBarEmpty + sl, kEngineThreads);
    }
}

// ------------------------------------------------------------------------------------
// Deredden / normalise (batched)
// ------------------------------------------------------------------------------------
struct TrialArrays {
    const size_t* len;       // [T]; null: one series, its lengths below and its offsets 0
    const size_t* off;       // [T] offsets into the packed series
    const size_t* lo_len;    // [T] scrunched lengths
    const size_t* lo_off;    // [T] offsets into the packed scrunched series
    size_t one_len, one_lo_len;

    __device__ size_t length(int t) const { return len ? len[t] : one_len; }
    __device__ size_t offset(int t) const { return len ? off[t] : 0; }
    __device__ size_t lo_length(int t) const { return len ? lo_len[t] : one_lo_len; }
    __device__ size_t lo_offset(int t) const { return len ? lo_off[t] : 0; }
};

// ---- numpy's pairwise summation -----------------------------------------------------
// The reference's scrunch is `data[:N].reshape(-1, k).mean(axis=1)` on float32 data
// (running_medians.py:40-46). numpy reduces each contiguous row with its pairwise sum in the
// input type (numpy/_core/src/umath/loops_utils.h.src, pairwise_sum): a block of n < 8
// values is summed in turn from -0.0; a block of 8 <= n <= 128 values in eight strided
// accumulators r[j] = a[j] + a[j+8] + ... over its first n - n%8 values, combined as
// ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)), with the n%8 trailing values then added in turn; a
// longer block is split at n2 = n/2 - (n/2)%8 and the two halves' sums are added. The mean is
// that float32 sum divided by k, correctly rounded (numpy divides in float64 and casts; a
// float64 quotient of float32 operands rounds to float32 exactly as a float32 division).
// Reproduced here in the same order, so the scrunched series is bit-identical.
constexpr int kPwLeaf = 128;

// Leaves (blocks of <= 128 values) of the recursion over n values, left to right.
static int pw_num_leaves(long long n)
{
    if (n <= kPwLeaf) return 1;
    long long n2 = n / 2;
    n2 -= n2 % 8;
    return pw_num_leaves(n2) + pw_num_leaves(n - n2);
}

// Fills leaves[] with (start, length) in recursion (left to right) order; explicit stack.
__device__ void pw_leaf_table(int n, int2* leaves)
{
    int st_s[40], st_n[40];
    int sp = 0, nl = 0;
    st_s[sp] = 0;
    st_n[sp++] = n;
    while (sp > 0) {
        --sp;
        const int s = st_s[sp], m = st_n[sp];
        if (m <= kPwLeaf) {
            leaves[nl++] = make_int2(s, m);
            continue;
        }
        int m2 = m / 2;
        m2 -= m2 % 8;
        // right half pushed first, so the left half is popped (and emitted) first
        st_s[sp] = s + m2;
        st_n[sp++] = m - m2;
        st_s[sp] = s;
        st_n[sp++] = m2;
    }
}

// Adds the leaf sums up the recursion tree of n values in numpy's order (left + right at
// every split); leaf sums are consumed left to right.
__device__ float pw_combine(const float* leaf_sums, int n)
{
    int fn[40], fstate[40];
    float fleft[40];
    int sp = 0, li = 0;
    float ret = 0.0f;
    fn[0] = n;
    fstate[0] = 0;
    sp = 1;
    while (sp > 0) {
        const int t = sp - 1;
        const int m = fn[t];
        if (m <= kPwLeaf) {
            ret = leaf_sums[li++];
            --sp;
            continue;
        }
        int m2 = m / 2;
        m2 -= m2 % 8;
        if (fstate[t] == 0) {  // descend left
            fstate[t] = 1;
            fn[sp] = m2;
            fstate[sp++] = 0;
        } else if (fstate[t] == 1) {  // left done: descend right
            fleft[t] = ret;
            fstate[t] = 2;
            fn[sp] = m - m2;
            fstate[sp++] = 0;
        } else {  // both done
            ret = __fadd_rn(fleft[t], ret);
            --sp;
        }
    }
    return ret;
}

// The recursion over k values of at most 32 leaves, and its additions as a program: nodes 0 ..
// L-1 are the leaves (left to right), node L + q = node a[q] + node b[q], in the order numpy
// adds them (children before parents); the root is node 2L - 2 (node 0 when L = 1).
constexpr int kScrunchBatchLeaves = 32;
struct ScrunchTab {
    int nleaves;
    unsigned short start[kScrunchBatchLeaves];
    unsigned char len[kScrunchBatchLeaves];
    unsigned char a[kScrunchBatchLeaves], b[kScrunchBatchLeaves];
};

static int scrunch_tab(ScrunchTab& T, int nleaves, int start, int n, int* leaf, int* add)
{
    if (n <= kPwLeaf) {
        T.start[*leaf] = (unsigned short)start;
        T.len[*leaf] = (unsigned char)n;
        return (*leaf)++;
    }
    int n2 = n / 2;
    n2 -= n2 % 8;
    const int l = scrunch_tab(T, nleaves, start, n2, leaf, add);
    const int r = scrunch_tab(T, nleaves, start + n2, n - n2, leaf, add);
    T.a[*add] = (unsigned char)l;
    T.b[*add] = (unsigned char)r;
    return nleaves + (*add)++;
}

// Scrunch for factors whose recursion has at most 32 leaves (k up to a few thousand): a warp
// takes `pts` scrunched points at a time; its four 8-lane groups compute their leaves (one leaf
// per group per step, one strided accumulator per lane), then one lane per point adds up the
// leaves along the program above. What bounds it is the latency of the loads: a lane issues all
// of a leaf's (at most 16) before it adds them in order, and points per warp are chosen for
// warps enough to fill the GPU. (32 points a warp with one load in flight took 117 us for one
// series of 2^22 samples.)
// Dynamic shared memory: per warp pts points x (2L - 1) node values.
__global__ void __launch_bounds__(256)
    k_scrunch_batched(const float* __restrict__ x, TrialArrays A, int k, ScrunchTab T, int pts,
                      float* __restrict__ lores)
{
    after_previous_kernel();
    extern __shared__ float sm_scb[];
    __shared__ ScrunchTab S;
    const int nleaves = T.nleaves;
    const int nn = 2 * nleaves - 1, vs = nn | 1;  // odd per-point stride: no bank conflicts
    float* V = sm_scb + (threadIdx.x >> 5) * pts * vs;
    if (threadIdx.x < kScrunchBatchLeaves) {
        S.start[threadIdx.x] = T.start[threadIdx.x];
        S.len[threadIdx.x] = T.len[threadIdx.x];
        S.a[threadIdx.x] = T.a[threadIdx.x];
        S.b[threadIdx.x] = T.b[threadIdx.x];
    }
    __syncthreads();
    const int trial = blockIdx.y;
    const size_t nl = A.lo_length(trial);
    const float* xr = x + A.offset(trial);
    float* o = lores + A.lo_offset(trial);
    const int lane = threadIdx.x & 31;
    const int grp = lane >> 3, c = lane & 7;
    const size_t w0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
    const size_t nwarp = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t p0 = w0 * pts; p0 < nl; p0 += nwarp * pts) {
        const int np = (int)min((size_t)pts, nl - p0);
        const int tasks = np * nleaves;
        for (int u0 = 0; u0 < tasks; u0 += 4) {
            const int u = u0 + grp;
            const bool ok = u < tasks;
            const int pt = ok ? u / nleaves : 0, l = ok ? u - pt * nleaves : 0;
            const int len = ok ? S.len[l] : 0, full = len & ~7;
            const float* a = xr + (p0 + pt) * (size_t)k + S.start[l];
            float r[kPwLeaf / 8];
#pragma unroll
            for (int q = 0; q < kPwLeaf / 8; ++q) r[q] = 8 * q < full ? __ldg(a + 8 * q + c) : 0.0f;
            const float tail = full + c < len ? __ldg(a + full + c) : 0.0f;
            float v = r[0];
#pragma unroll
            for (int q = 1; q < kPwLeaf / 8; ++q)
                if (8 * q < full) v = __fadd_rn(v, r[q]);
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            if (full == 0) v = -0.0f;
            if (__any_sync(0xffffffffu, full < len)) {
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    const float y = __shfl_sync(0xffffffffu, tail, q, 8);
                    if (full + q < len) v = __fadd_rn(v, y);
                }
            }
            if (ok && c == 0) V[pt * vs + l] = v;
        }
        __syncwarp();
        if (lane < np) {
            float* Vp = V + lane * vs;
            for (int q = 0; q + 1 < nleaves; ++q)
                Vp[nleaves + q] = __fadd_rn(Vp[S.a[q]], Vp[S.b[q]]);
            o[p0 + lane] = __fdiv_rn(Vp[nn - 1], (float)k);
        }
        __syncwarp();
    }
}

// lores[j] = float32 mean of x[j*k .. (j+1)*k), numpy's pairwise order (see above).
// One warp per scrunched value; the warp's four 8-lane groups take one leaf each, a lane
// one of the eight strided accumulators; lane 0 adds the leaf sums up the tree.
// Dynamic shared memory: the leaf table (int2 per leaf) and one leaf-sum row per warp.
__global__ void k_scrunch(const float* __restrict__ x, TrialArrays A, int k, int nleaves,
                          float* __restrict__ lores)
{
    extern __shared__ __align__(16) unsigned char sm_scrunch[];
    int2* leaves = reinterpret_cast<int2*>(sm_scrunch);
    float* sums = reinterpret_cast<float*>(leaves + nleaves) + (threadIdx.x >> 5) * nleaves;
    if (threadIdx.x == 0) pw_leaf_table(k, leaves);
    __syncthreads();
    const int trial = blockIdx.y;
    const size_t nl = A.lo_length(trial);
    const float* xr = x + A.offset(trial);
    float* o = lores + A.lo_offset(trial);
    const int lane = threadIdx.x & 31;
    const int grp = lane >> 3, c = lane & 7;
    const size_t w0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
    const size_t nwarp = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t j = w0; j < nl; j += nwarp) {
        const float* a = xr + j * (size_t)k;
        for (int l0 = 0; l0 < nleaves; l0 += 4) {
            const int l = l0 + grp;
            float v = 0.0f;
            int2 lf = make_int2(0, 0);
            if (l < nleaves) {
                lf = leaves[l];
                if (lf.y >= 8) {
                    const int full = lf.y - lf.y % 8;
                    v = __ldg(a + lf.x + c);
                    for (int i = 8; i < full; i += 8) v = __fadd_rn(v, __ldg(a + lf.x + i + c));
                }
            }
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            if (l < nleaves && c == 0) {
                int i = lf.y - lf.y % 8;
                if (lf.y < 8) {
                    v = -0.0f;
                    i = 0;
                }
                for (; i < lf.y; ++i) v = __fadd_rn(v, __ldg(a + lf.x + i));
                sums[l] = v;
            }
        }
        __syncwarp();
        if (lane == 0) o[j] = __fdiv_rn(pw_combine(sums, k), (float)k);
        __syncwarp();
    }
}

// Launch shape of k_scrunch for factor k: 256 threads while the leaf table and eight
// leaf-sum rows fit 48 KB, fewer warps above that (up to the opt-in shared-memory size).
static int launch_scrunch(const float* x, const TrialArrays& A, int k, int ntrials,
                          size_t max_lo, float* lores, cudaStream_t st)
{
    const int nleaves = pw_num_leaves(k);
    if (nleaves <= kScrunchBatchLeaves) {
        ScrunchTab T;
        memset(&T, 0, sizeof(T));
        int leaf = 0, add = 0;
        T.nleaves = nleaves;
        scrunch_tab(T, nleaves, 0, k, &leaf, &add);
        // 8 warps of `pts` points: as many points a warp as leave 32 warps per SM
        int pts = 32;
        while (pts > 1 && (size_t)ntrials * max_lo < (size_t)pts * 148 * 32) pts >>= 1;
        const size_t smem = 8 * (size_t)pts * ((2 * nleaves - 1) | 1) * sizeof(float);
        dim3 g((unsigned)std::max<size_t>(1, std::min<size_t>((max_lo + 8 * pts - 1) / (8 * pts), 1 << 16)),
               (unsigned)ntrials);
        if (smem > 48 * 1024)
            RT_TRY_CUDA(cudaFuncSetAttribute(k_scrunch_batched,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_scrunch_batched<<<g, 256, smem, st>>>(x, A, k, T, pts, lores);
        return check_cuda(cudaGetLastError(), "scrunch");
    }
    const size_t per_warp = (size_t)nleaves * sizeof(float);
    const size_t table = (size_t)nleaves * sizeof(int2);
    int warps = 8;
    while (warps > 1 && table + warps * per_warp > 48 * 1024) warps >>= 1;
    const size_t smem = table + warps * per_warp;
    if (smem > 200 * 1024) return set_error(RT_EINVAL, "scrunch factor too large");
    if (smem > 48 * 1024)
        RT_TRY_CUDA(cudaFuncSetAttribute(k_scrunch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem));
    const unsigned threads = 32u * warps;
    // every CTA builds the leaf table first, so CTAs are few and long-lived: about 8192 in
    // all (at least 16 per series), each warp taking many points
    const size_t per_trial = std::max<size_t>(16, 8192 / (size_t)std::max(ntrials, 1));
    dim3 g((unsigned)std::max<size_t>(1, std::min<size_t>((max_lo + 63) / 64, per_trial)),
           (unsigned)ntrials);
    k_scrunch<<<g, threads, smem, st>>>(x, A, k, nleaves, lores);
    return check_cuda(cudaGetLastError(), "scrunch");
}

constexpr int kStatThreads = 256;

// Unsigned 32-bit division by an invariant divisor d >= 1 with one multiply-high
// (Granlund & Montgomery, "Division by invariant integers using multiplication", PLDI 1994,
// figure 4.1): l = ceil(log2 d), m = floor(2^32 (2^l - d) / d) + 1,
// q = (t + ((n - t) >> min(l, 1))) >> max(l - 1, 0) with t = mulhi(m, n); exact for every
// 32-bit n.
struct DivMagic {
    unsigned m;
    int sh1, sh2;
};

inline DivMagic div_magic(unsigned d)
{
    int l = 0;
    while ((1ull << l) < d) ++l;
    DivMagic g;
    g.m = (unsigned)((((1ull << 32) * ((1ull << l) - d)) / d) + 1);
    g.sh1 = l < 1 ? l : 1;
    g.sh2 = l - 1 > 0 ? l - 1 : 0;
    return g;
}

__device__ __forceinline__ unsigned div_by_magic(unsigned n, const DivMagic& g)
{
    const unsigned t = __umulhi(g.m, n);
    return (t + ((n - t) >> g.sh1)) >> g.sh2;
}

// np.interp of the scrunched running median (running_medians.py:82-85) over kInterpSpan
// consecutive samples of a series: with v = 2 i - (k - 1) = 2 k j + 2 dx, sample i lies dx past
// point j, and the value is fp[j] + slope_j * dx in float64 as numpy evaluates it (fp[j] at
// dx = 0, the end values outside). The CTA puts the points and slopes under its span in shared
// memory first (one division each); positions are then relative to the span, in 32 bits.
constexpr int kInterpSpan = 4096;
constexpr int kInterpCoefs = kInterpSpan / 2 + 2;  // k >= 2

struct InterpSpan {
    long long vb;       // v of the span's first sample
    unsigned rel0;      // vb relative to its first point's v (vb >= 0)
    double first, last;
    long long vlast;    // v >= vlast is at or right of the last point

    __device__ __forceinline__ void load(const float* fp, size_t nl, int k, size_t i0, int n,
                                         double2* coef)
    {
        vb = 2LL * (long long)i0 - (k - 1);
        const long long j0 = vb > 0 ? vb / (2LL * k) : 0;
        rel0 = (unsigned)(vb - 2LL * k * j0);
        const int nj = n / k + 2;
        for (int j = threadIdx.x; j < nj; j += blockDim.x) {
            const size_t jj = (size_t)(j0 + j);
            double2 c = make_double2(0.0, 0.0);
            if (jj < nl) {
                c.x = (double)fp[jj];
                if (jj + 1 < nl) c.y = __ddiv_rn(__dsub_rn((double)fp[jj + 1], c.x), (double)k);
            }
            coef[j] = c;
        }
        vlast = 2LL * k * (long long)(nl - 1) - vb;  // relative to vb from here on
        first = (double)fp[0];
        last = (double)fp[nl - 1];
    }
    // sample i of the span
    __device__ __forceinline__ double value(int i, int k, const DivMagic& g2k,
                                            const double2* coef) const
    {
        const int v = 2 * i;
        if (v < -vb) return first;
        if (v >= vlast) return last;
        const unsigned rel = rel0 + (unsigned)v;  // below 2 kInterpSpan + 2 k
        const unsigned j = div_by_magic(rel, g2k);
        const unsigned twodx = rel - j * 2u * (unsigned)k;
        const double2 c = coef[j];
        // (an integer below 2^32 as a double by its bits: no conversion)
        const double dx2 = __dsub_rn(__hiloint2double(0x43300000, (int)twodx), 4503599627370496.0);
        return twodx == 0 ? c.x : __dadd_rn(__dmul_rn(c.y, 0.5 * dx2), c.x);
    }
};

// Sum of a CTA's two per-thread values, in a fixed order (thread 0 has it).
__device__ __forceinline__ double2 block_sum2(double a, double b)
{
    __shared__ double2 w[kStatThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = make_double2(a, b);
    __syncthreads();
    double2 r = w[0];
    if (threadIdx.x == 0)
#pragma unroll
        for (int i = 1; i < kStatThreads / 32; ++i) {
            r.x += w[i].x;
            r.y += w[i].y;
        }
    return r;
}

// CTAs of a series in k_dered, k_sums and k_interp_rmed.
RT_HD size_t interp_blocks(size_t n) { return (n + kInterpSpan - 1) / kInterpSpan; }

// y = float32(x - running median); per-CTA shifted sums for the statistics.
// k > 1: the interpolated scrunched running median (InterpSpan); k == 1: rmed is the
// full-resolution float32 running median (float32 subtraction).
// Bound by the float64 work between a 4-byte read and a 4-byte write: a CTA takes 4,096
// consecutive samples, 16 loads a thread in flight. (64 CTAs a series striding over it, with a
// 64-bit division per sample and the slopes in global memory, took 267 us for 16 series of
// ~2^22 samples, and left half the GPU idle for one series.)
__global__ void __launch_bounds__(kStatThreads)
    k_dered(const float* __restrict__ x, TrialArrays A, int k, DivMagic g2k,
            const float* __restrict__ rmed, float* __restrict__ y, double* __restrict__ part)
{
    after_previous_kernel();
    constexpr int Q = kInterpSpan / kStatThreads;
    __shared__ double2 coef[kInterpCoefs];
    const int trial = blockIdx.y;
    const size_t N = A.length(trial), i0 = blockIdx.x * (size_t)kInterpSpan;
    if (i0 >= N) return;
    const int n = (int)min((size_t)kInterpSpan, N - i0);
    const float* xr = x + A.offset(trial);
    float* yr = y + A.offset(trial) + i0;
    float xv[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * kStatThreads;
        xv[q] = i < n ? xr[i0 + i] : 0.0f;
    }
    const float* fp = rmed + (k > 1 ? A.lo_offset(trial) : A.offset(trial));
    // the sums are shifted by y[0] (x = 0 <= xp[0]: its running median is fp[0])
    const float shift = k > 1 ? __double2float_rn((double)xr[0] - (double)fp[0])
                              : __fsub_rn(xr[0], fp[0]);
    const double shift_d = (double)shift;
    InterpSpan S;
    if (k > 1) S.load(fp, A.lo_length(trial), k, i0, n, coef);
    __syncthreads();
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * kStatThreads;
        if (i >= n) continue;
        const float yv = k > 1 ? __double2float_rn(__dsub_rn((double)xv[q], S.value(i, k, g2k, coef)))
                               : __fsub_rn(xv[q], fp[i0 + i]);
        yr[i] = yv;
        const double d = (double)yv - shift_d;
        s1 += d;
        s2 += d * d;
    }
    const double2 s = block_sum2(s1, s2);
    if (threadIdx.x == 0) {
        double* p = part + ((size_t)trial * gridDim.x + blockIdx.x) * 3;
        p[0] = s.x;
        p[1] = s.y;
        p[2] = shift_d;
    }
}

// Same statistics without deredden (normalise only).
__global__ void __launch_bounds__(kStatThreads)
    k_sums(const float* __restrict__ x, TrialArrays A, double* __restrict__ part)
{
    constexpr int Q = kInterpSpan / kStatThreads;
    const int trial = blockIdx.y;
    const size_t N = A.length(trial), i0 = blockIdx.x * (size_t)kInterpSpan;
    if (i0 >= N) return;
    const int n = (int)min((size_t)kInterpSpan, N - i0);
    const float* xr = x + A.offset(trial);
    const double shift = (double)xr[0];
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = threadIdx.x + q * kStatThreads;
        const double d = i < n ? (double)xr[i0 + i] - shift : 0.0;
        s1 += d;
        s2 += d * d;
    }
    const double2 s = block_sum2(s1, s2);
    if (threadIdx.x == 0) {
        double* p = part + ((size_t)trial * gridDim.x + blockIdx.x) * 3;
        p[0] = s.x;
        p[1] = s.y;
        p[2] = shift;
    }
}

// mean and standard deviation per trial (population variance, ddof = 0), a warp per trial:
// `blocks` partial sums of it at most, in a fixed order.
__global__ void k_stats(const double* __restrict__ part, TrialArrays A, int blocks, int ntrials,
                        double* __restrict__ mean, double* __restrict__ norm)
{
    after_previous_kernel();
    const int lane = threadIdx.x & 31;
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= ntrials) return;
    const double* p = part + (size_t)t * blocks * 3;
    const int nb = (int)interp_blocks(A.length(t));
    double s1 = 0.0, s2 = 0.0;
    for (int b = lane; b < nb; b += 32) {
        s1 += p[3 * b];
        s2 += p[3 * b + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane != 0) return;
    const double N = (double)A.length(t);
    const double d = s1 / N;
    const double var = s2 / N - d * d;
    mean[t] = p[2] + d;
    norm[t] = sqrt(var);
}

// fast_running_median output (running_medians.py:82-85): float64 interpolation of the
// scrunched running median back to every sample, two samples a thread at a time, stored as one
// 16-byte unit. Bound by the 8 bytes a sample that it writes.
__global__ void __launch_bounds__(kStatThreads)
    k_interp_rmed(TrialArrays A, int k, DivMagic g2k, const float* __restrict__ rmed,
                  double* __restrict__ out)
{
    __shared__ double2 coef[kInterpCoefs];
    const int trial = blockIdx.y;
    const size_t N = A.length(trial);
    const float* fp = rmed + A.lo_offset(trial);
    const size_t i0 = blockIdx.x * (size_t)kInterpSpan;
    if (i0 >= N) return;
    double* o = out + A.offset(trial) + i0;
    const int n = (int)min((size_t)kInterpSpan, N - i0);
    if (k == 1) {  // every sample is a point of the running median
        for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = (double)fp[i0 + i];
        return;
    }
    InterpSpan S;
    S.load(fp, A.lo_length(trial), k, i0, n, coef);
    __syncthreads();
    if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
        for (int i = 2 * threadIdx.x; i < n; i += 2 * blockDim.x) {
            const double a = S.value(i, k, g2k, coef);
            if (i + 1 < n)
                *reinterpret_cast<double2*>(o + i) = make_double2(a, S.value(i + 1, k, g2k, coef));
            else
                o[i] = a;
        }
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = S.value(i, k, g2k, coef);
    }
}

// z = float32((x - mean) / norm) in float64 (time_series.py:91-93).
__global__ void k_normalise(const float* __restrict__ x, TrialArrays A, const double* mean,
                            const double* norm, float* __restrict__ z)
{
    const int trial = blockIdx.y;
    const size_t N = A.length(trial);
    const float* xr = x + A.offset(trial);
    float* zr = z + A.offset(trial);
    const double m = mean[trial], s = norm[trial];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
         i += (size_t)gridDim.x * blockDim.x)
        zr[i] = __double2float_rn(__ddiv_rn(__dsub_rn((double)xr[i], m), s));
}

// ------------------------------------------------------------------------------------
// Plan
// ------------------------------------------------------------------------------------
struct SearchPlan {
    // configuration
    rt_search_config cfg;
    rt_search_tuning tuning = {1.0, 0, 0, 0.0};
    std::vector<rt_tile_rule> rules;    // per (rows, bins) tile choices, first match wins
    std::vector<int> widths;
    int nfast = 0;
    int snr_kinds = 0;                // kinds of S/N code the transforms need (snr_kind)
    std::vector<size_t> lengths, offsets;
    size_t total_len = 0, max_len = 0;
    // cycles (cpp/periodogram.hpp:135-158)
    std::vector<double> f, tau, pms;
    std::vector<int> use_seg, skip;
    // per trial
    std::vector<size_t> out_rows_off;   // [T+1]
    std::vector<size_t> ds_off;         // [T * C] offsets into the downsample arena
    size_t ds_total = 0;
    bool has_unit_factor = false;       // a cycle folds the series itself (f == 1)
    // deredden
    int scrunch = 1, rmed_width = 0;
    std::vector<size_t> lo_len, lo_off;
    size_t lo_total = 0, max_lo = 0;
    // work
    std::vector<StagePlan> plans;
    std::vector<XformRec> xforms;
    std::vector<int2> xform_tc;          // (trial, cycle) of each transform
    std::vector<WorkItem> items;
    int nseq = 0;
    size_t slot_floats = 0;
    int slots = 0;                       // scratch slots of the ring, a power of two
    int item_slots = 0;                  // ... that the work items are made for
    FfaLayout layout{};                  // shared-memory layout of the persistent kernel
    // device buffers
    bool dev_ready = false;
    int* d_widths = nullptr;
    XformRec* d_xforms = nullptr;
    WorkItem* d_items = nullptr;
    StagePlan* d_plans = nullptr;
    float* d_scratch = nullptr;
    int* d_counters = nullptr;          // ticket (8 bytes) + done + slot_release + error
    float* d_ds = nullptr;
    float* d_y = nullptr;               // dereddened series
    float* d_norm = nullptr;            // normalised copy (when a cycle has f == 1)
    float* d_lores = nullptr;
    float* d_rmed = nullptr;
    double* d_part = nullptr;
    double* d_mean = nullptr;
    double* d_normv = nullptr;
    size_t* d_len = nullptr;
    size_t* d_off = nullptr;
    size_t* d_lo_len = nullptr;
    size_t* d_lo_off = nullptr;
    double* d_f = nullptr;
    int* d_useseg = nullptr;
    size_t* d_dsoff = nullptr;
    // optional per-stage CUDA-event timing: deredden+normalise, downsample, FFA + S/N
    bool timing = false;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    unsigned long long* d_phase = nullptr;  // in-kernel phase profile (optional)
    int launches_last_run = 0;
    // replay of the whole run as one CUDA graph (optional); the graph is keyed on the
    // run's device pointers and captured again when they change
    bool use_graph = false;
    // bounded waits and fault injection (rt_search_set_wait_limit, rt_search_inject_fault)
    long long spin_limit = kSpinLimit;
    int dep_bias = 0;
    int alloc_fail_at = 0;   // 1-based device allocation that fails; 0: none
    int alloc_calls = 0;
    int ring_fails_above = 0;  // slots of the largest ring that there is room for; 0: no limit
    cudaGraphExec_t gexec = nullptr;
    cudaStream_t cap_stream = nullptr;
    const void* gkey[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    int graph_captures = 0;
};

static int plan_cycles(SearchPlan& P)
{
    const rt_search_config& c = P.cfg;
    // periodogram.hpp:25-40, same messages and order
    if (!(c.tsamp > 0)) return set_error(RT_EINVAL, "tsamp must be > 0");
    if (!(c.period_min > 0)) return set_error(RT_EINVAL, "period_min must be > 0");
    if (!(c.period_max > c.period_min)) return set_error(RT_EINVAL, "period_max must be > period_min");
    if (!(c.bins_min > 1)) return set_error(RT_EINVAL, "bins_min must be > 1");
    if (!(c.bins_max >= c.bins_min)) return set_error(RT_EINVAL, "bins_max must be >= bins_min");
    if (!(c.period_min >= c.tsamp * c.bins_min))
        return set_error(RT_EINVAL, "Must have: period_min >= tsamp * bins_min ");
    if (c.bins_max > 4096) return set_error(RT_EINVAL, "bins_max above 4096 is not supported");
    const double ds_ini = c.period_min / (c.tsamp * c.bins_min);
    const double ds_geo = (c.bins_max + 1.0) / c.bins_min;
    const size_t nds = (size_t)ceil(log(c.period_max / c.period_min) / log(ds_geo));
    if (nds > (size_t)kDsMaxCycles)
        return set_error(RT_EINVAL, "too many downsampling cycles (%zu)", nds);
    for (size_t i = 0; i < nds; ++i) {
        const double f = ds_ini * pow(ds_geo, (double)i);
        P.f.push_back(f);
        P.tau.push_back(f * c.tsamp);
        P.pms.push_back(c.period_max / (f * c.tsamp));
        P.skip.push_back(f == 1 ? 1 : 0);
        P.use_seg.push_back((f != 1 && ds_use_segments(f)) ? 1 : 0);
        if (f == 1) P.has_unit_factor = true;
    }
    return RT_OK;
}

// Slots of the ring of stage outputs, a power of two: one per multi-stage transform, up to kSlots.
static int ring_slots(const SearchPlan& P)
{
    int n = 1;
    while (n < kSlots && n < P.nseq) n *= 2;
    return n;
}

// Emits the work items of all transforms, in order. For a transform that needs several stages,
// stage s + 1 is emitted at least kLagItems items after stage s, so that by the time a CTA takes
// it the previous stage has usually completed; the transform that reuses a scratch slot starts
// only after every stage of the previous occupant is emitted.
static void plan_items(SearchPlan& P)
{
    P.items.clear();
    P.item_slots = P.slots;
    const size_t lag_items = P.tuning.lag_items > 0 ? (size_t)P.tuning.lag_items : kLagItems;
    std::set<std::tuple<size_t, int, int>> deferred;  // (due item count, xform, stage)
    std::vector<std::tuple<size_t, int, int>> seq_pending(P.nseq);  // its deferred entry, if any
    std::vector<char> seq_has_pending(P.nseq, 0);

    auto emit_stage = [&](int xi, int stage) {
        const StagePlan& sp = P.plans[P.xforms[xi].plan];
        for (int j = 0; j < sp.jobs[stage]; ++j) P.items.push_back({xi, (stage << 24) | j});
        const int seq = P.xforms[xi].seq;
        if (seq >= 0) {
            if (stage + 1 < sp.nstages) {
                auto e = std::make_tuple(P.items.size() + lag_items, xi, stage + 1);
                deferred.insert(e);
                seq_pending[seq] = e;
                seq_has_pending[seq] = 1;
            } else {
                seq_has_pending[seq] = 0;
            }
        }
    };
    auto flush = [&]() {
        while (!deferred.empty() && std::get<0>(*deferred.begin()) <= P.items.size()) {
            const auto e = *deferred.begin();
            deferred.erase(deferred.begin());
            emit_stage(std::get<1>(e), std::get<2>(e));
        }
    };
    auto finish_seq = [&](int seq) {  // emit all remaining stages of `seq` now
        while (seq_has_pending[seq]) {
            const auto e = seq_pending[seq];
            deferred.erase(e);
            emit_stage(std::get<1>(e), std::get<2>(e));
        }
    };
    for (int xi = 0; xi < (int)P.xforms.size(); ++xi) {
        if (P.xforms[xi].seq >= P.slots) finish_seq(P.xforms[xi].seq - P.slots);
        emit_stage(xi, 0);
        flush();
    }
    while (!deferred.empty()) {
        const auto e = *deferred.begin();
        deferred.erase(deferred.begin());
        emit_stage(std::get<1>(e), std::get<2>(e));
    }
}

// The transforms of a plan, in the order (trial, cycle, bins), and their work items.
static int plan_build(SearchPlan& P)
{
    RT_TRY(plan_cycles(P));
    const rt_search_config& c = P.cfg;
    const int T = (int)P.lengths.size();
    const int C = (int)P.f.size();
    P.out_rows_off.assign(T + 1, 0);
    P.ds_off.assign((size_t)T * C, 0);
    std::map<std::pair<int, long long>, int> plan_index;

    // (the first cycle has the smallest factor, and so the most rows)
    const size_t most_rows = C > 0 ? downsampled_size(P.max_len, P.f[0]) / c.bins_min : 0;
    // Room behind the second level buffer for the reads of the S/N past its last row, by every
    // number of threads that a transform of the plan may be given. (A one-stage transform can fill
    // the buffer to its last row; the last stage of others has at most kThreads / tpr rows.)
    int pad = kPadFloats;
    for (int b = (int)c.bins_min; b <= (int)c.bins_max; ++b) {
        bool tuned = P.tuning.snr_threads == 16;
        for (const rt_tile_rule& R : P.rules)
            tuned |= R.snr_threads == 16 && (unsigned)b >= R.bins_min && (unsigned)b <= R.bins_max;
        pad = std::max({pad, snr_overread(b, snr_tpr(b)), tuned ? snr_overread(b, 16) : 0});
    }
    P.layout = ffa_layout(kEngineDynBytes, (int)c.bins_min, most_rows, pad);
    size_t ds_total = 0;
    for (int t = 0; t < T; ++t) {
        const size_t N = P.lengths[t];
        size_t rows_total = 0;
        for (int ci = 0; ci < C; ++ci) {
            const double f = P.f[ci];
            const size_t n = downsampled_size(N, f);
            if (f != 1) {
                // downsample.hpp:11-16 (the reference downsamples every cycle)
                if (!((f > 1.0) && (f <= (double)N)))
                    return set_error(RT_EINVAL, "Downsampling factor must verify: 1 < f <= size");
                P.ds_off[(size_t)t * C + ci] = ds_total;
                ds_total += n;
            }
            const size_t bstop = std::min({(size_t)c.bins_max, n, (size_t)P.pms[ci]});
            for (size_t b = c.bins_min; b <= bstop; ++b) {
                const size_t rows = n / b;
                const size_t re = rows_to_evaluate(rows, b, P.pms[ci]);
                if (re == 0) continue;
                if (rows >= (1u << 24))
                    return set_error(RT_EINVAL, "transform of %zu rows is too large", rows);
                // rows per job: the shared-memory capacity, scaled by the tuning (its own
                // fraction for transforms of more than 8 jobs' worth of rows)
                const int cap_full = ffa_cap_rows(P.layout, (int)b);
                double frac = P.tuning.rows_fraction > 0 ? std::min(1.0, P.tuning.rows_fraction) : 1.0;
                if (rows > 8 * (size_t)cap_full && P.tuning.rows_fraction_deep > 0)
                    frac = std::min(1.0, P.tuning.rows_fraction_deep);
                int tune_tpr = P.tuning.snr_threads, max_depth = kMaxJobDepth;
                for (const rt_tile_rule& R : P.rules) {
                    if (rows < R.rows_min || rows > R.rows_max || b < R.bins_min || b > R.bins_max)
                        continue;
                    if (R.rows_fraction > 0) frac = std::min(1.0, R.rows_fraction);
                    if (R.snr_threads) tune_tpr = R.snr_threads;
                    if (R.max_levels) max_depth = R.max_levels - 1;
                    break;
                }
                const int capr = std::max(4, (int)((double)cap_full * frac));
                // S/N threads per profile: the default for these bins, or 16 where that is tuned
                // and 16 segments hold a profile
                const int tpr = (tune_tpr == 16 && b <= 16 * kSnrPhases) ? 16 : snr_tpr((int)b);
                const auto key = std::make_pair((int)rows, (long long)re * 8192 + (long long)b);
                int pi;
                auto itp = plan_index.find(key);
                if (itp == plan_index.end()) {
                    StagePlan sp;
                    // a rule's level count that needs more stages than a plan holds falls back
                    // to the default depth
                    if (capr < 4 ||
                        (!plan_stages((int)rows, (int)b, (int)re, capr, kThreads / tpr, &sp, max_depth) &&
                         !plan_stages((int)rows, (int)b, (int)re, capr, kThreads / tpr, &sp)))
                        return set_error(RT_EINVAL, "no device plan for a %zu x %zu transform", rows, b);
                    pi = (int)P.plans.size();
                    P.plans.push_back(sp);
                    plan_index[key] = pi;
                } else {
                    pi = itp->second;
                }
                XformRec X;
                memset(&X, 0, sizeof(X));
                const bool multi = P.plans[pi].nstages > 1;
                X.src_off = (f != 1) ? P.ds_off[(size_t)t * C + ci] : P.offsets[t];
                X.src_norm = (f != 1) ? 0 : 1;
                X.out_row = P.out_rows_off[t] + rows_total;
                X.tau = P.tau[ci];
                X.b = (int)b;
                X.m = (int)rows;
                X.rows_eval = (int)re;
                X.stdnoise = (float)sqrt((double)rows * downsampled_variance(N, f));
                X.plan = pi;
                X.seq = -1;
                X.tune = capr | (tpr << 16);
                if (multi) {
                    X.seq = P.nseq++;
                    // stage outputs use the level stride (16-byte aligned rows)
                    P.slot_floats = std::max(P.slot_floats, rows * (size_t)ffa_stride((int)b));
                }
                P.xforms.push_back(X);
                P.snr_kinds |= snr_kind((int)b, tpr);
                P.xform_tc.push_back(make_int2(t, ci));
                rows_total += re;
            }
        }
        P.out_rows_off[t + 1] = P.out_rows_off[t] + rows_total;
    }
    P.ds_total = ds_total;
    P.slots = ring_slots(P);
    plan_items(P);

    // deredden geometry (time_series.py:119, running_medians.py:72-80)
    P.lo_len.assign(T, 0);
    P.lo_off.assign(T, 0);
    if (c.deredden) {
        const double ws = nearbyint(c.rmed_width / c.tsamp);  // Python round(): half to even
        if (!(ws >= 1)) return set_error(RT_EINVAL, "rmed_width is shorter than one sample");
        P.rmed_width = (int)ws;
        if (!(c.rmed_minpts % 2)) return set_error(RT_EINVAL, "min_points must be an odd number");
        const double sf = std::max(1.0, ws / (double)c.rmed_minpts);
        P.scrunch = (int)sf;
        const int w = P.scrunch == 1 ? P.rmed_width : (int)c.rmed_minpts;
        if (!(w % 2)) return set_error(RT_EINVAL, "width must be an odd number");
        size_t lo_total = 0;
        for (int t = 0; t < T; ++t) {
            const size_t nl = P.scrunch == 1 ? P.lengths[t] : P.lengths[t] / P.scrunch;
            if (!((size_t)w < nl)) return set_error(RT_EINVAL, "width must be < size");
            P.lo_len[t] = nl;
            P.lo_off[t] = lo_total;
            lo_total += nl;
            P.max_lo = std::max(P.max_lo, nl);
        }
        P.lo_total = lo_total;
    }
    return RT_OK;
}

template <class T>
static void dfree(T*& p)
{
    if (p) cudaFree(p);
    p = nullptr;
}

static void plan_free_device(SearchPlan& P)
{
    dfree(P.d_widths); dfree(P.d_xforms); dfree(P.d_items); dfree(P.d_plans);
    dfree(P.d_scratch); dfree(P.d_counters); dfree(P.d_ds); dfree(P.d_y);
    dfree(P.d_norm); dfree(P.d_lores); dfree(P.d_rmed); dfree(P.d_part);
    dfree(P.d_mean); dfree(P.d_normv); dfree(P.d_len); dfree(P.d_off); dfree(P.d_lo_len);
    dfree(P.d_lo_off); dfree(P.d_f); dfree(P.d_useseg); dfree(P.d_dsoff);
    P.dev_ready = false;
}

// Device allocation of one of the plan's buffers. With an injected allocation fault
// (rt_search_inject_fault, RT_FAULT_ALLOC) the chosen call fails as cudaMalloc would.
template <class T>
static int dalloc(SearchPlan& P, T** p, size_t n)
{
    if (n == 0) n = 1;
    ++P.alloc_calls;
    if (P.alloc_fail_at > 0 && P.alloc_calls == P.alloc_fail_at)
        return set_error(RT_ENOMEM, "device allocation %d of the plan failed (injected)",
                         P.alloc_calls);
    cudaError_t e = cudaMalloc((void**)p, n * sizeof(T));
    if (e == cudaErrorMemoryAllocation) {  // without the scratch pool's kept memory, then
        cudaGetLastError();
        release_scratch();
        e = cudaMalloc((void**)p, n * sizeof(T));
    }
    return check_cuda(e, "device allocation of the plan");
}

template <class T>
static int copy_up(T* p, const std::vector<T>& v)
{
    if (!v.empty()) RT_TRY_CUDA(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return RT_OK;
}

template <class T>
static int upload(SearchPlan& P, T** p, const std::vector<T>& v)
{
    RT_TRY(dalloc(P, p, v.size()));
    return copy_up(*p, v);
}

static int plan_alloc_device(SearchPlan& P);

// Counters of a run, in one array: the ticket, the stage counts, the slot releases, the error.
static size_t plan_counters(const SearchPlan& P)
{
    return 2 + (size_t)P.nseq * kMaxStages + P.slots + 1;
}

// Allocates and fills the plan's device buffers once. On failure every buffer allocated so
// far is released again, so a failed call leaks nothing and can be retried.
static int plan_prepare_device(SearchPlan& P)
{
    if (P.dev_ready) return RT_OK;
    P.alloc_calls = 0;
    const int s = plan_alloc_device(P);
    if (s != RT_OK) {
        plan_free_device(P);
        return s;
    }
    P.dev_ready = true;
    return RT_OK;
}

// The ring of stage outputs, with half the slots as often as there is no room for it. The halo of
// its rows adds 5% to the ring at 240 bins and 80% at 20 (a series of 2^26 samples: 247 GB). With
// half the slots a transform takes its slot over from one 128 back; kLagItems are those of 213
// transforms at most. The work items follow the slots.
static int plan_alloc_ring(SearchPlan& P)
{
    int s = RT_ENOMEM;
    for (P.slots = ring_slots(P);; P.slots /= 2) {
        const bool no_room = P.ring_fails_above > 0 && P.slots > P.ring_fails_above;
        if (!no_room) s = dalloc(P, &P.d_scratch, (size_t)P.slots * 2 * std::max<size_t>(P.slot_floats, 1));
        if (s != RT_ENOMEM || P.slots == 1 || P.alloc_calls == P.alloc_fail_at) break;
    }
    if (s == RT_OK && P.slots != P.item_slots) plan_items(P);
    return s;
}

static int plan_alloc_device(SearchPlan& P)
{
    const int T = (int)P.lengths.size();
    RT_TRY(upload(P, &P.d_widths, P.widths));
    RT_TRY(dalloc(P, &P.d_items, P.items.size()));
    RT_TRY(upload(P, &P.d_plans, P.plans));
    RT_TRY(dalloc(P, &P.d_xforms, P.xforms.size()));
    RT_TRY(dalloc(P, &P.d_counters, 2 + (size_t)P.nseq * kMaxStages + kSlots + 1));
    // + 16 floats: bulk copies read whole 16-byte units around a block of rows
    RT_TRY(dalloc(P, &P.d_ds, P.ds_total + 16));
    if (P.cfg.deredden) {
        RT_TRY(dalloc(P, &P.d_y, P.total_len));
        RT_TRY(dalloc(P, &P.d_rmed, P.scrunch > 1 ? P.lo_total : P.total_len));
        if (P.scrunch > 1) RT_TRY(dalloc(P, &P.d_lores, P.lo_total));
    }
    if (P.has_unit_factor) RT_TRY(dalloc(P, &P.d_norm, P.total_len));
    RT_TRY(dalloc(P, &P.d_part, (size_t)T * interp_blocks(P.max_len) * 3));
    RT_TRY(dalloc(P, &P.d_mean, T));
    RT_TRY(dalloc(P, &P.d_normv, T));
    RT_TRY(upload(P, &P.d_len, P.lengths));
    RT_TRY(upload(P, &P.d_off, P.offsets));
    RT_TRY(upload(P, &P.d_lo_len, P.lo_len));
    RT_TRY(upload(P, &P.d_lo_off, P.lo_off));
    RT_TRY(upload(P, &P.d_f, P.f));
    RT_TRY(upload(P, &P.d_useseg, P.use_seg));
    RT_TRY(upload(P, &P.d_dsoff, P.ds_off));
    RT_TRY(plan_alloc_ring(P));  // (last: the other buffers' sizes are fixed)
    RT_TRY(copy_up(P.d_items, P.items));
    RT_TRY(copy_up(P.d_xforms, P.xforms));
    // a copy from pageable memory returns when the data is staged; the run may be on a stream that
    // does not wait for the default stream, which the copies are on
    RT_TRY_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    return RT_OK;
}

// The instance of k_search_persistent for a plan whose transforms need the kinds of S/N code in
// `kinds`: the usual searches need one kind only.
static void (*search_kernel_for(int kinds))(EngineArgs)
{
    if (kinds == kSnr8) return k_search_persistent<kSnr8>;
    if (kinds == kSnr16) return k_search_persistent<kSnr16>;
    if (kinds == kSnr32) return k_search_persistent<kSnr32>;
    return k_search_persistent<kSnr4 | kSnr8 | kSnr16 | kSnr32 | kSnr32Loop>;
}

static int engine_grid(void (*kernel)(EngineArgs))
{
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kEngineThreads, kEngineDynBytes);
    return std::max(1, sms * std::max(per, 1));
}

// ------------------------------------------------------------------------------------
// One transform by the persistent kernel (ffa2 of a large block): its jobs are the work items,
// stage by stage, and its rows the result. Against a launch per stage, a job's node lists,
// staging and stores run beside the levels of the one before: 16,384 x 488 values 176 to 155 us a
// call, 8,000 x 1,000 198 to 162, 33,000 x 250 175 to 147. From kPersistentItems jobs: with fewer
// the waits between the stages cost more (8,000 x 488: 88 against 80 us). Nodes counted one by one,
// so that one may start before its whole stage is done, took as long and slowed the searches.
// ------------------------------------------------------------------------------------
struct TransformState {
    unsigned long long ticket;
    int error;
    int done[kMaxStages];
    int slot_release;  // (one transform, one slot)
    // (apart from the counters, which every CTA changes: on their cache line, 16,001 x 499 took
    // 169.8 instead of 167.4 us)
    alignas(256) XformRec xform;
    StagePlan plan;
};

// Work items of the transform, its record and cleared counters.
__global__ void k_transform_items(TransformState* S, WorkItem* items, XformRec X, StagePlan P)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
    if (t == 0) {
        S->ticket = 0;
        S->error = RT_OK;
        S->slot_release = 0;
        S->xform = X;
        S->plan = P;
    }
    if (t < kMaxStages) S->done[t] = 0;
    int first = 0;
    for (int s = 0; s < P.nstages; ++s) {
        for (int j = t; j < P.jobs[s]; j += n) items[first + j] = WorkItem{0, s << 24 | j};
        first += P.jobs[s];
    }
}

// A bounded wait that ran out leaves NaN, and the error where it is asked for.
__global__ void k_transform_check(const TransformState* S, float* out, size_t n, int* d_err)
{
    if (S->error == RT_OK) return;
    if (blockIdx.x == 0 && threadIdx.x == 0 && d_err) *d_err = S->error;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        out[i] = __int_as_float(0x7fffffff);
}

struct TransformPlan {
    FfaLayout layout;
    StagePlan plan;
    int cap, items;
    size_t slot_floats, state_bytes, item_bytes;
};

static bool transform_plan(int m, int b, int rows_out, TransformPlan& T)
{
    T.layout = ffa_layout(kEngineDynBytes, b, (size_t)m);
    T.cap = ffa_cap_rows(T.layout, b);
    if (T.cap < 4 || T.cap > 0xffff || !plan_stages(m, b, rows_out, T.cap, 0, &T.plan)) return false;
    if (T.plan.nstages < 2) return false;
    T.items = 0;
    for (int s = 0; s < T.plan.nstages; ++s) {
        if (T.plan.jobs[s] >= 1 << 24) return false;
        T.items += T.plan.jobs[s];
    }
    T.slot_floats = ((size_t)m * ffa_stride(b) + 3) & ~size_t(3);
    T.state_bytes = (sizeof(TransformState) + 255) & ~size_t(255);
    T.item_bytes = ((size_t)T.items * sizeof(WorkItem) + 255) & ~size_t(255);
    return true;
}

size_t ffa_persistent_bytes(int m, int b, int rows_out)
{
    TransformPlan T;
    if (!transform_plan(m, b, rows_out, T) || T.items < kPersistentItems) return 0;
    return T.state_bytes + T.item_bytes + 2 * T.slot_floats * sizeof(float);
}

int ffa_transform_persistent(const float* in, int m, int b, int rows_out, float* out, void* scratch,
                             int* d_err, cudaStream_t st, long long wait_polls, int dep_bias)
{
    TransformPlan T;
    if (!transform_plan(m, b, rows_out, T))
        return set_error(RT_EINTERNAL, "no plan for an FFA transform of %d x %d", m, b);
    unsigned char* base = static_cast<unsigned char*>(scratch);
    TransformState* S = reinterpret_cast<TransformState*>(base);
    WorkItem* items = reinterpret_cast<WorkItem*>(base + T.state_bytes);
    XformRec X;
    memset(&X, 0, sizeof(X));
    X.tau = 1.0;
    X.b = b;
    X.m = m;
    X.rows_eval = rows_out;
    X.stdnoise = 1.0f;
    // bulk copies of whole 16-byte units stay inside the block if it starts and ends with one
    X.src_norm = (reinterpret_cast<uintptr_t>(in) & 15) != 0 || ((size_t)m * b) % 4 != 0;
    X.tune = T.cap;
    k_transform_items<<<std::min(148, (T.items + 255) / 256 + 1), 256, 0, st>>>(S, items, X, T.plan);
    RT_TRY_CUDA(cudaGetLastError());
    EngineArgs A;
    memset(&A, 0, sizeof(A));
    A.ds = A.norm = in;
    A.rows_out = out;
    A.xforms = &S->xform;
    A.items = items;
    A.nitems = T.items;
    A.plans = &S->plan;
    A.scratch = reinterpret_cast<float*>(base + T.state_bytes + T.item_bytes);
    A.slot_floats = T.slot_floats;
    A.done = S->done;
    A.slot_release = &S->slot_release;
    A.error = &S->error;
    A.ticket = &S->ticket;
    A.spin_limit = wait_polls > 0 ? wait_polls : kSpinLimit;
    A.dep_bias = dep_bias;
    A.layout = T.layout;
    void (*kernel)(EngineArgs) = k_search_persistent<kRowsOnly>;
    RT_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kEngineDynBytes));
    kernel<<<std::min(engine_grid(kernel), T.items), kEngineThreads, kEngineDynBytes, st>>>(A);
    RT_TRY_CUDA(cudaGetLastError());
    k_transform_check<<<148, 256, 0, st>>>(S, out, (size_t)rows_out * b, d_err);
    RT_TRY_CUDA(cudaGetLastError());
    return RT_OK;
}

// Launches the whole search of the plan on `st`. data: packed input series (device).
static int plan_run(SearchPlan& P, const float* data, float* normalised_out, double* periods,
                    uint32_t* foldbins, float* snrs, cudaStream_t st)
{
    RT_TRY(plan_prepare_device(P));
    const int T = (int)P.lengths.size();
    const int C = (int)P.f.size();
    TrialArrays TA{P.d_len, P.d_off, P.d_lo_len, P.d_lo_off, 0, 0};
    const float* series = data;  // series before normalisation
    int launches = 0;
    const dim3 stat_grid((unsigned)interp_blocks(P.max_len), (unsigned)T);
    // (here, so that the kernels follow one another)
    RT_TRY_CUDA(cudaMemsetAsync(P.d_counters, 0, plan_counters(P) * sizeof(int), st));
    if (P.timing) RT_TRY_CUDA(cudaEventRecord(P.ev[0], st));
    if (P.cfg.deredden) {
        const int k = P.scrunch;
        if (k > 1) {
            RT_TRY(launch_scrunch(data, TA, k, T, P.max_lo, P.d_lores, st));
            RT_TRY(launch_running_median(P.d_lores, P.d_lo_len, P.d_lo_off, T, P.max_lo,
                                         (int)P.cfg.rmed_minpts, P.d_rmed, st, true));
            launches += 2;
        } else {
            RT_TRY(launch_running_median(data, P.d_len, P.d_off, T, P.max_len, P.rmed_width,
                                         P.d_rmed, st, true));
            launches += 1;
        }
        RT_TRY_CUDA(launch_dependent(k_dered, stat_grid, dim3(kStatThreads), 0, st, data, TA, k,
                                     div_magic(2u * (unsigned)k), P.d_rmed, P.d_y, P.d_part));
        launches += 1;
        series = P.d_y;
    } else if (!P.cfg.already_normalised) {
        k_sums<<<stat_grid, kStatThreads, 0, st>>>(data, TA, P.d_part);
        RT_TRY_CUDA(cudaGetLastError());
        launches += 1;
    }
    const bool affine = !P.cfg.already_normalised;
    if (affine) {
        RT_TRY_CUDA(launch_dependent(k_stats, dim3((T + 3) / 4), dim3(128), 0, st, P.d_part, TA,
                                     (int)stat_grid.x, T, P.d_mean, P.d_normv));
        launches += 1;
    }
    if (P.timing) RT_TRY_CUDA(cudaEventRecord(P.ev[1], st));
    // The normalised series is materialised by the downsampler when the caller wants it or
    // when a cycle folds it directly (f == 1); without normalisation it is `series` itself.
    float* zdst = normalised_out ? normalised_out : (P.has_unit_factor && affine ? P.d_norm : nullptr);
    const float* zsrc = affine ? (zdst ? zdst : series) : series;
    if (!affine && normalised_out && normalised_out != series)
        RT_TRY_CUDA(cudaMemcpyAsync(normalised_out, series, P.total_len * sizeof(float),
                                    cudaMemcpyDeviceToDevice, st));
    DsJob job;
    job.in = series;
    job.in_off = P.d_off;
    job.lengths = P.d_len;
    job.mean = affine ? P.d_mean : nullptr;
    job.norm = affine ? P.d_normv : nullptr;
    job.norm_out = affine ? zdst : nullptr;
    job.f = P.d_f;
    job.use_seg = P.d_useseg;
    job.out = P.d_ds;
    job.out_off = P.d_dsoff;
    job.ncycles = C;
    job.use_seg_host = P.use_seg.data();
    job.f_host = P.f.data();
    job.skip_host = P.skip.data();
    RT_TRY(launch_downsample(job, T, P.max_len, st));
    {
        bool seg = job.norm_out != nullptr;
        for (int c = 0; c < C; ++c) {
            seg |= P.use_seg[c] != 0;
            launches += (!P.use_seg[c] && !P.skip[c]) ? 1 : 0;
        }
        launches += seg ? 1 : 0;
    }
    if (P.timing) RT_TRY_CUDA(cudaEventRecord(P.ev[2], st));
    EngineArgs A;
    memset(&A, 0, sizeof(A));
    A.ds = P.d_ds;
    A.norm = zsrc;
    A.snrs = snrs;
    A.xforms = P.d_xforms;
    A.items = P.d_items;
    A.nitems = (long long)P.items.size();
    A.plans = P.d_plans;
    A.widths = P.d_widths;
    A.nw = (int)P.widths.size();
    A.nfast = P.nfast;
    A.scratch = P.d_scratch;
    A.slot_floats = P.slot_floats;
    A.done = P.d_counters + 2;
    A.slot_release = A.done + (size_t)P.nseq * kMaxStages;
    A.slot_mask = P.slots - 1;
    while ((P.slots >> A.slot_shift) > 1) ++A.slot_shift;
    A.error = A.slot_release + P.slots;
    A.ticket = reinterpret_cast<unsigned long long*>(P.d_counters);
    A.phase_cycles = P.d_phase;
    A.spin_limit = P.spin_limit;
    A.dep_bias = P.dep_bias;
    A.layout = P.layout;
    void (*kernel)(EngineArgs) = search_kernel_for(P.snr_kinds);
    RT_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kEngineDynBytes));
    if (A.nitems > 0) {
        const int nx = (int)P.xforms.size();
        RT_TRY_CUDA(launch_dependent(k_search_periods, dim3(std::min((nx + 7) / 8, 148 * 8)),
                                     dim3(256), 0, st, P.d_xforms, nx, periods, foldbins));
        launches += 1;
        RT_TRY_CUDA(launch_dependent(kernel, dim3(engine_grid(kernel)), dim3(kEngineThreads),
                                     kEngineDynBytes, st, A));
        launches += 1;
    }
    if (P.timing) RT_TRY_CUDA(cudaEventRecord(P.ev[3], st));
    P.launches_last_run = launches;
    return RT_OK;
}

static int plan_check_error(SearchPlan& P, cudaStream_t st)
{
    int err = 0;
    RT_TRY_CUDA(cudaMemcpyAsync(&err, P.d_counters + plan_counters(P) - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    RT_TRY_CUDA(cudaStreamSynchronize(st));
    if (err == RT_ETIMEOUT)
        return set_error(RT_ETIMEOUT, "a bounded wait in the search kernel ran out");
    if (err != RT_OK) return set_error(err, "the search kernel reported error %d", err);
    return RT_OK;
}

// ------------------------------------------------------------------------------------
// Sparse-row backward of a run: the gradient with respect to the searched (normalised)
// series of sum(gsnr * snrs), for gradients on few periodogram rows (a max-S/N loss has one
// per trial). Output row s of a transform is a sum of every input row i rolled by a total
// shift sigma_i(s) (the tail shifts met on the way from the root to leaf i); the row is
// recomputed from the downsampled series that the run left in its arena, its boxcar S/N is
// differentiated (the max routed to the first maximising phase), and the row gradient is
// scattered back through the same shifts, then through the downsampling.
// ------------------------------------------------------------------------------------
struct BwdJob {
    int m, b, s, pad;
    float stdnoise;
    int pad2;
    unsigned long long grow;  // row index into gsnr
};

struct BwdGroup {
    unsigned long long src;   // float offset of the folded series (arena or z)
    unsigned long long gds;   // float offset of this group's downsampled gradient
    unsigned long long gz;    // float offset of the trial's series in the packed gradient
    unsigned long long sig;   // int offset of this group's shift table
    int job0, njobs, src_is_z, pad;
    size_t n_ds, N;
    double f;
};

constexpr int kBwdThreads = 256;
constexpr int kBwdMaxBins = 4096;

// One CTA per group, its rows in turn: their sums keep the forward's order. Bound: the latency of
// a chain of phases; with the loads of a row's sum one behind the other and the scatter by flat
// index (a division each), four groups of one row of 200 x 250 took 62 us, now 30.
__global__ void __launch_bounds__(kBwdThreads)
    k_rows_backward(const BwdGroup* __restrict__ groups, const BwdJob* __restrict__ jobs,
                    const float* __restrict__ arena, const float* __restrict__ z,
                    const float* __restrict__ gsnr, const int* __restrict__ widths, int nw,
                    int wmax, float* __restrict__ gds_all, int* __restrict__ sig_all)
{
    extern __shared__ float sm[];
    float* F = sm;                       // kBwdMaxBins
    float* C = F + kBwdMaxBins;          // b + wmax
    __shared__ float s_g[kBwdMaxBins];
    __shared__ int s_best[64];
    const BwdGroup G = groups[blockIdx.x];
    const float* src = (G.src_is_z ? z : arena) + G.src;
    float* gds = gds_all + G.gds;
    int* sig = sig_all + G.sig;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int q = 0; q < G.njobs; ++q) {
        const BwdJob J = jobs[G.job0 + q];
        const int m = J.m, b = J.b;
        // total shift of every input row for output row s
        for (int i = tid; i < m; i += kBwdThreads) {
            int row0 = 0, n = m, r = J.s, sg = 0;
            while (n > 1) {
                const int nh = n >> 1;
                const MergeCoef mc = merge_coef(n);
                const int h = merge_row(mc.kh, r), t = merge_row(mc.kt, r);
                if (i < row0 + nh) {
                    n = nh;
                    r = h;
                } else {
                    sg += (r - t) % b;
                    sg -= (sg >= b) ? b : 0;
                    row0 += nh;
                    n -= nh;
                    r = t;
                }
            }
            sig[i] = sg;
        }
        __syncthreads();
        // the output row
        for (int c = tid; c < b; c += kBwdThreads) {
            float acc = 0.0f;
            int i = 0;
            for (; i + 16 <= m; i += 16) {  // (the rows in order; sixteen loads in flight)
                float v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    int idx = c + sig[i + u];
                    idx -= (idx >= b) ? b : 0;
                    v[u] = src[(size_t)(i + u) * b + idx];
                }
#pragma unroll
                for (int u = 0; u < 16; ++u) acc = __fadd_rn(acc, v[u]);
            }
            for (; i < m; ++i) {
                int idx = c + sig[i];
                idx -= (idx >= b) ? b : 0;
                acc = __fadd_rn(acc, src[(size_t)i * b + idx]);
            }
            F[c] = acc;
        }
        __syncthreads();
        // boxcar S/N backward of the row (one warp)
        if (tid < 32) {
            double carry = 0.0;
            for (int c0 = 0; c0 < b; c0 += 32) {
                const int c = c0 + lane;
                const double v = (c < b) ? (double)F[c] : 0.0;
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
                if (lane == 0) s_best[k] = bi;
            }
        }
        __syncthreads();
        const float* g = gsnr + (size_t)J.grow * nw;
        for (int c = tid; c < b; c += kBwdThreads) {
            double acc = 0.0;
            for (int k = 0; k < nw; ++k) {
                float hb, be;
                boxcar_coefs(b, widths[k], &hb, &be);
                acc -= (double)g[k] * (double)be;
                int off = c - s_best[k] - 1;
                off += (off < 0) ? b : 0;
                if (off < widths[k]) acc += (double)g[k] * (double)hb;
            }
            s_g[c] = (float)(acc / (double)J.stdnoise);
        }
        __syncthreads();
        // back through the shifts: row i reads the row gradient at c - sigma_i. A warp per row;
        // what the group's first row finds in gds are the zeros it was cleared to.
        for (int i = tid >> 5; i < m; i += kBwdThreads / 32) {
            const int sg = sig[i];
            float* to = gds + (size_t)i * b;
#pragma unroll 8
            for (int c = lane; c < b; c += 32) {
                int idx = c - sg;
                idx += (idx < 0) ? b : 0;
                to[c] = __fadd_rn(q == 0 ? 0.0f : to[c], s_g[idx]);
            }
        }
        __syncthreads();
    }
}

// Downsampling adjoint of the groups of one wave (each trial at most once per wave): a thread per
// sample gathers from the few outputs that reach it. Bound: FP64 and conversion instructions;
// four series of 2^20 samples took 108 us with 64 CTAs a series and two divisions a sample, 37
// as it is now.
__global__ void k_groups_ds_adjoint(const BwdGroup* __restrict__ groups, const int* __restrict__ wave,
                                    const float* __restrict__ gds_all, float* __restrict__ gz_all)
{
    const BwdGroup G = groups[wave[blockIdx.y]];
    const float* gout = gds_all + G.gds;
    float* gin = gz_all + G.gz;
    const size_t N = G.N, n = G.n_ds;
    const double f = G.f, rf = 1.0 / f, dn = (double)n, n1 = (double)N - 1.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N;
         i += (size_t)gridDim.x * blockDim.x) {
        if (G.src_is_z) {  // the cycle folds the series itself
            if (i < n) gin[i] = __fadd_rn(gin[i], gout[i]);
            continue;
        }
        // Outputs k with floor(k f) <= i <= floor(k f + f), k f <= i + 1: from the one before
        // i / f to the one after (i + 1) / f, all of them doubles that hold whole numbers.
        const double di = whole_double(i);
        double acc = 0.0;
        double dk = fmax(floor_double(di * rf) - 2.0, 0.0);
        for (; dk < dn; dk += 1.0) {
            const double start = __dmul_rn(dk, f);
            const double fs = floor_double(start);
            if (fs > di) break;
            const double end = __dadd_rn(start, f);
            const double fe = fmin(floor_double(end), n1);
            if (fe < di) continue;
            double c = 0.0;
            if (di == fs) c += (double)__double2float_rn((fs + 1.0) - start);
            if (di == fe) c += (double)__double2float_rn(end - fe);
            if (di > fs && di < fe) c += 1.0;
            if (fe == fs) c -= 1.0;
            if (c != 0.0) acc += c * (double)gout[(size_t)dk];
        }
        if (acc != 0.0) gin[i] = __fadd_rn(gin[i], (float)acc);
    }
}

__global__ void k_live_rows(const float* __restrict__ g, size_t rows, int nw,
                            unsigned long long* __restrict__ list, unsigned long long cap,
                            unsigned long long* __restrict__ count)
{
    for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < rows;
         r += (size_t)gridDim.x * blockDim.x) {
        bool live = false;
        for (int k = 0; k < nw; ++k) live |= g[r * nw + k] != 0.0f;
        if (live) {
            const unsigned long long slot = atomicAdd(count, 1ull);
            if (slot < cap) list[slot] = r;
        }
    }
}

static int plan_backward(SearchPlan& P, const float* d_z, const float* d_gsnr, float* d_gz,
                         size_t max_rows, cudaStream_t st)
{
    if (!P.dev_ready) return set_error(RT_EINVAL, "the plan has not run");
    const size_t L = P.out_rows_off.back();
    const int nw = (int)P.widths.size();
    RT_TRY_CUDA(cudaMemsetAsync(d_gz, 0, P.total_len * sizeof(float), st));
    if (L == 0 || nw == 0) return RT_OK;
    // rows that carry a gradient
    unsigned long long *d_list = nullptr, *d_count = nullptr;
    RT_TRY_CUDA(scratch_malloc((void**)&d_list, (max_rows + 1) * sizeof(unsigned long long), st));
    d_count = d_list + max_rows;
    RT_TRY_CUDA(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), st));
    k_live_rows<<<(unsigned)std::min<size_t>((L + 255) / 256, 148 * 16), 256, 0, st>>>(
        d_gsnr, L, nw, d_list, max_rows, d_count);
    unsigned long long count = 0;
    RT_TRY_CUDA(cudaMemcpyAsync(&count, d_count, sizeof(count), cudaMemcpyDeviceToHost, st));
    RT_TRY_CUDA(cudaStreamSynchronize(st));
    if (count > max_rows) {
        cudaFreeAsync(d_list, st);
        return set_error(RT_EINVAL, "%llu periodogram rows carry a gradient (at most %zu)", count,
                         max_rows);
    }
    std::vector<unsigned long long> rows(count);
    if (count)
        RT_TRY_CUDA(cudaMemcpyAsync(rows.data(), d_list, count * sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, st));
    RT_TRY_CUDA(cudaStreamSynchronize(st));
    cudaFreeAsync(d_list, st);
    if (count == 0) return RT_OK;
    std::sort(rows.begin(), rows.end());
    // rows -> (transform, s), grouped by (trial, cycle) in plan order
    const int C = (int)P.f.size();
    std::vector<BwdJob> jobs;
    std::vector<BwdGroup> groups;
    std::vector<int> group_trial;
    size_t xi = 0, gds_total = 0, sig_total = 0;
    int last_tc = -1;
    for (unsigned long long r : rows) {
        while (xi + 1 < P.xforms.size() && P.xforms[xi + 1].out_row <= r) ++xi;
        const XformRec& X = P.xforms[xi];
        if (r < X.out_row || r >= X.out_row + (unsigned long long)X.rows_eval) continue;
        if (X.b > kBwdMaxBins || X.b + (size_t)*std::max_element(P.widths.begin(), P.widths.end()) > 2 * kBwdMaxBins)
            return set_error(RT_EINVAL, "profiles of %d bins are too long for the backward", X.b);
        const int t = P.xform_tc[xi].x, c = P.xform_tc[xi].y;
        const int tc = t * C + c;
        if (tc != last_tc) {
            BwdGroup G;
            const double f = P.f[c];
            const size_t N = P.lengths[t];
            G.src_is_z = (f == 1) ? 1 : 0;
            G.src = G.src_is_z ? P.offsets[t] : P.ds_off[(size_t)tc];
            G.n_ds = G.src_is_z ? N : downsampled_size(N, f);
            G.N = N;
            G.f = f;
            G.gds = gds_total;
            gds_total += (G.n_ds + 3) & ~size_t(3);
            G.gz = P.offsets[t];
            G.sig = sig_total;
            G.job0 = (int)jobs.size();
            G.njobs = 0;
            G.pad = 0;
            groups.push_back(G);
            group_trial.push_back(t);
            last_tc = tc;
        }
        BwdGroup& G = groups.back();
        BwdJob J;
        J.m = X.m;
        J.b = X.b;
        J.s = (int)(r - X.out_row);
        J.stdnoise = X.stdnoise;
        J.grow = r;
        J.pad = J.pad2 = 0;
        jobs.push_back(J);
        ++G.njobs;
        sig_total = std::max<size_t>(sig_total, (size_t)G.sig + (size_t)X.m);
    }
    if (jobs.empty()) return RT_OK;
    // waves: the k-th group of every trial (a trial's groups accumulate into one series)
    std::vector<std::vector<int>> waves;
    {
        std::map<int, int> seen;
        for (size_t g = 0; g < groups.size(); ++g) {
            const int k = seen[group_trial[g]]++;
            if ((int)waves.size() <= k) waves.emplace_back();
            waves[k].push_back((int)g);
        }
    }
    int wmax = 1;
    for (int w : P.widths) wmax = std::max(wmax, w);
    unsigned char* blob = nullptr;
    const size_t nwave = groups.size();
    const size_t bytes = groups.size() * sizeof(BwdGroup) + jobs.size() * sizeof(BwdJob) +
                         nwave * sizeof(int) + (gds_total + 4) * sizeof(float) +
                         (sig_total + 4) * sizeof(int) + 64;
    RT_TRY_CUDA(scratch_malloc((void**)&blob, bytes, st));
    BwdGroup* d_groups = reinterpret_cast<BwdGroup*>(blob);
    BwdJob* d_jobs = reinterpret_cast<BwdJob*>(d_groups + groups.size());
    int* d_wave = reinterpret_cast<int*>(d_jobs + jobs.size());
    float* d_gds = reinterpret_cast<float*>(
        (reinterpret_cast<uintptr_t>(d_wave + nwave) + 15) & ~uintptr_t(15));
    int* d_sig = reinterpret_cast<int*>(d_gds + gds_total + 4);
    int s = RT_OK;
    auto ck = [&](cudaError_t e) { if (s == RT_OK && e != cudaSuccess) s = check_cuda(e, "search backward"); };
    ck(cudaMemcpyAsync(d_groups, groups.data(), groups.size() * sizeof(BwdGroup),
                       cudaMemcpyHostToDevice, st));
    ck(cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(BwdJob), cudaMemcpyHostToDevice, st));
    ck(cudaMemsetAsync(d_gds, 0, gds_total * sizeof(float), st));
    const size_t smem = (size_t)(2 * kBwdMaxBins + wmax) * sizeof(float);
    ck(cudaFuncSetAttribute(k_rows_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (s == RT_OK) {
        k_rows_backward<<<(unsigned)groups.size(), kBwdThreads, smem, st>>>(
            d_groups, d_jobs, P.d_ds, d_z, d_gsnr, P.d_widths, nw, wmax, d_gds, d_sig);
        ck(cudaGetLastError());
    }
    // every group of a kernel call uses its own shift table: the groups run concurrently
    (void)sig_total;
    for (const auto& w : waves) {
        if (s != RT_OK) break;
        ck(cudaMemcpyAsync(d_wave, w.data(), w.size() * sizeof(int), cudaMemcpyHostToDevice, st));
        dim3 grid(592, (unsigned)w.size());
        k_groups_ds_adjoint<<<grid, 256, 0, st>>>(d_groups, d_wave, d_gds, d_gz);
        ck(cudaGetLastError());
    }
    cudaFreeAsync(blob, st);
    return s;
}

}  // namespace rt

// ====================================================================================
// C ABI
// ====================================================================================
using namespace rt;

struct rt_search_plan {
    SearchPlan p;
};

static int plan_create(const uint64_t* lengths, size_t ntrials, const rt_search_config* cfg,
                       const uint64_t* widths, size_t num_widths,
                       const rt_search_tuning* tuning, rt_search_plan** out,
                       const rt_tile_rule* rules = nullptr, size_t num_rules = 0)
{
    if (!out || !cfg || (!lengths && ntrials) || (!widths && num_widths))
        return set_error(RT_EINVAL, "null argument");
    *out = nullptr;
    if (ntrials == 0) return set_error(RT_EINVAL, "at least one time series is required");
    if (num_widths == 0 || num_widths > (size_t)kMaxWidths)
        return set_error(RT_EINVAL, "between 1 and %d trial widths are supported", kMaxWidths);
    rt_search_plan* h = new (std::nothrow) rt_search_plan();
    if (!h) return set_error(RT_ENOMEM, "out of host memory");
    SearchPlan& P = h->p;
    P.cfg = *cfg;
    if (tuning) P.tuning = *tuning;
    if (rules) P.rules.assign(rules, rules + num_rules);
    for (size_t i = 0; i < num_widths; ++i) {
        // snr.hpp:21-31
        if (!(widths[i] > 0 && widths[i] < cfg->bins_min)) {
            delete h;
            return set_error(RT_EINVAL, "trial widths must be all > 0 and < columns");
        }
        P.widths.push_back((int)widths[i]);
    }
    P.nfast = detect_fast_widths(P.widths.data(), (int)P.widths.size());
    if (P.nfast && P.widths.size() > 10 && cfg->bins_min <= 42) P.nfast = 0;
    for (size_t t = 0; t < ntrials; ++t) {
        if (lengths[t] == 0 || lengths[t] >= (1ull << 40)) {
            delete h;
            return set_error(RT_EINVAL, "time series %zu has an unsupported length", t);
        }
        P.lengths.push_back((size_t)lengths[t]);
        P.offsets.push_back(P.total_len);
        P.total_len += lengths[t];
        P.max_len = std::max(P.max_len, (size_t)lengths[t]);
    }
    int s = plan_build(P);
    if (s != RT_OK) {
        delete h;
        return s;
    }
    *out = h;
    return RT_OK;
}

extern "C" int rt_search_plan_create(const uint64_t* lengths, size_t ntrials,
                                     const rt_search_config* cfg, const uint64_t* widths,
                                     size_t num_widths, rt_search_plan** out)
{
    return plan_create(lengths, ntrials, cfg, widths, num_widths, nullptr, out);
}

static int check_tuning(const rt_search_tuning* tuning)
{
    if (tuning && !(tuning->rows_fraction >= 0.0 && tuning->rows_fraction <= 1.0))
        return set_error(RT_EINVAL, "rows_fraction must be in [0, 1]");
    if (tuning && !(tuning->rows_fraction_deep >= 0.0 && tuning->rows_fraction_deep <= 1.0))
        return set_error(RT_EINVAL, "rows_fraction_deep must be in [0, 1]");
    if (tuning && tuning->snr_threads != 0 && tuning->snr_threads != 8 && tuning->snr_threads != 16)
        return set_error(RT_EINVAL, "snr_threads must be 0, 8 or 16");
    if (tuning && tuning->lag_items < 0) return set_error(RT_EINVAL, "lag_items must be >= 0");
    return RT_OK;
}

extern "C" int rt_search_plan_create_tuned(const uint64_t* lengths, size_t ntrials,
                                           const rt_search_config* cfg, const uint64_t* widths,
                                           size_t num_widths, const rt_search_tuning* tuning,
                                           rt_search_plan** out)
{
    RT_TRY(check_tuning(tuning));
    return plan_create(lengths, ntrials, cfg, widths, num_widths, tuning, out);
}

extern "C" int rt_search_plan_create_rules(const uint64_t* lengths, size_t ntrials,
                                           const rt_search_config* cfg, const uint64_t* widths,
                                           size_t num_widths, const rt_search_tuning* tuning,
                                           const rt_tile_rule* rules, size_t num_rules,
                                           rt_search_plan** plan)
{
    if (num_rules && !rules) return set_error(RT_EINVAL, "null argument");
    for (size_t i = 0; i < num_rules; ++i) {
        const rt_tile_rule& R = rules[i];
        if (R.rows_min > R.rows_max || R.bins_min > R.bins_max)
            return set_error(RT_EINVAL, "tile rule %zu: empty rows or bins range", i);
        if (!(R.rows_fraction >= 0.0 && R.rows_fraction <= 1.0))
            return set_error(RT_EINVAL, "tile rule %zu: rows_fraction must be in [0, 1]", i);
        if (R.snr_threads != 0 && R.snr_threads != 8 && R.snr_threads != 16)
            return set_error(RT_EINVAL, "tile rule %zu: snr_threads must be 0, 8 or 16", i);
        if (R.max_levels < 0 || R.max_levels > kMaxJobDepth + 1)
            return set_error(RT_EINVAL, "tile rule %zu: max_levels must be in [0, %d]", i,
                             kMaxJobDepth + 1);
    }
    RT_TRY(check_tuning(tuning));
    return plan_create(lengths, ntrials, cfg, widths, num_widths, tuning, plan, rules, num_rules);
}

extern "C" int rt_search_plan_rows(const rt_search_plan* plan, uint64_t* row_offsets)
{
    if (!plan || !row_offsets) return set_error(RT_EINVAL, "null argument");
    for (size_t i = 0; i < plan->p.out_rows_off.size(); ++i) row_offsets[i] = plan->p.out_rows_off[i];
    return RT_OK;
}

extern "C" int rt_search_plan_stats(const rt_search_plan* plan, rt_search_plan_stats_t* st)
{
    if (!plan || !st) return set_error(RT_EINVAL, "null argument");
    const SearchPlan& P = plan->p;
    memset(st, 0, sizeof(*st));
    st->num_trials = P.lengths.size();
    st->num_cycles = P.f.size();
    st->num_transforms = P.xforms.size();
    st->num_work_items = P.items.size();
    st->num_multistage = (uint64_t)P.nseq;
    st->total_rows = P.out_rows_off.back();
    st->total_samples = P.total_len;
    st->downsampled_samples = P.ds_total;
    uint64_t fold = 0;
    for (const XformRec& X : P.xforms) fold += (uint64_t)X.m * X.b;
    st->folded_samples = fold;
    st->scrunch_factor = (uint64_t)P.scrunch;
    return RT_OK;
}

extern "C" int rt_search_plan_memory(const rt_search_plan* plan, rt_search_memory_t* h_out)
{
    if (!plan || !h_out) return set_error(RT_EINVAL, "null argument");
    const SearchPlan& P = plan->p;
    h_out->ring_slots = (uint64_t)P.slots;
    h_out->ring_slot_bytes = 2 * P.slot_floats * sizeof(float);
    h_out->shared_bytes = kEngineDynBytes;
    h_out->ops_bytes = (uint64_t)P.layout.ops_units * 16;
    h_out->buffer_bytes = (uint64_t)P.layout.buf_floats * sizeof(float);
    return RT_OK;
}

// Graph replay of plan_run: captured on the plan's own stream (the legacy default stream
// cannot be captured), launched on the caller's.
static int plan_run_graph(SearchPlan& P, const float* data, float* normalised_out,
                          double* periods, uint32_t* foldbins, float* snrs, cudaStream_t st)
{
    const void* key[5] = {data, normalised_out, periods, foldbins, snrs};
    bool same = P.gexec != nullptr;
    for (int i = 0; i < 5; ++i) same = same && key[i] == P.gkey[i];
    if (!same) {
        RT_TRY(plan_prepare_device(P));  // allocations happen outside the capture
        if (!P.cap_stream)
            RT_TRY_CUDA(cudaStreamCreateWithFlags(&P.cap_stream, cudaStreamNonBlocking));
        if (P.gexec) {
            cudaGraphExecDestroy(P.gexec);
            P.gexec = nullptr;
        }
        RT_TRY_CUDA(cudaStreamBeginCapture(P.cap_stream, cudaStreamCaptureModeThreadLocal));
        const int rc = plan_run(P, data, normalised_out, periods, foldbins, snrs, P.cap_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t ec = cudaStreamEndCapture(P.cap_stream, &g);
        if (rc != RT_OK) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ec != cudaSuccess) return check_cuda(ec, "cudaStreamEndCapture");
        const cudaError_t ei = cudaGraphInstantiate(&P.gexec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) {
            P.gexec = nullptr;
            return check_cuda(ei, "cudaGraphInstantiate");
        }
        for (int i = 0; i < 5; ++i) P.gkey[i] = key[i];
        ++P.graph_captures;
    }
    RT_TRY_CUDA(cudaGraphLaunch(P.gexec, st));
    return RT_OK;
}

extern "C" int rt_search_run(rt_search_plan* plan, const float* data, float* normalised_out,
                             double* periods, uint32_t* foldbins, float* snrs, void* stream)
{
    if (!plan || !data || !periods || !foldbins || !snrs) return set_error(RT_EINVAL, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    SearchPlan& P = plan->p;
    if (P.use_graph && !P.timing)
        return plan_run_graph(P, data, normalised_out, periods, foldbins, snrs, st);
    return plan_run(P, data, normalised_out, periods, foldbins, snrs, st);
}

extern "C" int rt_search_set_graph(rt_search_plan* plan, int enable)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    P.use_graph = enable != 0;
    if (!P.use_graph && P.gexec) {
        RT_TRY_CUDA(cudaGraphExecDestroy(P.gexec));
        P.gexec = nullptr;
    }
    return RT_OK;
}

extern "C" int rt_search_graph_captures(const rt_search_plan* plan, int* h_count)
{
    if (!plan || !h_count) return set_error(RT_EINVAL, "null argument");
    *h_count = plan->p.graph_captures;
    return RT_OK;
}

extern "C" int rt_search_plan_transforms(const rt_search_plan* plan, rt_search_transform* h_out)
{
    if (!plan || !h_out) return set_error(RT_EINVAL, "null argument");
    const SearchPlan& P = plan->p;
    for (size_t i = 0; i < P.xforms.size(); ++i) {
        const XformRec& X = P.xforms[i];
        rt_search_transform& o = h_out[i];
        o.trial = (uint32_t)P.xform_tc[i].x;
        o.cycle = (uint32_t)P.xform_tc[i].y;
        o.bins = (uint32_t)X.b;
        o.rows = (uint32_t)X.m;
        o.rows_eval = (uint32_t)X.rows_eval;
        o.out_row = X.out_row;
        o.factor = P.f[P.xform_tc[i].y];
        o.tau = X.tau;
        o.stdnoise = X.stdnoise;
    }
    return RT_OK;
}

extern "C" int rt_search_normalisation(rt_search_plan* plan, double* h_mean, double* h_std,
                                       void* stream)
{
    if (!plan || !h_mean || !h_std) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    const size_t T = P.lengths.size();
    if (!P.dev_ready || P.cfg.already_normalised) {
        for (size_t t = 0; t < T; ++t) {
            h_mean[t] = 0.0;
            h_std[t] = 1.0;
        }
        return RT_OK;
    }
    cudaStream_t st = (cudaStream_t)stream;
    RT_TRY_CUDA(cudaMemcpyAsync(h_mean, P.d_mean, T * sizeof(double), cudaMemcpyDeviceToHost, st));
    RT_TRY_CUDA(cudaMemcpyAsync(h_std, P.d_normv, T * sizeof(double), cudaMemcpyDeviceToHost, st));
    RT_TRY_CUDA(cudaStreamSynchronize(st));
    return RT_OK;
}

extern "C" int rt_search_backward_rows(rt_search_plan* plan, const float* d_z,
                                       const float* d_gsnr, float* d_gz, size_t max_rows,
                                       void* stream)
{
    if (!plan || !d_z || !d_gsnr || !d_gz) return set_error(RT_EINVAL, "null argument");
    if (max_rows == 0) return set_error(RT_EINVAL, "max_rows must be positive");
    return plan_backward(plan->p, d_z, d_gsnr, d_gz, max_rows, (cudaStream_t)stream);
}

extern "C" int rt_search_plan_prepare(rt_search_plan* plan)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    return plan_prepare_device(plan->p);
}

extern "C" int rt_search_check(rt_search_plan* plan, void* stream)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    if (!plan->p.dev_ready) return RT_OK;
    return plan_check_error(plan->p, (cudaStream_t)stream);
}

// The kernel arguments and buffers are baked into a captured graph: drop it.
static void plan_drop_graph(SearchPlan& P)
{
    if (P.gexec) cudaGraphExecDestroy(P.gexec);
    P.gexec = nullptr;
    for (int i = 0; i < 5; ++i) P.gkey[i] = nullptr;
}

extern "C" int rt_search_set_wait_limit(rt_search_plan* plan, long long polls)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    if (polls < 1) return set_error(RT_EINVAL, "the wait limit must be at least one poll");
    cudaDeviceSynchronize();
    plan->p.spin_limit = polls;
    plan_drop_graph(plan->p);
    return RT_OK;
}

extern "C" int rt_search_inject_fault(rt_search_plan* plan, int kind, int arg)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    cudaDeviceSynchronize();
    switch (kind) {
        case RT_FAULT_NONE:
            P.dep_bias = 0;
            P.alloc_fail_at = 0;
            P.ring_fails_above = 0;
            break;
        case RT_FAULT_STAGE_WAIT:
            P.dep_bias = 1;
            break;
        case RT_FAULT_ALLOC:
            if (arg < 1) return set_error(RT_EINVAL, "the failing allocation is numbered from 1");
            P.alloc_fail_at = arg;
            plan_free_device(P);  // the next run allocates again
            break;
        case RT_FAULT_RING:
            if (arg < 1) return set_error(RT_EINVAL, "a ring has one slot or more");
            P.ring_fails_above = arg;
            plan_free_device(P);
            break;
        default:
            return set_error(RT_EINVAL, "unknown fault kind %d", kind);
    }
    plan_drop_graph(P);
    return RT_OK;
}

extern "C" int rt_search_set_timing(rt_search_plan* plan, int enable)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    if (enable && !P.ev[0])
        for (int i = 0; i < 4; ++i) RT_TRY_CUDA(cudaEventCreate(&P.ev[i]));
    P.timing = enable != 0;
    return RT_OK;
}

extern "C" int rt_search_last_timing(rt_search_plan* plan, float* h_ms, int* h_launches)
{
    if (!plan || !h_ms) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    if (!P.timing || !P.ev[0]) return set_error(RT_EINVAL, "timing is not enabled on this plan");
    RT_TRY_CUDA(cudaEventSynchronize(P.ev[3]));
    for (int i = 0; i < 3; ++i) RT_TRY_CUDA(cudaEventElapsedTime(&h_ms[i], P.ev[i], P.ev[i + 1]));
    if (h_launches) *h_launches = P.launches_last_run;
    return RT_OK;
}

extern "C" int rt_search_set_profiling(rt_search_plan* plan, int enable)
{
    if (!plan) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    if (enable && !P.d_phase) {
        RT_TRY_CUDA(cudaMalloc((void**)&P.d_phase, kCounters * sizeof(unsigned long long)));
        RT_TRY_CUDA(cudaMemset(P.d_phase, 0, kCounters * sizeof(unsigned long long)));
    } else if (!enable && P.d_phase) {
        cudaFree(P.d_phase);
        P.d_phase = nullptr;
    }
    return RT_OK;
}

extern "C" int rt_search_phase_cycles(rt_search_plan* plan, uint64_t* h_counters, int reset)
{
    if (!plan || !h_counters) return set_error(RT_EINVAL, "null argument");
    SearchPlan& P = plan->p;
    if (!P.d_phase) return set_error(RT_EINVAL, "profiling is not enabled on this plan");
    RT_TRY_CUDA(cudaDeviceSynchronize());
    RT_TRY_CUDA(cudaMemcpy(h_counters, P.d_phase, kCounters * sizeof(uint64_t), cudaMemcpyDeviceToHost));
    if (reset) RT_TRY_CUDA(cudaMemset(P.d_phase, 0, kCounters * sizeof(unsigned long long)));
    return RT_OK;
}

extern "C" void rt_search_plan_destroy(rt_search_plan* plan)
{
    if (!plan) return;
    cudaDeviceSynchronize();
    if (plan->p.d_phase) cudaFree(plan->p.d_phase);
    if (plan->p.gexec) cudaGraphExecDestroy(plan->p.gexec);
    if (plan->p.cap_stream) cudaStreamDestroy(plan->p.cap_stream);
    for (int i = 0; i < 4; ++i)
        if (plan->p.ev[i]) cudaEventDestroy(plan->p.ev[i]);
    plan_free_device(plan->p);
    delete plan;
}

// ------------------------------------------------------------------------------------
// Single-series deredden / normalise (TimeSeries.deredden / normalise, fast_running_median)
// ------------------------------------------------------------------------------------
static TrialArrays one_series(size_t N, size_t nl)
{
    return TrialArrays{nullptr, nullptr, nullptr, nullptr, N, nl};
}

// width_samples / min_points -> (scrunch factor, running-median width, scrunched length)
static int rmed_geometry(size_t N, size_t width_samples, size_t minpts, int* k, int* w, size_t* nl)
{
    // running_medians.py:72-80
    if (!(minpts % 2)) return set_error(RT_EINVAL, "min_points must be an odd number");
    *k = (int)std::max(1.0, (double)width_samples / (double)minpts);
    *w = (*k == 1) ? (int)width_samples : (int)minpts;
    *nl = (*k == 1) ? N : N / (size_t)*k;
    // running_median.hpp:103-107
    if (!(*w % 2)) return set_error(RT_EINVAL, "width must be an odd number");
    if (!((size_t)*w < *nl)) return set_error(RT_EINVAL, "width must be < size");
    return RT_OK;
}

extern "C" int rt_fast_running_median(const float* d_x, size_t size, size_t width_samples,
                                      size_t min_points, double* d_out, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    int k, w;
    size_t nl;
    RT_TRY(rmed_geometry(size, width_samples, min_points, &k, &w, &nl));
    const TrialArrays A = one_series(size, nl);
    float *lores = nullptr, *rmed = nullptr;
    int s = RT_OK;
    if (k > 1) {
        RT_TRY_CUDA(scratch_malloc((void**)&lores, nl * sizeof(float), st));
        RT_TRY_CUDA(scratch_malloc((void**)&rmed, nl * sizeof(float), st));
        s = launch_scrunch(d_x, A, k, 1, nl, lores, st);
        if (s == RT_OK) s = launch_running_median(lores, nullptr, nullptr, 1, nl, w, rmed, st);
        if (s == RT_OK) {
            k_interp_rmed<<<(unsigned)((size + kInterpSpan - 1) / kInterpSpan), 256, 0, st>>>(
                A, k, div_magic(2u * (unsigned)k), rmed, d_out);
            s = check_cuda(cudaGetLastError(), "fast_running_median");
        }
    } else {
        // no scrunching: the exact running median (float32), widened to float64
        RT_TRY_CUDA(scratch_malloc((void**)&rmed, size * sizeof(float), st));
        s = launch_running_median(d_x, nullptr, nullptr, 1, size, w, rmed, st);
        if (s == RT_OK) {
            k_interp_rmed<<<(unsigned)((size + kInterpSpan - 1) / kInterpSpan), 256, 0, st>>>(
                one_series(size, size), 1, div_magic(2), rmed, d_out);
            s = check_cuda(cudaGetLastError(), "fast_running_median");
        }
    }
    if (lores) cudaFreeAsync(lores, st);
    if (rmed) cudaFreeAsync(rmed, st);
    return s;
}

extern "C" int rt_deredden(const float* d_x, size_t size, double tsamp, double width,
                           size_t min_points, float* d_out, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    const double ws = nearbyint(width / tsamp);  // int(round(width / tsamp)), half to even
    if (!(ws >= 1)) return set_error(RT_EINVAL, "width is shorter than one sample");
    int k, w;
    size_t nl;
    RT_TRY(rmed_geometry(size, (size_t)ws, min_points, &k, &w, &nl));
    const TrialArrays A = one_series(size, nl);
    float *lores = nullptr, *rmed = nullptr;
    double* part = nullptr;
    int s = RT_OK;
    const size_t blocks = interp_blocks(size);
    RT_TRY_CUDA(scratch_malloc((void**)&part, blocks * 3 * sizeof(double), st));
    if (k > 1) {
        RT_TRY_CUDA(scratch_malloc((void**)&lores, nl * sizeof(float), st));
        RT_TRY_CUDA(scratch_malloc((void**)&rmed, nl * sizeof(float), st));
        s = launch_scrunch(d_x, A, k, 1, nl, lores, st);
        if (s == RT_OK) s = launch_running_median(lores, nullptr, nullptr, 1, nl, w, rmed, st);
    } else {
        RT_TRY_CUDA(scratch_malloc((void**)&rmed, size * sizeof(float), st));
        s = launch_running_median(d_x, nullptr, nullptr, 1, size, w, rmed, st);
    }
    if (s == RT_OK) {
        k_dered<<<(unsigned)blocks, kStatThreads, 0, st>>>(d_x, A, k, div_magic(2u * (unsigned)k),
                                                          rmed, d_out, part);
        s = check_cuda(cudaGetLastError(), "deredden");
    }
    if (lores) cudaFreeAsync(lores, st);
    if (rmed) cudaFreeAsync(rmed, st);
    cudaFreeAsync(part, st);
    return s;
}

extern "C" int rt_normalise(const float* d_x, size_t size, float* d_out, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (size == 0) return RT_OK;
    const TrialArrays A = one_series(size, 0);
    double* part = nullptr;
    const size_t blocks = interp_blocks(size);
    RT_TRY_CUDA(scratch_malloc((void**)&part, (blocks * 3 + 2) * sizeof(double), st));
    double* mean = part + blocks * 3;
    double* norm = mean + 1;
    k_sums<<<(unsigned)blocks, kStatThreads, 0, st>>>(d_x, A, part);
    k_stats<<<1, 32, 0, st>>>(part, A, (int)blocks, 1, mean, norm);
    k_normalise<<<dim3(std::max(1, (int)std::min<size_t>((size + 255) / 256, 4096)), 1), 256, 0, st>>>(
        d_x, A, mean, norm, d_out);
    int s = check_cuda(cudaGetLastError(), "normalise");
    cudaFreeAsync(part, st);
    return s;
}
