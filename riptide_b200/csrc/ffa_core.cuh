// FFA transform core: one CTA executes one "tree job" of an FFA transform in shared memory.
//
// The reference computes the transform of an m x b block (cpp/transforms.hpp:30-50) by
// recursive halving: head = rows >> 1 (cpp/block.hpp:30-31), tail = the rest, then
//     out[s] = head[h] + roll(tail[t], -(s - t)),   h = int(kh*s + .5f), t = int(kt*s + .5f)
// (transforms.hpp:13-27; the shift h + b_s of the reference equals s - t).
//
// Here the recursion tree is cut into jobs that fit one CTA's shared memory:
//   * a job has a root node (a subtree of the transform: first row, row count), the range of
//     root output rows it must produce, and a depth G: nodes at depth G below the root are
//     computed straight from a global source array whose row j holds the output of a node
//     at depth G+1 (or, for full-depth jobs, raw input row j);
//   * going down the tree, a contiguous output range of a node needs a contiguous range of
//     rows of each child, so every level is a list of (node, row range) stored back to back
//     in a shared-memory buffer; two buffers alternate between levels;
//   * the root rows are left in one of the two buffers, from where the caller writes them to
//     global memory (to feed a job higher in the tree, or as the ffa2 result) or turns them
//     into boxcar S/N (snr_core.cuh).
//
// What bounds the levels is shared memory: an output value of a level is two reads, an add and
// a write, and one warp-wide access of 32 words is one of the SM's cycles. Three choices
// follow:
//   * a lane owns kLaneCols = 9 consecutive columns (an odd stride, so the 32 lanes of an
//     access fall in 32 banks, and one warp covers the 240-279 bins of the usual searches,
//     two the 480-520). Rows s and s + 1 of a node mostly read the same head and tail rows,
//     the tail shifted by one more column for the second: computed together they take
//     9 + 10 reads for 18 values instead of 36;
//   * every row is stored with its first kHalo columns repeated after its last one, computed
//     as columns b .. b + 8 of the row, so that the 10 consecutive columns a lane reads from a
//     rolled row never wrap: one address per lane and row, then immediate offsets;
//   * the bottom three levels of a subtree of whole rows (nodes of 4 to 8 input rows) are
//     computed in registers from the input rows, one node per warp (ffa_nodes_fused): 92 reads
//     and 72 writes of a lane for 3 x 72 values. Above them, two levels are computed per pass
//     over shared memory where the row numbers follow the usual pattern (level_quads).
//
// Against one level per pass with lanes 32 columns apart (a wrap test per value, unrolled for
// each count of column chunks), the search kernel over 16 trials of ~2^22 samples, bins
// 240-260, went from 12.1 to 9.4 ms (411 to 290 M warp instructions a trial), and 3 trials of
// 2^21 samples at bins 960-1040, which had taken a loop without unrolling, from 13.0 to 6.5 ms.
// Additions are float32 and performed in exactly the reference's order, so the result is
// bit-identical to cpp/transforms.hpp.
#pragma once
#include "common.cuh"
#include "bulk_copy.cuh"

namespace rt {

constexpr int kMaxJobDepth = 7;      // levels below the root computed inside one job
constexpr int kMaxTreeDepth = 5;     // deepest level of a job with a node list
constexpr int kMaxJobNodes = (2 << kMaxTreeDepth) - 1;  // nodes of all listed levels of one job
constexpr int kThreads = 480;        // compute threads per CTA of every FFA kernel (1 CTA per SM)
constexpr int kWarps = kThreads / 32;

constexpr int kLaneCols = 9;         // consecutive columns of a lane
constexpr int kHalo = kLaneCols + 2; // columns repeated past the end of a row
// Below this many bins a column window of a lane can wrap twice: such transforms take the
// plain level loop (level_rows_direct) throughout.
constexpr int kWideMinBins = 17;

// Barrier of the compute threads only (named barrier 1). The persistent search kernel adds a
// scheduling warp that does not take part; in the other kernels every thread computes.
__device__ __forceinline__ void cta_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
}

struct Node {
    int row0;   // first row of the node in the transform
    int rows;   // node size
    int lo;     // first needed output row (node-local)
    int hi;     // one past the last needed output row
    int off;    // row of `lo` inside this level's shared buffer
    int goff;   // first row group of the node at its level
    int qoff;   // first row quad of the node at its level
    int hbias, tbias;  // row r of the head / tail child is row hbias + r / tbias + r of the
                       // level below's buffer, of the staged rows, or of the transform
    int thr;    // last even row s with h(s) = s / 2 (odd rows: see head_row)
    float kh;   // head slope of the node (merge_coef), where rows follow no pattern
};

// One pass over a job's shared-memory levels: level d from level d + 1 by row groups, or
// (`two`) from level d + 2 by row quads. Its operations start at 16-byte unit `unit`.
struct Step {
    int d, two, unit, count;
};

struct JobTree {
    Node nodes[kMaxJobNodes];           // node i of level d at (1 << d) - 1 + i
    int level_rows[kMaxTreeDepth + 1];    // rows stored for each level
    int level_groups[kMaxTreeDepth + 1];  // row groups of each level
    int level_tails[kMaxTreeDepth + 1];   // row groups of its tail children: quads a level up
    Step steps[kMaxTreeDepth + 1];      // levels first_op .. 0, deepest first
    int nsteps;
    int depth;                          // deepest level with a node list
    int first_op;                       // levels first_op .. 0 are computed by `steps`
    int fused;                          // level `depth` is computed from the raw input rows
    int regular;                        // the root has at most kRegularRows rows
    int error;                          // nonzero if the job does not fit
    // Source rows of level `depth` staged in shared memory (jobs of later stages, whose source
    // is the previous stage's output): node i reads its head child's source rows
    // src_rng[i].x + [0, src_rng[i].y) from staged rows src_off[i] + ..., and its tail child's
    // rows src_rng[i].z + [0, .w) right after them. pstaged = 0: the level reads global rows.
    int pstaged;
    int src_off[(1 << kMaxTreeDepth) + 1];
    int4 src_rng[1 << kMaxTreeDepth];
};

// Description of one job, produced by the planners (host).
struct JobSpec {
    int root_row0, root_rows;  // root node
    int lo, hi;                // root output range
    int G;                     // relative depth of the level computed from the global source
};

// Full-depth job: G = smallest depth d with ceil(M / 2^d) <= 2 (all nodes there have 1 or
// 2 rows, whose children are single input rows).
RT_HD int full_depth(int rows)
{
    int d = 0;
    while (((rows + (1 << d) - 1) >> d) > 2) ++d;
    return d;
}

// Whether the bottom three levels (G, G - 1, G - 2) of a full-depth job are computed together:
// the nodes of level G - 2 then have 4 to 8 rows.
RT_HD bool job_fused(int G, int b) { return G >= 2 && b >= kWideMinBins; }

// Largest full depth of a stage-0 job whose node lists fit a JobTree.
RT_HD int max_full_depth(int b) { return b >= kWideMinBins ? kMaxJobDepth : kMaxTreeDepth; }

// Rows of a node are computed in groups of two consecutive rows, aligned so that the two rows
// share their tail row (t(s) = t(s + 1), and mostly their head row): for a node of n rows the
// group of row s is (s + n % 2) / 2. For every n up to kRegularRows that number is t(s) itself,
// and h(s) is t(s) (n even), t(s) - 1 (n odd, s odd), or one of the two (n odd, s even: t(s) up
// to the middle row n / 2 or, where that is odd, the row before it, t(s) - 1 beyond it): the CPU
// tests check every n and s. From n = 8195 on the float32 slope moves that middle row, and only
// the row groups (which read each row's own numbers) are used.
constexpr int kRegularRows = 8192;
RT_HD int group_of(int n, int s) { return (s + (n & 1)) >> 1; }

// h(s) of a node of at most kRegularRows rows, thr as in Node.
__device__ __forceinline__ int head_threshold(int rows)
{
    return (rows & 1) ? (rows >> 1) & ~1 : 0x7fffffff;
}
__device__ __forceinline__ int head_row(int thr, int s)
{
    return (s >> 1) - (int)((s > thr) & ((s & 1) ^ 1));
}
__device__ __forceinline__ int head_row(const Node& nd, int s) { return head_row(nd.thr, s); }

// Node q of a job's node list in heap order (1: the root, 2 q and 2 q + 1: the head and tail
// children of q): its row range follows from the root's by the head/tail row maps along the
// path to it. Every lane of a warp walks to a node of its own. `regular`: at most kRegularRows
// rows, whole-number maps (with the slopes, a division per level, the walk was most of the node
// lists' time).
__device__ __forceinline__ Node walk_to_node(const JobSpec& J, int q, int maxdepth, bool regular)
{
    Node nd;
    nd.row0 = J.root_row0;
    nd.rows = J.root_rows;
    nd.lo = J.lo;
    nd.hi = J.hi;
    nd.kh = 0.0f;
    const int d = 31 - __clz(q);
    if (regular) {
        for (int k = 0; k < maxdepth; ++k) {
            if (k >= d) break;
            const int mh = nd.rows >> 1, thr = head_threshold(nd.rows);
            if ((q >> (d - 1 - k)) & 1) {
                nd.lo = group_of(nd.rows, nd.lo);
                nd.hi = group_of(nd.rows, nd.hi - 1) + 1;
                nd.row0 += mh;
                nd.rows -= mh;
            } else {
                nd.lo = head_row(thr, nd.lo);
                nd.hi = head_row(thr, nd.hi - 1) + 1;
                nd.rows = mh;
            }
        }
    } else {
        for (int k = 0; k < maxdepth; ++k) {
            if (k >= d) break;
            const int tail = (q >> (d - 1 - k)) & 1;
            const int mh = nd.rows >> 1;
            const int n = tail ? nd.rows - mh : mh;
            const float slope = __fdiv_rn((float)n - 1.0f, (float)nd.rows - 1.0f);  // merge_coef
            nd.row0 += tail ? mh : 0;
            nd.rows = n;
            nd.lo = merge_row(slope, nd.lo);
            nd.hi = merge_row(slope, nd.hi - 1) + 1;
        }
        nd.kh = merge_coef(nd.rows).kh;
    }
    nd.thr = head_threshold(nd.rows);
    nd.hbias = nd.row0;
    nd.tbias = nd.row0 + (nd.rows >> 1);
    nd.off = nd.goff = nd.qoff = 0;
    return nd;
}

// Builds the node lists of a job (one warp, no CTA barrier): every lane walks to its nodes (31
// of levels 0 to 4, 32 of level 5), then the rows, groups and quads before each node in its
// level come from one scan over all levels. Level by level, with a scan each, it took the
// scheduling warp 6,600 cycles a job and kept the compute warps waiting.
// `raw`: a stage-0 job (whole subtree over raw input rows); otherwise the level-G source rows
// are laid out for staging (src_off, pstaged): set when every level-G node has two children and
// the rows fit a level buffer.
__device__ inline void build_job_tree_warp(JobTree& T, const JobSpec& J, int b, int cap_rows,
                                           int ops_units, bool raw)
{
    const int lane = threadIdx.x & 31;
    const bool fused = raw && job_fused(J.G, b);
    const int depth = fused ? J.G - 2 : J.G;
    if (depth > kMaxTreeDepth) {
        if (lane == 0) T.error = 1;
        __syncwarp();
        return;
    }
    const bool regular = J.root_rows <= kRegularRows;
    if (lane == 0) {
        T.depth = depth;
        T.fused = fused ? 1 : 0;
        T.regular = regular ? 1 : 0;
        T.error = 0;
        T.pstaged = 0;
    }
    __syncwarp();
    int first_op = b < kWideMinBins ? -1 : depth - 1;
    const int halves = depth == kMaxTreeDepth ? 2 : 1;
    for (int half = 0; half < halves; ++half) {
        const int q = half ? 32 + lane : lane + 1;
        const int d = 31 - __clz(q), i = q - (1 << d);  // level, node of the level
        const bool live = d <= depth && d < (half ? 6 : 5);
        Node nd = walk_to_node(J, live ? q : 1, depth, regular);
        // rows stored, row groups, and row groups of tail children (the quads of the level
        // above) of the node, scanned together: 11, 10 and 10 bits. The fused level stores
        // whole nodes.
        unsigned v = 0;
        if (live) {
            const int rows = (fused && d == depth) ? nd.rows : nd.hi - nd.lo;
            const int grp = group_of(nd.rows, nd.hi - 1) - group_of(nd.rows, nd.lo) + 1;
            v = rows | (grp << 11) | ((i & 1) ? (unsigned)grp << 21 : 0u);
        }
        // rows each level-G node needs from its two children, as consecutive staged blocks
        const bool source = !raw && half == halves - 1;
        const bool mine = source && live && d == depth;
        int v2 = 0;
        bool two = true;
        int4 rg = make_int4(0, 0, 0, 0);
        if (mine) {
            rg = make_int4(nd.row0, 0, nd.row0 + (nd.rows >> 1), 0);
            two = nd.rows >= 2;
            if (two) {
                const float kt = regular ? 0.f : merge_coef(nd.rows).kt;
                const int hlo = regular ? head_row(nd, nd.lo) : merge_row(nd.kh, nd.lo);
                const int hhi = regular ? head_row(nd, nd.hi - 1) : merge_row(nd.kh, nd.hi - 1);
                const int tlo = regular ? group_of(nd.rows, nd.lo) : merge_row(kt, nd.lo);
                const int thi = regular ? group_of(nd.rows, nd.hi - 1) : merge_row(kt, nd.hi - 1);
                rg = make_int4(rg.x + hlo, hhi + 1 - hlo, rg.z + tlo, thi + 1 - tlo);
            }
            v2 = rg.y + rg.w;
        }
        // both scans along the nodes of a level, at most 2^depth of them
        unsigned incl = v;
        int incl2 = v2;
        for (int o = 1; o < (1 << depth); o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            const int y2 = __shfl_up_sync(0xffffffffu, incl2, o);
            if (i >= o) {
                incl += y;
                incl2 += y2;
            }
        }
        const unsigned excl = incl - v;
        bool staged = false;
        if (source) {
            const int total = __shfl_sync(0xffffffffu, incl2, half ? 31 : (2 << depth) - 2);
            staged = __all_sync(0xffffffffu, two) && total <= cap_rows;
            if (lane == 0) {
                T.src_off[1 << depth] = total;
                T.pstaged = staged ? 1 : 0;
            }
            if (mine) {
                T.src_rng[i] = rg;
                T.src_off[i] = incl2 - v2;
            }
            if (staged && mine) {
                nd.hbias += incl2 - v2 - rg.x;
                nd.tbias += incl2 - v2 + rg.y - rg.z;
            }
            if (staged && b >= kWideMinBins) first_op = depth;
        }
        if (live) {
            nd.off = excl & 0x7ff;
            nd.goff = (excl >> 11) & 0x3ff;
            T.nodes[q - 1] = nd;
            if (i == (1 << d) - 1) {  // last node of the level
                T.level_rows[d] = incl & 0x7ff;
                T.level_groups[d] = (incl >> 11) & 0x3ff;
                T.level_tails[d] = incl >> 21;
                if ((int)(incl & 0x7ff) > cap_rows) T.error = 2;
            }
        }
        __syncwarp();
        if (live && d > 0) {
            Node& parent = T.nodes[(q >> 1) - 1];
            if (i & 1) {
                parent.qoff = excl >> 21;
                parent.tbias = nd.off - nd.lo;
            } else {
                parent.hbias = nd.off - nd.lo;
            }
        }
    }
    // the passes over levels first_op .. 0: two levels at a time from the deepest up, a single
    // one last when their number is odd; lane j has pass j
    {
        const int width = regular ? 2 : 1, ns = (first_op + width) / width;
        int d = first_op - lane * width;
        const bool live = lane < ns, two = live && regular && d >= 1;
        const int count = !live ? 0 : two ? T.level_tails[d] : T.level_groups[d];
        const int units = two ? 2 * count : count;
        int end = units;
        for (int o = 1; o < 8; o <<= 1) {  // at most kMaxTreeDepth + 1 passes
            const int y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += y;
        }
        if (live) T.steps[lane] = Step{two ? d - 1 : d, two ? 1 : 0, end - units, count};
        if (lane == 7) {
            T.first_op = first_op;
            T.nsteps = ns;
            if (end > ops_units) T.error = 3;
        }
    }
    __syncwarp();
}

// Chunks of kLaneCols columns of a row with its halo, and the stride of level rows in shared
// memory and in stage outputs (whole chunks, 16-byte aligned rows).
RT_HD int ffa_chunks(int b) { return (b + kHalo + kLaneCols - 1) / kLaneCols; }
RT_HD int ffa_stride(int b) { return (ffa_chunks(b) * kLaneCols + 3) & ~3; }

// One group of a level: output rows `out` and, with kOpTwo, `out` + 1 of the level buffer;
// row i is head row h_i + roll(tail row t_i, -shift_i) of the level below.
struct GroupOp {
    unsigned h;      // h_0 | h_1 << 16
    unsigned t;      // t_0 | t_1 << 16
    unsigned shift;  // shift_0 | shift_1 << 13 | flags
    int out;
};
enum : unsigned {
    kOpTwo = 1u << 26,       // two rows
    kOpSameHead = 1u << 27,  // h_1 = h_0
    kOpSameTail = 1u << 28,  // t_1 = t_0 and shift_1 = shift_0 + 1
};

// One quad of a level: up to four consecutive output rows k = 0 .. 3 (row `out` + k of the
// level buffer for the k of the mask) that read tail rows T_0 (k < 2) and T_1 of the level
// below, shifted by sC, sC + 1, sC + 1, sC + 2, and head rows H_0 (k = 0; k = 1 without
// kQuadH1), H_1 (k = 2; k = 1 with kQuadH1; k = 3 without kQuadH2) and H_2 (k = 3 with
// kQuadH2). Those rows are not stored: each is formed from the level below it,
//     H_0 = A_a0 + roll(B_b0, -sB),  H_1 = A_a1 + roll(B_b0, -(sB + 1)),
//     H_2 = A_a2 + roll(B_b2, -sB2),
//     T_0 = C_c0 + roll(D_d0, -(sD - sC)),  T_1 = C_c1 + roll(D_d0, -(sD - sC + 1)).
struct QuadOp {
    unsigned a01, b0a2, b2c0, c1d0;  // 16-bit row numbers of level d + 2, low half first
    unsigned sB;                     // sB | sB2 << 13
    unsigned sCD;                    // sC | sD << 13
    unsigned flags;                  // mask of valid rows | flags
    int out;
};
enum : unsigned {
    kQuadSameA = 16u,  // a1 = a0
    kQuadSameC = 32u,  // c1 = c0
    kQuadH1 = 64u,
    kQuadH2 = 128u,
};
static_assert(sizeof(GroupOp) == 16 && sizeof(QuadOp) == 32, "operations are read as 16-byte units");

// Source row numbers and shift of output row s of a node.
__device__ __forceinline__ void source_rows(const JobTree& T, const Node& nd, int s, int* h, int* t,
                                            int* shift)
{
    const int hs = T.regular ? head_row(nd, s) : merge_row(nd.kh, s);
    const int ts = T.regular ? group_of(nd.rows, s) : merge_row(merge_coef(nd.rows).kt, s);
    *shift = s - ts;
    *h = nd.hbias + hs;
    *t = nd.tbias + ts;
}

// x mod b by one multiply-high, `inv` = ceil(2^32 / b): exact while x b < 2^32 (the shifts of a
// transform of at most kRegularRows rows); x >= -1.
__device__ __forceinline__ int mod_bins(int x, int b, unsigned inv)
{
    if (x < 0) x += b;
    return x - (int)__umulhi((unsigned)x, inv) * b;
}

// Row group r of level d.
__device__ inline GroupOp make_group(const JobTree& T, int d, int r, int b, unsigned inv)
{
    const Node* lvl = T.nodes + (1 << d) - 1;
    int lo = 0, hi = (1 << d) - 1;  // node holding group r (nodes sorted by goff)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (lvl[mid].goff <= r) lo = mid;
        else hi = mid - 1;
    }
    const Node nd = lvl[lo];
    const int q = group_of(nd.rows, nd.lo) + (r - nd.goff);
    const int s0 = max(nd.lo, 2 * q - (nd.rows & 1));
    const int s1 = min(nd.hi - 1, 2 * q - (nd.rows & 1) + 1);
    GroupOp op;
    int h0, t0, sh0;
    source_rows(T, nd, s0, &h0, &t0, &sh0);
    sh0 = T.regular ? mod_bins(sh0, b, inv) : sh0 % b;
    op.out = nd.off + s0 - nd.lo;
    op.h = h0;
    op.t = t0;
    op.shift = sh0;
    if (s1 > s0) {
        int h1, t1, sh1;
        source_rows(T, nd, s1, &h1, &t1, &sh1);
        sh1 = T.regular ? mod_bins(sh1, b, inv) : sh1 % b;
        op.h |= h1 << 16;
        op.t |= t1 << 16;
        op.shift |= (sh1 << 13) | kOpTwo | (h1 == h0 ? kOpSameHead : 0) |
                    (t1 == t0 && sh1 == (sh0 + 1 == b ? 0 : sh0 + 1) ? kOpSameTail : 0);
    }
    return op;
}

// Row quad r of level d (over level d + 1, whose rows are not stored).
__device__ __forceinline__ QuadOp make_quad(const JobTree& T, int d, int r, int b, unsigned inv)
{
    const Node* lvl = T.nodes + (1 << d) - 1;
    int i = 0, hi = (1 << d) - 1;  // node holding quad r (nodes sorted by qoff)
    while (i < hi) {
        const int mid = (i + hi + 1) >> 1;
        if (lvl[mid].qoff <= r) i = mid;
        else hi = mid - 1;
    }
    const Node& N = lvl[i];
    const Node& Hn = T.nodes[(2 << d) - 1 + 2 * i];
    const Node& Tn = T.nodes[(2 << d) + 2 * i];
    const int p = N.rows & 1, pT = Tn.rows & 1;
    const int gid = group_of(Tn.rows, Tn.lo) + (r - N.qoff);   // tail row of T_0 and T_1
    const int t0 = 2 * gid - pT, s0 = 2 * t0 - p;              // T_0 and output row k = 0
    const int k0 = max(0, N.lo - s0), k1 = min(4, N.hi - s0);  // rows [k0, k1) are wanted
    const int hb = t0 - p;                                     // H_0
    const bool v0 = k0 == 0, v1 = k0 <= 1 && k1 > 1, v2 = k0 <= 2 && k1 > 2, v3 = k1 > 3;
    const bool h1 = v1 && p && 2 * t0 <= N.thr;      // k = 1 reads H_1: h(s0 + 1) = hb + 1
    const bool h2 = v3 && p && 2 * t0 + 2 <= N.thr;  // k = 3 reads H_2: h(s0 + 3) = hb + 2
    const bool need0 = v0 || (v1 && !h1), need1 = h1 || v2 || (v3 && !h2);
    // a row that nothing reads stands in for another, so that every row number is valid
    const int r0 = need0 ? hb : need1 ? hb + 1 : hb + 2;
    const int r1 = need1 ? hb + 1 : r0;
    const int r2 = h2 ? hb + 2 : r0;
    const int u0 = (v0 || v1) ? t0 : t0 + 1, u1 = (v2 || v3) ? t0 + 1 : t0;
    const int gB = group_of(Hn.rows, r0), gB2 = group_of(Hn.rows, r2);
    const int a0 = Hn.hbias + head_row(Hn, r0), a1 = Hn.hbias + head_row(Hn, r1);
    const int a2 = Hn.hbias + head_row(Hn, r2);
    const int c0 = Tn.hbias + head_row(Tn, u0), c1 = Tn.hbias + head_row(Tn, u1);
    QuadOp op;
    op.a01 = a0 | (a1 << 16);
    op.b0a2 = (Hn.tbias + gB) | (a2 << 16);
    op.b2c0 = (Hn.tbias + gB2) | (c0 << 16);
    op.c1d0 = c1 | ((Tn.tbias + gid) << 16);
    op.sB = mod_bins(hb - gB, b, inv) | (mod_bins(r2 - gB2, b, inv) << 13);
    op.sCD = mod_bins(s0 - t0, b, inv) | (mod_bins(s0 - gid, b, inv) << 13);
    op.flags = (v0 ? 1u : 0) | (v1 ? 2u : 0) | (v2 ? 4u : 0) | (v3 ? 8u : 0) |
               (a1 == a0 ? kQuadSameA : 0) | (c1 == c0 ? kQuadSameC : 0) | (h1 ? kQuadH1 : 0) |
               (h2 ? kQuadH2 : 0);
    op.out = N.off + s0 - N.lo;  // negative when row 0 is not wanted
    return op;
}

// Operations of all steps of the job, one thread per operation, dealt from the last thread down
// (the boxcar S/N of the search's previous job keeps the first warps longest). Call after
// build_job_tree_warp; the caller synchronises before using `ops`.
__device__ __forceinline__ void build_ops(const JobTree& T, int b, uint4* ops)
{
    const unsigned inv = 0xffffffffu / (unsigned)b + 1u;
    const int nsteps = T.nsteps;
    for (int g = kThreads - 1 - (int)threadIdx.x;; g += kThreads) {
        int r = g, k = 0;
        while (k < nsteps && r >= T.steps[k].count) r -= T.steps[k++].count;
        if (k >= nsteps) break;
        const Step st = T.steps[k];
        if (st.two)
            *reinterpret_cast<QuadOp*>(ops + st.unit + 2 * r) = make_quad(T, st.d, r, b, inv);
        else
            *reinterpret_cast<GroupOp*>(ops + st.unit + r) = make_group(T, st.d, r, b, inv);
    }
}

// a + b of two values at once: two round-to-nearest float32 additions
__device__ __forceinline__ void add2(float a0, float a1, float b0, float b1, float& s0, float& s1)
{
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
        " add.rn.f32x2 d, a, b;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(s0), "=f"(s1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// First column of a lane's window in a rolled row: (c0 + shift) mod b, for c0 < b + kHalo and
// shift < b (b >= kWideMinBins, so two subtractions are enough).
__device__ __forceinline__ int rolled_col(int c0, int shift, int b)
{
    const unsigned i = (unsigned)(c0 + shift);
    const unsigned j = min(i, i - (unsigned)b);
    return (int)min(j, j - (unsigned)b);
}

// Computes one level by row groups, from rows of stride `stride` with halo to rows of the same
// layout. A warp takes one group (two rows) at a time, or 32 / W groups when a row has at most
// W = 16 or 8 chunks; rows of more than 32 chunks are several warp tasks.
__device__ __forceinline__ void level_groups(const uint4* ops, int ngroups,
                                             const float* __restrict__ src,
                                             float* __restrict__ dst, int stride, int b)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = ffa_chunks(b);
    const int lw = nq <= 8 ? 3 : nq <= 16 ? 4 : 5;  // log2 of the lanes of a group
    const int nblk = (nq + 31) >> 5;
    const unsigned inv = (65536u + nblk - 1) / nblk;  // task / nblk: exact, task * nblk < 65536
    const int ntask = (ngroups * nblk + (32 >> lw) - 1) >> (5 - lw);
    const int sub = lane >> lw, ql = lane & ((1 << lw) - 1);
    for (int task = warp; task < ntask; task += kWarps) {
        int g = task, q = ql;
        if (nblk > 1) {
            g = (int)(((unsigned)task * inv) >> 16);
            q += 32 * (task - g * nblk);
        } else {
            g = (task << (5 - lw)) + sub;
        }
        if (q >= nq || g >= ngroups) continue;
        const uint4 v = ops[g];  // a GroupOp
        const int c0 = kLaneCols * q;
        const float* ph = src + (int)(v.x & 0xffff) * stride + c0;
        float* po = dst + (int)v.w * stride + c0;
        float H[kLaneCols], Tl[kLaneCols + 1];
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k) H[k] = ph[k];
        const float* pt = src + (int)(v.y & 0xffff) * stride + rolled_col(c0, v.z & 0x1fff, b);
#pragma unroll
        for (int k = 0; k <= kLaneCols; ++k) Tl[k] = pt[k];
#pragma unroll
        for (int k = 0; k + 1 < kLaneCols; k += 2) {
            float s0, s1;
            add2(H[k], H[k + 1], Tl[k], Tl[k + 1], s0, s1);
            po[k] = s0;
            po[k + 1] = s1;
        }
        po[kLaneCols - 1] = __fadd_rn(H[kLaneCols - 1], Tl[kLaneCols - 1]);
        if (!(v.z & kOpTwo)) continue;
        if (!(v.z & kOpSameHead)) {
            const float* ph1 = src + (int)(v.x >> 16) * stride + c0;
#pragma unroll
            for (int k = 0; k < kLaneCols; ++k) H[k] = ph1[k];
        }
        if (!(v.z & kOpSameTail)) {
            const float* pt1 =
                src + (int)(v.y >> 16) * stride + rolled_col(c0, (v.z >> 13) & 0x1fff, b);
#pragma unroll
            for (int k = 0; k < kLaneCols; ++k) Tl[k + 1] = pt1[k];
        }
        po += stride;
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k) po[k] = __fadd_rn(H[k], Tl[k + 1]);
    }
}

// Computes level d from level d + 2 by row quads, both of stride `stride` with halo: 42 reads
// and 36 writes of a lane for the 4 x 9 values of level d and the as many of level d + 1 that
// stay in registers (two passes of level_groups: 76 and 72).
__device__ __forceinline__ void level_quads(const uint4* ops, int nquads,
                                            const float* __restrict__ src,
                                            float* __restrict__ dst, int stride, int b)
{
    constexpr int K = kLaneCols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = ffa_chunks(b);
    const int lw = nq <= 8 ? 3 : nq <= 16 ? 4 : 5;  // log2 of the lanes of a quad
    const int nblk = (nq + 31) >> 5;
    const unsigned inv = (65536u + nblk - 1) / nblk;  // task / nblk: exact, task * nblk < 65536
    const int ntask = (nquads * nblk + (32 >> lw) - 1) >> (5 - lw);
    const int sub = lane >> lw, ql = lane & ((1 << lw) - 1);
    for (int task = warp; task < ntask; task += kWarps) {
        int g = task, q = ql;
        if (nblk > 1) {
            g = (int)(((unsigned)task * inv) >> 16);
            q += 32 * (task - g * nblk);
        } else {
            g = (task << (5 - lw)) + sub;
        }
        if (q >= nq || g >= nquads) continue;
        const uint4 v = ops[2 * g], w = ops[2 * g + 1];  // a QuadOp
        const int c0 = K * q;
        float T0[K + 1], T1[K + 1];
        {
            const float* pc = src + (int)(v.z >> 16) * stride + rolled_col(c0, w.y & 0x1fff, b);
            const float* pd =
                src + (int)(v.w >> 16) * stride + rolled_col(c0, (w.y >> 13) & 0x1fff, b);
            float C[K + 2], D[K + 3];
#pragma unroll
            for (int k = 0; k < K + 2; ++k) C[k] = pc[k];
#pragma unroll
            for (int k = 0; k < K + 3; ++k) D[k] = pd[k];
#pragma unroll
            for (int k = 0; k < K + 1; ++k) T0[k] = __fadd_rn(C[k], D[k]);
            if (!(w.z & kQuadSameC)) {
                pc += ((int)(v.w & 0xffff) - (int)(v.z >> 16)) * stride;
#pragma unroll
                for (int k = 0; k < K + 1; ++k) C[k + 1] = pc[k + 1];
            }
#pragma unroll
            for (int k = 0; k < K + 1; ++k) T1[k] = __fadd_rn(C[k + 1], D[k + 2]);
        }
        float H0[K], H1[K];
        {
            const float* pa = src + (int)(v.x & 0xffff) * stride + c0;
            const float* pb = src + (int)(v.y & 0xffff) * stride + rolled_col(c0, w.x & 0x1fff, b);
            float A[K], B[K + 1];
#pragma unroll
            for (int k = 0; k < K; ++k) A[k] = pa[k];
#pragma unroll
            for (int k = 0; k < K + 1; ++k) B[k] = pb[k];
#pragma unroll
            for (int k = 0; k < K; ++k) H0[k] = __fadd_rn(A[k], B[k]);
            if (!(w.z & kQuadSameA)) {
                pa += ((int)(v.x >> 16) - (int)(v.x & 0xffff)) * stride;
#pragma unroll
                for (int k = 0; k < K; ++k) A[k] = pa[k];
            }
#pragma unroll
            for (int k = 0; k < K; ++k) H1[k] = __fadd_rn(A[k], B[k + 1]);
        }
        float* po = dst + (int)w.w * stride + c0;
        if (w.z & 1u) {
#pragma unroll
            for (int k = 0; k < K; ++k) po[k] = __fadd_rn(H0[k], T0[k]);
        }
        po += stride;
        if (w.z & 2u) {
            if (w.z & kQuadH1) {
#pragma unroll
                for (int k = 0; k < K; ++k) H0[k] = H1[k];
            }
#pragma unroll
            for (int k = 0; k < K; ++k) po[k] = __fadd_rn(H0[k], T0[k + 1]);
        }
        po += stride;
        if (w.z & 4u) {
#pragma unroll
            for (int k = 0; k < K; ++k) po[k] = __fadd_rn(H1[k], T1[k]);
        }
        po += stride;
        if (w.z & 8u) {
            if (w.z & kQuadH2) {
                const float* pa = src + (int)(v.y >> 16) * stride + c0;
                const float* pb =
                    src + (int)(v.z & 0xffff) * stride + rolled_col(c0, (w.x >> 13) & 0x1fff, b);
#pragma unroll
                for (int k = 0; k < K; ++k) H1[k] = __fadd_rn(pa[k], pb[k]);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) po[k] = __fadd_rn(H1[k], T1[k + 1]);
        }
    }
}

// One level row by row with a modulo per column: any bins, any source (raw rows or rows with
// halo, shared or global memory, `sstride` apart). For what the other two loops do not take:
// fewer than kWideMinBins bins, whole subtrees of at most 4 rows, and stages whose source rows
// do not fit a level buffer.
__device__ __forceinline__ void level_rows_direct(const JobTree& T, int d, const float* src,
                                               size_t sstride, float* dst, int stride, int b)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Node* lvl = T.nodes + (1 << d) - 1;
    for (int r = warp; r < T.level_rows[d]; r += kWarps) {
        int lo = 0, hi = (1 << d) - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (lvl[mid].off <= r) lo = mid;
            else hi = mid - 1;
        }
        const Node nd = lvl[lo];
        float* out = dst + (size_t)r * stride;
        if (nd.rows == 1) {
            const int h = nd.hbias;
            for (int c = lane; c < b + kHalo; c += 32) out[c] = src[(size_t)h * sstride + c % b];
            continue;
        }
        int h, t, shift;
        source_rows(T, nd, nd.lo + (r - nd.off), &h, &t, &shift);
        const float *H = src + (size_t)h * sstride, *Tl = src + (size_t)t * sstride;
        for (int c = lane; c < b + kHalo; c += 32)
            out[c] = __fadd_rn(H[c % b], Tl[(c + shift) % b]);
    }
}

// Head and tail rows of output row s of a node of n <= 8 rows, as merge_row gives them: the
// rounded quotients s (n_child - 1) / (n - 1).
__host__ __device__ constexpr int small_row(int n, int child, int s)
{
    return n < 2 ? 0 : (2 * s * (child - 1) + (n - 1)) / (2 * (n - 1));
}

// The transform of N input rows on LEN consecutive columns, entirely in registers (the row and
// column numbers are compile-time constants; values nothing uses are never computed). off[j]:
// offset of column c0 + j (mod b) in a row.
template <int N, int LEN>
struct SmallNode {
    static __device__ __forceinline__ void run(const float* x, int b, const int* off,
                                               float (&o)[N][LEN])
    {
        constexpr int NH = N / 2, NT = N - NH;
        float H[NH][LEN], Tl[NT][LEN + NH];  // the largest shift s - t(s) is N - NT = NH
        SmallNode<NH, LEN>::run(x, b, off, H);
        SmallNode<NT, LEN + NH>::run(x + NH * b, b, off, Tl);
#pragma unroll
        for (int s = 0; s < N; ++s) {
#pragma unroll
            for (int j = 0; j < LEN; ++j)
                o[s][j] = __fadd_rn(H[small_row(N, NH, s)][j],
                                    Tl[small_row(N, NT, s)][j + s - small_row(N, NT, s)]);
        }
    }
};
template <int LEN>
struct SmallNode<1, LEN> {
    static __device__ __forceinline__ void run(const float* x, int, const int* off,
                                               float (&o)[1][LEN])
    {
#pragma unroll
        for (int j = 0; j < LEN; ++j) o[0][j] = x[off[j]];
    }
};

constexpr int kFusedWindow = kLaneCols + 7;  // columns a lane reads from the last of 8 rows

template <int N>
__device__ __forceinline__ void fused_node(const float* x, int b, const int* off, float* out,
                                           int stride)
{
    float o[N][kLaneCols];
    SmallNode<N, kLaneCols>::run(x, b, off, o);
#pragma unroll
    for (int s = 0; s < N; ++s) {
#pragma unroll
        for (int k = 0; k < kLaneCols; ++k) out[s * stride + k] = o[s][k];
    }
}

// Level T.depth of a fused job: a warp computes all rows of one node from its 4 to 8 raw input
// rows (row j of the transform at raw + j * b, no halo: a lane's window wraps at a column that
// is the same for every row, so one offset per window column serves all rows).
__device__ __forceinline__ void ffa_nodes_fused(const JobTree& T, const float* raw, float* dst,
                                                int stride, int b)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = ffa_chunks(b);
    const int lw = nq <= 8 ? 3 : nq <= 16 ? 4 : 5;
    const int nblk = (nq + 31) >> 5;
    const unsigned inv = (65536u + nblk - 1) / nblk;
    const int nnodes = 1 << T.depth;
    const int ntask = (nnodes * nblk + (32 >> lw) - 1) >> (5 - lw);
    const int sub = lane >> lw, ql = lane & ((1 << lw) - 1);
    const Node* lvl = T.nodes + nnodes - 1;
    for (int task = warp; task < ntask; task += kWarps) {
        int i = task, q = ql;
        if (nblk > 1) {
            i = (int)(((unsigned)task * inv) >> 16);
            q += 32 * (task - i * nblk);
        } else {
            i = (task << (5 - lw)) + sub;
        }
        if (q >= nq || i >= nnodes) continue;
        const int c0 = kLaneCols * q;
        const int w0 = c0 < b ? c0 : c0 - b;
        int off[kFusedWindow];
#pragma unroll
        for (int j = 0; j < kFusedWindow; ++j) off[j] = w0 + j - (w0 + j >= b ? b : 0);
        const float* x = raw + (size_t)lvl[i].row0 * b;
        float* out = dst + (size_t)lvl[i].off * stride + c0;
        switch (lvl[i].rows) {
            case 4: fused_node<4>(x, b, off, out, stride); break;
            case 5: fused_node<5>(x, b, off, out, stride); break;
            case 6: fused_node<6>(x, b, off, out, stride); break;
            case 7: fused_node<7>(x, b, off, out, stride); break;
            default: fused_node<8>(x, b, off, out, stride); break;
        }
    }
}

// Where a job's levels read.
struct LevelIO {
    const float* src = nullptr;     // global source: row j at src + j * src_stride (used when
    size_t src_stride = 0;          // nothing is staged)
    const float* staged = nullptr;  // source rows in shared memory
    bool staged_rows = false;       // staged: true = rows of the layout in JobTree::src_off
                                    // (stride = the level stride, with halo); false = raw row
                                    // j at staged + j * b
    uint64_t* bar = nullptr;        // staged by a bulk copy that completes on phase *phase of
    uint32_t* phase = nullptr;      // bar (null: already in place)
};

// Runs all levels of the job; the operations are built (build_ops) and the CTA synchronised.
// `src` is the level buffer that holds the staged source rows, `dst` the other one. Returns
// the one that holds the root rows [lo, hi) (stride `stride`, row i of the buffer = root output
// row lo + i). *ok is cleared if the wait for staged rows ran out.
__device__ inline float* run_job_levels(const JobTree& T, int b, float* src, float* dst,
                                        int stride, const uint4* ops, const LevelIO& io, bool* ok)
{
    if (io.bar) {
        *ok = mbar_wait(io.bar, *io.phase);
        *io.phase ^= 1u;
    }
    for (int d = T.depth; d > T.first_op; --d) {
        const bool first = d == T.depth;
        if (T.fused) {
            ffa_nodes_fused(T, io.staged, dst, stride, b);
        } else {
            const float* from = src;
            size_t fstride = stride;
            if (first && !io.staged) {
                from = io.src;
                fstride = io.src_stride;
            } else if (first && !io.staged_rows) {
                from = io.staged;
                fstride = b;
            }
            level_rows_direct(T, d, from, fstride, dst, stride, b);
        }
        cta_sync();
        float* x = src;
        src = dst;
        dst = x;
    }
    for (int k = 0; k < T.nsteps; ++k) {
        const Step st = T.steps[k];
        if (st.two)
            level_quads(ops + st.unit, st.count, src, dst, stride, b);
        else
            level_groups(ops + st.unit, st.count, src, dst, stride, b);
        cta_sync();
        float* x = src;
        src = dst;
        dst = x;
    }
    return src;
}

// Issued by one warp: bulk copies of the level-G source rows of a job laid out by
// build_job_tree_warp (pstaged), from a global source of 16-byte aligned rows of `stride`
// floats into `sbuf` (same stride), completing on `bar` (one arrival with the byte count). The
// caller has ordered the source's writes before the copies (fence.proxy.async.global).
__device__ inline void stage_source_rows_async(const JobTree& T, const float* src, int stride,
                                               float* sbuf, uint64_t* bar)
{
    const int lane = threadIdx.x & 31;
    const int n = 1 << T.depth;
    const size_t row_bytes = (size_t)stride * sizeof(float);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)(T.src_off[n] * row_bytes));
    __syncwarp();
    constexpr uint32_t kChunk = 32768;
    for (int i = lane; i < n; i += 32) {
        const int4 rg = T.src_rng[i];
        const int r0[2] = {rg.x, rg.z};
        const int cnt[2] = {rg.y, rg.w};
        int off = T.src_off[i];
        for (int h = 0; h < 2; ++h) {
            const unsigned char* from =
                reinterpret_cast<const unsigned char*>(src + (size_t)r0[h] * stride);
            unsigned char* to = reinterpret_cast<unsigned char*>(sbuf + (size_t)off * stride);
            const size_t bytes = (size_t)cnt[h] * row_bytes;
            for (size_t o = 0; o < bytes; o += kChunk) {
                const uint32_t nb = (uint32_t)(bytes - o < kChunk ? bytes - o : kChunk);
                bulk_g2s(to + o, from + o, nb, bar);
            }
            off += cnt[h];
        }
    }
}

// Shared-memory layout of a CTA running FFA jobs: [fixed part][operations][buffer][buffer].
// Operations (in 16-byte units) of a job whose levels hold at most cap_rows rows. A node with L
// rows wanted has at most L / 2 + 1 groups, and at most L / 2 + 1 rows wanted of its tail child
// (t(s) = group_of) and so L / 4 + 3 / 2 quads. Levels 5 .. 0 by three passes of quads (two
// units each) or by two and a single level: at most 3 cap_rows / 2 + 80 units; by single levels
// (more than kRegularRows rows): 6 (cap_rows / 2) + 63.
RT_HD int ffa_ops_units(int cap_rows, bool regular)
{
    return regular ? 3 * cap_rows / 2 + 80
                   : (kMaxTreeDepth + 1) * ((cap_rows + 1) / 2) + (2 << kMaxTreeDepth);
}

constexpr int kPadFloats = 256;

struct FfaLayout {
    int ops_units;     // room for operations, in 16-byte units
    int buf_floats;    // floats per level buffer (a multiple of 16)
};

// Layout of `bytes` of shared memory for transforms of at least bmin bins and at most max_rows
// rows: fixed by the smallest b, which has the most rows per level. `pad` floats stay free behind
// the second buffer, for what the boxcar S/N reads past the end of its last row (snr_overread).
RT_HD FfaLayout ffa_layout(size_t bytes, int bmin, size_t max_rows, int pad = kPadFloats)
{
    FfaLayout L;
    const int most = (int)(bytes / (2 * sizeof(float) * ffa_stride(bmin)));
    L.ops_units = (ffa_ops_units(most, max_rows <= (size_t)kRegularRows) + 3) & ~3;
    L.buf_floats = (int)((bytes - (size_t)L.ops_units * 16 - pad * sizeof(float)) /
                         (2 * sizeof(float))) & ~15;
    return L;
}

// Rows per level buffer.
RT_HD int ffa_cap_rows(const FfaLayout& L, int b) { return L.buf_floats / ffa_stride(b); }

// ------------------------------------------------------------------------------------
// Host-side planning of the stages of one transform.
//
// Stage 0 computes nodes at depth D[0] fully (full-depth jobs from the raw rows); stage k
// computes the needed rows of nodes at depth D[k] from the outputs of depth D[k-1]; the
// last stage has D = 0 (the root) and produces rows [0, rows_out).
// ------------------------------------------------------------------------------------
constexpr int kMaxStages = 6;

struct StagePlan {
    int nstages;
    int D[kMaxStages];      // node depth produced by each stage
    int R[kMaxStages];      // output rows per job (per node) of each stage
    int jobs[kMaxStages];   // number of jobs of each stage
    int jobs_per_node[kMaxStages];
};

// Plans the stages of a transform with m rows whose root output is [0, rows_out), for
// level buffers of cap_rows rows. Uses the bound: a job whose root range has R rows holds at
// most R + 3 * 2^G rows at any level (a child range of an L-row range has <= (L + 3) / 2
// rows, since kh, kt <= 1/2).
// max_depth: the largest depth G of a job (G + 1 levels computed in shared memory); smaller
// values cut deep transforms into more stages, whose outputs pass through L2.
// snr_rows: most rows of a last-stage job (0: no limit but cap_rows).
bool plan_stages(int m, int b, int rows_out, int cap_rows, int snr_rows, StagePlan* P,
                 int max_depth = kMaxJobDepth);
// Job k of stage s of a transform (host or device).
RT_HD void node_at(int m, int d, int i, int* row0, int* rows)
{
    int r0 = 0, rr = m;
    for (int k = d - 1; k >= 0; --k) {
        const int mh = rr >> 1;
        if ((i >> k) & 1) {
            r0 += mh;
            rr -= mh;
        } else {
            rr = mh;
        }
    }
    *row0 = r0;
    *rows = rr;
}

RT_HD JobSpec stage_job(int m, int rows_out, const StagePlan& P, int stage, int job)
{
    JobSpec J;
    const int d = P.D[stage];
    if (stage == 0) {
        int r0, rr;
        node_at(m, d, job, &r0, &rr);
        J.root_row0 = r0;
        J.root_rows = rr;
        J.lo = 0;
        J.hi = (P.nstages == 1) ? rows_out : rr;
        J.G = full_depth(rr);
        return J;
    }
    const int node = job / P.jobs_per_node[stage];
    const int part = job - node * P.jobs_per_node[stage];
    int r0, rr;
    node_at(m, d, node, &r0, &rr);
    const int hi_node = (stage == P.nstages - 1) ? rows_out : rr;
    J.root_row0 = r0;
    J.root_rows = rr;
    J.lo = part * P.R[stage];
    J.hi = J.lo + P.R[stage] < hi_node ? J.lo + P.R[stage] : hi_node;
    J.G = P.D[stage - 1] - d - 1;
    return J;
}

}  // namespace rt
