// mcd_analytic.cu -- analytic PMF propagation on the GPU (the reference's
// src/mc_dagprop/analytic/, pure Python there), behind the mcd_analytic_* C ABI.
//
// A PMF is (first value, probabilities) on the context's step grid.  Events are
// processed level by level (longest path from a source), two launches a level:
// k_an_conv computes every convolution of the level, its outputs split into
// one-warp chunks of 8 dealt out costliest first across the warps (the FP64
// multiply-adds are the bulk of the work);
// k_an_fold then takes one event per cluster of CTAs:
//   convolution along each incoming activity       _pmf.py:107-125
//   maximum over the predecessors, pairwise in      _pmf.py:127-148
//   precedence order, by cumulative products
//   mass correction after each operation            _pmf.py:82-105
//   clipping to the event's bounds under the        _propagator.py:150-265
//   underflow/overflow rules
// The reference accumulates convolutions and cumulative sums in np.longdouble;
// here they run in FP64 (fused multiply-adds, blocked scans), so results agree
// with the reference to rounding, not bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <deque>
#include <limits>
#include <string>
#include <type_traits>
#include <vector>

#include "mcd_handle.hpp"

namespace mcd {
namespace {

constexpr int kAnThreads = 128;   // threads of a fold CTA
constexpr int kAnCluster = 8;     // most CTAs of a fold cluster (one event)
constexpr int kAnGroup = 4;       // predecessors folded between two cluster barriers
// Outputs (and threads) per convolution chunk and CTA, and convolution CTAs per SM.
constexpr int kConvLanes = 4;                 // lanes per output
constexpr int kConvOuts = 32 / kConvLanes;    // outputs per chunk (one warp)
constexpr int kConvWarpsPerSm = 32;
constexpr int64_t kAnSmemBins = 1024;  // bins of a CTA's segment kept in shared memory (10 arrays, 80 KB)
constexpr int64_t kSparse = 4;  // an activity PMF with a non-zero bin in kSparse or fewer is read as those
constexpr int kAnArrays = 2 + 2 * kAnGroup;  // a segment's arrays: r, Q, a group's predecessors and their sums

// Kernel-reported errors (the reference raises ValueError in each case).
enum : int32_t {
    AN_ERR_UNDER_TRUNC = 1,   // underflow mass but no lower-bound bin (_propagator.py:192-193)
    AN_ERR_OVER_TRUNC = 2,    // overflow mass but no upper-bound bin (:203-205)
    AN_ERR_EMPTY = 4,         // nothing left after clipping (:229-232)
    AN_ERR_BOUNDS = 8,        // lower bound above upper bound (:163-164)
    AN_ERR_GRID = 16,         // operands that do not fit their common grid (misaligned values)
    AN_ERR_CAPACITY = 32,     // internal: a support larger than planned
};

struct AnEv {
    int32_t pred_begin, pred_end;  // predecessor entries, precedence order
    int64_t lower, upper;          // event bounds (_propagator.py:150-156)
    int64_t pool_off;              // output probabilities
    int32_t cap;                   // output capacity (bins)
    int32_t gmax;                  // grid bound of the event's intermediate PMFs
    int64_t scratch_off;           // global scratch slice (kAnArrays x segment a CTA), -1: shared memory
    int32_t user;                  // event index
    int32_t pad;
};

// One predecessor entry: what its convolution and its place in the fold need.
struct AnEntry {
    int64_t p_off;    // the source's probabilities in the pool
    int64_t q_off;    // the activity's in pmf_probs
    int64_t nz_off;   // sparse: its non-zero ones in nz_val, nz_idx
    int64_t out_off;  // the convolution in convbuf
    double q_first, q_mass;
    int32_t src;
    int32_t m;        // bins of the activity's PMF
    int32_t nnz;      // sparse: its non-zero bins, else 0
    int32_t pad;
};

struct AnOut {
    double first;
    double under, over;
    double mass;  // total probability of the event's PMF
    int32_t len;
    int32_t pad;
};

struct AnArgs {
    const AnEntry *entries;
    const double *pmf_probs;
    const double *nz_val;
    const int32_t *nz_idx;
    AnOut *out;
    double *pool;
    double *scratch;
    double *convbuf;          // the level's convolutions
    int32_t *err;
    int32_t step;
    int32_t urule, orule;
};

// A dependent FP64 instruction is some 75 clocks away (a warp's 32 lanes pass its SM
// sub-partition's FP64 unit in 64), an integer one a few, so decisions are taken on
// the bits where they can be.
__device__ __forceinline__ bool close12(double a, double b) {  // np.isclose(a, b, rtol=1e-12, atol=1e-15)
    return fabs(a - b) <= 1e-15 + 1e-12 * fabs(b);
}
constexpr long long kOneBits = 0x3FF0000000000000ll;
__device__ __forceinline__ bool positive(double a) {  // a > 0.0
    const long long b = __double_as_longlong(a);
    return b > 0 && b <= 0x7FF0000000000000ll;
}
__device__ __forceinline__ bool is_one(double a) { return __double_as_longlong(a) == kOneBits; }
// close12(a, 1.0): |a - 1| <= 1.001e-12, which is 4508 steps of 2^-52 above one and
// 9016 of 2^-53 below it (a - 1 is exact there).
__device__ __forceinline__ bool near_one(double a) {
    const long long d = __double_as_longlong(a) - kOneBits;
    return d >= -9016 && d <= 4508;
}
__device__ __forceinline__ bool close_default(double a, double b) {  // np.isclose defaults
    return fabs(a - b) <= 1e-8 + 1e-5 * fabs(b);
}
__device__ __forceinline__ double expected_mass(double m1, double m2) {  // _pmf.py:96-105
    return (near_one(m1) && near_one(m2)) ? 1.0 : m1 * m2;
}

constexpr int kAnWarps = kAnThreads / 32;

// ---- thread-block clusters
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Every thread of every CTA of the cluster; shared-memory writes before it, remote
// ones too, are seen after it.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Stores v at p's place in the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ void put_remote(double *p, uint32_t rank, double v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ int64_t round_half_even(double x) { return (int64_t)rint(x); }

// Length of the convolution of a pred PMF of n entries with an activity PMF of m.
__device__ __forceinline__ int64_t conv_len(int64_t n, int64_t m) { return n == 1 ? m : (m == 1 ? n : n + m - 1); }

// One chunk of kConvOuts outputs of one convolution (predecessor entry c.x, chunk
// index c.y), computed by one warp: kConvLanes lanes per output split its terms
// and add their partial sums with shuffles.  A warp's FP64 multiply-adds issue at
// the SM sub-partition's FP64 rate (a warp instruction per 64 clocks), so chunks
// are kept small: the last chunks of a level then finish soon after the others.
// Operands are read through the L1 cache (every chunk of a convolution reads the
// same activity PMF and overlapping windows of the predecessor's).  An activity
// PMF most of whose bins are zero (empirical values on a fine grid) is read as its
// non-zero bins: the terms left out are exact zeros.
__device__ void conv_chunk(const AnArgs &A, int2 c) {
    const AnEntry &t = A.entries[c.x];
    const int64_t n = A.out[t.src].len, m = t.m;
    const int lane = threadIdx.x & 31, sub = lane % kConvLanes;
    const int64_t len = conv_len(n, m), j = (int64_t)c.y * kConvOuts + lane / kConvLanes;
    const double *p = A.pool + t.p_off, *q = A.pmf_probs + t.q_off;
    double *out = A.convbuf + t.out_off;
    if (n == 1 || m == 1) {  // the reference's scaled copies (_pmf.py:111-116)
        if (j < len && sub == 0) out[j] = n == 1 ? __ldg(q + j) * __ldg(p) : __ldg(p + j) * __ldg(q);
        return;
    }
    double acc = 0.0;
    if (t.nnz) {
        const int32_t *idx = A.nz_idx + t.nz_off;
        const double *val = A.nz_val + t.nz_off;
        for (int k = sub; k < t.nnz; k += kConvLanes) {
            const int64_t i = j - __ldg(idx + k);
            if (i >= 0 && i < n) acc = fma(__ldg(p + i), __ldg(val + k), acc);
        }
    } else if (j < len) {
        const int64_t i0 = j - (m - 1) > 0 ? j - (m - 1) : 0, i1 = j < n - 1 ? j : n - 1;
        for (int64_t i = i0 + sub; i <= i1; i += kConvLanes) acc = fma(__ldg(p + i), __ldg(q + (j - i)), acc);
    }
#pragma unroll
    for (int o = 1; o < kConvLanes; o <<= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if (j < len && sub == 0) out[j] = acc;
}

// Every convolution of a level.  A level's chunks differ in cost (a chunk at a
// convolution's edge has few terms); the host lists them costliest first and each
// warp takes every gridDim.x-th, so the warps' loads come out nearly equal without
// a shared counter (one counter's atomics serialise at its L2 slice).
__global__ void __launch_bounds__(32) k_an_conv(const AnArgs A, const int2 *__restrict__ chunks, int32_t n_chunks) {
    for (int32_t ci = blockIdx.x; ci < n_chunks; ci += gridDim.x) conv_chunk(A, chunks[ci]);
}

// Where the predecessors' convolutions lie on the event's grid.  The reference
// places the running maximum and the next convolution on np.arange(min start, max
// end + step, step), each start rounded to it (_pmf.py:129-134); `next` takes one
// entry: its place in the grid so far extended by it, and by how much the grid's
// start moved down (every earlier entry lies that much further up).  Starts that
// are integers a whole number of steps apart need no FP64 (whole, ifirst).
struct AnGrid {
    double first;    // grid start, unless exact
    int64_t ifirst;  // grid start, if exact
    int64_t n;       // grid points
    int32_t step;
    bool exact;      // every start so far is an integer
    static __device__ bool whole(double f) { return fabs(f) < 9.0e15 && (double)(int64_t)f == f; }
    __device__ void start(double f, int64_t fi, bool is_whole, int64_t len, int32_t s) {
        first = f;
        ifirst = fi;
        exact = is_whole;
        n = len;
        step = s;
    }
    __device__ double begin() const { return exact ? (double)ifirst : first; }
    __device__ bool next(double f, int64_t fi, bool is_whole, int64_t len, int64_t *at, int64_t *moved) {
        if (exact && is_whole) {
            const int64_t d = fi - ifirst, k = step == 1 ? d : d / step;
            if (k * step == d) {
                *at = k > 0 ? k : 0;
                *moved = k < 0 ? -k : 0;
                const int64_t a = *moved + n, b = *at + len;
                n = a > b ? a : b;
                ifirst = k < 0 ? fi : ifirst;
                return true;
            }
        }
        first = begin();
        exact = false;
        const double st = (double)step, lo = fmin(first, f);
        const double hi = fmax(first + st * (double)(n - 1), f + st * (double)(len - 1));
        const int64_t m = (int64_t)ceil((hi + st - lo) / st);
        *moved = round_half_even((first - lo) / st);
        *at = round_half_even((f - lo) / st);
        const bool fits = *moved + n <= m && *at + len <= m;
        first = lo;
        n = m;
        return fits;
    }
};

// What the fold of an event starts from, in one read: the event and its first
// predecessor entries.
struct AnFold {
    AnEv ev;
    AnEntry first[kAnGroup];
};

// What the clipping of an event decides, once per CTA.
struct AnClip {
    double u, o;              // mass reported below and above
    double add_lo, add_hi;    // mass put on the first and last kept bin
    double div, mul;          // every kept value v becomes v / div * mul, or (div 0) v + v * mul
    double single_v, single_p;  // single: one value instead of the kept range
    double mass;
    int32_t single, status;   // status: error flag, 0 for none
};

// The flow rules (_propagator.py:158-265) on the masses below (u), inside (kept) and
// above (o) of a PMF with nk bins kept; at_lower, at_upper: the first and last kept
// bin lie on the bounds.  The kept values' common factor is seldom other than one but
// for rounding, and then taken as its difference from one: rounded to a double it is off
// by up to half a unit the same way for every value (1,000 events: error against 64-bit
// arithmetic 6.0e-17, this way 3.0e-17, as with a division a value).  Where it is another
// it is applied as a division and a product, which hold for kept masses whose reciprocal
// is no double.
__device__ AnClip clip_rules(int urule, int orule, double u, double kept, double o, int64_t nk, bool at_lower,
                             bool at_upper, double lower, double upper) {
    AnClip c{};
    double redist = 0.0;
    if (urule == MCD_RULE_TRUNCATE && positive(u)) {
        if (nk > 0 && at_lower) {
            c.add_lo = u;
        } else if (nk == 0) {
            c.single = 1;
            c.single_v = lower;
            c.single_p = u;
        } else {
            c.status = AN_ERR_UNDER_TRUNC;
            return c;
        }
        u = 0.0;
    } else if (urule == MCD_RULE_REDISTRIBUTE && positive(u)) {
        redist += u;
        u = 0.0;
    }
    if (orule == MCD_RULE_TRUNCATE && positive(o)) {
        const bool any = c.single || nk > 0;
        if (any && (c.single ? close_default(c.single_v, upper) : at_upper)) {
            if (c.single) c.single_p += o;
            else c.add_hi = o;
        } else if (!any) {
            c.single = 1;
            c.single_v = upper;
            c.single_p = o;
        } else {
            c.status = AN_ERR_OVER_TRUNC;
            return c;
        }
        o = 0.0;
    } else if (orule == MCD_RULE_REDISTRIBUTE && positive(o)) {
        redist += o;
        o = 0.0;
    }
    double inside = c.single ? c.single_p : (kept + c.add_lo) + c.add_hi;
    c.div = inside;  // (what is spread over the kept values is so in proportion to them)
    if (positive(redist)) {
        if (inside == 0.0) {
            c.single = 1;
            c.single_v = lower;
            c.single_p = redist;
        }
        inside += redist;
    }
    if (!c.single && nk == 0) {
        c.status = AN_ERR_EMPTY;
        return c;
    }
    const bool outside = __double_as_longlong(u) != 0 || __double_as_longlong(o) != 0;
    const double target = outside ? fmax(0.0, 1.0 - (u + o)) : 1.0;
    c.mass = inside;
    c.mul = target;
    if (positive(inside)) {
        if (is_one(target) && near_one(c.div)) {  // (1 / (1 + d) = 1 - d to rounding)
            c.mul = 1.0 - c.div;
            c.div = 0.0;
        } else if (fabs(target - c.div) <= 1e-12 * c.div) {
            c.mul = (target - c.div) / c.div;
            c.div = 0.0;
        }
        c.mass = c.single_p = target;
    } else if (positive(target)) {
        c.single = 1;
        c.single_v = lower;
        c.mass = c.single_p = target;
    } else {
        c.div = c.mul = 1.0;
    }
    const double all = outside ? c.mass + u + o : c.mass;
    if (!is_one(all) && !near_one(all) && positive(all)) {  // (the kept values are then zeros, or as they were)
        const double corr = 1.0 / all;
        c.mul *= corr;
        c.single_p *= corr;
        c.mass *= corr;
    }
    c.u = u;
    c.o = o;
    return c;
}

// One event a cluster of CTAs.  The fold is a chain of dependent steps, so it is cut
// to as few as it can be: the cumulative sum of a maximum is the product of its
// operands' cumulative sums, and its mass the product of their masses, so only the
// convolutions are scanned -- up to kAnGroup of them at once -- and the maximum
// itself is elementwise,
//   r(x) <- r(x) C(x) + c(x) R(x - 1),   R(x - 1) <- R(x - 1) C(x - 1),
// every correction of mass a common factor.  Each CTA holds a segment of the grid,
// a thread a few consecutive bins of it; what crosses CTAs are the segments' sums
// (distributed shared memory, one cluster barrier a group of predecessors and one
// for the clipping).  The FP64 pipe (2 lanes per clock and SM) makes block-wide
// sums dear -- a shuffle tree costs five full instructions a warp -- so a sum is one
// partial a thread, summed by one warp.
// A level of 20 events with up to 4 predecessors of 900 bins: 10-13 us (one CTA an
// event, every sum and scan block-wide: 54 us); the 1,000-event network of such
// levels 2.92 -> 1.18 ms, a 60-event line 395 -> 148 us.
__global__ void __launch_bounds__(kAnThreads) k_an_fold(const AnArgs A, const AnFold *__restrict__ level_ev) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double s_first[kAnThreads], s_expct[kAnThreads];
    __shared__ int64_t s_ifirst[kAnThreads], s_len[kAnThreads], s_off[kAnThreads];
    __shared__ bool s_whole[kAnThreads];
    __shared__ double cta_tot[2][kAnGroup][kAnCluster];  // [parity]: every CTA's segment sums, written by it
    __shared__ double g_below[kAnGroup];                 // mass below this CTA's segment
    __shared__ double g_fc[kAnGroup], g_fr[kAnGroup];    // corrections of mass
    __shared__ bool g_scaled;
    __shared__ double part[3][kAnThreads];
    __shared__ double clip_tot[3][kAnCluster];
    __shared__ AnClip clip;
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_rank(), NC = cluster_size();
    const AnFold &rec = level_ev[blockIdx.x / NC];
    AnEntry mine;  // (read beside the event)
    if (tid < kAnGroup) mine = rec.first[tid];
    const AnEv ev = rec.ev;
    const int64_t G = ev.gmax;
    const int np = ev.pred_end - ev.pred_begin;
    // (every CTA of the cluster takes the same decisions from the same values, so all
    // of them return at a failure, or none)
#define fail(code)                                          \
    do {                                                    \
        if (tid == 0 && rank == 0) atomicOr(A.err, (code)); \
    } while (0)

    // entries [base, base + kAnThreads) into shared memory
    auto load_entries = [&](int base) {
        __syncthreads();
        if (base + tid < np) {
            if (base + tid >= kAnGroup) mine = A.entries[ev.pred_begin + base + tid];
            else if (np > kAnThreads) mine = rec.first[tid];
            const AnOut ps = A.out[mine.src];
            const double f = ps.first + mine.q_first;
            s_first[tid] = f;
            s_whole[tid] = AnGrid::whole(f);
            s_ifirst[tid] = s_whole[tid] ? (int64_t)f : 0;
            s_len[tid] = conv_len(ps.len, mine.m);
            s_off[tid] = mine.out_off;
            s_expct[tid] = expected_mass(ps.mass, mine.q_mass);
        }
        __syncthreads();
    };
    // entry k (in shared memory at k % kAnThreads) onto the grid
    auto place = [&](AnGrid &g, int k, int64_t *at, int64_t *moved) {
        const int t = k % kAnThreads;
        *at = *moved = 0;
        if (k == 0) {
            g.start(s_first[t], s_ifirst[t], s_whole[t], s_len[t], A.step);
            return true;
        }
        return g.next(s_first[t], s_ifirst[t], s_whole[t], s_len[t], at, moved);
    };

    // ---- the event's grid
    AnGrid grid;
    int64_t shift = 0;  // how far entry 0 lies up the final grid
    for (int base = 0; base < np; base += kAnThreads) {
        load_entries(base);
        if (base == 0)  // every CTA of the cluster runs before any writes into another
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        for (int k = base; k < np && k < base + kAnThreads; ++k) {
            int64_t at, moved;
            const bool fits = place(grid, k, &at, &moved);
            shift += moved;
            if (grid.n > G || !fits) {
                fail(grid.n > G ? AN_ERR_CAPACITY : AN_ERR_GRID);
                return;
            }
        }
    }
    const int64_t n = grid.n;
    // This CTA's segment of the grid, bins [b0, b0 + bins).  Elementwise steps take bin
    // i on thread i % kAnThreads; a scan takes one warp a predecessor, a lane the
    // `per` bins from lane * per on.  (An odd `per` keeps the lanes' bins in different
    // shared-memory banks.)
    const int64_t seg = (n + NC - 1) / NC, b0 = (int64_t)rank * seg;
    const int bins = (int)(b0 >= n ? 0 : b0 + seg < n ? seg : n - b0);
    const int per = (int)(((seg + 31) / 32) | 1), room = per * 32;  // room: of each array
    double *arrays = ev.scratch_off >= 0 ? A.scratch + ev.scratch_off + (int64_t)rank * kAnArrays * room : sm;
    double *r = arrays, *Q = r + room, *C = Q + room, *S = C + kAnGroup * room;  // C, S: [predecessor of the group][room]

    // ---- the maximum over the predecessors
    double mR = 0.0;  // mass of the maximum so far (warp 0)
    AnGrid walk;
    int64_t below = shift;  // how far the entries so far lie up the final grid
    int parity = 0;
    for (int g0 = 0; g0 < np; g0 += kAnGroup, parity ^= 1) {
        if (np > kAnThreads && g0 % kAnThreads == 0) load_entries(g0);
        const int gn = np - g0 < kAnGroup ? np - g0 : kAnGroup;
        int64_t pos = 0;  // where entry g0 + warp begins on the final grid
        for (int k = 0; k < gn; ++k) {
            int64_t at, moved;
            place(walk, g0 + k, &at, &moved);
            below -= moved;
            if (k == warp) pos = at + below;
        }
        if (warp < gn) {
            const int t = (g0 + warp) % kAnThreads;
            const int64_t lo = pos - b0, hi = lo + s_len[t];
            const double *conv = A.convbuf + s_off[t] - lo;
            double *c = C + warp * room, *cum = S + warp * room;
            for (int i = lane; i < room; i += 32) c[i] = i < bins && i >= lo && i < hi ? conv[i] : 0.0;
            __syncwarp();
            double sum = 0.0;
            for (int i = lane * per; i < lane * per + per; ++i) {
                cum[i] = sum;
                sum += c[i];
            }
            double incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += u;
            }
            const double up = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
            if (lane)
                for (int i = lane * per; i < lane * per + per; ++i) cum[i] += up;
            const double total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            if (lane < (int)NC) put_remote(&cta_tot[parity][warp][rank], lane, total);
        }
        cluster_barrier();
        if (warp == 0) {
            // lane (k, j): entry k's mass up to CTA j
            const int k = lane / kAnCluster, j = lane % kAnCluster;
            double upto = k < gn && j < (int)NC ? cta_tot[parity][k][j] : 0.0;
#pragma unroll
            for (int o = 1; o < kAnCluster; o <<= 1) {
                const double u = __shfl_up_sync(0xFFFFFFFFu, upto, o);
                if (j >= o) upto += u;
            }
            const double tot = __shfl_sync(0xFFFFFFFFu, upto, k * kAnCluster + kAnCluster - 1);
            const double off = __shfl_sync(0xFFFFFFFFu, upto, k * kAnCluster + (rank ? rank - 1 : 0));
            // the convolution's mass corrected to its expected value ...
            double mass = tot, fc = 1.0;
            if (k < gn) {
                const double expct = s_expct[(g0 + k) % kAnThreads];
                if (is_one(expct) ? !near_one(tot) : !close12(tot, expct)) {
                    if (tot > 0.0) {
                        fc = expct / tot;
                        mass = tot * fc;
                    }
                }
            }
            // ... and the maximum's: 1 where both operands' are, else their product, which
            // is what it has
            double fr = 1.0;
#pragma unroll
            for (int q = 0; q < kAnGroup; ++q) {
                const double m = __shfl_sync(0xFFFFFFFFu, mass, q * kAnCluster);
                if (q >= gn) continue;
                if (g0 + q == 0) {
                    mR = m;
                    continue;
                }
                const bool both_one = near_one(m) && near_one(mR);
                mR *= m;
                if (both_one && !near_one(mR)) {
                    const double f = 1.0 / mR;
                    mR *= f;
                    if (k == q) fr = f;
                }
            }
            if (j == 0 && k < gn) {
                g_below[k] = rank ? off : 0.0;
                g_fc[k] = fc;
                g_fr[k] = fr;
            }
            const bool scaled = __any_sync(0xFFFFFFFFu, !is_one(fc) || !is_one(fr));
            if (lane == 0) g_scaled = scaled;
        }
        __syncthreads();
        // r(x) <- r(x) C(x) + c(x) R(x - 1), R(x - 1) <- R(x - 1) C(x - 1)
        auto combine = [&](auto corrected) {
            for (int i = tid; i < bins; i += kAnThreads) {
                double v = 0.0, q = 0.0;
                if (g0) {
                    v = r[i];
                    q = Q[i];
                }
#pragma unroll
                for (int k = 0; k < kAnGroup; ++k) {
                    if (k >= gn) continue;
                    double c = C[k * room + i], lower = S[k * room + i] + g_below[k], upper = lower + c;
                    if (corrected.value) {
                        c *= g_fc[k];
                        lower *= g_fc[k];
                        upper *= g_fc[k];
                    }
                    if (g0 + k == 0) {
                        v = c;
                        q = lower;
                    } else {
                        v = fma(v, upper, c * q);
                        q *= lower;
                    }
                    if (corrected.value) {
                        v *= g_fr[k];
                        q *= g_fr[k];
                    }
                }
                r[i] = v;
                Q[i] = q;
            }
        };
        if (g_scaled) combine(std::true_type{});
        else combine(std::false_type{});
        if (g0 + kAnGroup < np) __syncthreads();  // this group's shared values are read before the next writes them
    }

    // ---- clipping to [lower, upper]; every thread touches only its own bins
    if (ev.lower > ev.upper) {
        fail(AN_ERR_BOUNDS);
        return;
    }
    int64_t ka, kb;
    const bool unit = grid.exact && A.step == 1;
    if (unit) {
        ka = ev.lower - grid.ifirst;
        kb = ev.upper - grid.ifirst + 1;
    } else {
        ka = (int64_t)ceil(((double)ev.lower - grid.begin()) / (double)A.step);
        kb = (int64_t)floor(((double)ev.upper - grid.begin()) / (double)A.step) + 1;
    }
    ka = ka < 0 ? 0 : (ka > n ? n : ka);
    kb = kb > n ? n : (kb < ka ? ka : kb);
    const double lower = (double)ev.lower, upper = (double)ev.upper, fX = grid.begin(), step = (double)A.step;
    const bool at_lower = (unit && grid.ifirst + ka == ev.lower) || close_default(fX + step * (double)ka, lower);
    const bool at_upper = (unit && grid.ifirst + kb - 1 == ev.upper) || close_default(fX + step * (double)(kb - 1), upper);
    const double first_kept = fX + step * (double)ka;
    {
        double s[3] = {0.0, 0.0, 0.0};  // mass below, inside, above
        for (int i = tid; i < bins; i += kAnThreads) {
            const double v = r[i];
            if (b0 + i < ka) s[0] += v;
            else if (b0 + i < kb) s[1] += v;
            else s[2] += v;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) part[q][tid] = s[q];
    }
    __syncthreads();
    if (warp < 3) {
        static_assert(kAnWarps == 4 && kAnGroup == 4, "a lane's four partial sums");
        double t = (part[warp][lane] + part[warp][32 + lane]) + (part[warp][64 + lane] + part[warp][96 + lane]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, d);
        if (lane < (int)NC) put_remote(&clip_tot[warp][rank], lane, t);
    }
    cluster_barrier();
    if (warp == 0) {
        // lane (q, j): the mass below, inside and above of CTA j, summed over the CTAs
        const int q = lane / kAnCluster, j = lane % kAnCluster;
        double t = q < 3 && j < (int)NC ? clip_tot[q][j] : 0.0;
#pragma unroll
        for (int d = 1; d < kAnCluster; d <<= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, d);
        const double u = __shfl_sync(0xFFFFFFFFu, t, 0), kept = __shfl_sync(0xFFFFFFFFu, t, kAnCluster),
                     over = __shfl_sync(0xFFFFFFFFu, t, 2 * kAnCluster);
        if (lane == 0) {
            clip = clip_rules(A.urule, A.orule, u, kept, over, kb - ka, at_lower, at_upper, lower, upper);
        }
    }
    __syncthreads();
    if (clip.status) {
        fail(clip.status);
        return;
    }
    // ---- output
    const bool single = clip.single != 0;
    const int64_t len = single ? 1 : kb - ka;
    if (len > ev.cap) {
        fail(AN_ERR_CAPACITY);
        return;
    }
    double *dst = A.pool + ev.pool_off;
    if (!single)
        for (int i = tid; i < bins; i += kAnThreads) {
            const int64_t x = b0 + i;
            if (x < ka || x >= kb) continue;
            double v = r[i];
            if (x == ka) v += clip.add_lo;
            if (x == kb - 1) v += clip.add_hi;
            dst[x - ka] = clip.div == 0.0 ? fma(v, clip.mul, v) : v / clip.div * clip.mul;
        }
    if (tid == 0 && rank == 0) {
        if (single) dst[0] = clip.single_p;
        AnOut w;
        w.first = single ? clip.single_v : first_kept;
        w.under = clip.u;
        w.over = clip.o;
        w.mass = clip.mass;
        w.len = (int32_t)len;
        w.pad = 0;
        A.out[ev.user] = w;
    }
#undef fail
}

}  // namespace
}  // namespace mcd

using namespace mcd;

struct mcd_analytic {
    int device = 0;
    cudaStream_t stream = nullptr;
    int32_t E = 0;
    AnArgs args{};
    std::vector<int32_t> level_off;    // non-origin levels: events level_ev[level_off[l] .. level_off[l+1])
    std::vector<int32_t> level_smem;   // dynamic shared memory per fold launch (bytes)
    std::vector<int32_t> level_ctas;   // CTAs per event (cluster size) of each fold launch
    std::vector<int32_t> chunk_off;    // convolution chunks of each level: chunks[chunk_off[l] .. chunk_off[l+1])
    AnFold *d_level_ev = nullptr;
    int2 *d_chunks = nullptr;
    cudaGraphExec_t graph = nullptr;   // every level's two launches
    const AnEv *d_ev = nullptr;        // [E], by event
    char *dmem = nullptr;
    int64_t bins = 0;                  // output pool size
    bool ran = false;
};

namespace {

int64_t py_round(double x) { return (int64_t)std::nearbyint(x); }  // half to even, as Python and numpy round

}  // namespace

extern "C" {

int mcd_analytic_create(const mcd_analytic_desc *d, mcd_analytic **out) {
    mcd_analytic *an = nullptr;
    const int rc = guarded([&] {
        if (!d || !out) throw McdError(MCD_ERR_INVALID, "null argument");
        *out = nullptr;
        const int32_t E = d->n_events, K = d->n_pmfs, T = d->n_targets;
        if (E < 0 || K < 0 || T < 0) throw McdError(MCD_ERR_INVALID, "negative array length");
        if (d->step <= 0) throw McdError(MCD_ERR_INVALID, "step_size must be positive");
        if (!(d->max_delay >= 0.0) && !std::isnan(d->max_delay))
            throw McdError(MCD_ERR_INVALID, "max_delay must be non-negative when provided");
        if (d->underflow_rule < 1 || d->underflow_rule > 3 || d->overflow_rule < 1 || d->overflow_rule > 3)
            throw McdError(MCD_ERR_INVALID, "unknown underflow/overflow rule");
        const int64_t P = T > 0 ? d->pred_off[T] : 0;
        if (d->pmf_off[0] != 0) throw McdError(MCD_ERR_INVALID, "pmf_off must start at 0");
        for (int32_t k = 0; k < K; ++k)
            if (d->pmf_off[k + 1] <= d->pmf_off[k]) throw McdError(MCD_ERR_INVALID, "PMF values cannot be empty");
        // predecessors by target, precedence order
        std::vector<int64_t> tstart((size_t)E, -1), tlen((size_t)E, 0);
        for (int32_t t = 0; t < T; ++t) {
            const int32_t tg = d->target[t];
            if (tg < 0 || tg >= E) throw McdError(MCD_ERR_INVALID, "target index out of range");
            if (tstart[tg] != -1) throw McdError(MCD_ERR_INVALID, "precedence_list names a target twice");
            tstart[tg] = d->pred_off[t];
            tlen[tg] = d->pred_off[t + 1] - d->pred_off[t];
            if (tlen[tg] < 0) throw McdError(MCD_ERR_INVALID, "pred_off must be non-decreasing");
            for (int64_t p = d->pred_off[t]; p < d->pred_off[t + 1]; ++p) {
                if (d->pred_src[p] < 0 || d->pred_src[p] >= E)
                    throw McdError(MCD_ERR_INVALID, "predecessor index out of range");
                if (d->pred_pmf[p] < 0 || d->pred_pmf[p] >= K)
                    throw McdError(MCD_ERR_INVALID, "missing activity for a predecessor entry");
            }
        }
        // Kahn order with levels (longest path from a source)
        std::vector<std::vector<int32_t>> adj((size_t)E);
        std::vector<int64_t> indeg(tlen);
        for (int32_t e = 0; e < E; ++e)
            for (int64_t k = 0; k < tlen[e]; ++k) adj[d->pred_src[tstart[e] + k]].push_back(e);
        std::vector<int32_t> level((size_t)E, 0), order;
        order.reserve((size_t)E);
        std::deque<int32_t> q;
        for (int32_t e = 0; e < E; ++e)
            if (indeg[e] == 0) q.push_back(e);
        while (!q.empty()) {
            const int32_t v = q.front();
            q.pop_front();
            order.push_back(v);
            for (int32_t w : adj[v]) {
                level[w] = std::max(level[w], level[v] + 1);
                if (--indeg[w] == 0) q.push_back(w);
            }
        }
        if ((int64_t)order.size() != E) throw McdError(MCD_ERR_RUNTIME, "Invalid DAG: cycle detected");

        // plan: bounds, value ranges of every event's PMF, grid bounds, pool offsets
        const double step = (double)d->step;
        std::vector<AnEv> ev((size_t)E);
        std::vector<double> vlo((size_t)E), vhi((size_t)E);  // value range of each event's PMF
        std::vector<double> pmf_mass((size_t)K), pmf_last((size_t)K);
        for (int32_t k = 0; k < K; ++k) {
            double s = 0.0;
            for (int64_t i = d->pmf_off[k]; i < d->pmf_off[k + 1]; ++i) s += d->pmf_probs[i];
            pmf_mass[k] = s;
            pmf_last[k] = d->pmf_first[k] + step * (double)(d->pmf_off[k + 1] - d->pmf_off[k] - 1);
        }
        std::vector<AnOut> init((size_t)E);
        int64_t pool = 0;
        for (int32_t e : order) {
            AnEv &r = ev[e];
            r.pred_begin = (int32_t)(tlen[e] > 0 ? tstart[e] : 0);
            r.pred_end = (int32_t)(tlen[e] > 0 ? tstart[e] + tlen[e] : 0);
            r.scratch_off = -1;
            r.user = e;
            r.pad = 0;
            if (tlen[e] == 0) {  // origin: a unit mass at the rounded earliest time (_propagator.py:105-111)
                const double v = (double)py_round(d->earliest[e] / step) * step;
                vlo[e] = vhi[e] = v;
                r.lower = r.upper = 0;
                r.cap = 1;
                r.gmax = 1;
                r.pool_off = pool;
                pool += 1;
                init[e] = AnOut{v, 0.0, 0.0, 1.0, 1, 0};
                continue;
            }
            const double lat = d->latest[e], ear = d->earliest[e];
            const double up = std::isnan(d->max_delay) ? lat : std::min(lat, ear + d->max_delay);
            r.lower = py_round(ear);
            r.upper = py_round(up);
            double glo = std::numeric_limits<double>::infinity(), ghi = -glo;
            for (int64_t p = tstart[e]; p < tstart[e] + tlen[e]; ++p) {
                const int32_t s = d->pred_src[p], k = d->pred_pmf[p];
                glo = std::min(glo, vlo[s] + d->pmf_first[k]);
                ghi = std::max(ghi, vhi[s] + pmf_last[k]);
            }
            const double span = std::floor((ghi - glo) / step) + 3.0;  // + grid rounding margin
            if (!(span < 2.0e9)) throw McdError(MCD_ERR_INVALID, "an event's PMF grid is too large");
            r.gmax = (int32_t)span;
            const double win = (double)(r.upper - r.lower);
            const double capd = win >= 0.0 ? std::floor(win / step) + 1.0 : 1.0;
            r.cap = (int32_t)std::max(1.0, std::min(capd, span));
            r.pool_off = pool;
            pool += r.cap;
            // the clipped PMF lies in [lower, upper] (a kept range or one bound value)
            vlo[e] = (double)r.lower;
            vhi[e] = (double)std::max(r.lower, r.upper);
            init[e] = AnOut{0.0, 0.0, 0.0, 0.0, 0, 0};
        }
        // levels of non-origin events, scratch per level
        int32_t n_levels = 0;
        for (int32_t e = 0; e < E; ++e)
            if (tlen[e] > 0) n_levels = std::max(n_levels, level[e]);
        std::vector<std::vector<int32_t>> by_level((size_t)n_levels + 1);
        for (int32_t e : order)
            if (tlen[e] > 0) by_level[level[e]].push_back(e);
        an = new mcd_analytic();
        an->E = E;
        std::vector<AnFold> level_ev;
        std::vector<int2> chunks;
        std::vector<AnEntry> entries((size_t)P);
        // activity PMFs most of whose bins are zero, as their non-zero bins (all PMFs
        // finite: zero times infinity is not a term to leave out)
        bool finite = true;
        for (int64_t i = 0; i < d->pmf_off[K]; ++i) finite = finite && std::isfinite(d->pmf_probs[i]);
        std::vector<double> nz_val;
        std::vector<int32_t> nz_idx, nz_n((size_t)K, 0);
        std::vector<int64_t> nz_off((size_t)K, 0);
        for (int32_t k = 0; k < K; ++k) {
            const int64_t m = d->pmf_off[k + 1] - d->pmf_off[k];
            const double *q = d->pmf_probs + d->pmf_off[k];
            int64_t nz = 0;
            for (int64_t i = 0; i < m; ++i) nz += q[i] != 0.0;
            if (!finite || m < 2 || nz == 0 || kSparse * nz > m) continue;
            nz_off[(size_t)k] = (int64_t)nz_val.size();
            nz_n[(size_t)k] = (int32_t)nz;
            for (int64_t i = 0; i < m; ++i)
                if (q[i] != 0.0) {
                    nz_val.push_back(q[i]);
                    nz_idx.push_back((int32_t)i);
                }
        }
        an->level_off.push_back(0);
        an->chunk_off.push_back(0);
        int64_t scratch_max = 0, conv_max = 0;
        for (int32_t l = 1; l <= n_levels; ++l) {
            int64_t scratch = 0, smem_bins = 0, conv = 0;
            std::vector<std::pair<int64_t, int2>> level_chunks;  // (estimated multiply-adds, chunk)
            // CTAs an event: a bin a thread, up to the largest cluster
            int64_t widest = 1;
            for (int32_t e : by_level[l]) widest = std::max<int64_t>(widest, ev[e].gmax);
            int32_t ctas = 1;
            while (ctas < kAnCluster && (int64_t)ctas * kAnThreads < widest) ctas *= 2;
            for (int32_t e : by_level[l]) {
                AnEv &r = ev[e];
                const int64_t seg = (r.gmax + ctas - 1) / ctas, room = (((seg + 31) / 32) | 1) * 32;
                if (room <= kAnSmemBins) {
                    smem_bins = std::max<int64_t>(smem_bins, room);
                } else {
                    r.scratch_off = scratch;
                    scratch += (int64_t)kAnArrays * room * ctas;
                }
                for (int64_t p = tstart[e]; p < tstart[e] + tlen[e]; ++p) {  // each convolution's slot and chunks
                    const int32_t src = d->pred_src[p], pk = d->pred_pmf[p];
                    const int64_t n = ev[src].cap, m = d->pmf_off[pk + 1] - d->pmf_off[pk];
                    const int64_t len = n == 1 ? m : (m == 1 ? n : n + m - 1);
                    const int32_t nnz = nz_n[(size_t)pk];
                    entries[(size_t)p] = AnEntry{ev[src].pool_off, d->pmf_off[pk], nz_off[(size_t)pk], conv,
                                                 d->pmf_first[pk], pmf_mass[pk], src, (int32_t)m, nnz, 0};
                    conv += (len + 1) / 2 * 2;
                    for (int64_t c = 0; c * kConvOuts < len; ++c) {
                        const int64_t jm = c * kConvOuts + kConvOuts / 2;  // the chunk's middle output
                        const int64_t terms = (n == 1 || m == 1) ? 1
                                              : nnz              ? nnz
                                                    : (std::min(jm, n - 1) - std::max<int64_t>(0, jm - (m - 1)) + 1);
                        level_chunks.emplace_back(std::max<int64_t>(terms, 1) * kConvOuts, make_int2((int)p, (int)c));
                    }
                }
                AnFold f{};
                f.ev = r;
                for (int64_t k = 0; k < kAnGroup && k < tlen[e]; ++k) f.first[k] = entries[(size_t)(tstart[e] + k)];
                level_ev.push_back(f);
            }
            std::stable_sort(level_chunks.begin(), level_chunks.end(),
                             [](const auto &x, const auto &y) { return x.first > y.first; });
            for (const auto &lc : level_chunks) chunks.push_back(lc.second);
            scratch_max = std::max(scratch_max, scratch);
            conv_max = std::max(conv_max, conv);
            an->level_off.push_back((int32_t)level_ev.size());
            an->chunk_off.push_back((int32_t)chunks.size());
            an->level_smem.push_back((int32_t)(kAnArrays * smem_bins * (int64_t)sizeof(double)));
            an->level_ctas.push_back(ctas);
        }
        an->bins = pool;
        // device layout: one allocation
        cuda_check(cudaGetDevice(&an->device), "cudaGetDevice");
        cuda_check(cudaStreamCreateWithFlags(&an->stream, cudaStreamNonBlocking), "stream create");
        const size_t s_ev = align_up((size_t)E * sizeof(AnEv), 256),
                     s_entry = align_up(std::max<size_t>(entries.size(), 1) * sizeof(AnEntry), 256),
                     s_probs = align_up((size_t)std::max<int64_t>(d->pmf_off[K], 1) * 8, 256),
                     s_nzv = align_up(std::max<size_t>(nz_val.size(), 1) * 8, 256),
                     s_nzi = align_up(std::max<size_t>(nz_idx.size(), 1) * 4, 256),
                     s_out = align_up((size_t)std::max(E, 1) * sizeof(AnOut), 256),
                     s_pool = align_up((size_t)std::max<int64_t>(pool, 1) * 8, 256),
                     s_scr = align_up((size_t)std::max<int64_t>(scratch_max, 1) * 8, 256),
                     s_lev = align_up(std::max<size_t>(level_ev.size(), 1) * sizeof(AnFold), 256), s_err = 256,
                     s_conv = align_up((size_t)std::max<int64_t>(conv_max, 1) * 8, 256),
                     s_chunk = align_up(std::max<size_t>(chunks.size(), 1) * sizeof(int2), 256);
        const size_t total = s_ev + s_entry + s_probs + s_nzv + s_nzi + s_out + s_pool + s_scr + s_lev + s_err + s_conv + s_chunk;
        cuda_check(cudaMalloc(&an->dmem, total), "analytic allocation");
        char *p = an->dmem;
        auto put = [&](const void *src, size_t bytes, size_t slot) -> char * {
            char *at = p;
            if (bytes) cuda_check(cudaMemcpy(at, src, bytes, cudaMemcpyHostToDevice), "analytic upload");
            p += slot;
            return at;
        };
        AnArgs &a = an->args;
        an->d_ev = reinterpret_cast<const AnEv *>(put(ev.data(), (size_t)E * sizeof(AnEv), s_ev));
        a.entries = reinterpret_cast<const AnEntry *>(put(entries.data(), entries.size() * sizeof(AnEntry), s_entry));
        a.pmf_probs = reinterpret_cast<const double *>(put(d->pmf_probs, (size_t)d->pmf_off[K] * 8, s_probs));
        a.nz_val = reinterpret_cast<const double *>(put(nz_val.data(), nz_val.size() * 8, s_nzv));
        a.nz_idx = reinterpret_cast<const int32_t *>(put(nz_idx.data(), nz_idx.size() * 4, s_nzi));
        a.out = reinterpret_cast<AnOut *>(put(init.data(), (size_t)E * sizeof(AnOut), s_out));
        a.pool = reinterpret_cast<double *>(p);
        {  // origins' unit masses
            std::vector<double> ones((size_t)std::max<int64_t>(pool, 1), 0.0);
            for (int32_t e = 0; e < E; ++e)
                if (tlen[e] == 0) ones[(size_t)ev[e].pool_off] = 1.0;
            cuda_check(cudaMemcpy(p, ones.data(), (size_t)pool * 8, cudaMemcpyHostToDevice), "analytic upload");
        }
        p += s_pool;
        a.scratch = reinterpret_cast<double *>(p);
        p += s_scr;
        an->d_level_ev = reinterpret_cast<AnFold *>(put(level_ev.data(), level_ev.size() * sizeof(AnFold), s_lev));
        a.convbuf = reinterpret_cast<double *>(p);
        p += s_conv;
        an->d_chunks = reinterpret_cast<int2 *>(put(chunks.data(), chunks.size() * sizeof(int2), s_chunk));
        a.err = reinterpret_cast<int32_t *>(p);
        cuda_check(cudaMemset(a.err, 0, 4), "analytic error flag");
        a.step = d->step;
        a.urule = d->underflow_rule;
        a.orule = d->overflow_rule;
        cuda_check(cudaFuncSetAttribute(k_an_fold, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(kAnArrays * kAnSmemBins * sizeof(double))),
                   "analytic shared memory");
        int sms = 0;
        cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, an->device), "device query");
        // every level's launches, captured once into a graph
        cuda_check(cudaStreamBeginCapture(an->stream, cudaStreamCaptureModeThreadLocal), "graph capture");
        for (size_t l = 0; l + 1 < an->level_off.size(); ++l) {
            const int32_t nc = an->chunk_off[l + 1] - an->chunk_off[l], ne = an->level_off[l + 1] - an->level_off[l];
            if (nc > 0)
                k_an_conv<<<std::min(nc, sms * kConvWarpsPerSm), 32, 0, an->stream>>>(
                    an->args, an->d_chunks + an->chunk_off[l], nc);
            if (ne > 0) {
                cudaLaunchAttribute at{};
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = (unsigned)an->level_ctas[l];
                at.val.clusterDim.y = at.val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3((unsigned)(ne * an->level_ctas[l]));
                cfg.blockDim = dim3(kAnThreads);
                cfg.dynamicSmemBytes = (size_t)an->level_smem[l];
                cfg.stream = an->stream;
                cfg.attrs = &at;
                cfg.numAttrs = 1;
                const AnFold *first = an->d_level_ev + an->level_off[l];
                (void)cudaLaunchKernelEx(&cfg, k_an_fold, an->args, first);  // (an error ends the capture)
            }
        }
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(an->stream, &g);
        cuda_check(ce, "graph capture");
        const cudaError_t ie = cudaGraphInstantiate(&an->graph, g, 0);
        cudaGraphDestroy(g);
        cuda_check(ie, "graph instantiate");
        *out = an;
    });
    if (rc != MCD_OK && an) mcd_analytic_destroy(an);
    return rc;
}

void mcd_analytic_destroy(mcd_analytic *an) {
    if (!an) return;
    if (an->stream) cudaStreamSynchronize(an->stream);
    if (an->graph) cudaGraphExecDestroy(an->graph);
    if (an->stream) cudaStreamDestroy(an->stream);
    if (an->dmem) cudaFree(an->dmem);
    delete an;
}

int mcd_analytic_run(mcd_analytic *an) {
    return guarded([&] {
        if (!an) throw McdError(MCD_ERR_INVALID, "null handle");
        cuda_check(cudaSetDevice(an->device), "cudaSetDevice");
        cuda_check(cudaGraphLaunch(an->graph, an->stream), "analytic launch");
        cuda_check(cudaStreamSynchronize(an->stream), "analytic run");
        int32_t flags = 0;
        cuda_check(cudaMemcpy(&flags, an->args.err, 4, cudaMemcpyDeviceToHost), "analytic error flag");
        if (flags) {
            cuda_check(cudaMemset(an->args.err, 0, 4), "analytic error flag");
            if (flags & AN_ERR_BOUNDS) throw McdError(MCD_ERR_INVALID, "min_value must not exceed max_value");
            if (flags & AN_ERR_UNDER_TRUNC)
                throw McdError(MCD_ERR_INVALID, "Underflow mass cannot be truncated: no lower-bound bin present.");
            if (flags & AN_ERR_OVER_TRUNC)
                throw McdError(MCD_ERR_INVALID, "Overflow mass cannot be truncated: no upper-bound bin present.");
            if (flags & AN_ERR_EMPTY) throw McdError(MCD_ERR_INVALID, "PMF must not be empty after clipping");
            if (flags & AN_ERR_GRID)
                throw McdError(MCD_ERR_INVALID, "PMF values do not fit their common grid (values off the step grid)");
            throw McdError(MCD_ERR_RUNTIME, "analytic kernel: a PMF exceeded its planned support");
        }
        an->ran = true;
    });
}

int64_t mcd_analytic_bins(const mcd_analytic *an) { return an ? an->bins : 0; }

int mcd_analytic_fetch(const mcd_analytic *an, double *first, int64_t *offset, int64_t *length, double *probs,
                       double *underflow, double *overflow) {
    return guarded([&] {
        if (!an) throw McdError(MCD_ERR_INVALID, "null handle");
        if (!an->ran) throw McdError(MCD_ERR_INVALID, "run() has not completed");
        cuda_check(cudaSetDevice(an->device), "cudaSetDevice");
        std::vector<AnOut> o((size_t)an->E);
        std::vector<AnEv> ev((size_t)an->E);
        if (an->E) {
            cuda_check(cudaMemcpy(o.data(), an->args.out, o.size() * sizeof(AnOut), cudaMemcpyDeviceToHost),
                       "analytic fetch");
            cuda_check(cudaMemcpy(ev.data(), an->d_ev, ev.size() * sizeof(AnEv), cudaMemcpyDeviceToHost),
                       "analytic fetch");
        }
        if (probs && an->bins)
            cuda_check(cudaMemcpy(probs, an->args.pool, (size_t)an->bins * 8, cudaMemcpyDeviceToHost),
                       "analytic fetch");
        for (int32_t e = 0; e < an->E; ++e) {
            if (first) first[e] = o[e].first;
            if (offset) offset[e] = ev[e].pool_off;
            if (length) length[e] = o[e].len;
            if (underflow) underflow[e] = o[e].under;
            if (overflow) overflow[e] = o[e].over;
        }
    });
}

}  // extern "C"
