// mcd_inspect.cu -- per-type delay histograms of sampled durations, the GPU form of
// the reference's delay inspection (demo/inspection.py:11-29: durations - base per
// activity type, absolute and relative to the base).
//
// A histogram needs the draws and nothing of the propagation, so one kernel draws
// every link's durations (the sampled propagation's own draws: same Philox block,
// word and arithmetic) and bins them in registers and shared memory; no duration
// goes to memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "mcd_device.cuh"
#include "mcd_handle.hpp"

namespace mcd {

namespace {

// Bin of x in [lo, hi) with nb bins: 0 below lo, 1 + floor((x - lo) * nb / (hi - lo))
// inside, nb + 1 at or above hi.
__device__ __forceinline__ int delay_bin(double x, double lo, double hi, int nb) {
    if (!(x >= lo)) return 0;
    if (!(x < hi)) return nb + 1;
    const int b = (int)((x - lo) * (double)nb / (hi - lo));
    return 1 + (b < nb ? b : nb - 1);
}

// Per link class: the ranges, and what bins a delay in single precision -- bin
// q = (x - lo) * scale, off from the exact quotient by less than eps bins.
struct DelayBins {
    double lo, hi;
    float flo, scale, eps;
};

// The float nearest below |x| in magnitude with x's sign, by integer operations
// (a conversion would occupy the FP64 pipe, 2 lanes per clock and SM); NaN for a
// magnitude outside the normal floats, zero included.
__device__ __forceinline__ float narrow(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const uint32_t mag = hi & 0x7FFFFFFFu;
    if (mag - 0x38100000u >= 0x47F00000u - 0x38100000u) return __int_as_float(0x7FC00000);
    return __uint_as_float((hi & 0x80000000u) | ((mag - 0x38000000u) << 3) | (lo >> 29));
}

// delay_bin of the double that f approximates (relative error below 2^-22), or -1
// when a bin's edge is nearer than the error.
__device__ __forceinline__ int quick_bin(float f, const DelayBins &d, int nb) {
    const float q = (f - d.flo) * d.scale;
    if (!(fabsf(q - rintf(q)) > d.eps)) return -1;  // (NaN too)
    return q < 0.0f ? 0 : q > (float)nb ? nb + 1 : 1 + (int)q;
}

// Whether the square of base b or its reciprocal's is so far out that a link's relative
// moments cannot be had from its absolute ones.
__host__ __device__ inline bool far_base(double b) { return b != 0.0 && !(fabs(b) >= 1e-100 && fabs(b) <= 1e100); }

struct HistArgs {
    const int32_t *cls;      // [L] class of each link, -1: none
    const double *base;      // [L]
    const double *ranges;    // [class][abs lo, abs hi, rel lo, rel hi]
    int32_t nc, nb;
    unsigned long long *counts;  // [class][abs, rel][nb + 2]
    double *moments;             // [class][abs, rel][count, sum, sum of squares]
    int32_t rounds;              // 128-sample rounds of an item
};

// The tables block's room in shared memory (16-byte aligned).
__host__ __device__ constexpr size_t hist_tables_bytes(int32_t n_dist, int32_t n_alias) {
    return (n_dist * sizeof(DistParam) + n_alias * (sizeof(AliasEntry) + sizeof(AliasPick)) + 15) / 16 * 16;
}

constexpr int kHistThreads = 256;
constexpr int kHistWarps = kHistThreads / 32;
constexpr int kHistLanes = 4;  // samples a lane draws at a time

// Bound by the issue of the draws (65 warp instructions a warp-draw) with the FP64
// pipe behind it.  A warp takes one Philox block's links for `rounds` x 128
// samples, four samples a lane at a time.  What a delay costs depends on its kind:
//   fixed links          one value: its bin is found once per item and counted n times;
//   tables of <= 32 bins the entries drawn are counted (shared memory), and each
//                        entry's delay is binned once per item;
//   other draws          the delay and its two sums in FP64 (four operations), its
//                        bins in single precision, the exact quotient only where an
//                        edge is near.
// Relative sums follow per link from the absolute ones (the base divides out), so
// they cost one division a link and item; of bases beyond 1e-100 to 1e100 every delay
// is divided (far_base).
// 10,000 samples of 1,000 events (2,400 links, five kinds): 0.39 ms; as a
// propagation with a durations output and a kernel that binned those with FP64
// divisions and FP64 shared-memory atomics the whole call took 12.4 ms more.
// FAR: some link has a far base (the check in the draws' loop costs the others 13 %).
template <bool TSMEM, bool FAR>
__global__ void __launch_bounds__(kHistThreads) k_delay_hist(const KArgs a, const HistArgs h) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int nh = h.nc * 2 * (h.nb + 2);
    const size_t tables = TSMEM ? hist_tables_bytes(a.n_dist, a.n_alias) : 0;
    double2 *acc = reinterpret_cast<double2 *>(sm + tables);                   // [warp][link of the group][lane]
    double *smom = reinterpret_cast<double *>(acc + kHistWarps * kGroupLinks * 32);  // [class][6]
    DelayBins *bins = reinterpret_cast<DelayBins *>(smom + h.nc * 6);          // [class][abs, rel]
    unsigned *entries = reinterpret_cast<unsigned *>(bins + h.nc * 2);         // [warp][link of the group][32]
    unsigned *shist = entries + kHistWarps * kGroupLinks * 32;
    if (TSMEM) {
        const int n8 = (a.n_dist * (int)sizeof(DistParam) + a.n_alias * (int)(sizeof(AliasEntry) + sizeof(AliasPick))) / 8;
        for (int i = threadIdx.x; i < n8; i += kHistThreads)
            reinterpret_cast<uint2 *>(sm)[i] = reinterpret_cast<const uint2 *>(a.dist)[i];
    }
    for (int i = threadIdx.x; i < kHistWarps * kGroupLinks * 32; i += kHistThreads) {
        acc[i] = make_double2(0.0, 0.0);
        entries[i] = 0u;
    }
    for (int i = threadIdx.x; i < nh; i += kHistThreads) shist[i] = 0u;
    for (int i = threadIdx.x; i < h.nc * 6; i += kHistThreads) smom[i] = 0.0;
    for (int i = threadIdx.x; i < h.nc * 2; i += kHistThreads) {
        DelayBins d;
        d.lo = h.ranges[2 * i];
        d.hi = h.ranges[2 * i + 1];
        const double w = d.hi - d.lo;
        d.flo = (float)d.lo;
        d.scale = (float)((double)h.nb / w);
        // rounding of x (2^-22), of lo, of the difference and of the product, each
        // relative to the largest magnitude inside the range, times four
        d.eps = (float)((double)h.nb * ((fabs(d.lo) + fabs(d.hi)) / w + 1.0) * 1.9073486328125e-06);
        bins[i] = d;
    }
    __syncthreads();
    const DistParam *dists = TSMEM ? reinterpret_cast<const DistParam *>(sm) : a.dist;
    const AliasEntry *alias = reinterpret_cast<const AliasEntry *>(dists + a.n_dist);
    const AliasPick *picks = reinterpret_cast<const AliasPick *>(alias + a.n_alias);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double2 *wacc = acc + warp * kGroupLinks * 32;
    unsigned *went = entries + warp * kGroupLinks * 32;
    auto count = [&](int c, int which, int bin, unsigned m) { atomicAdd(&shist[(c * 2 + which) * (h.nb + 2) + bin], m); };
    auto exact = [&](int c, int which, double x) {
        const DelayBins &d = bins[c * 2 + which];
        return delay_bin(x, d.lo, d.hi, h.nb);
    };
    const int64_t item = (int64_t)h.rounds * 32 * kHistLanes;
    for (int64_t block0 = (int64_t)blockIdx.y * item; block0 < a.n; block0 += (int64_t)gridDim.y * item) {
        const int64_t end = block0 + item < a.n ? block0 + item : a.n;
        for (int g = blockIdx.x * kHistWarps + warp; g < a.n_groups; g += gridDim.x * kHistWarps) {
            const int4 grp = __ldg(reinterpret_cast<const int4 *>(a.groups + g));  // block, first, n
#pragma unroll 1
            for (int64_t s0 = block0; grp.x >= 0 && s0 < end; s0 += 32 * kHistLanes) {
                uint64_t seed[kHistLanes];
                U4 w[kHistLanes];
                bool on[kHistLanes];
#pragma unroll
                for (int j = 0; j < kHistLanes; ++j) {
                    const int64_t s = s0 + 32 * j + lane;
                    on[j] = s < end;
                    seed[j] = on[j] ? (uint64_t)__ldg(a.seeds + s) : 0ull;
                    w[j] = draw_words(seed[j], (uint32_t)grp.x, 0u, 0u);
                }
#pragma unroll 1
                for (int i = 0; i < grp.z; ++i) {
                    const int4 *q = reinterpret_cast<const int4 *>(a.draws + grp.y + i);
                    const int4 r0 = __ldg(q);
                    const int vt = __ldg(&q[1].x);
                    const double v = __hiloint2double(r0.w, r0.z);
                    const int kd = r0.y, kind = kd & KD_KIND_MASK, wsel = (kd >> KD_WORD_SHIFT) & 3;
                    const int c = __ldg(h.cls + r0.x);
                    const DistParam &p = dists[kd >> 8];
                    // (a gamma link outside every class is drawn all the same: its rejection cap is an error)
                    if (c < 0 && kind != K_GAMMA) continue;
                    if (vt >= 0 && p.tab_n <= 32) {
#pragma unroll
                        for (int j = 0; j < kHistLanes; ++j)
                            if (on[j]) atomicAdd(&went[i * 32 + pick_bin(p, picks, word_of(w[j], wsel), w[j].y, (kd & KD_TWO_WORD) != 0)], 1u);
                        continue;
                    }
                    const double b = __ldg(h.base + r0.x);
                    // (NaN, so every bin exact, where the base is no finite float)
                    const bool far = FAR && far_base(b);
                    const float invb = fabsf((float)b) < 3e38f ? 1.0f / (float)b : __int_as_float(0x7FC00000);
                    double sum = 0.0, sq = 0.0;
#pragma unroll
                    for (int j = 0; j < kHistLanes; ++j) {
                        if (!on[j]) continue;
                        float dfac;
                        double d;
                        if (kind == K_EXP) d = draw_exponential(p, v, word_of(w[j], wsel), dfac);
                        else if (kind == K_GAMMA)
                            d = p.erlang ? draw_erlang(p, v, (uint32_t)r0.x, seed[j], w[j], wsel, a.err, &dfac)
                                         : draw_gamma(p, v, (uint32_t)grp.x, seed[j], a.err, &dfac);
                        else
                            d = draw_empirical(p, alias, picks, nullptr, v, kind == K_EMP_REL, word_of(w[j], wsel), w[j].y,
                                               (kd & KD_TWO_WORD) != 0, dfac);
                        if (c < 0) continue;
                        const double delta = d - b;  // demo/inspection.py:23-24
                        sum += delta;
                        sq = fma(delta, delta, sq);
                        const float f = narrow(delta);
                        int k = quick_bin(f, bins[c * 2], h.nb);
                        if (k < 0) k = exact(c, 0, delta);
                        count(c, 0, k, 1u);
                        if (b != 0.0) {  // relative delays of links with a non-zero base (:25-26)
                            k = quick_bin(f * invb, bins[c * 2 + 1], h.nb);
                            if (k < 0) k = exact(c, 1, delta / b);
                            count(c, 1, k, 1u);
                            if (far) {
                                const double x = delta / b;
                                atomicAdd(&smom[c * 6 + 4], x);
                                atomicAdd(&smom[c * 6 + 5], x * x);
                            }
                        }
                    }
                    if (c >= 0) {
                        double2 &t = wacc[i * 32 + lane];
                        t.x += sum;
                        t.y += sq;
                    }
                }
            }
            __syncwarp();
            // the item's links: entry counts binned, sums over the lanes into the class's moments
            for (int i = 0; i < grp.z; ++i) {
                const int4 *q = reinterpret_cast<const int4 *>(a.draws + grp.y + i);
                const int4 r0 = __ldg(q);
                const int vt = __ldg(&q[1].x);
                const int c = __ldg(h.cls + r0.x), kind = r0.y & KD_KIND_MASK;
                if (c < 0) continue;
                const double b = __ldg(h.base + r0.x);
                const double m = (double)(end - block0);
                double sum, sq, rel = 0.0, rel_sq = 0.0;  // (the latter two of far bases)
                const bool fixed = kind == K_FIXED, far = FAR && far_base(b);
                if (fixed || (vt >= 0 && dists[r0.y >> 8].tab_n <= 32)) {
                    unsigned n_k;  // this lane's value and how often it was drawn
                    double delta = 0.0;
                    if (fixed) {
                        n_k = lane == 0 ? (unsigned)(end - block0) : 0u;
                        if (n_k) delta = __hiloint2double(r0.w, r0.z) - b;
                    } else {
                        n_k = went[i * 32 + lane];
                        went[i * 32 + lane] = 0u;
                        if (n_k) delta = a.vals[vt + lane] - b;
                    }
                    if (n_k) {
                        count(c, 0, exact(c, 0, delta), n_k);
                        if (b != 0.0) count(c, 1, exact(c, 1, delta / b), n_k);
                    }
                    sum = (double)n_k * delta;
                    sq = sum * delta;
                    if (far && n_k) {
                        const double x = delta / b;
                        rel = (double)n_k * x;
                        rel_sq = rel * x;
                    }
                } else {
                    double2 &t = wacc[i * 32 + lane];
                    sum = t.x;
                    sq = t.y;
                    t = make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                    sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
                }
                if (far) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        rel += __shfl_xor_sync(0xFFFFFFFFu, rel, o);
                        rel_sq += __shfl_xor_sync(0xFFFFFFFFu, rel_sq, o);
                    }
                }
                if (lane < (b != 0.0 ? 6 : 3)) {  // lanes 0-2: count, sum, squares of the delays; 3-5: relative
                    const double s = lane >= 3 ? 1.0 / b : 1.0;
                    const int k = lane % 3;
                    const double first = far && lane >= 3 ? rel : sum * s, second = far && lane >= 3 ? rel_sq : sq * s * s;
                    atomicAdd(&smom[c * 6 + lane], k == 0 ? m : k == 1 ? first : second);
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nh; i += kHistThreads)
        if (shist[i]) atomicAdd(&h.counts[i], (unsigned long long)shist[i]);
    for (int i = threadIdx.x; i < h.nc * 6; i += kHistThreads)
        if (smom[i] != 0.0) atomicAdd(&h.moments[i], smom[i]);
}

}  // namespace
}  // namespace mcd

using namespace mcd;

extern "C" {

int mcd_delay_histograms(mcd_dag *g, const int64_t *seeds, int64_t n, const int32_t *link_class,
                         const double *link_base, int32_t n_classes, int32_t n_bins, const double *ranges,
                         uint64_t *counts, double *moments) {
    return guarded([&] {
        if (!g || !link_class || !link_base || !ranges || !counts || !moments)
            throw McdError(MCD_ERR_INVALID, "null argument");
        if (n < 0) throw McdError(MCD_ERR_INVALID, "negative sample count");
        if (n > 0 && !seeds) throw McdError(MCD_ERR_INVALID, "null seeds");
        if (n_classes < 1 || n_bins < 1 || (size_t)n_classes * 2 * (n_bins + 2) * 4 + (size_t)n_classes * 48 > 48 * 1024)
            throw McdError(MCD_ERR_INVALID, "n_classes * 2 * (n_bins + 2) counters must fit 48 KB");
        const int32_t L = g->h.L;
        for (int32_t l = 0; l < L; ++l)
            if (link_class[l] < -1 || link_class[l] >= n_classes) throw McdError(MCD_ERR_INVALID, "link class out of range");
        for (int32_t c = 0; c < n_classes; ++c)
            if (!(ranges[4 * c] < ranges[4 * c + 1]) || !(ranges[4 * c + 2] < ranges[4 * c + 3]))
                throw McdError(MCD_ERR_INVALID, "each histogram range needs lo < hi");
        cuda_check(cudaSetDevice(g->device), "cudaSetDevice");
        cudaStream_t st = g->stream[0];
        const size_t nh = (size_t)n_classes * 2 * (n_bins + 2), nm = (size_t)n_classes * 6;
        // samples per launch: a launch's draws fit the 32-bit counters of any one CTA
        const int64_t C = std::max<int64_t>(1, std::min<int64_t>(n, ((int64_t)1 << 31) / std::max(L, 1)));
        const size_t o_cls = 0, o_base = align_up((size_t)L * 4, 256), o_rng = o_base + align_up((size_t)L * 8, 256),
                     o_cnt = o_rng + align_up((size_t)n_classes * 32, 256), o_mom = o_cnt + align_up(nh * 8, 256),
                     o_seed = o_mom + align_up(nm * 8, 256), total = o_seed + align_up((size_t)C * 8, 256);
        ensure_ws(g, total);
        char *w = g->ws;
        cuda_check(cudaMemcpyAsync(w + o_cls, link_class, (size_t)L * 4, cudaMemcpyHostToDevice, st), "upload");
        cuda_check(cudaMemcpyAsync(w + o_base, link_base, (size_t)L * 8, cudaMemcpyHostToDevice, st), "upload");
        cuda_check(cudaMemcpyAsync(w + o_rng, ranges, (size_t)n_classes * 32, cudaMemcpyHostToDevice, st), "upload");
        cuda_check(cudaMemsetAsync(w + o_cnt, 0, nh * 8, st), "reset");
        cuda_check(cudaMemsetAsync(w + o_mom, 0, nm * 8, st), "reset");
        const HostDag &hd = g->h;
        const size_t tables = hd.tables_in_smem ? hist_tables_bytes((int32_t)hd.dist.size(), (int32_t)hd.alias.size()) : 0;
        const size_t smem = tables + kHistWarps * kGroupLinks * 32 * (sizeof(double2) + 4) +
                            (size_t)n_classes * (48 + 2 * sizeof(DelayBins)) + nh * 4;
        bool far = false;
        for (int32_t l = 0; l < L; ++l) far = far || far_base(link_base[l]);
        void (*fn)(const KArgs, const HistArgs) =
            hd.tables_in_smem ? far ? k_delay_hist<true, true> : k_delay_hist<true, false>
                              : far ? k_delay_hist<false, true> : k_delay_hist<false, false>;
        cuda_check(raise_smem_limit((const void *)fn, smem), "histogram shared memory");
        int sms = 0, per_sm = 0;
        cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device), "device query");
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kHistThreads, smem), "occupancy query");
        HistArgs ha{};
        ha.cls = reinterpret_cast<const int32_t *>(w + o_cls);
        ha.base = reinterpret_cast<const double *>(w + o_base);
        ha.ranges = reinterpret_cast<const double *>(w + o_rng);
        ha.nc = n_classes;
        ha.nb = n_bins;
        ha.counts = reinterpret_cast<unsigned long long *>(w + o_cnt);
        ha.moments = reinterpret_cast<double *>(w + o_mom);
        KArgs drawn = base_args(g);
        image_draws(g, drawn);
        const int64_t groups = drawn.n_groups, slots = (int64_t)std::max(per_sm, 1) * sms;
        for (int64_t off = 0; off < n && groups > 0; off += C) {
            const int64_t m = std::min(C, n - off);
            cuda_check(cudaMemcpyAsync(w + o_seed, seeds + off, (size_t)m * 8, cudaMemcpyHostToDevice, st), "seeds");
            KArgs a = drawn;
            a.seeds = reinterpret_cast<const int64_t *>(w + o_seed);
            a.n = m;
            // an item's fixed costs (binning table entries, reducing sums) want many
            // samples, the last wave wants several items a warp
            int64_t blocks = 1;
            ha.rounds = 8;
            for (; ha.rounds > 1; ha.rounds /= 2) {
                blocks = (m + ha.rounds * 32 * kHistLanes - 1) / (ha.rounds * 32 * kHistLanes);
                if (blocks * groups >= 4 * slots * kHistWarps) break;
            }
            blocks = (m + ha.rounds * 32 * kHistLanes - 1) / (ha.rounds * 32 * kHistLanes);
            const int64_t gy = std::min<int64_t>(blocks, std::min<int64_t>(slots, 65535));
            const int64_t gx = std::max<int64_t>(1, std::min((groups + kHistWarps - 1) / kHistWarps, slots / gy));
            fn<<<dim3((unsigned)gx, (unsigned)gy), kHistThreads, smem, st>>>(a, ha);
            cuda_check(cudaGetLastError(), "histogram launch");
        }
        cuda_check(cudaMemcpyAsync(counts, w + o_cnt, nh * 8, cudaMemcpyDeviceToHost, st), "download");
        cuda_check(cudaMemcpyAsync(moments, w + o_mom, nm * 8, cudaMemcpyDeviceToHost, st), "download");
        check_device_error(g);
    });
}

}  // extern "C"
