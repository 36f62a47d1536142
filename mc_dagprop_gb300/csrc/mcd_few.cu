// mcd_few.cu -- few samples: lanes over predecessors or events, a CTA a sample.
//
// A tile of 32 samples an SM leaves most of the chip idle when few samples are run, and
// its levels are then a chain: an event's entries one after another, each a Philox block
// and a sampler, some 5,000 clocks a stage.  Here the draws come first, on all SMs
// (k_few_draw), into a scratch in the order in which the propagation reads them; then a
// CTA of one to twenty samples walks the stages (k_few).  What is left of a stage is a
// barrier, one add and a maximum, and nothing else may lie on that path: records and
// durations come through a ring of stage buffers that a warp of its own fills by bulk
// copies several stages ahead.  It is bound by that chain, about 1,800 clocks a stage of
// 100 events, and by the draws' instructions as the samples grow.
// Measured, before and after: 1,000 events, one seed through host buffers 168 -> 62 us;
// 200,000 events, one seed 13.1 -> 1.5 ms; on the device, 10,000 events x 152 samples
// 642 -> 111 us, 20,017 x 608 1,757 -> 560, 200,000 x 608 12.8 -> 3.8 ms.
#include "mcd_device.cuh"

namespace mcd {

constexpr int kFewDrawThreads = 128;

// First element of a stage's durations in KArgs-wide numbering, samples aside: even, so
// that a copy starts on a 16-byte boundary (stages' ranges stay apart: each stage moves
// the numbering on by one).
__device__ __forceinline__ int64_t few_first(int stage, int first_entry) {
    return (int64_t)((uint32_t)(first_entry + stage + 1) & ~1u);
}

// Durations of the stage blockIdx.x.  A warp's lanes are the samples of a block of 32 S
// (S a lane: a record is read and decoded once for them, and their chains overlap) and,
// when n is smaller, several entries; a lane takes kFewDrawRun entries one after another
// where n fills the lanes (one otherwise: latency), drawing a Philox block once for the
// entries that share it.  The last CTAs draw the links no entry references.  The draws are
// the sampled propagation's own (same records, blocks, words and arithmetic): equal bits.
// Bound by instructions (per 32 draws 148 at one sample a lane, 109 at four).  Both
// kernels, 20,017 events: x 1,216 832 us with one sample a lane, 750 with two, 742 with
// four; x 2,432 1,388, 1,256, 1,197; x 152 412, 411, 419.
constexpr int kFewDrawRun = 4;
template <bool GIVEN, int S>
__global__ void __launch_bounds__(kFewDrawThreads) k_few_draw(const KArgs a, const FewArgs f) {
    const int stage = blockIdx.x, n = f.n, ns = f.ns, lane = threadIdx.x & 31;
    const DistParam *dists = a.dist;
    const AliasEntry *alias = reinterpret_cast<const AliasEntry *>(dists + a.n_dist);
    const AliasPick *picks = reinterpret_cast<const AliasPick *>(alias + a.n_alias);
    const int lanes_log = n > 16 ? 5 : n > 8 ? 4 : n > 4 ? 3 : n > 2 ? 2 : n > 1 ? 1 : 0;  // of a lane's samples
    const int run = n >= 32 ? kFewDrawRun : 1;
    const int blocks = (n + 32 * S - 1) / (32 * S);  // of samples
    const int per_warp = run << (5 - lanes_log);     // entries a warp takes
    U4 words[S];
    uint32_t drawn = 0xFFFFFFFFu;  // the block `words` are of (no block has this number)
    uint64_t seed[S];
    auto draw = [&](int kd, double v, const double *vt, uint32_t block, uint32_t link, double (&d)[S]) {
        const int kind = kd & KD_KIND_MASK;
#pragma unroll
        for (int j = 0; j < S; ++j) d[j] = v;
        if (kind == K_FIXED) return;
        const DistParam &p = dists[kd >> 8];
        float dfac;
        if (kind == K_GAMMA && !p.erlang) {
#pragma unroll
            for (int j = 0; j < S; ++j) d[j] = draw_gamma(p, v, block, seed[j], a.err, &dfac);
            return;
        }
        if (block != drawn) {
#pragma unroll
            for (int j = 0; j < S; ++j) words[j] = draw_words(seed[j], block, 0u, 0u);
        }
        drawn = block;
        const int w = (kd >> KD_WORD_SHIFT) & 3;
        if (kind == K_GAMMA) {
#pragma unroll
            for (int j = 0; j < S; ++j) d[j] = draw_erlang(p, v, link, seed[j], words[j], w, a.err, &dfac);
        } else if (kind == K_EXP) {
#pragma unroll
            for (int j = 0; j < S; ++j) d[j] = draw_exponential(p, v, word_of(words[j], w), dfac);
        } else {
#pragma unroll
            for (int j = 0; j < S; ++j)
                d[j] = draw_empirical(p, alias, picks, vt, v, kind == K_EMP_REL, word_of(words[j], w), words[j].y,
                                      (kd & KD_TWO_WORD) != 0, dfac);
        }
    };
    const bool aux = stage >= a.n_stages;
    const int4 *sm = reinterpret_cast<const int4 *>(a.stage_meta + kStageMetaInts * stage);
    const int4 meta = aux ? make_int4(0, 0, 0, a.n_aux) : __ldg(sm), mv = aux ? meta : __ldg(sm + 1);
    double *out = aux ? nullptr : f.entry_dur + few_first(stage, meta.z) * ns;
    const int cta = blockIdx.y + (aux ? (stage - a.n_stages) * gridDim.y : 0);
    const int ctas = aux ? (gridDim.x - a.n_stages) * gridDim.y : gridDim.y;
    const int items = (meta.w + per_warp - 1) / per_warp * blocks;
    constexpr int kWarps = kFewDrawThreads / 32;
    for (int item = cta * kWarps + (threadIdx.x >> 5); item < items; item += ctas * kWarps) {
        const int g = item / blocks;
        const int s = (item - g * blocks) * (32 * S) + (lane & ((1 << lanes_log) - 1));
        if (s >= n) continue;
        int64_t of_cta[S], col[S];  // (a CTA of the propagation reads its own samples)
        bool in[S];
#pragma unroll
        for (int j = 0; j < S; ++j) {
            const int sj = s + 32 * j;
            in[j] = sj < n;
            seed[j] = !in[j] ? 0 : f.seeds ? (uint64_t)__ldg(f.seeds + sj) : (uint64_t)f.seed[sj & (kFewInline - 1)];
            of_cta[j] = (int64_t)(sj / ns) * f.cta_entries + sj % ns;
            col[j] = sj * f.dur_col;
        }
        drawn = 0xFFFFFFFFu;
        const int first = g * per_warp + (lane >> lanes_log) * run;
        for (int i = first; i < first + run && i < meta.w; ++i) {
            double dur[S];
            if (aux) {
                const LinkRec lr = a.aux[i];  // (owns its block)
                draw(lr.kd, lr.v, nullptr, (uint32_t)lr.link, (uint32_t)lr.link, dur);
#pragma unroll
                for (int j = 0; j < S; ++j)
                    if (in[j]) f.durations[(int64_t)lr.link * f.dur_row + col[j]] = dur[j];
                continue;
            }
            const int4 *q = reinterpret_cast<const int4 *>(a.pred + meta.z + i);
            const int4 r0 = __ldg(q);  // src_slot, src_user, link, kd
            if (GIVEN) {
#pragma unroll
                for (int j = 0; j < S; ++j)
                    dur[j] = r0.z >= 0 && in[j] ? __ldg(f.dur_in + (int64_t)r0.z * f.dur_row + col[j]) : 0.0;
            } else {
                const int4 r1 = __ldg(q + 1);  // v, dvo, block
                const double *vt = nullptr;
                if (r1.z >= 0 && (r0.w & KD_KIND_MASK) != K_FIXED)
                    vt = meta.y >= 0 ? a.vals + mv.x + (r1.z - mv.w) / (int)sizeof(double) : a.vals + (r1.z ^ kVtGlobal);
                draw(r0.w, __hiloint2double(r1.y, r1.x), vt, (uint32_t)r1.w, (uint32_t)r0.z, dur);
                if (f.durations && (r0.w & KD_WRITE)) {
#pragma unroll
                    for (int j = 0; j < S; ++j)
                        if (in[j]) f.durations[(int64_t)r0.z * f.dur_row + col[j]] = dur[j];
                }
            }
#pragma unroll
            for (int j = 0; j < S; ++j)
                if (in[j]) out[of_cta[j] + (int64_t)i * ns] = dur[j];
        }
    }
}

// One CTA for ns samples, its last warp the producer.  Of the others' threads, G lanes
// take a sample of an event, and every step-th event of a stage.  An entry's place in its
// list decides ties as in the sequential loop (_core.cpp:338-347: a later equal time
// takes over), so the maximum over (key, place), taken where its key reaches the event's
// own, is the loop's result.
// One lane an event: entries are read kAhead at a time, their loads and adds overlapping
// (20,017 events x 608 samples 692 -> 589 us).  Several lanes: a thread's first unit of a
// stage is read before the barrier that ends the stage before, so that the chain is the
// window's read, the add, the maximum and the window's write (x 32 397 -> 358; one lane an
// event gained nothing by it).  The copies of two stages ahead have then landed at each
// barrier, of a ring of three buffers at least.
template <bool POSITIVE, int G>
__global__ void __launch_bounds__(G == 1 ? 896 : 544, 1) k_few(const KArgs a, const FewArgs f) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bars[kFewRing];
    __shared__ int2 head[kFewRing];  // of the stage in a buffer: events, first entry
    constexpr int kAhead = 4;
    constexpr bool kEarly = G > 1;
    constexpr int ahead = kEarly ? 2 : 1; // stages whose copies have landed at a barrier
    double *win = reinterpret_cast<double *>(smem);
    unsigned char *ring = smem + f.ring_off;
    const int lane = threadIdx.x & 31, R = f.ring, NS = a.n_stages, ns = f.ns;
    const bool producer = threadIdx.x == blockDim.x - 32, worker = (int)threadIdx.x < f.workers;
    const double *entry_dur = f.entry_dur + (int64_t)blockIdx.x * f.cta_entries;
    const int4 *meta = reinterpret_cast<const int4 *>(a.stage_meta);
    constexpr int kVecs = kStageMetaInts / 4;
    int4 m_next[2] = {};  // the producer's next two stages: first event, events, first entry, entries
    auto fill = [&](int l, int4 m) {
        const int b = l % R;
        const int n_ev = m.y >= 0 ? m.y : -m.y;
        head[b] = make_int2(n_ev, m.z);
        const uint32_t ev_bytes = (uint32_t)n_ev * (uint32_t)sizeof(EvRec);
        const uint32_t pr_bytes = (uint32_t)m.w * (uint32_t)sizeof(PredRec);
        const uint32_t du_bytes = ((uint32_t)(m.w + 1) & ~1u) * (uint32_t)ns * (uint32_t)sizeof(double);
        unsigned char *buf = ring + b * f.buf_bytes;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&bars[b], ev_bytes + pr_bytes + du_bytes);
        bulk_g2s(buf, a.ev + m.x, ev_bytes, &bars[b]);
        if (m.w) bulk_g2s(buf + f.pred_off, a.pred + m.z, pr_bytes, &bars[b]);
        if (m.w) bulk_g2s(buf + f.dur_off, entry_dur + few_first(l, m.z) * ns, du_bytes, &bars[b]);
    };
    // (the workers are a multiple of G * ns: a thread's units are all of one sample)
    const int j = ((int)threadIdx.x / G) % ns, s = blockIdx.x * ns + j;
    const int first = (int)threadIdx.x / (G * ns), step = f.workers / (G * ns);
    double *wcol = win + j, *rcol = f.realized && s < f.n ? f.realized + s * f.out_col : nullptr;
    int32_t *ccol = f.cause && s < f.n ? f.cause + s * f.out_col : nullptr;
    bool ok = true;
    int issued = 0, waits = 0;  // the producer's: stages copied, and the one last waited for
    if (producer) {
        for (int k = 0; k < R; ++k) mbar_init(&bars[k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (; issued < R && issued < NS; ++issued) fill(issued, __ldg(meta + kVecs * issued));
        for (int k = 0; k < 2; ++k)
            if (R + k < NS) m_next[k] = __ldg(meta + kVecs * (R + k));
        for (; waits < ahead && waits < NS && ok; ++waits) ok = stage_wait(&bars[waits], 0u, a.err);
        --waits;
    }
    // A thread's unit: its event, and its first entry with its duration (kEarly).
    EvRec ev{};
    int2 src{};  // src_slot, src_user
    double dur = 0.0;
    int p0 = 0, pe = 0;  // its first entry, and its event's end, in the stage's entries
    const PredRec *pred = nullptr;
    const double *dcol = nullptr;
    auto fetch = [&](int b, int e) {  // event e of the stage in buffer b
        const unsigned char *buf = ring + b * f.buf_bytes;
        pred = reinterpret_cast<const PredRec *>(buf + f.pred_off);
        dcol = reinterpret_cast<const double *>(buf + f.dur_off) + j;
        ev = load_ev(reinterpret_cast<const EvRec *>(buf) + e);
        p0 = ev.pred_begin - head[b].y + (lane & (G - 1));
        pe = ev.pred_end - head[b].y;
        if (kEarly && p0 < pe) {
            src = *reinterpret_cast<const int2 *>(pred + p0);
            dur = dcol[p0 * ns];
        }
    };
    const unsigned group = ((1u << G) - 1u) << (lane & ~(G - 1));
    auto run = [&]() {
        const long long init_key = POSITIVE ? ev.init_bits : ev.init_key;
        const long long ub_key = POSITIVE ? ev.ub_bits : ev.ub_key;
        long long key = (long long)0x8000000000000000ull, bits = 0;  // (below any event's own key)
        int place = -1, cause = -1;
        if constexpr (kEarly) {
            for (int p = p0;;) {
                bool clamp;
                if (p < pe && relax_time<POSITIVE>(wcol[window_row<1>(src.x) * ns] + dur, ub_key, ev.ub_bits, key,
                                                   bits, clamp)) {
                    place = p;
                    cause = src.y;
                }
                p += G;
                if (p >= pe) break;
                src = *reinterpret_cast<const int2 *>(pred + p);
                dur = dcol[p * ns];
            }
        } else {
            for (int p = p0; p < pe; p += kAhead) {
                int2 from[kAhead];
                double t[kAhead];
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (p + k < pe) {
                        from[k] = *reinterpret_cast<const int2 *>(pred + p + k);
                        t[k] = wcol[window_row<1>(from[k].x) * ns] + dcol[(p + k) * ns];
                    }
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    bool clamp;
                    if (p + k < pe && relax_time<POSITIVE>(t[k], ub_key, ev.ub_bits, key, bits, clamp)) cause = from[k].y;
                }
            }
        }
        long long best = key;
        int at = place;
#pragma unroll
        for (int m = 1; m < G; m *= 2) {
            const long long k = __shfl_xor_sync(group, best, m);
            const int q = __shfl_xor_sync(group, at, m);
            if (k > best || (k == best && q > at)) {
                best = k;
                at = q;
            }
        }
        const bool taken = best >= init_key;  // (an event without entries has none: its key is above)
        if (G == 1 || (taken ? place == at : (lane & (G - 1)) == 0)) {
            if (!taken) {
                cause = -1;
                bits = ub_key < init_key ? ev.ub_bits : ev.init_bits;  // realized = std::min(latest, ub)
            }
            const double v = __longlong_as_double(bits);
            const int slot = window_row<1>(ev.slot);
            if (slot >= 0) wcol[slot * ns] = v;
            if (rcol) *at_row(rcol, ev.user, (uint32_t)f.out_row * 8u) = v;
            if (ccol) *at_row(ccol, ev.user, (uint32_t)f.out_row * 4u) = cause;
        }
    };
    if (!__syncthreads_or(!ok)) {
        int b = 0, b2 = ahead;  // buffers of stages l and l + ahead
        uint32_t phase2 = 0;    // phase of the latter
        if (kEarly && worker && first < head[0].x) fetch(0, first);
        for (int l = 0; l < NS; ++l) {
            const int nb = b + 1 == R ? 0 : b + 1;
            if (worker) {
                const int n_ev = head[b].x;
                if (kEarly && first < n_ev) run();
                for (int e = first + (kEarly ? step : 0); e < n_ev; e += step) {
                    fetch(b, e);
                    run();
                }
                // the next stage's first unit: its records have landed, and off its chain
                if (kEarly && l + 1 < NS && first < head[nb].x) fetch(nb, first);
            }
            if (producer && l + ahead < NS) {
                waits = l + ahead;
                ok = stage_wait(&bars[b2], phase2, a.err);
            }
            if (__syncthreads_or(!ok)) break;
            if (producer && l + R < NS) {
                fill(l + R, m_next[0]);
                issued = l + R + 1;
                m_next[0] = m_next[1];
                if (l + R + 2 < NS) m_next[1] = __ldg(meta + kVecs * (l + R + 2));
            }
            b = nb;
            if (++b2 == R) {
                b2 = 0;
                phase2 ^= 1u;
            }
        }
    }
    if (producer && !ok)  // a copy that never landed: drain the others in flight, then leave
        for (int l = waits + 1; l < issued; ++l) stage_wait(&bars[l % R], (uint32_t)((l / R) & 1), a.err);
}

int sm_count();

// The layout of a launch of n samples; false where this path does not apply: a window that
// the caller wants off chip, warps per CTA that the caller fixed, stages that leave no
// ring, more scratch than kFewScratch, and sizes where it measured no faster.  (A window
// too large for rows of 32 samples is no obstacle: 50,000 events in levels of 200 x 152
// samples 3,690 -> 645 us.)  With `work` the stages plus a 64th of the events: samples
// drawn, general and few,
//   100 events in 2 stages (work 4)    8.3 and 12.7 us: the second launch is not repaid
//   150 in 7 (10)        x 40 18.6, 17.0    x 608 18.6, 20.6
//   203 in 11 (14)       x 152 24.7, 20.5   x 608 24.7, 22.6   x 2,432 24.7, 26.1
//   2,000 in 34 (65)     x 608 122, 51      x 2,432 123, 111
//   20,017 in 493 (805)  x 608 1,755, 560   x 2,432 1,757, 1,196   x 3,001 1,758, 1,506
// and durations given, whose general kernel has less to do a stage,
//   203  x 608 20.6, 23.1;  600 in 20 (29)  x 608 45, 31   x 1,824 45, 39   x 2,432 45, 46
//   20,017  x 1,216 1,424, 769   x 1,824 1,426, 1,017;  50,000 in 833  x 2,432 2,889, 2,929
// What the last samples an SM gain, as the time of the general kernels over that of
// these, at 12 to 100 events a level in 13 to 455 stages:
//   drawn, up to 30 stages   16 an SM 1.02-1.29, 18 0.97-1.29;
//                            20 up to 20 events a level 1.00-1.26, 30 to 100 0.93-1.06
//   40 stages and more       18 1.01-1.97;
//                            20 where four fifths of the entries draw 1.01-1.73; where half
//                            of them do, up to 30 events a level 1.11-1.89, 44 to 100 0.94-1.03
// (the draws are dealt out evenly here and lie on the stages' chain there; narrow levels
// leave the general kernels' warps idle).
// direct: the rows go straight to the host, which saves more launches than this adds.
bool few_layout(const KArgs &a, int64_t n, bool given, bool direct, FewArgs &f) {
    const int sms = sm_count();
    if (n < 1 || !a.rows_planned || a.avg_units <= 0 || a.n_stages <= 0 || sms <= 0) return false;
    const int64_t work = a.n_stages + a.n_events / 64;
    if (!direct && work < (given ? 24 : 8)) return false;
    const int64_t width = a.n_events / a.n_stages;
    const bool drawing = 3 * (int64_t)a.n_sampled >= 2 * (int64_t)a.n_entries;
    const int most = given             ? 12
                     : work < 12       ? 1
                     : work < 24       ? 4
                     : width <= 24     ? 20
                     : a.n_stages < 40 ? 16
                     : width <= 36 || drawing ? 20 : 18;
    if (n > (int64_t)most * sms) return false;
    f.given = given;
    f.n = (int32_t)n;
    f.ns = (int32_t)((n + sms - 1) / sms);
    f.ctas = (int32_t)((n + f.ns - 1) / f.ns);
    f.cta_entries = ((int64_t)a.n_entries + a.n_stages + 2) / 2 * 2 * f.ns;
    f.scratch = (size_t)f.ctas * (size_t)f.cta_entries * sizeof(double);
    if (f.scratch > kFewScratch) return false;
    const size_t win = ((size_t)a.window_slots * f.ns * sizeof(double) + 127) / 128 * 128;
    const size_t ev = (size_t)a.stage_events * sizeof(EvRec), pred = (size_t)a.stage_entries * sizeof(PredRec);
    const size_t dur = (size_t)(a.stage_entries + 1) / 2 * 2 * f.ns * sizeof(double);
    const size_t buf = (ev + pred + dur + 127) / 128 * 128;
    const int64_t units = (int64_t)a.stage_events * f.ns;
    // Lanes over an event's entries shorten its chain while the stage's warps are few; past
    // some 16 warps their reductions cost more issue than they save (50,000 events in stages
    // of up to 128: one sample a CTA 1 lane 681 us, 4 lanes 594; 20,017 in stages of 37,
    // eight samples: 1 lane 568, 4 lanes 627).
    f.lanes = units <= 128 ? 4 : 1;
    if (win + (f.lanes > 1 ? 3 : 2) * buf > kFewSmem) return false;
    f.ring_off = (int32_t)win;
    f.pred_off = (int32_t)ev;
    f.dur_off = (int32_t)(ev + pred);
    f.buf_bytes = (int32_t)buf;
    f.ring = (int32_t)((kFewSmem - win) / buf < (size_t)kFewRing ? (kFewSmem - win) / buf : kFewRing);
    f.smem = (int32_t)(win + f.ring * buf);
    const int unit = f.lanes * f.ns;  // threads an event
    const int64_t all = (int64_t)a.stage_events * unit;
    f.workers = (int32_t)(all < 864 ? all : 864 / unit * unit);
    f.threads = (f.workers + 31) / 32 * 32 + 32;
    return true;
}

cudaError_t launch_few(const KArgs &a, const FewArgs &f, cudaStream_t st) {
    // CTAs along y: a warp for each item of the largest stage, up to 64 CTAs an SM in all
    const int64_t lanes = f.n >= 32 ? 32 : f.n, run = f.n >= 32 ? kFewDrawRun : 1;
    const int per_lane = f.n <= 64 ? 1 : f.n <= 1024 || f.given ? 2 : 4;  // samples a lane
    const int64_t blocks = (f.n + 32 * per_lane - 1) / (32 * per_lane);
    const int64_t items = ((int64_t)a.stage_entries * lanes + 32 * run - 1) / (32 * run) * blocks;
    const int64_t per = (items + kFewDrawThreads / 32 - 1) / (kFewDrawThreads / 32);
    const int64_t most = (int64_t)64 * sm_count() / a.n_stages + 1;
    const unsigned gy = (unsigned)(per < 1 ? 1 : per < most ? per : most);
    const int64_t per_cta = kFewDrawThreads * run * gy;
    const int64_t aux = f.durations && a.n_aux > 0 ? ((int64_t)a.n_aux * f.n + per_cta - 1) / per_cta : 0;
    void (*draw)(const KArgs, const FewArgs) =
        f.given ? per_lane == 1 ? k_few_draw<true, 1> : k_few_draw<true, 2>
                 : per_lane == 1 ? k_few_draw<false, 1> : per_lane == 2 ? k_few_draw<false, 2> : k_few_draw<false, 4>;
    draw<<<dim3((unsigned)(a.n_stages + (aux < 64 ? aux : 64)), gy), kFewDrawThreads, 0, st>>>(a, f);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const bool pos = a.positive && !f.given;
    void (*fn)(const KArgs, const FewArgs) =
        f.lanes == 4 ? pos ? k_few<true, 4> : k_few<false, 4> : pos ? k_few<true, 1> : k_few<false, 1>;
    e = raise_smem_limit((const void *)fn, (size_t)f.smem);
    if (e != cudaSuccess) return e;
    fn<<<(unsigned)f.ctas, (unsigned)f.threads, (size_t)f.smem, st>>>(a, f);
    return cudaGetLastError();
}

}  // namespace mcd
