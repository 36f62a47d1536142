// mcd_prop_given.cu -- the propagation of given durations.
#include "mcd_device.cuh"

namespace mcd {

// Durations of fewer bytes are taken to be in L2 (129 MB): at 90 MB the form for those
// takes 5 % less time on average when they are and the same when not, at 100 to 200 MB
// 3 % more.
constexpr int64_t kGivenHotBytes = (int64_t)96 << 20;

cudaError_t launch_prop_given(const KArgs &a, bool win_smem, cudaStream_t st) {
    const bool wide = win_smem && use_wide(a);
    const KArgs w = wide ? wide_args(a) : a;
    const int tile = wide ? kWideTile : kTile;
    const dim3 grid((unsigned)((a.n + tile - 1) / tile));
    // (4,000 events x 4,864 samples, 8 warps: of 3.9 predecessors 742 us ahead, 758 in
    // groups; of 4.4 858 and 820; 32 warps, whose reads overlap more, of 2.5 217 and 223,
    // of 3.5 296 and 283.  Wide tiles have no registers left for groups.)
    const bool lists = (int64_t)a.n_entries > (int64_t)kGivenAhead * a.n_events;
    const bool hot = (int64_t)a.n_entries * a.n * (int64_t)sizeof(double) < kGivenHotBytes;
    constexpr int kCold = kGivenGroups, kHot = kGivenGroupsHot;
    void (*fn)(const KArgs) = wide        ? k_propagate_given<true, 2, kGivenAheadOnce>
                              : !win_smem ? hot ? k_propagate_given<false, 1, kHot> : k_propagate_given<false, 1, kCold>
                              : hot       ? k_propagate_given<true, 1, kHot>
                              : lists     ? k_propagate_given<true, 1, kCold>
                                          : k_propagate_given<true, 1, kGivenAheadOnce>;
    const cudaError_t e = raise_smem_limit((const void *)fn, (size_t)w.smem_total);
    if (e != cudaSuccess) return e;
    fn<<<grid, (unsigned)(pick_warps(w, grid.x, kGivenWarps, kGivenWarps) * 32), (size_t)w.smem_total, st>>>(w);
    return cudaGetLastError();
}

}  // namespace mcd
