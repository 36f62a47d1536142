// mcd_prop_given.cu -- the propagation of given durations.
#include "mcd_device.cuh"

namespace mcd {

cudaError_t launch_prop_given(const KArgs &a, bool win_smem, cudaStream_t st) {
    const bool wide = win_smem && use_wide(a);
    const KArgs w = wide ? wide_args(a) : a;
    const int tile = wide ? kWideTile : kTile;
    const dim3 grid((unsigned)((a.n + tile - 1) / tile));
    // (4,000 events x 4,864 samples, 8 warps: of 3.5 predecessors 627 us by the short form,
    // 659 by the long one; of 4.5 851 and 800.  Wide tiles have no registers left for it.)
    const bool lists = (int64_t)a.n_entries > (int64_t)kGivenAhead * a.n_events;
    void (*fn)(const KArgs) = wide       ? k_propagate_given<true, 2, false>
                              : win_smem ? lists ? k_propagate_given<true, 1, true> : k_propagate_given<true, 1, false>
                              : lists    ? k_propagate_given<false, 1, true>
                                         : k_propagate_given<false, 1, false>;
    const cudaError_t e = raise_smem_limit((const void *)fn, (size_t)w.smem_total);
    if (e != cudaSuccess) return e;
    fn<<<grid, (unsigned)(pick_warps(w, grid.x, kGivenWarps, kGivenWarps) * 32), (size_t)w.smem_total, st>>>(w);
    return cudaGetLastError();
}

}  // namespace mcd
