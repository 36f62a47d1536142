// mcd_prop_wide.cu -- instantiations of k_propagate over wide tiles: two samples a
// lane, 64 a tile (a separate translation unit keeps the build parallel).
#include "mcd_device.cuh"

namespace mcd {

// For DAGs of non-negative finite times whose tables block sits in shared memory
// (use_wide).
cudaError_t launch_prop_wide(const KArgs &w, bool stats, dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
    void (*fn)(const KArgs) = stats ? k_propagate<true, true, true, kTablesSmem, 2>
                                    : k_propagate<true, false, true, kTablesSmem, 2>;
    const cudaError_t e = raise_smem_limit((const void *)fn, smem);
    if (e != cudaSuccess) return e;
    fn<<<grid, block, smem, st>>>(w);
    return cudaGetLastError();
}

}  // namespace mcd
