// The voxel-scattering gather, one CTA per chain of a voxel tile.
#include "confocal_launch.cuh"

namespace fbp {
fbp_status gather_scatter_split(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                                  int sp, bool free_walk, bool bounce, bool capped) {
    return dispatch_scatter<true>(ctx, p, grid, smem, stream, sp, free_walk, bounce, capped);
}
}  // namespace fbp
