// The voxel-scattering gather, 16 voxels per thread.
#include "confocal_launch.cuh"

namespace fbp {
fbp_status gather_scatter_wide(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                               cudaStream_t stream, int sp, bool bounce, bool capped) {
    return dispatch_scatter<false, kKVFull>(ctx, p, grid, smem, stream, sp, true, bounce, capped);
}
}  // namespace fbp
