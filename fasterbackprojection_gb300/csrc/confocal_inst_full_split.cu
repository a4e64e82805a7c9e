// The gather over all scan points, one CTA per chain of a voxel tile.
#include "confocal_launch.cuh"

namespace fbp {
fbp_status gather_full_split(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                             bool bounce, float t0, bool capped) {
    return dispatch_confocal<false, true>(ctx, p, grid, smem, stream, bounce, t0, capped);
}
}  // namespace fbp
