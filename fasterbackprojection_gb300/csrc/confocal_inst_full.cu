// The gather over all scan points, one CTA per voxel tile.
#include "confocal_launch.cuh"

namespace fbp {
fbp_status gather_full(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                       bool bounce, float t0, bool capped) {
    return dispatch_confocal<false, false>(ctx, p, grid, smem, stream, bounce, t0, capped);
}
}  // namespace fbp
