// Persistent multi-capture gather kernels.
#include "batch_launch.cuh"

namespace fbp {
fbp_status batch_prepare_kernel(const BatchLaunch& b, int* ctas_per_sm) {
    return batch_dispatch(nullptr, b, 0, nullptr, ctas_per_sm);
}
fbp_status batch_launch(fbp_context* ctx, const BatchLaunch& b, int ctas, cudaStream_t s) {
    return batch_dispatch(ctx, b, ctas, s, nullptr);
}
}  // namespace fbp
