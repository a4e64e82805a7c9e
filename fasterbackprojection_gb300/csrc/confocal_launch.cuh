// Launchers of the confocal gather, one translation unit per family so that
// the variants compile in parallel.
#pragma once

#include "bp_gather.cuh"

namespace fbp {

// Voxels per thread along x: 16 (the scan point's geometry and the stage's
// bookkeeping amortised over more pairs: 2.67e12 -> 2.74e12 pairs/s at 256^3
// with the gather as it then was; the voxel-scattering walk 52.2 -> 48.8 ms
// for 64^2 x 1024 -> 256^3), 8 for the sampled gather (its tiles are the MIS
// sampling tiles).
constexpr int kKV = 8, kKVFull = 16, kWY = 2, kWZ = 4;

fbp_status gather_full(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                       bool bounce, float t0, bool capped);
fbp_status gather_sampled(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                          bool bounce, float t0, bool capped);
// sp: steps every walk may take unrolled (2..4); free_walk: every walk takes
// them all.
fbp_status gather_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                          int sp, bool free_walk, bool bounce, bool capped);
// The same with p.chains CTAs per tile, in clusters.
fbp_status gather_full_cluster(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                               cudaStream_t stream, bool bounce, float t0, bool capped);
fbp_status gather_scatter_cluster(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                                  cudaStream_t stream, int sp, bool free_walk, bool bounce, bool capped);

// One launch of the gather; CLUSTER: clusters of p.chains CTAs along x.
template <int PATH, bool BOUNCE, bool SAMPLED, bool CLAMP, bool CLUSTER>
fbp_status go_confocal(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream) {
    constexpr int KV = SAMPLED ? kKV : kKVFull;
    auto kernel = confocal_gather_kernel<KV, kWY, kWZ, PATH, BOUNCE, SAMPLED, CLAMP, CLUSTER>;
    FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if constexpr (!CLUSTER) {
        kernel<<<grid, 32 * kWY * kWZ, smem, stream>>>(p);
    } else {
        FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = p.chains;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid.x * p.chains, grid.y, grid.z);
        cfg.blockDim = dim3(32 * kWY * kWZ);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        FBP_TRY_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    }
    FBP_CHECK_LAUNCH(ctx, "confocal_gather_kernel");
    return FBP_OK;
}

template <bool SAMPLED, bool CLUSTER>
fbp_status dispatch_confocal(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                             cudaStream_t stream, bool bounce, float t0, bool capped) {
    if (!bounce && t0 == 0.f) {
        if (capped) return go_confocal<PATH_2D, false, SAMPLED, true, CLUSTER>(ctx, p, grid, smem, stream);
        return go_confocal<PATH_2D, false, SAMPLED, false, CLUSTER>(ctx, p, grid, smem, stream);
    }
    switch ((t0 > 0.f ? 4 : 0) + (bounce ? 2 : 0) + (capped ? 1 : 0)) {
        case 0: return go_confocal<PATH_FAST, false, SAMPLED, false, CLUSTER>(ctx, p, grid, smem, stream);
        case 1: return go_confocal<PATH_FAST, false, SAMPLED, true, CLUSTER>(ctx, p, grid, smem, stream);
        case 2: return go_confocal<PATH_FAST, true, SAMPLED, false, CLUSTER>(ctx, p, grid, smem, stream);
        case 3: return go_confocal<PATH_FAST, true, SAMPLED, true, CLUSTER>(ctx, p, grid, smem, stream);
        case 4: return go_confocal<PATH_EXACT, false, SAMPLED, false, CLUSTER>(ctx, p, grid, smem, stream);
        case 5: return go_confocal<PATH_EXACT, false, SAMPLED, true, CLUSTER>(ctx, p, grid, smem, stream);
        case 6: return go_confocal<PATH_EXACT, true, SAMPLED, false, CLUSTER>(ctx, p, grid, smem, stream);
        default: return go_confocal<PATH_EXACT, true, SAMPLED, true, CLUSTER>(ctx, p, grid, smem, stream);
    }
}

// The voxel-scattering walks of prefix SP: predicated steps (clamped window
// index), or unconditional ones, clamped only where the window is the row.
template <int SP, bool CLUSTER>
fbp_status dispatch_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                            cudaStream_t stream, bool free_walk, bool bounce, bool capped) {
    constexpr int W = PATH_SCATTER + SP - 2, F = W + kScatterForms;
    if (!free_walk) {
        if (bounce) return go_confocal<W, true, false, true, CLUSTER>(ctx, p, grid, smem, stream);
        return go_confocal<W, false, false, true, CLUSTER>(ctx, p, grid, smem, stream);
    }
    if (bounce) {
        if (capped) return go_confocal<F, true, false, true, CLUSTER>(ctx, p, grid, smem, stream);
        return go_confocal<F, true, false, false, CLUSTER>(ctx, p, grid, smem, stream);
    }
    if (capped) return go_confocal<F, false, false, true, CLUSTER>(ctx, p, grid, smem, stream);
    return go_confocal<F, false, false, false, CLUSTER>(ctx, p, grid, smem, stream);
}

template <bool CLUSTER>
fbp_status dispatch_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                            cudaStream_t stream, int sp, bool free_walk, bool bounce, bool capped) {
    static_assert(kScatterMaxPrefix == 4, "one case per prefix");
    switch (sp) {
        case 2: return dispatch_scatter<2, CLUSTER>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        case 3: return dispatch_scatter<3, CLUSTER>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        case 4: return dispatch_scatter<4, CLUSTER>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        default: return set_error(FBP_ERR_INTERNAL, "voxel scattering: no kernel for this step prefix");
    }
}

}  // namespace fbp
