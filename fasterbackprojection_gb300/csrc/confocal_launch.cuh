// Launchers of the confocal gather, one translation unit per family so that
// the variants compile in parallel.
#pragma once

#include "bp_gather.cuh"

namespace fbp {

// Voxels per thread along x: 16 (the scan point's geometry and the stage's
// bookkeeping amortised over more pairs: 2.67e12 -> 2.74e12 pairs/s at 256^3
// with the gather as it then was), 8 for the sampled gather (its tiles are the MIS
// sampling tiles) and for the voxel-scattering walk, which takes 16 only where
// every walk is as long as its unrolled steps and the volume needs no chains:
// 64^2 x 1024 -> 256^3 50.8 against 53.5 ms, but with longer walks (64^2 x 2048)
// 118.0 against 116.2, and 40^2 x 1024 -> 160^3 10.26 against 9.76.
constexpr int kKV = 8, kKVFull = 16, kWY = 2, kWZ = 4;

fbp_status gather_full(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                       bool bounce, float t0, bool capped);
fbp_status gather_sampled(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                          bool bounce, float t0, bool capped);
// sp: steps every walk may take unrolled (2..4); free_walk: every walk takes
// them all.
fbp_status gather_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem, cudaStream_t stream,
                          int sp, bool free_walk, bool bounce, bool capped);
// 16 voxels per thread: free walks.
fbp_status gather_scatter_wide(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                               cudaStream_t stream, int sp, bool bounce, bool capped);
// The same with p.chains CTAs per tile.
fbp_status gather_full_split(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                             cudaStream_t stream, bool bounce, float t0, bool capped);
fbp_status gather_scatter_split(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                                cudaStream_t stream, int sp, bool free_walk, bool bounce, bool capped);

// One launch of the gather; SPLIT: p.chains CTAs per tile, then the fold.
template <int PATH, bool BOUNCE, bool SAMPLED, bool CLAMP, bool SPLIT, int KV = SAMPLED ? kKV : kKVFull>
fbp_status go_confocal(fbp_context* ctx, ConfocalGatherParams p, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kernel = confocal_gather_kernel<KV, kWY, kWZ, PATH, BOUNCE, SAMPLED, CLAMP, SPLIT>;
    FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t n = (uint64_t)p.Vx * p.Vy * p.Vz;
    if (SPLIT) grid.x *= p.chains;
    kernel<<<grid, 32 * kWY * kWZ, smem, stream>>>(p);
    FBP_CHECK_LAUNCH(ctx, "confocal_gather_kernel");
    return SPLIT ? fold_chains(ctx, p.chain_sums, p.chains, n, p.volume, stream) : FBP_OK;
}

template <bool SAMPLED, bool SPLIT>
fbp_status dispatch_confocal(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                             cudaStream_t stream, bool bounce, float t0, bool capped) {
    if (!bounce && t0 == 0.f) {
        if (capped) return go_confocal<PATH_2D, false, SAMPLED, true, SPLIT>(ctx, p, grid, smem, stream);
        return go_confocal<PATH_2D, false, SAMPLED, false, SPLIT>(ctx, p, grid, smem, stream);
    }
    switch ((t0 > 0.f ? 4 : 0) + (bounce ? 2 : 0) + (capped ? 1 : 0)) {
        case 0: return go_confocal<PATH_FAST, false, SAMPLED, false, SPLIT>(ctx, p, grid, smem, stream);
        case 1: return go_confocal<PATH_FAST, false, SAMPLED, true, SPLIT>(ctx, p, grid, smem, stream);
        case 2: return go_confocal<PATH_FAST, true, SAMPLED, false, SPLIT>(ctx, p, grid, smem, stream);
        case 3: return go_confocal<PATH_FAST, true, SAMPLED, true, SPLIT>(ctx, p, grid, smem, stream);
        case 4: return go_confocal<PATH_EXACT, false, SAMPLED, false, SPLIT>(ctx, p, grid, smem, stream);
        case 5: return go_confocal<PATH_EXACT, false, SAMPLED, true, SPLIT>(ctx, p, grid, smem, stream);
        case 6: return go_confocal<PATH_EXACT, true, SAMPLED, false, SPLIT>(ctx, p, grid, smem, stream);
        default: return go_confocal<PATH_EXACT, true, SAMPLED, true, SPLIT>(ctx, p, grid, smem, stream);
    }
}

// The voxel-scattering walks of prefix SP: predicated steps (clamped window
// index), or unconditional ones, clamped only where the window is the row.
template <int SP, bool SPLIT, int KV>
fbp_status dispatch_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                            cudaStream_t stream, bool free_walk, bool bounce, bool capped) {
    constexpr int W = PATH_SCATTER + SP - 2, F = W + kScatterForms;
    if constexpr (KV == kKV) {
        if (!free_walk) {
            if (bounce) return go_confocal<W, true, false, true, SPLIT, KV>(ctx, p, grid, smem, stream);
            return go_confocal<W, false, false, true, SPLIT, KV>(ctx, p, grid, smem, stream);
        }
    }
    if (bounce) {
        if (capped) return go_confocal<F, true, false, true, SPLIT, KV>(ctx, p, grid, smem, stream);
        return go_confocal<F, true, false, false, SPLIT, KV>(ctx, p, grid, smem, stream);
    }
    if (capped) return go_confocal<F, false, false, true, SPLIT, KV>(ctx, p, grid, smem, stream);
    return go_confocal<F, false, false, false, SPLIT, KV>(ctx, p, grid, smem, stream);
}

template <bool SPLIT, int KV = kKV>
fbp_status dispatch_scatter(fbp_context* ctx, const ConfocalGatherParams& p, dim3 grid, size_t smem,
                            cudaStream_t stream, int sp, bool free_walk, bool bounce, bool capped) {
    static_assert(kScatterMaxPrefix == 4, "one case per prefix");
    switch (sp) {
        case 2: return dispatch_scatter<2, SPLIT, KV>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        case 3: return dispatch_scatter<3, SPLIT, KV>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        case 4: return dispatch_scatter<4, SPLIT, KV>(ctx, p, grid, smem, stream, free_walk, bounce, capped);
        default: return set_error(FBP_ERR_INTERNAL, "voxel scattering: no kernel for this step prefix");
    }
}

}  // namespace fbp
