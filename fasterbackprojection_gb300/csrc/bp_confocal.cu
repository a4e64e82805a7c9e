// Confocal backprojection as a voxel-tiled gather.
//
// Replaces Laser::reconstructAABBConfocal (Laser.cu:482-498) and
// backprojectConfocalVoxel (transient_reconstruction.cuh:93-136).  The
// reference launches one thread per (voxel, scan point) pair and adds each
// contribution with a global FP32 atomic.  Here one CTA owns a tile of voxels
// and walks all scan points; for every scan point it stages only the window
// of time bins the tile can reach into shared memory (one bulk copy), so each
// pair costs a shared-memory load instead of a global gather + atomic, and the
// sum order is fixed (reproducible run to run).  Volumes with few tiles walk
// the scan points in several chains, one CTA each, folded afterwards.
//
// Data layout in HBM (per call, in the context's scratch):
//   rows   [L][row_pitch] FP32: one padded row per scan point, time
//          innermost, values <= 1e-5 already replaced by 0 (the reference
//          skips them), zeros in [T, row_pitch).  BF16 / FP16 captures are
//          widened here (exactly), so the pair loop reads FP32 with no
//          per-pair conversion; the gather is bound by instruction issue, not
//          by the bytes of its windows.
//   scan   [L] float4 (x, y, z, bounce)   bounce = |l-laser|+|l-sensor| or 0
//   axes   xs[Vx], ys[Vz], zs[Vy]         voxel-centre coordinates
#include "fbp_internal.cuh"
#include "bp_common.cuh"
#include "bp_gather.cuh"
#include "confocal_launch.cuh"

#include <algorithm>
#include <cmath>

namespace fbp {

// ------------------------------------------------------------ prep kernels --

__global__ void axis_tables_kernel(float* __restrict__ xs, float* __restrict__ ys, float* __restrict__ zs,
                                   uint32_t Vx, uint32_t Vy, uint32_t Vz, float mnx, float mny, float mnz, float sx,
                                   float sy, float sz) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // transient_reconstruction.cuh:106: (vx, vz, vy) drive world (x, y, z).
    if (i < Vx) xs[i] = ref_voxel_coord(i, sx, mnx);
    if (i < Vz) ys[i] = ref_voxel_coord(i, sy, mny);
    if (i < Vy) zs[i] = ref_voxel_coord(i, sz, mnz);
}

// Per scan point (x, y, z, bounce): transient_reconstruction.cuh:109-110.
__global__ void scan_table_kernel(float4* __restrict__ out, const float* __restrict__ xyz, uint32_t n, int discard,
                                  float ax, float ay, float az, float bx, float by, float bz, int confocal_pair) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = xyz[3 * (size_t)i], y = xyz[3 * (size_t)i + 1], z = xyz[3 * (size_t)i + 2];
    float b = 0.f;
    if (discard == 0) {
        // confocal: |l - laserPos| + |l - sensorPos|; exhaustive tables carry
        // one distance each (|l - laserPos| or |s - sensorPos|).
        const float d1 = ref_distance(x, y, z, ax, ay, az);
        b = confocal_pair ? add_rn(d1, ref_distance(x, y, z, bx, by, bz)) : d1;
    }
    out[i] = make_float4(x, y, z, b);
}

namespace {

// Depth slices [z_begin, z_end) of the volume (the whole volume by default)
// into `volume` ([z_end - z_begin][Vy][Vx]).  The window plan and the voxel
// tables are those of the whole volume, so with z_begin a multiple of the
// tile depth a slab is bitwise the same rows of the full result.
fbp_status launch_confocal(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                           const float* laser_xyz, float* volume, cudaStream_t stream, const SampleParams* smp,
                           uint32_t z_begin = 0, uint32_t z_end = 0xFFFFFFFFu, bool scatter = false) {
    const uint32_t L = in.num_laser_targets, T = in.num_time_bins;
    const uint32_t Vx = in.voxel_res[0], Vy = in.voxel_res[1], Vz = in.voxel_res[2];
    if (z_end > Vz) z_end = Vz;
    if (z_begin >= z_end) return FBP_OK;
    constexpr int ALIGN = 4;  // FP32 rows

    // The voxel-scattering variant reads every bin of dist -/+ half the voxel
    // diagonal, one step past the end (up to max(step, diagonal) from 0 where
    // a walk is clipped at 0).
    const double vdiag = std::sqrt((double)in.voxel_size[0] * in.voxel_size[0] +
                                   (double)in.voxel_size[1] * in.voxel_size[1] +
                                   (double)in.voxel_size[2] * in.voxel_size[2]);
    const double extra = scatter ? 1.52 * vdiag + 2.0 * std::fabs((double)in.time_step) : 0.0;
    // Steps per (voxel, scan point): at most ceil(diagonal / (dt + EPS)),
    // one more where rounding lands on the end; the kernel unrolls 2..4
    // of them and loops over the rest.  Where even the shortest walk
    // takes all the unrolled steps (a 1e-4 m margin over the rounding of
    // the path arithmetic below 64 m) they need no end test, and the
    // unclamped window index of the other paths applies.
    const double step = (double)in.time_step + (double)FBP_EPS;
    const int sp = (int)std::min(std::max(std::ceil(vdiag / step), 2.0), (double)kScatterMaxPrefix);
    const bool free_walk = scatter && (sp - 1) * step + 1e-4 < vdiag;
    // ... and where none takes more (sp steps already pass the far end).
    const bool exact_walk = free_walk && sp * step > vdiag + 1e-4;

    // Windows of the largest tile (clamped to the volume) of kv voxels along x.
    // The sampled kernel also holds its cluster list in static shared memory.
    WindowPlan wp, wide;
    auto plan = [&](uint32_t kv, bool narrow, WindowPlan* out) -> fbp_status {
        const double ex = (double)std::min<uint32_t>(kv, Vx) * std::fabs(in.voxel_size[0]);
        const double ey = (double)std::min<uint32_t>(4 * kWZ, Vz) * std::fabs(in.voxel_size[1]);
        const double ez = (double)std::min<uint32_t>(8 * kWY, Vy) * std::fabs(in.voxel_size[2]);
        return plan_window(ctx, ex, ey, ez, in.time_step, T, ALIGN, sizeof(float),
                           ConfocalGatherParams::meta_bytes((int)kv) + (smp ? kSampledStaticSmem : 0) +
                               kahan_smem_bytes((int)kv, 32 * kWY * kWZ, scatter) + 16,
                           out, "fbp_backproject_confocal", extra, gather_ctas(32 * kWY * kWZ, narrow),
                           ConfocalGatherParams::kWindowBufs);
    };
    ConfocalGatherParams p{};
    uint32_t kv = smp || scatter ? kKV : kKVFull;
    FBP_TRY(plan(kv, scatter, &wp));
    if (smp) wp.smem -= kSampledStaticSmem;
    p.chains = smp ? 1 : scatter ? scatter_chains(ctx, in, wp.smem, vdiag / step) : gather_chains(ctx, in, wp.smem);
    if (exact_walk) {
        if (plan(kKVFull, false, &wide) != FBP_OK) {
            clear_error();
        } else if (gather_chains(ctx, in, wide.smem) == 1) {
            kv = kKVFull;
            wp = wide;
            p.chains = 1;
        }
    }
    float* rows = nullptr;
    FBP_TRY(gather_scratch(ctx, (size_t)L * wp.pitch * sizeof(float), &p.chains, (uint64_t)Vx * Vy * (z_end - z_begin), stream,
                           &rows, &p.chain_sums));
    PrepTables tables{};
    FBP_TRY(table_buffers(ctx, in, laser_xyz, nullptr, true, stream, &tables));
    FBP_TRY(prepare_gather(ctx, dtype, PrepRows{cube, rows, L, T, wp.pitch, layout == FBP_LAYOUT_TIME_MAJOR}, tables, stream));

    p.scan = tables.lasers;
    p.xs = tables.axes;
    p.ys = p.xs + Vx;
    p.zs = p.ys + Vz;
    p.rows = rows;
    p.volume = volume;
    p.status = ctx->status_dev;
    p.ys += z_begin;
    p.Vx = Vx; p.Vy = Vy; p.Vz = z_end - z_begin; p.L = L; p.T = T;
    p.t0 = in.time_offset;
    p.dt = in.time_step;
    p.row_pitch = wp.pitch;
    p.slot_w = wp.slot_w;
    p.ch = wp.ch;
    for (int k = 0; k < 3; ++k) p.vs[k] = in.voxel_size[k];
    p.exact_weights = ctx->weight_mode == FBP_WEIGHTS_REFERENCE;
    if (smp) p.smp = *smp;
    dim3 grid(cdiv(Vx, kv), cdiv(Vy, 8 * kWY), cdiv(z_end - z_begin, 4 * kWZ));
    const bool bounce = in.discard_first_last_bounces == 0;
    if (scatter) {
        p.scat_exact = exact_walk;
        if (kv == kKVFull) return gather_scatter_wide(ctx, p, grid, wp.smem, stream, sp, bounce, wp.capped);
        if (p.chains > 1) return gather_scatter_split(ctx, p, grid, wp.smem, stream, sp, free_walk, bounce, wp.capped);
        return gather_scatter(ctx, p, grid, wp.smem, stream, sp, free_walk, bounce, wp.capped);
    }
    if (smp) return gather_sampled(ctx, p, grid, wp.smem, stream, bounce, in.time_offset, wp.capped);
    if (p.chains > 1) return gather_full_split(ctx, p, grid, wp.smem, stream, bounce, in.time_offset, wp.capped);
    return gather_full(ctx, p, grid, wp.smem, stream, bounce, in.time_offset, wp.capped);
}

}  // namespace

// The most scratch that chains may ask for (volumes beyond 16 M voxels have tiles
// enough for every SM).
constexpr size_t kChainSumBytes = (size_t)128 << 20;

// Chains (CTAs per tile) of a gather: 1 where the tiles alone keep every SM
// busy, else as many as a model of the launch asks for.  The model, in units of
// one group at an SM's full rate: the busiest SM's CTAs, each with its share of
// the groups and half a group of set-up, at the rate of the CTAs resident
// together (one or two reach 0.68 and 0.88 of three; 0.55, 0.8 and 0.93 of four),
// the uneven end (a whole CTA where tiles differ in their idle warps), and the
// sums' way through memory and the fold's launch.  One CTA per tile against this rule (both with the
// tables' launches of their own, which one launch for rows and tables has since
// taken 8-28 us off): 32^2 x 256 -> 32^3 328 -> 45 us (16 chains), 64^2 x 512 ->
// 64^3 1264 -> 432 us (7), 90^2 x 700 -> 75 x 101 x 83 4028 -> 2189 us (16),
// 128^2 x 1024 -> 128^3 14.2 -> 11.5 ms (5), 8^2 x 16^2 x 512 -> 48^3 2251 ->
// 666 us (14).  The sums through the
// shared memory of a cluster instead (at most 16 chains, and clusters leave
// part of a GPC's slots empty): 48, 483, 2596 us, 11.9 ms, 728 us.
uint32_t split_chains(const fbp_context* ctx, uint64_t tiles, double busy, uint64_t groups, int occ, double group_us,
                      uint64_t n) {
    constexpr double kRates[2][kScatterCtasPerSm] = {{0.68, 0.88, 1.0}, {0.55, 0.8, 0.93, 1.0}};
    const double* const kRate = kRates[occ > kGatherCtasPerSm];
    constexpr uint32_t kMaxChains = 32;
    uint32_t best = 1;
    double best_t = 0.0;
    const uint64_t most = std::min<uint64_t>(std::min<uint64_t>(kMaxChains, groups), kChainSumBytes / (8 * n));
    for (uint32_t c = 1; c <= std::max<uint64_t>(most, 1); ++c) {
        const uint64_t per_sm = cdiv(tiles * c, (uint64_t)ctx->sm_count);
        const double rate = kRate[std::min<uint64_t>(per_sm, (uint64_t)occ) - 1] / kRate[occ - 1];
        const double ctas = busy < 1.0 ? (double)(tiles * c) * busy / ctx->sm_count + 1.0 : (double)per_sm + 0.3;
        double t = ctas * ((double)((groups + c - 1) / c) + 0.5) / rate;
        if (c > 1) t += (3.0 + 0.2 * c + (double)c * (double)n * 16.0 / 5.0e6) / group_us;  // 5 TB/s
        if (c == 1 || t < 0.98 * best_t) {
            best = c;
            best_t = t;
        }
    }
    return best;
}

double busy_warps(const uint32_t res[3]) {
    return (double)cdiv(res[1], 8) * cdiv(res[2], 4) / ((double)cdiv(res[1], 16) * 2 * cdiv(res[2], 16) * 4);
}

uint32_t gather_chains(const fbp_context* ctx, const fbp_recon_info& in, size_t smem) {
    static_assert(kWY == 2 && kWZ == 4, "busy_warps counts warps of 8 x 4 in tiles of 16 x 16");
    const uint64_t tiles = (uint64_t)cdiv(in.voxel_res[0], kKVFull) * cdiv(in.voxel_res[1], 8 * kWY) *
                           cdiv(in.voxel_res[2], 4 * kWZ);
    return split_chains(ctx, tiles, busy_warps(in.voxel_res),
                        cdiv(in.num_laser_targets, ConfocalGatherParams::kGroup), resident_ctas(smem, kGatherCtasPerSm),
                        kGatherGroupUs, (uint64_t)in.voxel_res[0] * in.voxel_res[1] * in.voxel_res[2]);
}

uint32_t scatter_chains(const fbp_context* ctx, const fbp_recon_info& in, size_t smem, double steps) {
    const uint64_t tiles = (uint64_t)cdiv(in.voxel_res[0], kKV) * cdiv(in.voxel_res[1], 8 * kWY) *
                           cdiv(in.voxel_res[2], 4 * kWZ);
    return split_chains(ctx, tiles, busy_warps(in.voxel_res),
                        cdiv(in.num_laser_targets, ConfocalGatherParams::kGroup), resident_ctas(smem, kScatterCtasPerSm),
                        kScatterStepUs * std::max(steps, 2.0), (uint64_t)in.voxel_res[0] * in.voxel_res[1] * in.voxel_res[2]);
}

fbp_status gather_scratch(fbp_context* ctx, size_t row_bytes, uint32_t* chains, uint64_t n, cudaStream_t stream,
                          float** rows, float** sums) {
    void* r = nullptr;
    const size_t at = (row_bytes + 255) & ~size_t(255), bytes = *chains > 1 ? (size_t)2 * *chains * n * sizeof(float) : 0;
    size_t& have = ctx->ws_bytes[WS_CHAIN_SUMS];
    void*& ws = ctx->ws[WS_CHAIN_SUMS];
    // A context's first call makes one allocation for both (each costs tens of
    // microseconds); later ones use what is behind the rows where it is enough.
    if (ctx->ws_bytes[WS_CUBE_ROWS] < row_bytes && have < bytes) {
        const fbp_status st = workspace(ctx, WS_CUBE_ROWS, at + bytes, stream, &r);
        if (st != FBP_OK && st != FBP_ERR_OOM) return st;
        if (st == FBP_ERR_OOM) {
            cudaGetLastError();
            clear_error();
        }
    }
    FBP_TRY(workspace(ctx, WS_CUBE_ROWS, row_bytes, stream, &r));
    *rows = static_cast<float*>(r);
    if (*chains <= 1) return FBP_OK;
    if (ctx->ws_bytes[WS_CUBE_ROWS] >= at + bytes) {
        *sums = reinterpret_cast<float*>(static_cast<char*>(r) + at);
        return FBP_OK;
    }
    if (have < bytes) {
        // A smaller volume may want more of this than a larger one, so a graph
        // captured before must not lose its buffer to a later call: an outgrown
        // one lives as long as the context.  Each at least doubles the last, and one
        // of more than half of kChainSumBytes is that large at once and the last of
        // all: together they stay below twice kChainSumBytes.
        const size_t grown = bytes > kChainSumBytes / 2 ? kChainSumBytes : std::max(bytes, 2 * have);
        void* p = nullptr;
        if (!workspace_ready(ctx, WS_CHAIN_SUMS, bytes, stream)) {
            *chains = 1;
            return FBP_OK;
        }
        const cudaError_t e = cudaMalloc(&p, grown);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            *chains = 1;
            return FBP_OK;
        }
        FBP_TRY_CUDA(e);
        if (ws) ctx->ws_outgrown.push_back(ws);
        ws = p;
        have = grown;
    }
    *sums = static_cast<float*>(ws);
    return FBP_OK;
}

__global__ void fold_chains_kernel(const float* __restrict__ sums, uint32_t chains, uint64_t n, float* __restrict__ out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        float sum = 0.f, comp = 0.f;
#pragma unroll 4
        for (uint32_t c = 0; c < chains; ++c) {
            const float s = sums[2 * c * n + i], e = sums[(2 * c + 1) * n + i];
            kahan_fold(s, e, sum, comp);
        }
        out[i] = sum;
    }
}

fbp_status fold_chains(fbp_context* ctx, const float* sums, uint32_t chains, uint64_t n, float* out,
                       cudaStream_t stream) {
    const unsigned blocks = (unsigned)std::min<uint64_t>(cdiv(n, 256), (uint64_t)ctx->sm_count * 8);
    fold_chains_kernel<<<blocks, 256, 0, stream>>>(sums, chains, n, out);
    FBP_CHECK_LAUNCH(ctx, "fold_chains_kernel");
    return FBP_OK;
}

// Tile grid of the confocal gather (also the MIS sampling tiles).
void confocal_tile_grid(const fbp_recon_info& in, uint32_t out[3]) {
    out[0] = cdiv(in.voxel_res[0], kKV);
    out[1] = cdiv(in.voxel_res[1], 8 * kWY);
    out[2] = cdiv(in.voxel_res[2], 4 * kWZ);
}

fbp_status confocal_gather(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                           const float* laser_xyz, float* volume, cudaStream_t s, const SampleParams* smp) {
    return launch_confocal(ctx, in, cube, dtype, layout, laser_xyz, volume, s, smp);
}

fbp_status confocal_gather_scatter(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype,
                                   int layout, const float* laser_xyz, float* volume, cudaStream_t s) {
    return launch_confocal(ctx, in, cube, dtype, layout, laser_xyz, volume, s, nullptr, 0, 0xFFFFFFFFu, true);
}

fbp_status confocal_gather_slab(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                                const float* laser_xyz, uint32_t z_begin, uint32_t z_end, float* volume,
                                cudaStream_t s) {
    return launch_confocal(ctx, in, cube, dtype, layout, laser_xyz, volume, s, nullptr, z_begin, z_end);
}

fbp_status build_tables(fbp_context* ctx, const fbp_recon_info& in, const float* laser_xyz, cudaStream_t stream,
                        const float4** scan, const float** xs, const float** ys, const float** zs) {
    const uint32_t L = in.num_laser_targets;
    const uint32_t Vx = in.voxel_res[0], Vy = in.voxel_res[1], Vz = in.voxel_res[2];
    void* sp = nullptr;
    void* ap = nullptr;
    FBP_TRY(workspace(ctx, WS_SCAN_TABLE, (size_t)L * sizeof(float4), stream, &sp));
    FBP_TRY(workspace(ctx, WS_AXIS_TABLES, (size_t)(Vx + Vy + Vz) * sizeof(float), stream, &ap));
    float4* s = static_cast<float4*>(sp);
    float* a = static_cast<float*>(ap);
    scan_table_kernel<<<cdiv(L, 256), 256, 0, stream>>>(
        s, laser_xyz, L, (int)in.discard_first_last_bounces, in.laser_position[0], in.laser_position[1],
        in.laser_position[2], in.sensor_position[0], in.sensor_position[1], in.sensor_position[2], 1);
    FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
    const uint32_t vmax = std::max(Vx, std::max(Vy, Vz));
    axis_tables_kernel<<<cdiv(vmax, 256), 256, 0, stream>>>(a, a + Vx, a + Vx + Vz, Vx, Vy, Vz, in.hidden_min[0],
                                                            in.hidden_min[1], in.hidden_min[2], in.voxel_size[0],
                                                            in.voxel_size[1], in.voxel_size[2]);
    FBP_CHECK_LAUNCH(ctx, "axis_tables_kernel");
    *scan = s;
    *xs = a;
    *ys = a + Vx;
    *zs = a + Vx + Vz;
    return FBP_OK;
}

fbp_status plan_window(const fbp_context* ctx, double ex, double ey, double ez, double time_step, uint32_t T, int align,
                       size_t elem_bytes, size_t meta_bytes, WindowPlan* out, const char* who, double extra_path,
                       int ctas_per_sm, int window_bufs) {
    const double diag = std::sqrt(ex * ex + ey * ey + ez * ez);
    // Round trip across the tile (plus any extra path range), a 2-bin margin
    // on each side, alignment slack.
    const double span = (2.0 * diag + extra_path) / std::fabs(time_step) + 8.0 + align;
    const uint32_t t_round = (T + align - 1) / align * align;
    const uint32_t cap = t_round + align;
    uint32_t slot_w = span < (double)cap ? ((uint32_t)std::ceil(span) + align - 1) / align * align : cap;
    if (slot_w > cap) slot_w = cap;
    out->slot_w = slot_w;
    out->capped = slot_w == cap;
    out->pitch = t_round + slot_w;
    const size_t per_stage = (size_t)window_bufs * (slot_w + align) * elem_bytes;  // per scan point of a stage
    // Points per stage: 32, halved down to 8 where that lets one more CTA share
    // the SM (at 128^2 x 1024 -> 128^3 a stage of 16 keeps three CTAs instead
    // of two), below 8 only where not even one CTA fits otherwise.
    int ch = 0;
    for (int n = ctas_per_sm; n >= 2 && !ch; --n) {
        const size_t room = kSmSharedBytes / n - kCtaReservedShared;
        for (int c = 32; c >= 8 && !ch; c >>= 1)
            if (meta_bytes + (size_t)c * per_stage <= room) ch = c;
    }
    if (!ch) {
        ch = 32;
        while (ch > 1 && meta_bytes + (size_t)ch * per_stage > (size_t)ctx->smem_optin) ch >>= 1;
    }
    if (meta_bytes + (size_t)ch * per_stage > (size_t)ctx->smem_optin)
        return set_error(FBP_ERR_UNSUPPORTED, std::string(who) + ": time-bin window too large for shared memory");
    out->ch = ch;
    out->smem = meta_bytes + (size_t)ch * per_stage;
    return FBP_OK;
}

fbp_status validate_info(const fbp_recon_info* info, bool need_sensors, const char* who) {
    if (!info) return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": null info");
    const fbp_recon_info& in = *info;
    if (in.num_laser_targets == 0 || in.num_time_bins == 0 || (need_sensors && in.num_sensor_targets == 0))
        return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": empty capture (zero scan points or bins)");
    if (in.voxel_res[0] == 0 || in.voxel_res[1] == 0 || in.voxel_res[2] == 0)
        return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": zero voxel resolution");
    if (!(std::isfinite(in.time_step) && in.time_step > 0.f))
        return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": time_step must be finite and > 0");
    if (in.num_time_bins >= (1u << 22))
        return set_error(FBP_ERR_UNSUPPORTED, std::string(who) + ": more than 2^22 time bins");
    const uint64_t V = (uint64_t)in.voxel_res[0] * in.voxel_res[1] * in.voxel_res[2];
    if (V >= (1ull << 32)) return set_error(FBP_ERR_UNSUPPORTED, std::string(who) + ": more than 2^32 voxels");
    for (int k = 0; k < 3; ++k)
        if (!std::isfinite(in.hidden_min[k]) || !std::isfinite(in.voxel_size[k]))
            return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": non-finite volume geometry");
    if (!std::isfinite(in.time_offset)) return set_error(FBP_ERR_INVALID_ARG, std::string(who) + ": non-finite time_offset");
    return FBP_OK;
}

}  // namespace fbp

using namespace fbp;

extern "C" fbp_status fbp_backproject_confocal_scatter(fbp_context* ctx, const fbp_recon_info* info,
                                                       const void* cube, int dtype, int layout,
                                                       const float* laser_xyz, float* volume, void* stream) {
    return guarded("fbp_backproject_confocal_scatter", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, false, "fbp_backproject_confocal_scatter"));
        if (!cube || !laser_xyz || !volume)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_confocal_scatter: null buffer");
        if (layout != FBP_LAYOUT_TIME_MAJOR && layout != FBP_LAYOUT_TIME_INNER)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_confocal_scatter: unknown layout");
        if (!(info->time_step > 1e-4f))
            return set_error(FBP_ERR_UNSUPPORTED, "fbp_backproject_confocal_scatter: time_step must exceed 0.1 mm");
        return confocal_gather_scatter(ctx, *info, cube, dtype, layout, laser_xyz, volume, (cudaStream_t)stream);
    });
}

extern "C" fbp_status fbp_backproject_confocal(fbp_context* ctx, const fbp_recon_info* info, const void* cube,
                                               int dtype, int layout, const float* laser_xyz, float* volume,
                                               void* stream) {
    return guarded("fbp_backproject_confocal", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, false, "fbp_backproject_confocal"));
        if (!cube || !laser_xyz || !volume) return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_confocal: null buffer");
        if (layout != FBP_LAYOUT_TIME_MAJOR && layout != FBP_LAYOUT_TIME_INNER)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_confocal: unknown layout");
        if (dtype != FBP_F32 && dtype != FBP_BF16 && dtype != FBP_F16)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_confocal: unknown dtype");
        return confocal_gather(ctx, *info, cube, dtype, layout, laser_xyz, volume, (cudaStream_t)stream, nullptr);
    });
}

// ------------------------------------------------------------ diagnostics --

namespace fbp {

__device__ __forceinline__ void voxel_of(int64_t v, uint32_t Vx, uint32_t Vy, uint32_t& vx, uint32_t& vy, uint32_t& vz) {
    const uint64_t slice = (uint64_t)Vx * Vy;
    vz = (uint32_t)(v / slice);
    const uint32_t r = (uint32_t)(v % slice);
    vy = r / Vx;
    vx = r % Vx;
}

__global__ void debug_confocal_bins_kernel(fbp_recon_info in, const float4* __restrict__ scan,
                                           const int64_t* __restrict__ vidx, uint64_t nv, int32_t* __restrict__ bins) {
    const uint64_t L = in.num_laser_targets;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= nv * L) return;
    const uint64_t vi = i / L, l = i % L;
    uint32_t vx, vy, vz;
    voxel_of(vidx[vi], in.voxel_res[0], in.voxel_res[1], vx, vy, vz);
    const float px = ref_voxel_coord(vx, in.voxel_size[0], in.hidden_min[0]);
    const float py = ref_voxel_coord(vz, in.voxel_size[1], in.hidden_min[1]);
    const float pz = ref_voxel_coord(vy, in.voxel_size[2], in.hidden_min[2]);
    const float4 g = scan[l];
    float dist = fma_rn(sqrt_approx(ref_dot3(sub_rn(px, g.x), sub_rn(py, g.y), sub_rn(pz, g.z))), 2.f, -in.time_offset);
    if (in.discard_first_last_bounces == 0) dist = add_rn(dist, g.w);
    const int b = __float2int_rz(ref_bin_ratio(dist, rcp_approx(in.time_step)));
    bins[i] = (b >= 0 && b < (int)in.num_time_bins) ? b : -1;
}

// The path (dist) of each pair in the gathers' FP32 expression, and the two
// per-call constants of the scattering walk: rcp.approx(timeStep) and half the
// voxel diagonal.
__global__ void debug_confocal_paths_kernel(fbp_recon_info in, const float4* __restrict__ scan,
                                            const int64_t* __restrict__ vidx, uint64_t nv, float* __restrict__ paths,
                                            float* __restrict__ consts) {
    const uint64_t L = in.num_laser_targets;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i == 0 && consts) {
        consts[0] = rcp_approx(in.time_step);
        consts[1] = mul_rn(0.5f, sqrt_approx(ref_dot3(in.voxel_size[0], in.voxel_size[1], in.voxel_size[2])));
    }
    if (i >= nv * L) return;
    const uint64_t vi = i / L, l = i % L;
    uint32_t vx, vy, vz;
    voxel_of(vidx[vi], in.voxel_res[0], in.voxel_res[1], vx, vy, vz);
    const float px = ref_voxel_coord(vx, in.voxel_size[0], in.hidden_min[0]);
    const float py = ref_voxel_coord(vz, in.voxel_size[1], in.hidden_min[1]);
    const float pz = ref_voxel_coord(vy, in.voxel_size[2], in.hidden_min[2]);
    const float4 g = scan[l];
    float dist = fma_rn(sqrt_approx(ref_dot3(sub_rn(px, g.x), sub_rn(py, g.y), sub_rn(pz, g.z))), 2.f, -in.time_offset);
    if (in.discard_first_last_bounces == 0) dist = add_rn(dist, g.w);
    paths[i] = dist;
}

__global__ void debug_exhaustive_bins_kernel(fbp_recon_info in, const float4* __restrict__ lscan,
                                             const float4* __restrict__ sscan, const int64_t* __restrict__ vidx,
                                             uint64_t nv, int32_t* __restrict__ bins) {
    const uint64_t L = in.num_laser_targets, S = in.num_sensor_targets;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= nv * L * S) return;
    const uint64_t vi = i / (L * S), l = (i / S) % L, s = i % S;
    uint32_t vx, vy, vz;
    voxel_of(vidx[vi], in.voxel_res[0], in.voxel_res[1], vx, vy, vz);
    const float px = ref_voxel_coord(vx, in.voxel_size[0], in.hidden_min[0]);
    const float py = ref_voxel_coord(vz, in.voxel_size[1], in.hidden_min[1]);
    const float pz = ref_voxel_coord(vy, in.voxel_size[2], in.hidden_min[2]);
    const float4 lg = lscan[l], sg = sscan[s];
    const float dl = sqrt_approx(ref_dot3(sub_rn(px, lg.x), sub_rn(py, lg.y), sub_rn(pz, lg.z)));
    const float ds = sqrt_approx(ref_dot3(sub_rn(px, sg.x), sub_rn(py, sg.y), sub_rn(pz, sg.z)));
    float dist = sub_rn(add_rn(dl, ds), in.time_offset);
    if (in.discard_first_last_bounces == 0) dist = add_rn(dist, add_rn(lg.w, sg.w));
    const int b = __float2int_rz(ref_bin_ratio(dist, rcp_approx(in.time_step)));
    bins[i] = (b >= 0 && b < (int)in.num_time_bins) ? b : -1;
}

}  // namespace fbp

extern "C" fbp_status fbp_debug_confocal_bins(fbp_context* ctx, const fbp_recon_info* info, const float* laser_xyz,
                                              const int64_t* voxel_idx, uint64_t num_voxels, int32_t* bins,
                                              void* stream) {
    return guarded("fbp_debug_confocal_bins", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, false, "fbp_debug_confocal_bins"));
        if (!laser_xyz || !voxel_idx || !bins) return set_error(FBP_ERR_INVALID_ARG, "fbp_debug_confocal_bins: null buffer");
        cudaStream_t s = (cudaStream_t)stream;
        const float4* scan;
        const float *xs, *ys, *zs;
        FBP_TRY(build_tables(ctx, *info, laser_xyz, s, &scan, &xs, &ys, &zs));
        const uint64_t n = num_voxels * info->num_laser_targets;
        if (n == 0) return FBP_OK;
        debug_confocal_bins_kernel<<<cdiv(n, 256), 256, 0, s>>>(*info, scan, voxel_idx, num_voxels, bins);
        FBP_CHECK_LAUNCH(ctx, "debug_confocal_bins_kernel");
        return FBP_OK;
    });
}

extern "C" fbp_status fbp_debug_confocal_paths(fbp_context* ctx, const fbp_recon_info* info, const float* laser_xyz,
                                               const int64_t* voxel_idx, uint64_t num_voxels, float* paths,
                                               float* consts, void* stream) {
    return guarded("fbp_debug_confocal_paths", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, false, "fbp_debug_confocal_paths"));
        if (!laser_xyz || !voxel_idx || !paths || !consts)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_debug_confocal_paths: null buffer");
        cudaStream_t s = (cudaStream_t)stream;
        const float4* scan;
        const float *xs, *ys, *zs;
        FBP_TRY(build_tables(ctx, *info, laser_xyz, s, &scan, &xs, &ys, &zs));
        const uint64_t n = std::max<uint64_t>(num_voxels * info->num_laser_targets, 1);
        debug_confocal_paths_kernel<<<cdiv(n, 256), 256, 0, s>>>(*info, scan, voxel_idx, num_voxels, paths, consts);
        FBP_CHECK_LAUNCH(ctx, "debug_confocal_paths_kernel");
        return FBP_OK;
    });
}

extern "C" fbp_status fbp_debug_exhaustive_bins(fbp_context* ctx, const fbp_recon_info* info, const float* laser_xyz,
                                                const float* sensor_xyz, const int64_t* voxel_idx, uint64_t num_voxels,
                                                int32_t* bins, void* stream) {
    return guarded("fbp_debug_exhaustive_bins", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, true, "fbp_debug_exhaustive_bins"));
        if (!laser_xyz || !sensor_xyz || !voxel_idx || !bins)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_debug_exhaustive_bins: null buffer");
        cudaStream_t s = (cudaStream_t)stream;
        const uint32_t L = info->num_laser_targets, Sn = info->num_sensor_targets;
        void* lp = nullptr;
        void* sp = nullptr;
        FBP_TRY(workspace(ctx, WS_SCAN_TABLE, (size_t)L * sizeof(float4), s, &lp));
        FBP_TRY(workspace(ctx, WS_SENSOR_TABLE, (size_t)Sn * sizeof(float4), s, &sp));
        scan_table_kernel<<<cdiv(L, 256), 256, 0, s>>>(static_cast<float4*>(lp), laser_xyz, L,
                                                      (int)info->discard_first_last_bounces, info->laser_position[0],
                                                      info->laser_position[1], info->laser_position[2], 0.f, 0.f, 0.f, 0);
        FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
        scan_table_kernel<<<cdiv(Sn, 256), 256, 0, s>>>(static_cast<float4*>(sp), sensor_xyz, Sn,
                                                       (int)info->discard_first_last_bounces, info->sensor_position[0],
                                                       info->sensor_position[1], info->sensor_position[2], 0.f, 0.f, 0.f, 0);
        FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
        const uint64_t n = num_voxels * L * Sn;
        if (n == 0) return FBP_OK;
        debug_exhaustive_bins_kernel<<<cdiv(n, 256), 256, 0, s>>>(*info, static_cast<const float4*>(lp),
                                                                 static_cast<const float4*>(sp), voxel_idx, num_voxels,
                                                                 bins);
        FBP_CHECK_LAUNCH(ctx, "debug_exhaustive_bins_kernel");
        return FBP_OK;
    });
}
