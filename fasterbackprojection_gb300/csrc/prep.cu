// The gathers' inputs in one launch: padded, thresholded FP32 rows of the
// capture, the scan and SPAD tables, the voxel-centre coordinates.
#include "fbp_internal.cuh"
#include "bp_common.cuh"

#include <algorithm>

namespace fbp {

namespace {

constexpr int kPrepThreads = 256, kPrepWarps = kPrepThreads / 32;
constexpr int kTileBins = 128;  // time-major tiles: 32 points x 128 bins

template <typename S>
__device__ __forceinline__ float thresholded(S v) {
    const float c = to_f32(v);
    return c > FBP_EPS ? c : 0.f;
}

// Four consecutive samples at src (aligned to four of them).
__device__ __forceinline__ float4 load4(const float* src) { return *reinterpret_cast<const float4*>(src); }
template <typename S>
__device__ __forceinline__ float4 load4(const S* src) {
    const uint2 b = *reinterpret_cast<const uint2*>(src);
    S h[4];
    memcpy(h, &b, 8);
    return make_float4(to_f32(h[0]), to_f32(h[1]), to_f32(h[2]), to_f32(h[3]));
}

// Blocks [0, row_blocks): rows.  Time inner: a warp per row, 16-byte stores (and
// loads where VEC).  Time major: tiles of 32 points x 128 bins transposed
// through shared memory (16 loads a thread in flight; 32 x 32 tiles took 296
// us).  Blocks from row_blocks: one table entry per thread.  Bound by memory:
// 256^2 points x 1024 bins, rows of 2 KB + window, FP32 240 -> 129 us (6.2
// TB/s), FP16 238 -> 111 us, time major 217 -> 145 us; small calls gain the two
// launches that the tables had of their own (32^3 volume 43.4 -> 37.5 us).
template <typename S, bool TIME_MAJOR, bool VEC>
__global__ void __launch_bounds__(kPrepThreads) prepare_kernel(PrepRows r, PrepTables t, uint32_t row_blocks) {
    const S* cube = static_cast<const S*>(r.cube);
    if (blockIdx.x < row_blocks) {
        if (TIME_MAJOR) {
            __shared__ float tile[kTileBins][33];
            const uint32_t across = (uint32_t)((r.count + 31) / 32);
            const uint32_t l0 = blockIdx.x % across * 32, t0 = blockIdx.x / across * kTileBins;
            const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
            const bool inside = l0 + tx < r.count;
#pragma unroll
            for (int k = 0; k < kTileBins / kPrepWarps; ++k) {
                const uint32_t b = t0 + ty + k * kPrepWarps;
                tile[ty + k * kPrepWarps][tx] = inside && b < r.T ? thresholded(cube[(uint64_t)b * r.count + l0 + tx]) : 0.f;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 32 / kPrepWarps; ++j) {
                const uint32_t l = l0 + ty + j * kPrepWarps;
                if (l >= r.count) break;
                float* dst = r.rows + (uint64_t)l * r.pitch;
#pragma unroll
                for (int k = 0; k < kTileBins; k += 32) {
                    const uint32_t b = t0 + k + tx;
                    if (b < r.pitch) dst[b] = tile[k + tx][ty + j * kPrepWarps];
                }
            }
        } else {
            const uint32_t lane = threadIdx.x & 31;
            const uint64_t warps = (uint64_t)row_blocks * kPrepWarps;
            for (uint64_t l = blockIdx.x * (uint64_t)kPrepWarps + (threadIdx.x >> 5); l < r.count; l += warps) {
                const S* src = cube + l * r.T;
                float* dst = r.rows + l * r.pitch;
#pragma unroll 4
                for (uint32_t b = lane * 4; b < r.pitch; b += 128) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (VEC) {
                        if (b < r.T) {  // T is a multiple of 4
                            v = load4(src + b);
                            v = make_float4(thresholded(v.x), thresholded(v.y), thresholded(v.z), thresholded(v.w));
                        }
                    } else {
                        if (b < r.T) v.x = thresholded(src[b]);
                        if (b + 1 < r.T) v.y = thresholded(src[b + 1]);
                        if (b + 2 < r.T) v.z = thresholded(src[b + 2]);
                        if (b + 3 < r.T) v.w = thresholded(src[b + 3]);
                    }
                    *reinterpret_cast<float4*>(dst + b) = v;
                }
            }
        }
        return;
    }
    const uint64_t i = (uint64_t)(blockIdx.x - row_blocks) * kPrepThreads + threadIdx.x;
    // transient_reconstruction.cuh:109-110: (x, y, z, bounce distances) per point.
    auto point = [&](const float* xyz, const float (&a)[3], const float* b) {
        const float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
        float w = 0.f;
        if (t.discard == 0) {
            w = ref_distance(x, y, z, a[0], a[1], a[2]);
            if (b) w = add_rn(w, ref_distance(x, y, z, b[0], b[1], b[2]));
        }
        return make_float4(x, y, z, w);
    };
    if (i < t.num_lasers) t.lasers[i] = point(t.laser_xyz, t.laser_pos, t.num_sensors ? nullptr : t.sensor_pos);
    if (i < t.num_sensors) t.sensors[i] = point(t.sensor_xyz, t.sensor_pos, nullptr);
    // transient_reconstruction.cuh:106: (vx, vz, vy) drive world (x, y, z).
    if (i < t.res[0]) t.axes[i] = ref_voxel_coord((uint32_t)i, t.size[0], t.min[0]);
    if (i < t.res[2]) t.axes[t.res[0] + i] = ref_voxel_coord((uint32_t)i, t.size[1], t.min[1]);
    if (i < t.res[1]) t.axes[t.res[0] + t.res[2] + i] = ref_voxel_coord((uint32_t)i, t.size[2], t.min[2]);
}

template <typename S>
fbp_status launch(fbp_context* ctx, const PrepRows& r, const PrepTables& t, cudaStream_t stream) {
    const uint64_t entries = std::max<uint64_t>(std::max<uint64_t>(t.num_lasers, t.num_sensors),
                                                std::max(t.res[0], std::max(t.res[1], t.res[2])));
    const unsigned tables = cdiv(entries, kPrepThreads);
    if (r.time_major) {
        const uint64_t tiles = (uint64_t)cdiv(r.count, 32) * cdiv(r.pitch, kTileBins);
        if (tiles + tables > 0x7FFFFFFFull) return set_error(FBP_ERR_UNSUPPORTED, "capture too large for one launch");
        prepare_kernel<S, true, false><<<(unsigned)tiles + tables, kPrepThreads, 0, stream>>>(r, t, (unsigned)tiles);
    } else {
        const unsigned blocks = (unsigned)std::min<uint64_t>(cdiv(r.count, kPrepWarps), (uint64_t)ctx->sm_count * 16);
        const bool vec = r.T % 4 == 0 && reinterpret_cast<uintptr_t>(r.cube) % (4 * sizeof(S)) == 0;
        if (vec) prepare_kernel<S, false, true><<<blocks + tables, kPrepThreads, 0, stream>>>(r, t, blocks);
        else prepare_kernel<S, false, false><<<blocks + tables, kPrepThreads, 0, stream>>>(r, t, blocks);
    }
    FBP_CHECK_LAUNCH(ctx, "prepare_kernel");
    return FBP_OK;
}

}  // namespace

fbp_status prepare_gather(fbp_context* ctx, int dtype, const PrepRows& r, const PrepTables& t, cudaStream_t stream) {
    switch (dtype) {
        case FBP_F32: return launch<float>(ctx, r, t, stream);
        case FBP_BF16: return launch<__nv_bfloat16>(ctx, r, t, stream);
        case FBP_F16: return launch<__half>(ctx, r, t, stream);
        default: return set_error(FBP_ERR_INVALID_ARG, "unknown dtype");
    }
}

fbp_status table_buffers(fbp_context* ctx, const fbp_recon_info& in, const float* laser_xyz, const float* sensor_xyz,
                         bool axes, cudaStream_t stream, PrepTables* t) {
    const uint32_t L = in.num_laser_targets, Sn = sensor_xyz ? in.num_sensor_targets : 0;
    void *lp = nullptr, *sp = nullptr, *ap = nullptr;
    FBP_TRY(workspace(ctx, WS_SCAN_TABLE, (size_t)L * sizeof(float4), stream, &lp));
    if (Sn) FBP_TRY(workspace(ctx, WS_SENSOR_TABLE, (size_t)Sn * sizeof(float4), stream, &sp));
    if (axes) {
        const size_t n = (size_t)in.voxel_res[0] + in.voxel_res[1] + in.voxel_res[2];
        FBP_TRY(workspace(ctx, WS_AXIS_TABLES, n * sizeof(float), stream, &ap));
    }
    t->laser_xyz = laser_xyz;
    t->sensor_xyz = sensor_xyz;
    t->num_lasers = L;
    t->num_sensors = Sn;
    t->discard = (int)in.discard_first_last_bounces;
    t->lasers = static_cast<float4*>(lp);
    t->sensors = static_cast<float4*>(sp);
    t->axes = static_cast<float*>(ap);
    for (int k = 0; k < 3; ++k) {
        t->laser_pos[k] = in.laser_position[k];
        t->sensor_pos[k] = in.sensor_position[k];
        t->min[k] = in.hidden_min[k];
        t->size[k] = in.voxel_size[k];
        t->res[k] = axes ? in.voxel_res[k] : 0;
    }
    return FBP_OK;
}

}  // namespace fbp
