// Pieces shared by the backprojection gathers.
#pragma once

#include "fbp_internal.cuh"

namespace fbp {

// ---------------------------------------------- bulk copies and mbarriers --

// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) from
// global to shared memory, completing on the mbarrier at shared address `bar`.
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* gmem_src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst),
                 "l"(gmem_src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint32_t bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase with this parity, at most kWaitLimit polls (each
// suspends for a while in hardware; the longest wait in earnest is one
// stage); false when they ran out.
constexpr uint32_t kWaitLimit = 1u << 22;
__device__ __forceinline__ bool mbar_wait_parity(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// One FP32 element of shared memory at a shared-state-space byte address.
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// The sample of the bin floor(x) of a window that starts at bin a, from
// biased = x + (2^23 - a) rounded towards zero: its low bits are floor(x) - a,
// with no conversion.
//   CLAMP   clamped to the slot at shared address `slot` (its sentinel, a zero,
//           sits at slot_w).
//   else    the planner guarantees a <= x < a + slot_w; `slot` is the address
//           less the exponent's bits (kBiasBits).
constexpr uint32_t kBiasBits = 0x4B000000u << 2;  // 2^23 as float bits, in bytes
template <bool CLAMP>
__device__ __forceinline__ float read_bin(float biased, int slot, uint32_t slot_w) {
    if (CLAMP) return lds_f32((uint32_t)slot + (min(__float_as_uint(biased) - 0x4B000000u, slot_w) << 2));
    return lds_f32((uint32_t)slot + (__float_as_uint(biased) << 2));
}

// ------------------------------------------------------ confocal gather --

// Scan-point sampling for the unbiased MIS estimator: each voxel tile draws
// K scan points i.i.d. from a proposal p(l | tile) and weights each pair by
// 1 / (K p(l | tile)), so sum_k f(v, l_k) / (K p(l_k)) is an unbiased estimate
// of the full backprojection sum at every voxel of the tile.
enum SampleMode { SAMPLE_UNIFORM = 0, SAMPLE_ALIAS = 1, SAMPLE_CLUSTERS = 2 };
// Cluster samples per tile (SAMPLE_CLUSTERS) and the static shared memory the
// sampled gather keeps for them.
constexpr uint32_t kMaxClusterSamples = 256;
constexpr size_t kSampledStaticSmem = kMaxClusterSamples * 8 + 64;
struct SampleParams {
    int mode;
    uint32_t K;              // samples per tile
    unsigned long long seed;
    const float* prob;       // SAMPLE_ALIAS: Vose tables over scan points
    const uint32_t* alias;
    const float* pl;         // SAMPLE_ALIAS: p(l)
    const float* tile_cdf;   // SAMPLE_CLUSTERS: [tiles][G] inclusive CDF over clusters (null: uniform)
    uint32_t G;              // clusters
    uint32_t cluster_side;   // scan points per cluster side
    uint32_t n_side;         // scan grid side (scan point l = iz * n_side + ix)
};

// Counter-based uniforms in [0, 1): a 64-bit mix of (seed, tile, k, stream).
__device__ __forceinline__ float hash_uniform(unsigned long long seed, unsigned long long tile, unsigned k, unsigned s) {
    unsigned long long x = seed ^ (tile * 0x9E3779B97F4A7C15ull) ^ ((unsigned long long)k << 32 | s) * 0xD1B54A32D192ED03ull;
    x ^= x >> 31;
    x *= 0x7FB5D329728EA185ull;
    x ^= x >> 27;
    x *= 0x81DADEF4BC2DD44Dull;
    x ^= x >> 33;
    return (float)(x >> 40) * (1.0f / 16777216.0f);
}

struct ConfocalGatherParams {
    const float4* scan;
    const float* xs;
    const float* ys;
    const float* zs;
    float* volume;
    int* status;
    uint32_t Vx, Vy, Vz, L, T;
    float t0, dt;
    uint32_t row_pitch;  // elements per padded row
    uint32_t slot_w;     // window width in elements (the sentinel zero sits at slot_w)
    int ch;              // scan points per window stage (a power of two <= 32)
    uint32_t chains;     // contiguous ranges of scan-point groups with compensated sums of their own
    float* chain_sums;   // split tiles: [chains][sum, compensation][volume]
    const void* rows;    // [L][row_pitch] FP32
    SampleParams smp;    // used by the sampled (MIS) variant only
    float vs[3];         // voxel size (the voxel-scattering variant's extent)
    int exact_weights;   // 1: every weight by its own rcp.approx (FBP_WEIGHTS_REFERENCE)
    int scat_exact;      // voxel scattering: every walk is exactly the unrolled steps long (no tail loop)

    // Shared memory in front of the windows: the pipeline's barriers, then per
    // scan point of kPlanBufs groups: (x, y, z, bounce), (bias, bias, slot
    // address), the x differences to the tile's kv columns, the window's source
    // and length, the sample weight; two words per group.
    static constexpr int kGroup = 32;
    static constexpr int kWindowBufs = 2;  // stages of windows
    static constexpr int kPlanBufs = 4;    // groups of plans
    __host__ __device__ static constexpr size_t meta_bytes(int kv) {
        return 64 +
               (size_t)kPlanBufs * kGroup * (sizeof(float4) + sizeof(int4) + (kv + 1) * sizeof(float) + sizeof(void*) +
                                             sizeof(int)) +
               (size_t)kPlanBufs * sizeof(int2);
    }
};

// Shared memory holding the compensated (Kahan) sums of a CTA's voxels when a
// thread owns 16 of them, or walks 8 of the voxel-scattering variant (sum and
// compensation per voxel, [2 KV][threads]): kept there instead of in 64 (or 16)
// registers, so three (or four) CTAs fit per SM.
__host__ __device__ constexpr size_t kahan_smem_bytes(int kv, int threads, bool scatter = false) {
    return kv >= 16 || scatter ? (size_t)2 * kv * threads * sizeof(float) : 0;
}

// Window geometry shared by the gathers: the widest bin span a tile of the
// given world extents can need, capped at the whole row (T bins plus one
// alignment step), the padded row pitch, and the stage size that fits the
// shared-memory budget.
struct WindowPlan {
    uint32_t slot_w, pitch;
    int ch;
    bool capped;  // slot_w is the whole row: bins past a window must be clamped
    size_t smem;
};
fbp_status plan_window(const fbp_context* ctx, double ex, double ey, double ez, double time_step, uint32_t T, int align,
                       size_t elem_bytes, size_t meta_bytes, WindowPlan* out, const char* who,
                       double extra_path = 0.0, int ctas_per_sm = 1, int window_bufs = 2);
// The confocal gather's chains for a volume and a capture (of the whole
// volume, whatever part of it a launch computes, so that slabs and batches sum
// like the single call).
uint32_t gather_chains(const fbp_context* ctx, const fbp_recon_info& in, size_t smem);
// The same for the voxel-scattering variant, whose walks take `steps` steps.
uint32_t scatter_chains(const fbp_context* ctx, const fbp_recon_info& in, size_t smem, double steps);
// Chains for a launch of `tiles` tiles (whose warps are `busy` to that part)
// that each walk `groups` groups of `group_us` microseconds (at an SM's full
// rate) into n outputs, occ CTAs to an SM.
uint32_t split_chains(const fbp_context* ctx, uint64_t tiles, double busy, uint64_t groups, int occ, double group_us,
                      uint64_t n);
// Part of the warps of 16 x 16 (rows, slices) tiles that own voxels of a volume.
double busy_warps(const uint32_t res[3]);
constexpr double kGatherGroupUs = 6.3;  // 32 scan points x 4096 voxels
constexpr double kScatterStepUs = 2.5;  // 32 scan points x 2048 voxels, per step of the walk
// Scratch of a gather: its rows and, for n outputs in several chains, their sums
// ([chains][2][n]; *chains becomes 1 where there is no room for them: no memory,
// or a stream under capture and too small a buffer).
fbp_status gather_scratch(fbp_context* ctx, size_t row_bytes, uint32_t* chains, uint64_t n, cudaStream_t stream,
                          float** rows, float** sums);
// out[i] = the chains' sums [chains][sum, compensation][n], folded in order.
fbp_status fold_chains(fbp_context* ctx, const float* sums, uint32_t chains, uint64_t n, float* out, cudaStream_t stream);
// CTAs of `smem` bytes of dynamic shared memory an SM holds, at most `most`.
inline int resident_ctas(size_t smem, int most) {
    const size_t n = kSmSharedBytes / (smem + kCtaReservedShared);
    return n < 1 ? 1 : (n < (size_t)most ? (int)n : most);
}
constexpr int kGatherCtasPerSm = 3;   // 256 threads of 80 registers
constexpr int kScatterCtasPerSm = 4;  // ... of 64: the voxel-scattering walk of 8 voxels

// The confocal gather over all scan points (smp == nullptr) or over K sampled
// scan points per tile (the unbiased MIS estimator).
fbp_status confocal_gather_scatter(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype,
                                   int layout, const float* laser_xyz, float* volume, cudaStream_t s);
fbp_status confocal_gather_slab(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                                const float* laser_xyz, uint32_t z_begin, uint32_t z_end, float* volume,
                                cudaStream_t s);
fbp_status confocal_gather(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                           const float* laser_xyz, float* volume, cudaStream_t s, const SampleParams* smp);
void confocal_tile_grid(const fbp_recon_info& in, uint32_t out[3]);

// The gathers' inputs, made by one launch (prepare_gather).
// Rows [count][pitch] FP32 (pitch a multiple of 4), time innermost, values
// <= 1e-5 replaced by 0 (the reference skips them), zeros in [T, pitch); 16-bit
// captures are widened exactly.
struct PrepRows {
    const void* cube;
    float* rows;
    uint64_t count;
    uint32_t T, pitch;
    int time_major;  // cube[t][row] instead of cube[row][t]
};
// Scan tables (x, y, z, bounce distances) and voxel-centre coordinates
// [Vx + Vz + Vy]; zero counts leave a table out.
struct PrepTables {
    const float *laser_xyz, *sensor_xyz;
    float4 *lasers, *sensors;
    float* axes;
    uint32_t num_lasers, num_sensors;  // no sensors: confocal, both bounces with the lasers
    int discard;
    float laser_pos[3], sensor_pos[3], min[3], size[3];
    uint32_t res[3];
};
fbp_status prepare_gather(fbp_context* ctx, int dtype, const PrepRows& rows, const PrepTables& tables, cudaStream_t stream);
// The tables' part of the request, in the context's scratch (sensor_xyz null:
// confocal; axes: a volume's coordinates too).
fbp_status table_buffers(fbp_context* ctx, const fbp_recon_info& in, const float* laser_xyz, const float* sensor_xyz,
                         bool axes, cudaStream_t stream, PrepTables* t);

__global__ void axis_tables_kernel(float* __restrict__ xs, float* __restrict__ ys, float* __restrict__ zs,
                                   uint32_t Vx, uint32_t Vy, uint32_t Vz, float mnx, float mny, float mnz, float sx,
                                   float sy, float sz);

// Shared host helpers.
fbp_status build_tables(fbp_context* ctx, const fbp_recon_info& in, const float* laser_xyz, cudaStream_t stream,
                        const float4** scan, const float** xs, const float** ys, const float** zs);
fbp_status validate_info(const fbp_recon_info* info, bool need_sensors, const char* who);

__global__ void scan_table_kernel(float4* __restrict__ out, const float* __restrict__ xyz, uint32_t n, int discard,
                                  float ax, float ay, float az, float bx, float by, float bz, int confocal_pair);

}  // namespace fbp
