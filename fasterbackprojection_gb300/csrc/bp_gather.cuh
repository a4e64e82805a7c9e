// Device code of the confocal gather, shared by the one-capture kernel
// (bp_confocal.cu) and the persistent multi-capture kernel (batch.cu).
#pragma once

#include "bp_common.cuh"

namespace fbp {

// Arithmetic paths of the pair loop (all reproduce the reference's bins):
//   PATH_2D     time_offset == 0, no bounce terms: dist = 2d exactly, so
//               x = d * (2 rcp(dt)) and the weight is rcp(d^2) = 4 rcp(dist^2);
//               the stage's partial sum is scaled by 1/4 (exact).
//   PATH_FAST   time_offset <= 0 (every path >= 0): dist = fma(d, 2, -t0) [+ bounce].
//   PATH_EXACT  time_offset > 0: negative paths possible.  Groups with a path
//               near or below zero take the guarded loop and bin by
//               conversion (int() truncates towards zero); the others run
//               PATH_FAST's arithmetic, whose floor is the same for x > 0
//               (a conversion is a third MUFU-pipe operation per pair).
// CLAMP: windows that are the whole row, whose bins are clamped to the slot;
// otherwise the planner guarantees that every bin lies inside its window.
//   PATH_SCATTER + j  the reference's ACCUMULATE_VOXEL_SCATTERING variant
//               (transient_reconstruction.cuh:112-126): every bin of the
//               path range dist -/+ the voxel's half diagonal, stepped by
//               (dt + EPS) in float like the reference.  The first 2 + j
//               steps run unrolled and predicated (the voxels' walks
//               interleave), any further ones in a loop; bins by the same
//               round-toward-zero add (the path is never negative).
//   PATH_SCATTER + 3 + j  the same where every walk takes at least 2 + j
//               steps: the host checks (1 + j) (dt + EPS) + 1e-4 m < the
//               voxel diagonal, and stages with a path under 3.5 mm past
//               the half diagonal or of 64 m or more take the predicated
//               reference loop, so the unrolled steps add unconditionally
//               (the rounding of dd over four steps stays below 2e-5 m).
enum { PATH_2D = 0, PATH_FAST = 1, PATH_EXACT = 2, PATH_SCATTER = 3 };
constexpr int kScatterMaxPrefix = 4;
constexpr int kScatterForms = kScatterMaxPrefix - 1;  // prefixes 2, 3, 4
__host__ __device__ constexpr bool is_scatter(int path) { return path >= PATH_SCATTER; }
__host__ __device__ constexpr int scatter_prefix(int path) { return (path - PATH_SCATTER) % kScatterForms + 2; }
__host__ __device__ constexpr bool scatter_free(int path) { return path - PATH_SCATTER >= kScatterForms; }
// The scattering walk of 8 voxels per thread.  It is bound by the latency of its
// dependent steps, so four CTAs of 64 registers count for more than what 16
// voxels share (their plan reads and stages); it keeps its voxels' x instead
// of reading planned differences, the shared-memory pipe being half full.
__host__ __device__ constexpr bool scatter_narrow(int kv, int path) { return is_scatter(path) && kv == 8; }

// What the pair loop reads of a planned scan point (broadcast shared loads).
// dx: the x differences to the tile's KV voxel columns, as packed pairs: the
// same for every thread, so the planner makes them once (the subtractions were
// an eighth of the loop's issue slots).
struct ScanPlan {
    const float4* geo;      // (x, y, z, bounce)
    const int4* meta;       // (bias, bias, slot address, 0); see read_bin
    const ulonglong2* dx;   // [KV / 4] per point
    const float* weight;    // WEIGHTED: the sample's weight
};

// One staged stage of scan points against a thread's KV voxels (consecutive
// along x, sharing the y/z offsets).
template <int KV, int PATH, bool BOUNCE, bool CLAMP, bool SAFE, bool WEIGHTED>
__device__ __forceinline__ void confocal_stage(const ScanPlan pl, int nl, float py,
                                               float pz, float neg_t0, float rcp_dt, uint32_t slot_w,
                                               float (&acc)[KV], float ext = 0.f, float step = 0.f,
                                               bool tail = true, const f32x2_t* px = nullptr) {
    const float rcp2 = 2.f * rcp_dt;  // exact
    if constexpr (is_scatter(PATH)) {
        constexpr int SP = scatter_prefix(PATH);
        static_assert(SP >= 1 && SP <= kScatterMaxPrefix, "prefix within the step bound");
        const int max_it = (int)(2.f * ext / step) + 4;  // >= 4 >= SP
        // The reference adds I * w per bin with an atomic: one rounding for
        // the product, one for the sum, in bin order.  The count bound only
        // matters where dist is so large that adding the step no longer
        // changes it (no such path reaches a bin).  Once dd >= dmax it stays
        // there, so a predicated step past the end only reads (the clamped
        // index keeps it inside the slot).
        for (int i = 0; i < nl; ++i) {
            const float4 g = pl.geo[i];
            const int4 m = pl.meta[i];
            const float bias = __int_as_float(m.x);
            const float wl = WEIGHTED ? pl.weight[i] : 1.f;
            const float dy = sub_rn(py, g.y), dz = sub_rn(pz, g.z);
            const float dy2 = mul_rn(dy, dy);
            f32x2_t dxp[KV / 2];
            if constexpr (scatter_narrow(KV, PATH)) {
                const f32x2_t gxp = pack2(g.x, g.x);
#pragma unroll
                for (int j = 0; j < KV / 2; ++j) dxp[j] = sub_rn2(px[j], gxp);
            } else {
#pragma unroll
                for (int j = 0; j < KV / 4; ++j) {
                    const ulonglong2 v = pl.dx[(size_t)i * (KV / 4) + j];
                    dxp[2 * j] = v.x;
                    dxp[2 * j + 1] = v.y;
                }
            }
            auto bin_at = [&](float dd) -> float {
                const float x = ref_bin_ratio(dd, rcp_dt);
                return read_bin<CLAMP>(add_rz(x, bias), m.z, slot_w);
            };
            // Steps SP.. of one walk (rare: a diagonal longer than the planned steps).
            auto walk_rest = [&](float a, float dd, float dmax, float w) -> float {
                for (int it = SP; dd < dmax && it < max_it; ++it) {
                    float I = bin_at(dd);
                    if (WEIGHTED) I *= wl;
                    a = add_rn(a, mul_rn(I, w));
                    dd = add_rn(dd, step);
                }
                return a;
            };
            if constexpr (!SAFE) {
                // Voxel pairs (k, k + 1) in packed FP32 pairs, step by step.
                const f32x2_t dy2p = pack2(dy2, dy2), dzp = pack2(dz, dz);
                const f32x2_t gwp = pack2(g.w, g.w), extp = pack2(ext, ext), stepp = pack2(step, step);
                const f32x2_t rdp = pack2(rcp_dt, rcp_dt), biasp = pack2(bias, bias), wlp = pack2(wl, wl);
#pragma unroll
                for (int j = 0; j < KV / 2; ++j) {
                    const f32x2_t dx = dxp[j];
                    float q0, q1, s0, s1, e0, e1, h0, h1;
                    unpack2(fma_rn2(dzp, dzp, fma_rn2(dx, dx, dy2p)), q0, q1);
                    f32x2_t dist = fma_rn2(pack2(sqrt_approx(q0), sqrt_approx(q1)), pack2(2.f, 2.f),
                                           pack2(neg_t0, neg_t0));
                    if (BOUNCE) dist = add_rn2(dist, gwp);
                    unpack2(mul_rn2(dist, dist), s0, s1);
                    const f32x2_t w = pack2(rcp_approx(s0), rcp_approx(s1));
                    unpack2(sub_rn2(dist, extp), e0, e1);
                    unpack2(add_rn2(dist, extp), h0, h1);  // dmax
                    f32x2_t dd = pack2(fmaxf(0.f, e0), fmaxf(0.f, e1));
                    float a0 = acc[2 * j], a1 = acc[2 * j + 1];
#pragma unroll
                    for (int it = 0; it < SP; ++it) {
                        float d0, d1, b0, b1, p0, p1;
                        unpack2(dd, d0, d1);
                        unpack2(add_rz2(mul_rn2(dd, rdp), biasp), b0, b1);
                        f32x2_t I = pack2(read_bin<CLAMP>(b0, m.z, slot_w), read_bin<CLAMP>(b1, m.z, slot_w));
                        if (WEIGHTED) I = mul_rn2(I, wlp);
                        unpack2(mul_rn2(I, w), p0, p1);
                        if constexpr (scatter_free(PATH)) {
                            a0 = add_rn(a0, p0);  // dd < dmax holds for every unrolled step
                            a1 = add_rn(a1, p1);
                        } else {
                            a0 = add_rn_if_lt(a0, p0, d0, h0);
                            a1 = add_rn_if_lt(a1, p1, d1, h1);
                        }
                        dd = add_rn2(dd, stepp);
                    }
                    if (scatter_free(PATH) && !tail) {
                        // Every walk is exactly the unrolled steps long.
                        acc[2 * j] = a0;
                        acc[2 * j + 1] = a1;
                        continue;
                    }
                    float d0, d1, w0, w1;
                    unpack2(dd, d0, d1);
                    unpack2(w, w0, w1);
                    acc[2 * j] = walk_rest(a0, d0, h0, w0);
                    acc[2 * j + 1] = walk_rest(a1, d1, h1, w1);
                }
            } else {
#pragma unroll
                for (int k = 0; k < KV; ++k) {
                    float dx2[2];
                    unpack2(dxp[k / 2], dx2[0], dx2[1]);
                    const float dx = dx2[k & 1];
                    const float d = sqrt_approx(fma_rn(dz, dz, fma_rn(dx, dx, dy2)));
                    float dist = fma_rn(d, 2.f, neg_t0);
                    if (BOUNCE) dist = add_rn(dist, g.w);
                    const float w = ref_safe_rcp(mul_rn(dist, dist));
                    float dd = fmaxf(0.f, sub_rn(dist, ext));
                    const float dmax = add_rn(dist, ext);
                    float a = acc[k];
#pragma unroll
                    for (int it = 0; it < SP; ++it) {
                        float I = bin_at(dd);
                        if (WEIGHTED) I *= wl;
                        a = add_rn_if_lt(a, mul_rn(I, w), dd, dmax);
                        dd = add_rn(dd, step);
                    }
                    acc[k] = walk_rest(a, dd, dmax, w);
                }
            }
        }
        return;
    } else if constexpr (!SAFE) {
        // Voxel pairs (k, k + 1) in packed FP32 pairs: the bins are the scalar
        // loop's operations, bit for bit, in half the instructions.  A packed
        // instruction holds the issue port for two cycles, and the port is what
        // bounds this loop: issue 66 % and second cycles 34 % of all cycles, MUFU
        // pipe 76 % (362 ms with the x differences worked out here, 347 with the
        // planner's).
        //
        // Weights by simultaneous inversion (P. L. Montgomery, "Speeding the
        // Pollard and elliptic curve methods of factorization", Math. Comp. 48
        // (1987), section 10.3.1): the squared paths of G packed pairs share
        // ONE reciprocal per lane (G = 2: r = 1 / (s_0 s_1), 1 / s_0 = r s_1;
        // G = 4: r = 1 / (s_0 s_1 s_2 s_3), 1 / s_0 = (r s_2 s_3) s_1).
        // Without bounces and time offset (PATH_2D) the squared distance is
        // there already as the root's argument, which saves the product and
        // the root's error and pays for G = 4's two more roundings: 8.9e-8 rms
        // against 64 bits, 1.06e-7 with G = 2 and d * d; 1.25 MUFU operations
        // per voxel.  The other paths have to square the path and keep G = 2
        // (1.05e-7 rms; G = 4 would have 1.11e-7).  Groups with a path under
        // 3.5 mm or over 10 km, whose products could leave the normal FP32
        // range, take the scalar loop with the reference's safeRCP.
        constexpr int G = PATH == PATH_2D && KV % 8 == 0 ? 4 : 2;
        f32x2_t accp[KV / 2];
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) accp[j] = pack2(acc[2 * j], acc[2 * j + 1]);
        const f32x2_t rcp2p = pack2(rcp2, rcp2), rdp = pack2(rcp_dt, rcp_dt), two = pack2(2.f, 2.f);
        const f32x2_t nt0p = pack2(neg_t0, neg_t0);
#pragma unroll 4
        for (int i = 0; i < nl; ++i) {
            const float4 g = pl.geo[i];
            const int4 m = pl.meta[i];
            const f32x2_t biasp = pack2(__int_as_float(m.x), __int_as_float(m.y));
            const float dy = sub_rn(py, g.y), dz = sub_rn(pz, g.z);
            const float dy2 = mul_rn(dy, dy);
            const f32x2_t dy2p = pack2(dy2, dy2), dzp = pack2(dz, dz);
            const f32x2_t gwp = pack2(g.w, g.w);
            f32x2_t wlp = 0ull;
            if (WEIGHTED) {
                const float wl = pl.weight[i];
                wlp = pack2(wl, wl);
            }
#pragma unroll
            for (int j0 = 0; j0 < KV / 2; j0 += G) {
                f32x2_t sq[G], Iq[G], dx[G];
#pragma unroll
                for (int jj = 0; jj < G; jj += 2) {
                    const ulonglong2 v = pl.dx[(size_t)i * (KV / 4) + (j0 + jj) / 2];
                    dx[jj] = v.x;
                    dx[jj + 1] = v.y;
                }
#pragma unroll
                for (int jj = 0; jj < G; ++jj) {
                    const f32x2_t q = fma_rn2(dzp, dzp, fma_rn2(dx[jj], dx[jj], dy2p));
                    float q0, q1, b0, b1;
                    unpack2(q, q0, q1);
                    const f32x2_t d = pack2(sqrt_approx(q0), sqrt_approx(q1));
                    f32x2_t x;
                    if (PATH == PATH_2D) {
                        x = mul_rn2(d, rcp2p);
                        sq[jj] = q;
                    } else {
                        f32x2_t dist = fma_rn2(d, two, nt0p);
                        if (BOUNCE) dist = add_rn2(dist, gwp);
                        x = mul_rn2(dist, rdp);
                        sq[jj] = mul_rn2(dist, dist);
                    }
                    unpack2(add_rz2(x, biasp), b0, b1);
                    Iq[jj] = pack2(read_bin<CLAMP>(b0, m.z, slot_w), read_bin<CLAMP>(b1, m.z, slot_w));
                    if (WEIGHTED) Iq[jj] = mulf2(Iq[jj], wlp);
                }
                float m0, m1;
                if constexpr (G == 4) {
                    const f32x2_t p01 = mul_rn2(sq[0], sq[1]), p23 = mul_rn2(sq[2], sq[3]);
                    unpack2(mul_rn2(p01, p23), m0, m1);
                    const f32x2_t r = pack2(rcp_approx(m0), rcp_approx(m1));
                    const f32x2_t r01 = mul_rn2(r, p23), r23 = mul_rn2(r, p01);  // 1/(s0 s1), 1/(s2 s3)
                    accp[j0 + 0] = fmaf2(Iq[0], mul_rn2(r01, sq[1]), accp[j0 + 0]);
                    accp[j0 + 1] = fmaf2(Iq[1], mul_rn2(r01, sq[0]), accp[j0 + 1]);
                    accp[j0 + 2] = fmaf2(Iq[2], mul_rn2(r23, sq[3]), accp[j0 + 2]);
                    accp[j0 + 3] = fmaf2(Iq[3], mul_rn2(r23, sq[2]), accp[j0 + 3]);
                } else {
                    unpack2(mul_rn2(sq[0], sq[1]), m0, m1);
                    const f32x2_t r = pack2(rcp_approx(m0), rcp_approx(m1));
                    accp[j0 + 0] = fmaf2(Iq[0], mul_rn2(r, sq[1]), accp[j0 + 0]);
                    accp[j0 + 1] = fmaf2(Iq[1], mul_rn2(r, sq[0]), accp[j0 + 1]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) unpack2(accp[j], acc[2 * j], acc[2 * j + 1]);
    } else {
        // Guarded: every weight by the reference's own safeRCP, and with
        // PATH_EXACT the bin by conversion, like the reference's static_cast.
#pragma unroll 2
        for (int i = 0; i < nl; ++i) {
            const float4 g = pl.geo[i];
            const int4 m = pl.meta[i];
            const float wl = WEIGHTED ? pl.weight[i] : 1.f;
            const float dy = sub_rn(py, g.y), dz = sub_rn(pz, g.z);
            const float dy2 = mul_rn(dy, dy);
#pragma unroll
            for (int k = 0; k < KV; ++k) {
                const float dx = reinterpret_cast<const float*>(pl.dx)[i * KV + k];
                const float d = sqrt_approx(fma_rn(dz, dz, fma_rn(dx, dx, dy2)));
                float dist = fma_rn(d, 2.f, neg_t0);
                if (BOUNCE) dist = add_rn(dist, g.w);
                const float x = ref_bin_ratio(dist, rcp_dt);
                float I;
                if (PATH == PATH_EXACT) {
                    I = lds_f32((uint32_t)m.z + (min((uint32_t)(__float2int_rz(x) - m.x), slot_w) << 2));
                } else {
                    const float bias = __int_as_float(m.x);
                    I = read_bin<CLAMP>(add_rz(x, bias), m.z, slot_w);
                }
                if (WEIGHTED) I *= wl;
                acc[k] = fmaf(I, ref_safe_rcp(mul_rn(dist, dist)), acc[k]);
            }
        }
    }
}

// The main kernel.  One CTA of 32*WY*WZ threads (or several, one per chain)
// owns a tile of KV (x) x 8*WY (rows) x 4*WZ (depth slices) voxels; a warp
// covers 8 rows x 4 slices, a thread KV consecutive voxels along x.  Scan
// points (or, SAMPLED, K scan points drawn per tile) are taken in groups of 32:
// FP32 sums inside a group, a Kahan fold per group.
//
// Pipeline: one warp plans a group's bin windows two groups ahead (barrier
// `plan`); the windows arrive in stages of p.ch scan points, double buffered,
// each window one bulk copy that completes on the stage's `full` barrier; a
// warp that is through with a stage arrives on its `empty` barrier.  The warps
// take turns at planning and at copying, so no warp waits for another's
// planning and no barrier spans the CTA.
//
// Chains: the groups are cut into p.chains contiguous ranges, each with its
// own compensated sums; the chains' sums are folded, compensated, in order.
// SPLIT: one CTA per chain, which leaves its sums in p.chain_sums for
// fold_chains.  Otherwise one CTA walks the chains one after the other with the
// totals in `totals` (global, [2 KV][threads] per CTA): the same operations in
// the same order, so the volume is the same bit for bit.
template <int KV, int WY, int WZ, int PATH, bool BOUNCE, bool SAMPLED, bool CLAMP, bool SPLIT>
__device__ __forceinline__ void confocal_tile(const ConfocalGatherParams& p, uint32_t bx, uint32_t by, uint32_t bz,
                                              unsigned long long tile_id, float* totals = nullptr) {
    constexpr int NT = 32 * WY * WZ, NW = WY * WZ;
    constexpr int GRP = ConfocalGatherParams::kGroup;
    constexpr int ALIGN = 4;  // floats per 16-byte copy
    constexpr int TY = 8 * WY, TZ = 4 * WZ;
    const uint32_t CH = p.ch;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t slot_stride = p.slot_w + ALIGN;  // sentinel element(s) at slot_w
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem_raw);
    constexpr uint32_t NB = ConfocalGatherParams::kWindowBufs, MB = ConfocalGatherParams::kPlanBufs;
    const uint32_t bar_full = sbase, bar_empty = sbase + 8 * NB, bar_plan = sbase + 16 * NB;  // NB, NB and MB of 8 bytes
    float4* s_geo = reinterpret_cast<float4*>(smem_raw + 64);            // [MB][GRP]
    int4* s_meta = reinterpret_cast<int4*>(s_geo + MB * GRP);            // [MB][GRP]
    ulonglong2* s_dx = reinterpret_cast<ulonglong2*>(s_meta + MB * GRP);  // [MB][GRP][KV / 4]
    const float** s_src = reinterpret_cast<const float**>(s_dx + MB * GRP * (KV / 4));  // [MB][GRP]
    int* s_cnt = reinterpret_cast<int*>(s_src + MB * GRP);               // [MB][GRP]
    float* s_w = reinterpret_cast<float*>(s_cnt + MB * GRP);             // [MB][GRP]
    int2* s_group = reinterpret_cast<int2*>(s_w + MB * GRP);             // [MB] (points kept, guarded)
    constexpr size_t slots_off = ConfocalGatherParams::meta_bytes(KV);
    float* s_slots = reinterpret_cast<float*>(smem_raw + slots_off);     // [NB][CH][slot_stride]

    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int wy = warp % WY, wz = warp / WY;

    const uint32_t tx0 = bx * KV, ty0 = by * TY, tz0 = bz * TZ;
    const uint32_t vy = ty0 + wy * 8 + (lane & 7);
    const uint32_t vz = tz0 + wz * 4 + (lane >> 3);
    const bool row_ok = vy < p.Vy && vz < p.Vz;

    // Tile AABB of voxel centres (clamped to the volume).
    const uint32_t tx1 = min(tx0 + KV, p.Vx) - 1, ty1 = min(ty0 + TY, p.Vy) - 1, tz1 = min(tz0 + TZ, p.Vz) - 1;
    const float bx0 = fminf(p.xs[tx0], p.xs[tx1]), bx1 = fmaxf(p.xs[tx0], p.xs[tx1]);
    const float by0 = fminf(p.ys[tz0], p.ys[tz1]), by1 = fmaxf(p.ys[tz0], p.ys[tz1]);
    const float bz0 = fminf(p.zs[ty0], p.zs[ty1]), bz1 = fmaxf(p.zs[ty0], p.zs[ty1]);

    const float py = p.ys[min(vz, p.Vz - 1)];
    const float pz = p.zs[min(vy, p.Vy - 1)];

    constexpr bool PX = scatter_narrow(KV, PATH);
    f32x2_t px[PX ? KV / 2 : 1];
#pragma unroll
    for (int j = 0; j < (PX ? KV / 2 : 0); ++j)
        px[j] = pack2(p.xs[min(tx0 + 2 * j, p.Vx - 1)], p.xs[min(tx0 + 2 * j + 1, p.Vx - 1)]);

    const float rcp_dt = rcp_approx(p.dt);
    const float neg_t0 = -p.t0;
    // PATH_SCATTER: length(voxelSize) / 2 and the step timeStep + EPS, in the
    // reference's FP32 arithmetic (transient_reconstruction.cuh:113-125).
    const float scat_ext = is_scatter(PATH) ? mul_rn(0.5f, sqrt_approx(ref_dot3(p.vs[0], p.vs[1], p.vs[2]))) : 0.f;
    const float scat_step = is_scatter(PATH) ? add_rn(p.dt, FBP_EPS) : 0.f;

    const uint32_t rank = SPLIT ? blockIdx.x % p.chains : 0;  // this CTA's chain
    if (tid == 0) {
        for (uint32_t b = 0; b < NB; ++b) {
            mbar_init(bar_full + 8 * b, 1);
            mbar_init(bar_empty + 8 * b, NW);
        }
        for (uint32_t b = 0; b < MB; ++b) mbar_init(bar_plan + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // Sentinel of every slot.
    for (uint32_t i = tid; i < NB * CH * ALIGN; i += NT)
        s_slots[(size_t)(i / ALIGN) * slot_stride + p.slot_w + i % ALIGN] = 0.f;

    // SAMPLE_CLUSTERS: this tile's clusters, drawn by systematic sampling from
    // its CDF (K positions (k + u) / K), duplicates merged; each chosen
    // cluster is gathered whole with weight hits / (K p_c).
    uint32_t nitems = SAMPLED ? p.smp.K : p.L;
    const uint32_t* s_clu = nullptr;
    const float* s_cw = nullptr;
    if constexpr (SAMPLED) {
        __shared__ uint32_t clu[kMaxClusterSamples];
        __shared__ float cw[kMaxClusterSamples];
        __shared__ uint32_t ncl;
        if (p.smp.mode == SAMPLE_CLUSTERS) {
            const uint32_t K = p.smp.K, G = p.smp.G;
            const float* cdf = p.smp.tile_cdf ? p.smp.tile_cdf + tile_id * G : nullptr;
            if (warp == 0) {
                const float u = hash_uniform(p.smp.seed, tile_id, 0xFFFFFFFFu, 2);
                for (uint32_t k = lane; k < K; k += 32) {
                    const float x = ((float)k + u) / (float)K;
                    uint32_t c;
                    if (cdf) {
                        uint32_t lo = 0, hi = G - 1;  // first c with x < cdf[c]
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if (x < cdf[mid]) hi = mid; else lo = mid + 1;
                        }
                        c = lo;
                    } else {
                        c = min((uint32_t)(x * (float)G), G - 1);
                    }
                    clu[k] = c;
                }
                __syncwarp();
                if (lane == 0) {
                    uint32_t n = 0;
                    for (uint32_t k = 0; k < K; ++k) {
                        const uint32_t c = clu[k];
                        if (n > 0 && clu[n - 1] == c) {
                            cw[n - 1] += 1.f;
                        } else {
                            clu[n] = c;
                            cw[n] = 1.f;
                            ++n;
                        }
                    }
                    for (uint32_t j = 0; j < n; ++j) {
                        const uint32_t c = clu[j];
                        const float pc = cdf ? cdf[c] - (c > 0 ? cdf[c - 1] : 0.f) : 1.f / (float)G;
                        cw[j] = pc > 0.f ? cw[j] / ((float)K * pc) : 0.f;
                    }
                    ncl = n;
                }
            }
            __syncthreads();
            nitems = ncl * p.smp.cluster_side * p.smp.cluster_side;
            s_clu = clu;
            s_cw = cw;
        }
    }
    const uint32_t ngroups = (nitems + GRP - 1) / GRP;
    // Chain k: groups [k ngroups / chains, (k + 1) ngroups / chains).
    auto chain_begin = [&](uint32_t k) { return (uint32_t)((uint64_t)k * ngroups / p.chains); };
    const uint32_t g0 = SPLIT ? chain_begin(rank) : 0;
    const uint32_t mine = SPLIT ? chain_begin(rank + 1) - g0 : ngroups;  // groups of this CTA, from g0
    const uint32_t sub = GRP / CH;                                 // stages per group
    const uint32_t nstages = mine * sub;
    const bool warp_ok = __any_sync(0xffffffffu, row_ok);          // the warp owns voxels of the volume

    // Plan this CTA's group gi (one warp): bin window of each scan point.  Its
    // buffer held group gi - MB, which every warp is past: this runs once the
    // first stage of group gi - 2 is full, so once all were through with a
    // stage of group gi - 3 or, with one stage per group, all of gi - 4.
    auto plan_group = [&](uint32_t gi) {
        const uint32_t gb = (gi % MB) * GRP;
        {
            const uint32_t item = (g0 + gi) * GRP + lane;
            uint32_t l = item;
            float wgt = 1.f;
            if (SAMPLED && item < nitems) {
                const float u1 = hash_uniform(p.smp.seed, tile_id, item, 0);
                const float u2 = hash_uniform(p.smp.seed, tile_id, item, 1);
                float pl;
                if (p.smp.mode == SAMPLE_UNIFORM) {
                    l = min((uint32_t)(u1 * (float)p.L), p.L - 1);
                    pl = 1.f / (float)p.L;
                } else if (p.smp.mode == SAMPLE_ALIAS) {
                    const uint32_t kk = min((uint32_t)(u1 * (float)p.L), p.L - 1);
                    l = u2 < p.smp.prob[kk] ? kk : p.smp.alias[kk];
                    pl = p.smp.pl[l];
                } else {
                    // Point `inner` of the j-th chosen cluster (outside the grid
                    // for a ragged edge cluster: skipped).
                    const uint32_t cs = p.smp.cluster_side, cpr = (p.smp.n_side + cs - 1) / cs;
                    const uint32_t j = item / (cs * cs), inner = item - j * (cs * cs);
                    const uint32_t cl = s_clu[j];
                    const uint32_t ix = (cl % cpr) * cs + inner % cs, iz = (cl / cpr) * cs + inner / cs;
                    l = (ix < p.smp.n_side && iz < p.smp.n_side) ? iz * p.smp.n_side + ix : 0xFFFFFFFFu;
                    pl = 0.f;
                    wgt = s_cw[j];
                }
                if (p.smp.mode != SAMPLE_CLUSTERS) wgt = pl > 0.f ? 1.f / ((float)nitems * pl) : 0.f;
            }
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            int cnt = 0, near = 0, a = 0;
            bool skip = true;
            // l >= L: a point of a ragged edge cluster, outside the scan grid.
            if (item < nitems && l < p.L) {
                g = p.scan[l];
                // Nearest and farthest voxel-centre distance of the tile.
                const float cx = fminf(fmaxf(g.x, bx0), bx1), cy = fminf(fmaxf(g.y, by0), by1),
                            cz = fminf(fmaxf(g.z, bz0), bz1);
                const float dmin = sqrtf((g.x - cx) * (g.x - cx) + (g.y - cy) * (g.y - cy) + (g.z - cz) * (g.z - cz));
                const float fx = fmaxf(fabsf(g.x - bx0), fabsf(g.x - bx1)), fy = fmaxf(fabsf(g.y - by0), fabsf(g.y - by1)),
                            fz = fmaxf(fabsf(g.z - bz0), fabsf(g.z - bz1));
                const float dmax = sqrtf(fx * fx + fy * fy + fz * fz);
                const float bnc = BOUNCE ? g.w : 0.f;
                float pmin = 2.f * dmin + neg_t0 + bnc, pmax = 2.f * dmax + neg_t0 + bnc;
                if (is_scatter(PATH)) {
                    // The bins of dist -/+ ext, read one step past dist + ext;
                    // a walk clipped at 0 reads up to max(step, 2 ext).
                    pmin = fmaxf(0.f, pmin - 1.01f * scat_ext);
                    pmax = fmaxf(pmax + 1.01f * scat_ext, 2.02f * scat_ext) + scat_step;
                }
                // Paths this short make dist^2 <= EPS possible: use safeRCP's
                // branch.  Paths this long (or NaN) could take the batched
                // reciprocal's products out of the FP32 range: also per voxel.
                // The unconditional scattering walk also wants paths under
                // 64 m (its rounding bound) and dist - ext > 0 (pmin above).
                near = pmin < 0.0035f || !(pmax < (scatter_free(PATH) ? 64.f : 1.0e4f));
                // Conservative bin range with a 2-bin margin for rounding.
                const int blo = (int)fmaxf(fminf(floorf(pmin * rcp_dt), 1.0e9f), -1.0e9f) - 2;
                const int bhi = (int)fmaxf(fminf(floorf(pmax * rcp_dt), 1.0e9f), -1.0e9f) + 2;
                a = max(blo, 0) & ~(ALIGN - 1);
                skip = bhi < 0 || blo >= (int)p.T;  // no bin of this tile is inside [0, T)
                if (!skip) {
                    if (CLAMP) a = min(a, (int)(p.row_pitch - p.slot_w));
                    const int hi = min(bhi + 1, (int)p.row_pitch);
                    cnt = (max(hi - a, 0) + ALIGN - 1) & ~(ALIGN - 1);
                    if (cnt > (int)p.slot_w) {
                        if (CLAMP) {
                            // Capped window: bins past it map to the sentinel; only an
                            // uncovered valid bin would be an error.
                            if (min(bhi + 1, (int)p.T) - a > (int)p.slot_w) atomicExch(p.status, (int)FBP_ERR_DEVICE);
                            cnt = (int)p.slot_w;
                        } else {
                            // The planner's span bound failed: skip, report.
                            atomicExch(p.status, (int)FBP_ERR_DEVICE);
                            skip = true;
                            cnt = 0;
                        }
                    }
                }
            }
            // Points with nothing to read (also those with a NaN path) drop out;
            // the others keep their order.
            const unsigned kept = __ballot_sync(0xffffffffu, !skip);
            const uint32_t pos = __popc(kept & ((1u << lane) - 1u));
            const bool guarded = __any_sync(0xffffffffu, near && !skip) || p.exact_weights;
            if (!skip) {
                const uint32_t st = gi * sub + pos / CH;
                const uint32_t slot_elem = ((st % NB) * CH + pos % CH) * slot_stride;
                uint32_t slot = sbase + (uint32_t)slots_off + (slot_elem << 2);
                int bias = a;  // PATH_EXACT, guarded
                if (!(PATH == PATH_EXACT && guarded)) {
                    bias = __float_as_int((float)(8388608 - a));
                    if (!CLAMP) slot -= kBiasBits;
                }
                s_geo[gb + pos] = g;
                s_meta[gb + pos] = make_int4(bias, bias, (int)slot, 0);
                float* dx = reinterpret_cast<float*>(s_dx + (gb + pos) * (KV / 4));
#pragma unroll
                for (int k = 0; k < (PX ? 0 : KV); ++k) dx[k] = sub_rn(p.xs[min(tx0 + k, p.Vx - 1)], g.x);
                s_cnt[gb + pos] = cnt;
                s_src[gb + pos] = static_cast<const float*>(p.rows) + (size_t)l * p.row_pitch + a;
                s_w[gb + pos] = wgt;
            }
            if (lane == 0) s_group[gi % MB] = make_int2(__popc(kept), guarded);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_plan + 8 * (gi % MB));
        }
    };

    // A wait that ran out of polls (status FBP_ERR_TIMEOUT): the warp keeps
    // arriving at the CTA's barriers but touches nothing else.
    bool dead = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (!dead && !mbar_wait_parity(bar, parity)) {
            dead = true;
            if (lane == 0) atomicExch(p.status, (int)FBP_ERR_TIMEOUT);
        }
    };

    // Fill stage st (one warp): one bulk copy per window.
    auto produce = [&](uint32_t st) {
        const uint32_t buf = st % NB, gi = st / sub, first = (st % sub) * CH;
        wait(bar_plan + 8 * (gi % MB), (gi / MB) & 1);
        if (st >= NB) wait(bar_empty + 8 * buf, (st / NB - 1) & 1);
        if (dead) return;
        const uint32_t gb = (gi % MB) * GRP, n = (uint32_t)s_group[gi % MB].x;
        const uint32_t bytes = lane - first < CH && (uint32_t)lane < n ? (uint32_t)s_cnt[gb + lane] * 4u : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_arrive_expect_tx(bar_full + 8 * buf, total);
        __syncwarp();
        if (bytes)
            bulk_load(sbase + (uint32_t)slots_off + (((buf * CH + lane - first) * slot_stride) << 2), s_src[gb + lane],
                      bytes, bar_full + 8 * buf);
    };

    // Compensated sums: in registers, or (16 voxels per thread, the scattering
    // walk) in shared memory behind the windows, [2 KV][NT] so a warp's accesses
    // are consecutive words.
    constexpr bool KSMEM = kahan_smem_bytes(KV, NT, is_scatter(PATH)) > 0;
    static_assert(!SPLIT || KSMEM, "a split tile keeps its compensated sums in shared memory");
    float* s_kahan = reinterpret_cast<float*>(
        smem_raw + ((slots_off + (size_t)NB * CH * slot_stride * sizeof(float) + 15) & ~size_t(15)));
    float acc[KV], ksum[KSMEM ? 1 : KV], kcomp[KSMEM ? 1 : KV];
#pragma unroll
    for (int k = 0; k < KV; ++k) acc[k] = 0.f;
    if constexpr (KSMEM) {
#pragma unroll
        for (int k = 0; k < 2 * KV; ++k) s_kahan[k * NT + tid] = 0.f;
    } else {
#pragma unroll
        for (int k = 0; k < KV; ++k) ksum[k] = kcomp[k] = 0.f;
    }
    // A previous tile's writes to this memory before the bulk copies' writes.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // barriers initialised, sentinels written
    if (warp < 2 && (uint32_t)warp < mine) plan_group(warp);
    if (warp == 0 && nstages > 0) produce(0);
    uint32_t chain = 0;

    for (uint32_t gi = 0; gi < mine; ++gi) {
        const uint32_t gb = (gi % MB) * GRP;
        float scale = 1.f;
        for (uint32_t h = 0; h < sub; ++h) {
            const uint32_t st = gi * sub + h, buf = st % NB;
            wait(bar_full + 8 * buf, (st / NB) & 1);
            if (st + 1 < nstages && warp == (int)((st + 1) % NW)) produce(st + 1);
            if (h == 0 && gi + 2 < mine && !dead && warp == (int)((st + NW / 2) % NW)) plan_group(gi + 2);
            const int2 grp = s_group[gi % MB];
            const int nl = min((int)CH, grp.x - (int)(h * CH));
            if (warp_ok && !dead) {
                const uint32_t o = gb + h * CH;
                const ScanPlan plan{s_geo + o, s_meta + o, s_dx + o * (KV / 4), s_w + o};
                if (!grp.y) {
                    confocal_stage<KV, PATH, BOUNCE, CLAMP, false, SAMPLED>(plan, nl, py, pz, neg_t0, rcp_dt, p.slot_w,
                                                                            acc, scat_ext, scat_step, !p.scat_exact, px);
                    if (PATH == PATH_2D) scale = 0.25f;  // w was rcp(d^2) = 4 rcp(dist^2)
                } else {
                    confocal_stage<KV, PATH, BOUNCE, CLAMP, true, SAMPLED>(plan, nl, py, pz, neg_t0, rcp_dt, p.slot_w,
                                                                           acc, scat_ext, scat_step, true, px);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * buf);
        }
#pragma unroll
        for (int k = 0; k < KV; ++k) {
            if constexpr (KSMEM) {
                float sk = s_kahan[(2 * k) * NT + tid], ck = s_kahan[(2 * k + 1) * NT + tid];
                kahan_add(mul_rn(acc[k], scale), sk, ck);
                s_kahan[(2 * k) * NT + tid] = sk;
                s_kahan[(2 * k + 1) * NT + tid] = ck;
            } else {
                kahan_add(mul_rn(acc[k], scale), ksum[k], kcomp[k]);
            }
            acc[k] = 0.f;
        }
        if constexpr (KSMEM && !SPLIT) {
            // The end of a chain, of several: its sums to the totals.
            while (p.chains > 1 && chain < p.chains && gi + 1 == chain_begin(chain + 1)) {
                for (int k = 0; k < KV; ++k) {
                    float* t = totals + ((size_t)blockIdx.x * KV + k) * (2 * NT) + tid;
                    float sum = chain ? t[0] : 0.f, comp = chain ? t[NT] : 0.f;
                    kahan_fold(s_kahan[(2 * k) * NT + tid], s_kahan[(2 * k + 1) * NT + tid], sum, comp);
                    t[0] = sum;
                    t[NT] = comp;
                    s_kahan[(2 * k) * NT + tid] = s_kahan[(2 * k + 1) * NT + tid] = 0.f;
                }
                ++chain;
            }
        }
    }

    if constexpr (SPLIT) {
        if (row_ok) {
            const size_t n = (size_t)p.Vx * p.Vy * p.Vz;
            float* sums = p.chain_sums + (size_t)rank * 2 * n + ((size_t)vz * p.Vy + vy) * p.Vx + tx0;
#pragma unroll
            for (int k = 0; k < KV; ++k)
                if (tx0 + k < p.Vx) {
                    sums[k] = s_kahan[(2 * k) * NT + tid];
                    sums[n + k] = s_kahan[(2 * k + 1) * NT + tid];
                }
        }
    } else if (row_ok) {
        float* out = p.volume + ((size_t)vz * p.Vy + vy) * p.Vx + tx0;
#pragma unroll
        for (int k = 0; k < KV; ++k)
            if (tx0 + k < p.Vx)
                out[k] = !KSMEM ? ksum[KSMEM ? 0 : k]
                                : (p.chains > 1 ? totals[((size_t)blockIdx.x * KV + k) * (2 * NT) + tid] : s_kahan[(2 * k) * NT + tid]);
    }
    __syncthreads();  // every warp is through with the barriers
    if (tid == 0) {   // (a persistent kernel sets them up again for its next tile)
        for (uint32_t b = 0; b < 2 * NB + MB; ++b) mbar_inval(bar_full + 8 * b);
    }
}

// Registers for three CTAs of 256 threads (80 each), or four (64).
constexpr int gather_ctas(int threads, bool narrow = false) {
    return threads > 256 ? 1 : narrow ? kScatterCtasPerSm : kGatherCtasPerSm;
}

template <int KV, int WY, int WZ, int PATH, bool BOUNCE, bool SAMPLED, bool CLAMP, bool SPLIT = false>
__global__ void __launch_bounds__(32 * WY * WZ, gather_ctas(32 * WY * WZ, scatter_narrow(KV, PATH)))
confocal_gather_kernel(ConfocalGatherParams p) {
    const uint32_t cs = SPLIT ? p.chains : 1, bx = blockIdx.x / cs;
    const unsigned long long tile_id = ((unsigned long long)blockIdx.z * gridDim.y + blockIdx.y) * (gridDim.x / cs) + bx;
    confocal_tile<KV, WY, WZ, PATH, BOUNCE, SAMPLED, CLAMP, SPLIT>(p, bx, blockIdx.y, blockIdx.z, tile_id);
}

// Persistent form for a batch of captures: CTAs pull (capture, tile) work items
// from an atomic counter until the list is exhausted.  Items are sorted by
// decreasing cost on the host, so the long tiles start first.
struct BatchItem {
    uint32_t capture, bx, by, bz;
};

template <int KV, int WY, int WZ, int PATH, bool BOUNCE, bool CLAMP>
__global__ void __launch_bounds__(32 * WY * WZ, gather_ctas(32 * WY * WZ))
confocal_batch_kernel(const ConfocalGatherParams* __restrict__ caps, const BatchItem* __restrict__ items,
                      uint32_t nitems, unsigned int* __restrict__ counter, float* __restrict__ totals) {
    __shared__ uint32_t s_item;
    for (;;) {
        __syncthreads();  // the previous tile is done with shared memory and s_item
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const BatchItem w = items[it];
        confocal_tile<KV, WY, WZ, PATH, BOUNCE, false, CLAMP, false>(caps[w.capture], w.bx, w.by, w.bz, it, totals);
    }
}

}  // namespace fbp
