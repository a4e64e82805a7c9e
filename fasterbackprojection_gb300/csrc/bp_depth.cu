// Depth-plane backprojection (the reference's non-AABB mode).
//
// Replaces Laser::reconstructDepthConfocal / reconstructDepthExhaustive
// (Laser.cu:379-480) and backprojectConfocal / backprojectExhaustive
// (transient_reconstruction.cuh:41-91).  Test points are
//   laser_xyz[c] + wall_normal * float(depths[d])
// and contributions are unweighted, summed in a fixed order instead of by one
// atomic per pair.  Time bins follow the reference's FP32 expression exactly.
//   Confocal: depth_tile_kernel, a thread for 16 test points of a tile, windows
//   of the rows in shared memory, FP32 sums of 32 scan points folded with
//   compensation.
//   Few planes of many scan points (tiles_pay), rows too long for the tiles'
//   windows, no memory for FP32 rows, and every exhaustive capture: a thread per
//   test point that reads the rows from global memory (FP32 sums of 64, Kahan
//   across them).
#include "fbp_internal.cuh"
#include "bp_common.cuh"

#include <algorithm>
#include <cmath>

namespace fbp {

struct DepthTileParams {
    const float4* scan;      // [L] (x, y, z, bounce)
    const float* xyz;        // [L][3]
    const double* depths;    // [D]
    const float* rows;       // [L][pitch]
    float* act;              // [L][D]
    int* status;
    uint32_t L, D, T, pitch;
    uint32_t side;           // > 0: the scan points are a side x side grid (tiles of 16 x 16), else runs of 256
    float nx, ny, nz, t0, dt;
    uint32_t chains;         // CTAs per tile, one per range of scan-point groups
    float* chain_sums;       // chains > 1: [chains][sum, compensation][L][D]

    static constexpr int kGroup = 32, kPlanBufs = 4, kThreads = 256, kDepths = 16;
    static constexpr uint32_t kSlot = 256;           // widest window that is not the whole row
    // Barriers, per scan point of kPlanBufs groups (x, y, z, bounce), (bias,
    // bias, slot address), the window's source and length, two words per group.
    // (A lattice's x differences, 16 floats, per scan point too.)
    static constexpr size_t kMeta = 64 + (size_t)kPlanBufs * kGroup * (16 + 16 + 64 + 8 + 4) + kPlanBufs * 8;
    static constexpr size_t kSums = (size_t)2 * kDepths * kThreads * sizeof(float);
    static constexpr size_t kSmem = kSmSharedBytes / 3 - kCtaReservedShared - 512;  // three CTAs per SM
    static constexpr uint32_t kWindowFloats = (uint32_t)((kSmem - kMeta - kSums) / sizeof(float));
    // Longest row whose whole-row windows fit, one scan point to a stage.
    static constexpr uint32_t kMaxBins = (kWindowFloats / 2 - 8) / 4 * 4;
    static uint32_t pitch_of(uint32_t T) { return (T + 3) / 4 * 4 + kSlot; }
    static size_t row_bytes(const fbp_recon_info& in) {
        return (size_t)in.num_laser_targets * pitch_of(in.num_time_bins) * sizeof(float);
    }
};

// A CTA (or p.chains of them, one per range of scan-point groups) owns 256
// scan points' test points at 16 consecutive depths.  Pipeline, groups and
// folds as in the confocal gather; the window width is the CTA's own, from the
// box of its points (the host does not know the positions), and windows wider
// than kSlot are whole rows, like those of a CTA with a non-finite point
// (int(NaN) is bin 0).
// YONLY: the wall normal has only a y component, so x and z do not depend on
// the depth (adding 0 * depth changes no bit).  If the CTA's 16 x 16 scan
// points are then also a lattice (x by column, z by row, one y), a thread takes
// the 16 columns of one row at one depth, so that the x differences are common
// to the CTA (made by the planner) and a warp, 2 rows x 16 depths, reads few
// neighbouring bins; otherwise a thread takes the 16 depths of one scan point,
// a warp 8 x 4 of the grid.
// Bound by the issue port (a packed FP32 instruction holds it two cycles):
// about 20 cycles per packed pair on a lattice, 30 otherwise.  64^2 x 512, 200
// planes: one thread per point with rows in global memory 2867 us, a thread
// per scan point 1200 us, the lattice 898 us.
// PLAIN: no time offset and no bounces.
template <bool YONLY, bool BOUNCE, bool PLAIN>
__global__ void __launch_bounds__(DepthTileParams::kThreads, YONLY ? 3 : 2) depth_tile_kernel(DepthTileParams p) {
    using P = DepthTileParams;
    constexpr int NT = P::kThreads, NW = NT / 32, KV = P::kDepths;
    constexpr uint32_t GRP = P::kGroup, NB = 2, MB = P::kPlanBufs;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float s_box[6][NW];
    __shared__ float s_lat[33];  // x of the columns, z of the rows, y
    __shared__ float s_df[KV];   // the depths
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t bar_full = sbase, bar_empty = sbase + 8 * NB, bar_plan = sbase + 16 * NB;  // NB, NB and MB of 8 bytes
    float4* s_geo = reinterpret_cast<float4*>(smem_raw + 64);              // [MB][GRP]
    int4* s_meta = reinterpret_cast<int4*>(s_geo + MB * GRP);              // [MB][GRP]
    ulonglong2* s_dx = reinterpret_cast<ulonglong2*>(s_meta + MB * GRP);   // [MB][GRP][KV / 4]
    const float** s_src = reinterpret_cast<const float**>(s_dx + MB * GRP * (KV / 4));  // [MB][GRP]
    int* s_cnt = reinterpret_cast<int*>(s_src + MB * GRP);                 // [MB][GRP]
    int2* s_group = reinterpret_cast<int2*>(s_cnt + MB * GRP);             // [MB] (points kept, guarded)
    float* s_sums = reinterpret_cast<float*>(smem_raw + P::kMeta);         // [2 KV][NT]
    float* s_slots = s_sums + 2 * KV * NT;                                 // [NB][CH][slot_stride]
    const uint32_t slots_at = sbase + (uint32_t)(P::kMeta + P::kSums);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = blockIdx.x % p.chains, tile = blockIdx.x / p.chains;
    // This thread's scan point (unless the tile is a lattice).
    const uint32_t cx = (warp & 1) * 8 + (lane & 7), cz = (warp >> 1) * 4 + (lane >> 3), sx = p.side ? (p.side + 15) / 16 : 1;
    uint32_t c = tile * NT + tid;
    bool ok = c < p.L;
    if (p.side) {
        const uint32_t ix = tile % sx * 16 + cx, iz = tile / sx * 16 + cz;
        ok = ix < p.side && iz < p.side;
        c = min(iz, p.side - 1) * p.side + min(ix, p.side - 1);
    }
    c = min(c, p.L - 1);
    const uint32_t d0 = blockIdx.y * KV;

    if (tid < KV) s_df[tid] = (float)p.depths[min(d0 + tid, p.D - 1)];
    __syncthreads();
    // Test points (transient_reconstruction.cuh:51) and their box.
    const float lx = p.xyz[3 * (size_t)c], ly = p.xyz[3 * (size_t)c + 1], lz = p.xyz[3 * (size_t)c + 2];
    float box[6] = {INFINITY, -INFINITY, INFINITY, -INFINITY, INFINITY, -INFINITY};
    bool finite = true;
    // YONLY: x and z are the scan point's at every depth; 0 * depth, NaN where the
    // depth is not finite, is put into y (any NaN makes the path one).
    auto point = [&](int k, float& x, float& y, float& z) {
        const float df = s_df[k];
        x = YONLY ? lx : fma_rn(p.nx, df, lx);
        y = YONLY && !isfinite(df) ? NAN : fma_rn(p.ny, df, ly);
        z = YONLY ? lz : fma_rn(p.nz, df, lz);
    };
    for (int k = 0; k < KV; ++k) {
        float x, y, z;
        point(k, x, y, z);
        finite = finite && isfinite(x) && isfinite(y) && isfinite(z);
        box[0] = fminf(box[0], x); box[1] = fmaxf(box[1], x);
        box[2] = fminf(box[2], y); box[3] = fmaxf(box[3], y);
        box[4] = fminf(box[4], z); box[5] = fmaxf(box[5], z);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, box[i], o);
            box[i] = i & 1 ? fmaxf(box[i], v) : fminf(box[i], v);
        }
        if (lane == 0) s_box[i][warp] = box[i];
    }
    if (tid == 0) {
        for (uint32_t b = 0; b < NB; ++b) {
            mbar_init(bar_full + 8 * b, 1);
            mbar_init(bar_empty + 8 * b, NW);
        }
        for (uint32_t b = 0; b < MB; ++b) mbar_init(bar_plan + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
#pragma unroll
    for (int k = 0; k < 2 * KV; ++k) s_sums[k * NT + tid] = 0.f;
    if (cz == 0) s_lat[cx] = lx;
    if (cx == 0) s_lat[16 + cz] = lz;
    if (tid == 0) s_lat[32] = ly;
    const bool odd = __syncthreads_or(!finite);
    const bool lattice = __syncthreads_and(YONLY && p.side > 0 && !odd && lx == s_lat[cx] && lz == s_lat[16 + cz] &&
                                           ly == s_lat[32]);
    // On a lattice: this thread's depth and row.
    const uint32_t ld = d0 + (lane & 15), lr = (uint32_t)warp * 2 + (lane >> 4);
    if (lattice) ok = ld < p.D && tile / sx * 16 + lr < p.side;
    const bool warp_ok = __any_sync(0xffffffffu, ok);
#pragma unroll
    for (int i = 0; i < 6; ++i)
        for (int w = 0; w < NW; ++w) box[i] = i & 1 ? fmaxf(box[i], s_box[i][w]) : fminf(box[i], s_box[i][w]);

    // Window width: the round trip across the box and a 2-bin margin on each
    // side, or the whole row; scan points per stage: what fits twice.
    const float rcp_dt = rcp_approx(p.dt);
    const float ex = box[1] - box[0], ey = box[3] - box[2], ez = box[5] - box[4];
    const float span = 2.01f * sqrtf(ex * ex + ey * ey + ez * ez) / p.dt + 12.f;
    const uint32_t t_round = (p.T + 3) & ~3u;
    const bool whole = odd || !(span < (float)P::kSlot) || t_round + 4 <= (uint32_t)span;
    const uint32_t slot_w = whole ? t_round + 4 : ((uint32_t)span + 4) & ~3u;
    const uint32_t slot_stride = slot_w + 4;  // sentinel at slot_w
    uint32_t CH = GRP;
    while (CH > 1 && NB * CH * slot_stride > P::kWindowFloats) CH >>= 1;
    for (uint32_t i = tid; i < NB * CH * 4; i += NT) s_slots[(size_t)(i / 4) * slot_stride + slot_w + i % 4] = 0.f;

    const uint32_t ngroups = (p.L + GRP - 1) / GRP;
    const uint32_t g0 = (uint32_t)((uint64_t)rank * ngroups / p.chains);
    const uint32_t mine = (uint32_t)((uint64_t)(rank + 1) * ngroups / p.chains) - g0;
    const uint32_t sub = GRP / CH, nstages = mine * sub;
    const float neg_t0 = -p.t0;

    // Plan this CTA's group gi (one warp): see the confocal gather.
    auto plan_group = [&](uint32_t gi) {
        const uint32_t gb = (gi % MB) * GRP, l = (g0 + gi) * GRP + lane;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        int a = 0, cnt = 0, near = 0;
        bool keep = l < p.L;
        if (keep) {
            g = p.scan[l];
            const float cx = fminf(fmaxf(g.x, box[0]), box[1]), cy = fminf(fmaxf(g.y, box[2]), box[3]),
                        cz = fminf(fmaxf(g.z, box[4]), box[5]);
            const float dmin = sqrtf((g.x - cx) * (g.x - cx) + (g.y - cy) * (g.y - cy) + (g.z - cz) * (g.z - cz));
            const float fx = fmaxf(fabsf(g.x - box[0]), fabsf(g.x - box[1])),
                        fy = fmaxf(fabsf(g.y - box[2]), fabsf(g.y - box[3])),
                        fz = fmaxf(fabsf(g.z - box[4]), fabsf(g.z - box[5]));
            const float dmax = sqrtf(fx * fx + fy * fy + fz * fz);
            const float bnc = BOUNCE ? g.w : 0.f;
            const float pmin = 2.f * dmin + neg_t0 + bnc, pmax = 2.f * dmax + neg_t0 + bnc;
            if (odd || !isfinite(pmax) || !isfinite(pmin)) {
                near = 1;  // int() of every path, over the row from bin 0
                cnt = (int)slot_w;
            } else {
                near = pmin < 0.0035f && (p.t0 > 0.f || BOUNCE);  // int() truncates towards zero
                const int blo = (int)fmaxf(fminf(floorf(pmin * rcp_dt), 1.0e9f), -1.0e9f) - 2;
                const int bhi = (int)fmaxf(fminf(floorf(pmax * rcp_dt), 1.0e9f), -1.0e9f) + 2;
                keep = bhi >= 0 && blo < (int)p.T;  // a bin of the tile is inside [0, T)
                a = whole ? 0 : max(blo, 0) & ~3;
                cnt = whole ? (int)slot_w : (max(bhi + 1 - a, 0) + 3) & ~3;
                if (keep && cnt > (int)slot_w) {  // the span bound failed: skip, report
                    atomicExch(p.status, (int)FBP_ERR_DEVICE);
                    keep = false;
                }
            }
            cnt = min(cnt, (int)p.pitch - a);
        }
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        const bool guarded = __any_sync(0xffffffffu, near && keep);
        const uint32_t pos = __popc(kept & ((1u << lane) - 1u));
        if (keep) {
            const uint32_t st = gi * sub + pos / CH;
            uint32_t slot = slots_at + (((st % NB) * CH + pos % CH) * slot_stride << 2);
            int bias = a;
            if (!guarded) {
                bias = __float_as_int((float)(8388608 - a));
                if (!whole) slot -= kBiasBits;
            }
            s_geo[gb + pos] = g;
            s_meta[gb + pos] = make_int4(bias, bias, (int)slot, 0);
            if (lattice) {
                float* dx = reinterpret_cast<float*>(s_dx + (gb + pos) * (KV / 4));
#pragma unroll
                for (int k = 0; k < KV; ++k) dx[k] = sub_rn(s_lat[k], g.x);
            }
            s_cnt[gb + pos] = cnt;
            s_src[gb + pos] = p.rows + (size_t)l * p.pitch + a;
        }
        if (lane == 0) s_group[gi % MB] = make_int2(__popc(kept), guarded);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_plan + 8 * (gi % MB));
    };
    bool dead = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (!dead && !mbar_wait_parity(bar, parity)) {
            dead = true;
            if (lane == 0) atomicExch(p.status, (int)FBP_ERR_TIMEOUT);
        }
    };
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
            bulk_load(slots_at + ((buf * CH + lane - first) * slot_stride << 2), s_src[gb + lane], bytes, bar_full + 8 * buf);
    };

    f32x2_t accp[KV / 2];
#pragma unroll
    for (int j = 0; j < KV / 2; ++j) accp[j] = 0ull;
    const f32x2_t xs = PLAIN ? pack2(2.f * rcp_dt, 2.f * rcp_dt) : pack2(rcp_dt, rcp_dt);  // (2 d) rcp = d (2 rcp)
    const f32x2_t two = pack2(2.f, 2.f), nt0p = pack2(neg_t0, neg_t0);
    // Path ratio of a packed pair of squared distances.
    auto ratio = [&](f32x2_t q, float bounce) -> f32x2_t {
        float q0, q1;
        unpack2(q, q0, q1);
        f32x2_t d = pack2(sqrt_approx(q0), sqrt_approx(q1));
        if (!PLAIN) {
            d = fma_rn2(d, two, nt0p);
            if (BOUNCE) d = add_rn2(d, pack2(bounce, bounce));
        }
        return mul_rn2(d, xs);
    };
    const float lpy = fma_rn(p.ny, s_df[lane & 15], s_lat[32]), lpz = s_lat[16 + lr];
    auto walk_lattice = [&](uint32_t o, int n, auto&& sample) {
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const float4 g = s_geo[o + i];
            const int4 m = s_meta[o + i];
            const float dy = sub_rn(lpy, g.y), dz = sub_rn(lpz, g.z);
            const float dy2 = mul_rn(dy, dy);
            const f32x2_t dy2p = pack2(dy2, dy2), dzp = pack2(dz, dz);
#pragma unroll
            for (int j = 0; j < KV / 4; ++j) {
                const ulonglong2 dx = s_dx[(o + i) * (KV / 4) + j];
                accp[2 * j] = add_rn2(accp[2 * j], sample(ratio(fma_rn2(dzp, dzp, fma_rn2(dx.x, dx.x, dy2p)), g.w), m));
                accp[2 * j + 1] =
                    add_rn2(accp[2 * j + 1], sample(ratio(fma_rn2(dzp, dzp, fma_rn2(dx.y, dx.y, dy2p)), g.w), m));
            }
        }
    };
    auto walk_points = [&](uint32_t o, int n, auto&& sample) {
        float px[YONLY ? 1 : KV], pz[YONLY ? 1 : KV];  // (made per stage: they would hold the lattice's registers)
        f32x2_t pyp[KV / 2];
#pragma unroll
        for (int k = 0; k < KV; k += 2) {
            float y0, y1;
            point(k, px[YONLY ? 0 : k], y0, pz[YONLY ? 0 : k]);
            point(k + 1, px[YONLY ? 0 : k + 1], y1, pz[YONLY ? 0 : k + 1]);
            pyp[k / 2] = pack2(y0, y1);
        }
#pragma unroll 2
        for (int i = 0; i < n; ++i) {
            const float4 g = s_geo[o + i];
            const int4 m = s_meta[o + i];
            const float dx = sub_rn(px[0], g.x), dz = sub_rn(pz[0], g.z);
#pragma unroll
            for (int j = 0; j < KV / 2; ++j) {
                const f32x2_t dy = sub_rn2(pyp[j], pack2(g.y, g.y));
                f32x2_t dxp = pack2(dx, dx), dzp = pack2(dz, dz);
                if (!YONLY) {
                    dxp = sub_rn2(pack2(px[YONLY ? 0 : 2 * j], px[YONLY ? 0 : 2 * j + 1]), pack2(g.x, g.x));
                    dzp = sub_rn2(pack2(pz[YONLY ? 0 : 2 * j], pz[YONLY ? 0 : 2 * j + 1]), pack2(g.z, g.z));
                }
                accp[j] = add_rn2(accp[j], sample(ratio(fma_rn2(dzp, dzp, fma_rn2(dxp, dxp, mul_rn2(dy, dy))), g.w), m));
            }
        }
    };
    auto fast = [&](f32x2_t x, const int4& m) -> f32x2_t {
        float b0, b1;
        unpack2(add_rz2(x, pack2(__int_as_float(m.x), __int_as_float(m.y))), b0, b1);
        return pack2(read_bin<false>(b0, m.z, slot_w), read_bin<false>(b1, m.z, slot_w));
    };
    auto clamped = [&](f32x2_t x, const int4& m) -> f32x2_t {
        float b0, b1;
        unpack2(add_rz2(x, pack2(__int_as_float(m.x), __int_as_float(m.y))), b0, b1);
        return pack2(read_bin<true>(b0, m.z, slot_w), read_bin<true>(b1, m.z, slot_w));
    };
    auto converted = [&](f32x2_t x, const int4& m) -> f32x2_t {  // static_cast<int>, like the reference
        float x0, x1;
        unpack2(x, x0, x1);
        return pack2(lds_f32((uint32_t)m.z + (min((uint32_t)(__float2int_rz(x0) - m.x), slot_w) << 2)),
                     lds_f32((uint32_t)m.z + (min((uint32_t)(__float2int_rz(x1) - m.x), slot_w) << 2)));
    };

    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // sentinels written
    if (warp < 2 && (uint32_t)warp < mine) plan_group(warp);
    if (warp == 0 && nstages > 0) produce(0);
    for (uint32_t gi = 0; gi < mine; ++gi) {
        const uint32_t gb = (gi % MB) * GRP;
        for (uint32_t h = 0; h < sub; ++h) {
            const uint32_t st = gi * sub + h, buf = st % NB;
            wait(bar_full + 8 * buf, (st / NB) & 1);
            if (st + 1 < nstages && warp == (int)((st + 1) % NW)) produce(st + 1);
            if (h == 0 && gi + 2 < mine && !dead && warp == (int)((st + NW / 2) % NW)) plan_group(gi + 2);
            const int2 grp = s_group[gi % MB];
            const int n = min((int)CH, grp.x - (int)(h * CH));
            if (warp_ok && !dead) {
                const uint32_t o = gb + h * CH;
                if (YONLY && lattice && !whole && !grp.y) walk_lattice(o, n, fast);
                else if (YONLY && lattice && !grp.y) walk_lattice(o, n, clamped);
                else if (YONLY && lattice) walk_lattice(o, n, converted);
                else if (grp.y) walk_points(o, n, converted);
                else if (whole) walk_points(o, n, clamped);
                else walk_points(o, n, fast);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * buf);
        }
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) {
            float part[2];
            unpack2(accp[j], part[0], part[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float* s = s_sums + (2 * (2 * j + h)) * NT + tid;
                float sum = s[0], comp = s[NT];
                kahan_add(part[h], sum, comp);
                s[0] = sum;
                s[NT] = comp;
            }
            accp[j] = 0ull;
        }
    }

    if (!ok) return;
    const size_t n = (size_t)p.L * p.D;
    float* out = p.chains == 1 ? p.act : p.chain_sums + (size_t)rank * 2 * n;
    for (uint32_t k = 0; k < (uint32_t)KV; ++k) {
        const uint32_t ix = tile % sx * 16 + k, iz = tile / sx * 16 + lr;
        if (lattice ? ix >= p.side : d0 + k >= p.D) continue;
        const size_t at = lattice ? ((size_t)iz * p.side + ix) * p.D + ld : (size_t)c * p.D + d0 + k;
        out[at] = s_sums[(2 * k) * NT + tid];
        if (p.chains > 1) out[n + at] = s_sums[(2 * k + 1) * NT + tid];
    }
}

template <bool YONLY, bool BOUNCE, bool PLAIN>
fbp_status go_depth_tiles(fbp_context* ctx, DepthTileParams p, dim3 grid, cudaStream_t stream) {
    auto kernel = depth_tile_kernel<YONLY, BOUNCE, PLAIN>;
    const size_t smem = DepthTileParams::kMeta + DepthTileParams::kSums + DepthTileParams::kWindowFloats * sizeof(float);
    FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t n = (uint64_t)p.L * p.D;
    grid.x *= p.chains;
    kernel<<<grid, DepthTileParams::kThreads, smem, stream>>>(p);
    FBP_CHECK_LAUNCH(ctx, "depth_tile_kernel");
    return p.chains > 1 ? fold_chains(ctx, p.chain_sums, p.chains, n, p.act, stream) : FBP_OK;
}

// The confocal planes by tiles of 256 scan points x 16 depths.
fbp_status launch_depth_tiles(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, int layout,
                              const float* laser_xyz, const double* depths, uint32_t D, float* act,
                              cudaStream_t stream) {
    const uint32_t L = in.num_laser_targets, T = in.num_time_bins;
    DepthTileParams p{};
    p.pitch = DepthTileParams::pitch_of(T);
    const uint32_t side = (uint32_t)std::lround(std::sqrt((double)L));
    p.side = (uint64_t)side * side == L ? side : 0;
    p.nx = in.wall_normal[0]; p.ny = in.wall_normal[1]; p.nz = in.wall_normal[2];
    const uint64_t tiles = p.side ? (uint64_t)cdiv(side, 16) * cdiv(side, 16) : cdiv(L, DepthTileParams::kThreads);
    const dim3 grid((unsigned)tiles, cdiv(D, DepthTileParams::kDepths));
    const bool yonly = p.nx == 0.f && p.nz == 0.f, bounce = in.discard_first_last_bounces == 0;
    p.chains = split_chains(ctx, tiles * grid.y, 1.0, cdiv(L, DepthTileParams::kGroup), yonly ? 3 : 2, 5.0, (uint64_t)L * D);
    float* rows = nullptr;
    FBP_TRY(gather_scratch(ctx, DepthTileParams::row_bytes(in), &p.chains, (uint64_t)L * D, stream, &rows, &p.chain_sums));
    PrepTables tables{};
    FBP_TRY(table_buffers(ctx, in, laser_xyz, nullptr, false, stream, &tables));
    FBP_TRY(prepare_gather(ctx, dtype,
                           PrepRows{cube, rows, L, T, p.pitch, layout == FBP_LAYOUT_TIME_MAJOR}, tables, stream));
    p.scan = tables.lasers;
    p.xyz = laser_xyz;
    p.depths = depths;
    p.rows = rows;
    p.act = act;
    p.status = ctx->status_dev;
    p.L = L; p.D = D; p.T = T;
    p.t0 = in.time_offset;
    p.dt = in.time_step;
    const bool plain = !bounce && p.t0 == 0.f;
    if (yonly) {
        if (bounce) return go_depth_tiles<true, true, false>(ctx, p, grid, stream);
        if (plain) return go_depth_tiles<true, false, true>(ctx, p, grid, stream);
        return go_depth_tiles<true, false, false>(ctx, p, grid, stream);
    }
    if (bounce) return go_depth_tiles<false, true, false>(ctx, p, grid, stream);
    if (plain) return go_depth_tiles<false, false, true>(ctx, p, grid, stream);
    return go_depth_tiles<false, false, false>(ctx, p, grid, stream);
}

template <typename S>
__global__ void depth_confocal_kernel(const S* __restrict__ rows, uint32_t pitch, const float4* __restrict__ scan,
                                      const float* __restrict__ laser_xyz, const double* __restrict__ depths,
                                      uint32_t L, uint32_t D, uint32_t T, float nx, float ny, float nz, float t0,
                                      float dt, int bounce, float* __restrict__ act) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= (uint64_t)L * D) return;
    const uint32_t c = (uint32_t)(i / D), d = (uint32_t)(i % D);
    const float df = (float)depths[d];
    // transient_reconstruction.cuh:51
    const float px = fma_rn(nx, df, laser_xyz[3 * (size_t)c]);
    const float py = fma_rn(ny, df, laser_xyz[3 * (size_t)c + 1]);
    const float pz = fma_rn(nz, df, laser_xyz[3 * (size_t)c + 2]);
    const float rcp_dt = rcp_approx(dt);
    float ksum = 0.f, kcomp = 0.f;
    for (uint32_t l0 = 0; l0 < L; l0 += 64) {
        const uint32_t l1 = min(L, l0 + 64);
        float acc = 0.f;
        for (uint32_t l = l0; l < l1; ++l) {
            const float4 g = scan[l];
            const float dist0 = sqrt_approx(ref_dot3(sub_rn(px, g.x), sub_rn(py, g.y), sub_rn(pz, g.z)));
            float dist = fma_rn(dist0, 2.f, -t0);
            if (bounce) dist = add_rn(dist, g.w);
            const int b = __float2int_rz(ref_bin_ratio(dist, rcp_dt));
            if (b < 0 || b >= (int)T) continue;
            acc += to_f32(rows[(size_t)l * pitch + b]);
        }
        const float y = sub_rn(acc, kcomp);
        const float t = add_rn(ksum, y);
        kcomp = sub_rn(sub_rn(t, ksum), y);
        ksum = t;
    }
    act[i] = ksum;
}

template <typename S>
__global__ void depth_exhaustive_kernel(const S* __restrict__ rows, uint32_t pitch, const float4* __restrict__ lscan,
                                        const float4* __restrict__ sscan, const float* __restrict__ laser_xyz,
                                        const double* __restrict__ depths, uint32_t L, uint32_t Sn, uint32_t D,
                                        uint32_t T, float nx, float ny, float nz, float t0, float dt, int bounce,
                                        float* __restrict__ act) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= (uint64_t)L * D) return;
    const uint32_t c = (uint32_t)(i / D), d = (uint32_t)(i % D);
    const float df = (float)depths[d];
    // transient_reconstruction.cuh:78
    const float px = fma_rn(nx, df, laser_xyz[3 * (size_t)c]);
    const float py = fma_rn(ny, df, laser_xyz[3 * (size_t)c + 1]);
    const float pz = fma_rn(nz, df, laser_xyz[3 * (size_t)c + 2]);
    const float rcp_dt = rcp_approx(dt);
    float ksum = 0.f, kcomp = 0.f;
    for (uint32_t l = 0; l < L; ++l) {
        const float4 lg = lscan[l];
        const float dl = sqrt_approx(ref_dot3(sub_rn(px, lg.x), sub_rn(py, lg.y), sub_rn(pz, lg.z)));
        for (uint32_t s0 = 0; s0 < Sn; s0 += 64) {
            const uint32_t s1 = min(Sn, s0 + 64);
            float acc = 0.f;
            for (uint32_t s = s0; s < s1; ++s) {
                const float4 sg = sscan[s];
                const float ds = sqrt_approx(ref_dot3(sub_rn(sg.x, px), sub_rn(sg.y, py), sub_rn(sg.z, pz)));
                // transient_reconstruction.cuh:80-82
                float dist = sub_rn(add_rn(dl, ds), t0);
                if (bounce) dist = add_rn(dist, add_rn(lg.w, sg.w));
                const int b = __float2int_rz(ref_bin_ratio(dist, rcp_dt));
                if (b < 0 || b >= (int)T) continue;
                acc += to_f32(rows[((size_t)l * Sn + s) * pitch + b]);
            }
            const float y = sub_rn(acc, kcomp);
            const float t = add_rn(ksum, y);
            kcomp = sub_rn(sub_rn(t, ksum), y);
            ksum = t;
        }
    }
    act[i] = ksum;
}

// Thresholded copy into [R][pitch] rows (time innermost).  Confocal
// time-major cubes are transposed.
template <typename S>
__global__ void depth_rows_kernel(S* __restrict__ rows, const S* __restrict__ cube, uint64_t R, uint32_t T,
                                  uint32_t pitch, int time_major) {
    const uint64_t n = R * pitch;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / pitch;
        const uint32_t t = (uint32_t)(i % pitch);
        S v = from_f32<S>(0.f);
        if (t < T) {
            const S c = time_major ? cube[(uint64_t)t * R + r] : cube[r * T + t];
            if (to_f32(c) > FBP_EPS) v = c;
        }
        rows[i] = v;
    }
}

// Whether the tiles beat the row kernel for D planes.  Tiles always work on 16
// planes and on whole 16 x 16 (or 256) scan points, so few planes of many scan
// points are cheaper by rows, one thread per test point, which take about as
// long for any number of points that fit the GPU at once.  Both in nanoseconds
// per scan point walked, from measurements on 144^2 .. 240^2 points: rows 140
// while they stay in the L2 and up to 215 from memory, for each 1536 points on
// every SM; tiles 1.1 each with windows (1.5 for a tilted normal), 1.35, 1.65 or
// 2.45 where whole rows leave room for 4, 2 or 1 scan points to a stage, as a few
// planes far apart need.  Tiles against rows: 176^2 points, 512 bins, 2 planes 3.8
// and 5.5 ms; 240^2, 512 bins, 2 planes 13.1 and 11.8 ms; 240^2, 2048 bins, 4
// planes 30.3 and 14.0 ms.
bool tiles_pay(const fbp_context* ctx, const fbp_recon_info& in, uint32_t D, size_t elem_bytes) {
    using P = DepthTileParams;
    const uint32_t L = in.num_laser_targets, T = in.num_time_bins;
    const uint32_t side = (uint32_t)std::lround(std::sqrt((double)L));
    const double tiles = (uint64_t)side * side == L ? (double)cdiv(side, 16) * cdiv(side, 16) : (double)cdiv(L, P::kThreads);
    const bool yonly = in.wall_normal[0] == 0.f && in.wall_normal[2] == 0.f;
    const bool plain = in.discard_first_last_bounces != 0 && in.time_offset == 0.f;
    const uint32_t staged = P::kWindowFloats / 2 / (T + 8);  // whole rows to a stage
    double tile = yonly ? (plain ? 1.1 : 1.2) : (plain ? 1.5 : 1.65);
    if (D > 1 && T > 600) tile = (staged >= 4 ? 1.35 : staged >= 2 ? 1.65 : 2.45) * (yonly ? 1.0 : 1.3);
    const double waves = std::ceil((double)L * D / (1536.0 * ctx->sm_count));
    const double row = std::min(140.0 + 0.55e-6 * L * T * elem_bytes, 215.0) * (waves > 1.0 ? 1.2 * waves : 1.0);
    return tiles * cdiv(D, P::kDepths) * tile * 152.0 / ctx->sm_count <= row;
}

template <typename S>
fbp_status launch_depths(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int layout,
                         const float* laser_xyz, const float* sensor_xyz, const double* depths, uint32_t D,
                         float* act, cudaStream_t stream) {
    const bool exhaustive = in.capture_system == FBP_EXHAUSTIVE;
    if (!exhaustive && in.num_time_bins <= DepthTileParams::kMaxBins && cdiv(D, DepthTileParams::kDepths) <= 65535 &&
        tiles_pay(ctx, in, D, sizeof(S)) && workspace_ready(ctx, WS_CUBE_ROWS, DepthTileParams::row_bytes(in), stream)) {
        const fbp_status st = launch_depth_tiles(ctx, in, cube, dtype_of<S>(), layout, laser_xyz, depths, D, act, stream);
        if (st != FBP_ERR_OOM) return st;
        cudaGetLastError();  // no memory for FP32 rows: the kernel below needs the capture's own bytes
        clear_error();
    }
    const uint32_t L = in.num_laser_targets, Sn = exhaustive ? in.num_sensor_targets : 1, T = in.num_time_bins;
    const uint32_t pitch = (T + 7) / 8 * 8;
    const uint64_t R = (uint64_t)L * Sn;
    void* rows = nullptr;
    FBP_TRY(workspace(ctx, WS_CUBE_ROWS, R * pitch * sizeof(S), stream, &rows));
    {
        const uint64_t n = R * pitch;
        const unsigned blocks = (unsigned)std::min<uint64_t>(cdiv(n, 256), (uint64_t)ctx->sm_count * 16);
        depth_rows_kernel<S><<<blocks, 256, 0, stream>>>(static_cast<S*>(rows), static_cast<const S*>(cube), R, T,
                                                         pitch, !exhaustive && layout == FBP_LAYOUT_TIME_MAJOR);
        FBP_CHECK_LAUNCH(ctx, "depth_rows_kernel");
    }
    const int bounce = in.discard_first_last_bounces == 0;
    const uint64_t npts = (uint64_t)L * D;
    if (!exhaustive) {
        void* sp = nullptr;
        FBP_TRY(workspace(ctx, WS_SCAN_TABLE, (size_t)L * sizeof(float4), stream, &sp));
        scan_table_kernel<<<cdiv(L, 256), 256, 0, stream>>>(static_cast<float4*>(sp), laser_xyz, L,
                                                           (int)in.discard_first_last_bounces, in.laser_position[0],
                                                           in.laser_position[1], in.laser_position[2],
                                                           in.sensor_position[0], in.sensor_position[1],
                                                           in.sensor_position[2], 1);
        FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
        depth_confocal_kernel<S><<<cdiv(npts, 128), 128, 0, stream>>>(
            static_cast<const S*>(rows), pitch, static_cast<const float4*>(sp), laser_xyz, depths, L, D, T,
            in.wall_normal[0], in.wall_normal[1], in.wall_normal[2], in.time_offset, in.time_step, bounce, act);
        FBP_CHECK_LAUNCH(ctx, "depth_confocal_kernel");
        return FBP_OK;
    }
    void* lp = nullptr;
    void* sp = nullptr;
    FBP_TRY(workspace(ctx, WS_SCAN_TABLE, (size_t)L * sizeof(float4), stream, &lp));
    FBP_TRY(workspace(ctx, WS_SENSOR_TABLE, (size_t)Sn * sizeof(float4), stream, &sp));
    scan_table_kernel<<<cdiv(L, 256), 256, 0, stream>>>(static_cast<float4*>(lp), laser_xyz, L,
                                                       (int)in.discard_first_last_bounces, in.laser_position[0],
                                                       in.laser_position[1], in.laser_position[2], 0.f, 0.f, 0.f, 0);
    FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
    scan_table_kernel<<<cdiv(Sn, 256), 256, 0, stream>>>(static_cast<float4*>(sp), sensor_xyz, Sn,
                                                        (int)in.discard_first_last_bounces, in.sensor_position[0],
                                                        in.sensor_position[1], in.sensor_position[2], 0.f, 0.f, 0.f, 0);
    FBP_CHECK_LAUNCH(ctx, "scan_table_kernel");
    depth_exhaustive_kernel<S><<<cdiv(npts, 128), 128, 0, stream>>>(
        static_cast<const S*>(rows), pitch, static_cast<const float4*>(lp), static_cast<const float4*>(sp), laser_xyz,
        depths, L, Sn, D, T, in.wall_normal[0], in.wall_normal[1], in.wall_normal[2], in.time_offset, in.time_step,
        bounce, act);
    FBP_CHECK_LAUNCH(ctx, "depth_exhaustive_kernel");
    return FBP_OK;
}

}  // namespace fbp

using namespace fbp;

extern "C" fbp_status fbp_backproject_depths(fbp_context* ctx, const fbp_recon_info* info, const void* cube, int dtype,
                                             int layout, const float* laser_xyz, const float* sensor_xyz,
                                             const double* depths, uint32_t num_depths, float* activation,
                                             void* stream) {
    return guarded("fbp_backproject_depths", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        if (!info) return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: null info");
        const bool exhaustive = info->capture_system == FBP_EXHAUSTIVE;
        if (info->capture_system != FBP_CONFOCAL && !exhaustive)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: unknown capture system");
        if (info->num_laser_targets == 0 || info->num_time_bins == 0 || (exhaustive && info->num_sensor_targets == 0))
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: empty capture");
        if (!(info->time_step > 0.f)) return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: time_step must be > 0");
        if (!cube || !laser_xyz || !depths || !activation || (exhaustive && !sensor_xyz))
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: null buffer");
        if (num_depths == 0) return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: num_depths == 0");
        if (layout != FBP_LAYOUT_TIME_MAJOR && layout != FBP_LAYOUT_TIME_INNER)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: unknown layout");
        cudaStream_t s = (cudaStream_t)stream;
        switch (dtype) {
            case FBP_F32:
                return launch_depths<float>(ctx, *info, cube, layout, laser_xyz, sensor_xyz, depths, num_depths, activation, s);
            case FBP_BF16:
                return launch_depths<__nv_bfloat16>(ctx, *info, cube, layout, laser_xyz, sensor_xyz, depths, num_depths,
                                                    activation, s);
            case FBP_F16:
                return launch_depths<__half>(ctx, *info, cube, layout, laser_xyz, sensor_xyz, depths, num_depths, activation, s);
            default: return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_depths: unknown dtype");
        }
    });
}
