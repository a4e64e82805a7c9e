// Exhaustive (laser x SPAD) backprojection as a voxel-tiled gather.
//
// Replaces Laser::reconstructAABBExhaustive (Laser.cu:500-516) and
// backprojectExhaustiveVoxel (transient_reconstruction.cuh:138-166).  Same
// structure as the confocal gather: a CTA, or several, per voxel tile, the
// (laser, SPAD) pairs walked in groups, each pair's reachable time-bin window
// copied to shared memory.  The pair index splits as l = ls / S, s = ls % S;
// the reference splits by L (transient_reconstruction.cuh:147-148), which is
// the same only when L == S and reads past the laser table otherwise.
#include "fbp_internal.cuh"
#include "bp_common.cuh"

#include <algorithm>
#include <cmath>

namespace fbp {

struct ExhaustiveGatherParams {
    const float4* lscan;  // [L] (x, y, z, |l - laserPos| or 0)
    const float4* sscan;  // [S] (x, y, z, |s - sensorPos| or 0)
    const float* xs;
    const float* ys;
    const float* zs;
    float* volume;
    int* status;
    const float* rows;  // [L*S][row_pitch] FP32 (16-bit cubes are widened, exactly, when the rows are made)
    uint32_t Vx, Vy, Vz, L, S, T;
    float t0, dt;
    uint32_t row_pitch, slot_w;
    int ch;             // pairs per window stage (a power of two up to 32; at least 4 in blocks of 4 lasers)
    uint32_t chains;    // contiguous ranges of pair groups with compensated sums of their own, one CTA each
    float* chain_sums;  // chains > 1: [chains][sum, compensation][volume]
    int exact_weights;  // 1: every weight by its own rcp.approx (FBP_WEIGHTS_REFERENCE)

    // Shared memory in front of the windows: the pipeline's barriers, then per
    // pair of kPlanBufs groups: SPAD (x, y, z) and laser index, (bias, bias, slot address,
    // bounces), the SPAD's x differences to the tile's kv columns, the window's
    // source and length; two words per group.
    static constexpr int kGroup = 32;
    static constexpr int kWindowBufs = 3;  // two (5 % slower) where a window leaves no room for three
    static constexpr int kPlanBufs = 8;
    __host__ __device__ static constexpr size_t meta_bytes(int kv) {
        return 128 +
               (size_t)kPlanBufs * kGroup * (sizeof(float4) + sizeof(int4) + kv * sizeof(float) + sizeof(void*) +
                                             sizeof(int)) +
               (size_t)kPlanBufs * sizeof(int2);
    }
};

// Arithmetic of the triple loop (all reproduce the reference's bins):
//   EX_T0ZERO  time_offset == 0: dist = dl + ds [+ bounces]; the reference's
//              "- t0" subtracts zero, which changes no bit, so it is skipped.
//   EX_FAST    time_offset < 0: dist = (dl + ds) - t0 [+ bounces].
//   EX_EXACT   time_offset > 0: negative paths possible.  Groups with a path
//              near or below zero bin by conversion, like the reference's
//              static_cast; the others run EX_FAST's arithmetic.
// CLAMP: windows that are the whole row, whose bins are clamped to the slot;
// otherwise the planner guarantees that every bin lies inside its window.
enum { EX_T0ZERO = 0, EX_FAST = 1, EX_EXACT = 2 };

// One CTA of 32*WY*WZ threads (or p.chains of them, one per range of pair
// groups, their sums folded afterwards) owns a tile of KV x 8*WY x 4*WZ
// voxels, like the confocal gather, with its pipeline: plans two groups ahead,
// windows by bulk copies, no barrier across the CTA.
// LB = 4: pairs are walked as (laser block of 4, SPAD, laser in block), so
// the SPAD-to-voxel distance is computed once per SPAD for 4 lasers (the 4
// laser distances are kept per block); a last block short of lasers reads
// zeros.  LB = 1: pairs in (laser, SPAD) order.
// Bound by the issue port, which a packed FP32 instruction holds for two
// cycles: 16.2 instructions and 7.3 second cycles of the 25.5 cycles a packed
// pair of triples takes (8^2 x 32^2 x 1024 -> 128^3: 43.4 ms).  Reciprocals of
// their own for half or all of the weights (fewer products, more MUFU work)
// take the same time; blocks of 1, 2 and 8 lasers 78, 58 and 46 ms.
template <int KV, int WY, int WZ, int MODE, bool BOUNCE, bool CLAMP, int LB, uint32_t NB = ExhaustiveGatherParams::kWindowBufs>
__global__ void __launch_bounds__(32 * WY * WZ, 2)
exhaustive_gather_kernel(ExhaustiveGatherParams p) {
    static_assert(KV % 8 == 0, "voxels per thread in packed pairs, four to a weight group");
    using P = ExhaustiveGatherParams;
    constexpr int NT = 32 * WY * WZ, NW = WY * WZ, ALIGN = 4;
    constexpr uint32_t GRP = P::kGroup, MB = P::kPlanBufs;
    static_assert(NB <= P::kWindowBufs, "the barriers fit in front of the plans");
    constexpr int TY = 8 * WY, TZ = 4 * WZ;
    const uint32_t CH = p.ch;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t slot_stride = p.slot_w + ALIGN;  // sentinel elements at slot_w
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t bar_full = sbase, bar_empty = sbase + 8 * NB, bar_plan = sbase + 16 * NB;  // NB, NB and MB of 8 bytes
    float4* s_geo = reinterpret_cast<float4*>(smem_raw + 128);                          // [MB][GRP]
    int4* s_meta = reinterpret_cast<int4*>(s_geo + MB * GRP);                          // [MB][GRP]
    ulonglong2* s_dx = reinterpret_cast<ulonglong2*>(s_meta + MB * GRP);               // [MB][GRP][KV / 4]
    const float** s_src = reinterpret_cast<const float**>(s_dx + MB * GRP * (KV / 4));  // [MB][GRP]
    int* s_cnt = reinterpret_cast<int*>(s_src + MB * GRP);                             // [MB][GRP]
    int2* s_group = reinterpret_cast<int2*>(s_cnt + MB * GRP);                         // [MB] (pairs, guarded)
    constexpr size_t slots_off = P::meta_bytes(KV);
    float* s_slots = reinterpret_cast<float*>(smem_raw + slots_off);                   // [NB][CH][slot_stride]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wy = warp % WY, wz = warp / WY;
    const uint32_t rank = blockIdx.x % p.chains;
    const uint32_t tx0 = blockIdx.x / p.chains * KV, ty0 = blockIdx.y * TY, tz0 = blockIdx.z * TZ;
    const uint32_t vy = ty0 + wy * 8 + (lane & 7);
    const uint32_t vz = tz0 + wz * 4 + (lane >> 3);
    const bool row_ok = vy < p.Vy && vz < p.Vz;
    const bool warp_ok = __any_sync(0xffffffffu, row_ok);

    const uint32_t tx1 = min(tx0 + KV, p.Vx) - 1, ty1 = min(ty0 + TY, p.Vy) - 1, tz1 = min(tz0 + TZ, p.Vz) - 1;
    const float bx0 = fminf(p.xs[tx0], p.xs[tx1]), bx1 = fmaxf(p.xs[tx0], p.xs[tx1]);
    const float by0 = fminf(p.ys[tz0], p.ys[tz1]), by1 = fmaxf(p.ys[tz0], p.ys[tz1]);
    const float bz0 = fminf(p.zs[ty0], p.zs[ty1]), bz1 = fmaxf(p.zs[ty0], p.zs[ty1]);
    const float py = p.ys[min(vz, p.Vz - 1)];
    const float pz = p.zs[min(vy, p.Vy - 1)];
    const float rcp_dt = rcp_approx(p.dt);

    // Items: pairs in walking order (LB = 4: lasers padded to whole blocks).
    const uint64_t nitems = (uint64_t)((p.L + LB - 1) / LB * LB) * p.S;
    const uint64_t ngroups = (nitems + GRP - 1) / GRP;
    const uint64_t g0 = rank * ngroups / p.chains;
    const uint32_t mine = (uint32_t)((rank + 1) * ngroups / p.chains - g0);
    const uint32_t sub = GRP / CH;
    const uint64_t nstages = (uint64_t)mine * sub;

    if (tid == 0) {
        for (uint32_t b = 0; b < NB; ++b) {
            mbar_init(bar_full + 8 * b, 1);
            mbar_init(bar_empty + 8 * b, NW);
        }
        for (uint32_t b = 0; b < MB; ++b) mbar_init(bar_plan + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t i = tid; i < NB * CH * ALIGN; i += NT)  // sentinel of every slot
        s_slots[(size_t)(i / ALIGN) * slot_stride + p.slot_w + i % ALIGN] = 0.f;

    auto box_range = [&](const float4& g, float& dmin, float& dmax) {
        const float cx = fminf(fmaxf(g.x, bx0), bx1), cy = fminf(fmaxf(g.y, by0), by1), cz = fminf(fmaxf(g.z, bz0), bz1);
        dmin = sqrtf((g.x - cx) * (g.x - cx) + (g.y - cy) * (g.y - cy) + (g.z - cz) * (g.z - cz));
        const float fx = fmaxf(fabsf(g.x - bx0), fabsf(g.x - bx1)), fy = fmaxf(fabsf(g.y - by0), fabsf(g.y - by1)),
                    fz = fmaxf(fabsf(g.z - bz0), fabsf(g.z - bz1));
        dmax = sqrtf(fx * fx + fy * fy + fz * fz);
    };

    // Plan this CTA's group gi (one warp): bin window of each pair.  Its buffer
    // held group gi - MB, which every warp is past (see the confocal gather).
    auto plan_group = [&](uint32_t gi) {
        const uint32_t gb = (gi % MB) * GRP;
        const uint64_t item = (g0 + gi) * GRP + lane;
        float4 sg = make_float4(0.f, 0.f, 0.f, 0.f);
        float bnc = 0.f;
        uint32_t laser = 0;
        int cnt = 0, near = 0, a = 0;
        bool read = false;  // the window holds samples of the row
        uint64_t src = p.row_pitch - p.slot_w;  // else: the zeros after the row
        if (item < nitems) {
            const uint64_t spads = item / LB, block = spads / p.S;  // (LB = 4: past L - 1 in a short last block)
            const uint32_t lp = (uint32_t)block * LB + (uint32_t)(item % LB), l = min(lp, p.L - 1);
            const uint32_t s = (uint32_t)(spads - block * p.S);
            const float4 lg = p.lscan[l];
            sg = p.sscan[s];
            laser = lp;
            float dl0, dl1, ds0, ds1;
            box_range(lg, dl0, dl1);
            box_range(sg, ds0, ds1);
            bnc = BOUNCE ? add_rn(lg.w, sg.w) : 0.f;  // transient_reconstruction.cuh:161
            const float pmin = dl0 + ds0 - p.t0 + bnc, pmax = dl1 + ds1 - p.t0 + bnc;
            const int blo = (int)fmaxf(fminf(floorf(pmin * rcp_dt), 1.0e9f), -1.0e9f) - 2;
            const int bhi = (int)fmaxf(fminf(floorf(pmax * rcp_dt), 1.0e9f), -1.0e9f) + 2;
            // Paths this short make dist^2 <= EPS possible, paths this long
            // (or NaN) could take the shared reciprocal's product out of the
            // FP32 range, bins this high lie past any row: those groups weigh
            // each triple on its own and clamp each bin.
            near = pmin < 0.0035f || !(pmax < 1.0e4f) || bhi >= (1 << 22);
            a = max(blo, 0) & ~(ALIGN - 1);
            read = bhi >= 0 && blo < (int)p.T && lp < p.L;
            if (read) {
                if (CLAMP) a = min(a, (int)(p.row_pitch - p.slot_w));
                src = a;
            }
            cnt = (max(min(bhi + 1, read ? (int)p.row_pitch : bhi + 1) - a, 0) + ALIGN - 1) & ~(ALIGN - 1);
            if (cnt > (int)p.slot_w) {
                // CLAMP: bins past a capped window map to the sentinel; only an
                // uncovered valid bin would be an error.  Otherwise the planner's
                // span bound failed: read zeros, report.
                if (read && (!CLAMP || min(bhi + 1, (int)p.T) - a > (int)p.slot_w)) {
                    atomicExch(p.status, (int)FBP_ERR_DEVICE);
                    if (!CLAMP) read = false;
                }
                if (!CLAMP) near = 1;
                cnt = (int)p.slot_w;
            }
            src += (uint64_t)((size_t)l * p.S + s) * p.row_pitch;
        }
        const bool guarded = __any_sync(0xffffffffu, near) || p.exact_weights;
        const uint32_t st = gi * sub + lane / CH;
        const uint32_t slot_elem = ((st % NB) * CH + lane % CH) * slot_stride;
        uint32_t slot = sbase + (uint32_t)slots_off + (slot_elem << 2);
        int bias;
        if (MODE == EX_EXACT && guarded) {
            bias = read ? a : 0x40000000;  // (b - bias) past the slot: the sentinel
        } else if (CLAMP || guarded) {
            bias = __float_as_int((float)(8388608 - (read ? a : -(int)p.slot_w)));
        } else {
            bias = __float_as_int((float)(8388608 - a));
            slot -= kBiasBits;
            read = true;  // zeros are copied too
        }
        s_geo[gb + lane] = make_float4(sg.x, sg.y, sg.z, __uint_as_float(laser));
        s_meta[gb + lane] = make_int4(bias, bias, (int)slot, __float_as_int(bnc));
        if (LB == 1 || lane % LB == 0) {
            float* dx = reinterpret_cast<float*>(s_dx + (gb + lane) * (KV / 4));
#pragma unroll
            for (int k = 0; k < KV; ++k) dx[k] = sub_rn(p.xs[min(tx0 + k, p.Vx - 1)], sg.x);
        }
        s_cnt[gb + lane] = read && item < nitems ? cnt : 0;
        s_src[gb + lane] = p.rows + src;
        if (lane == 0) s_group[gi % MB] = make_int2((int)min((uint64_t)GRP, nitems - (g0 + gi) * GRP), guarded);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_plan + 8 * (gi % MB));
    };

    // A wait that ran out of polls (status FBP_ERR_TIMEOUT): the warp walks on
    // but touches nothing else.
    bool dead = false;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (!dead && !mbar_wait_parity(bar, parity)) {
            dead = true;
            if (lane == 0) atomicExch(p.status, (int)FBP_ERR_TIMEOUT);
        }
    };

    // Fill stage st (one warp): one bulk copy per window.
    auto produce = [&](uint64_t st) {
        const uint32_t buf = st % NB, gi = (uint32_t)(st / sub), first = (uint32_t)(st % sub) * CH;
        wait(bar_plan + 8 * (gi % MB), (gi / MB) & 1);
        if (st >= NB) wait(bar_empty + 8 * buf, (uint32_t)(st / NB - 1) & 1);
        if (dead) return;
        const uint32_t gb = (gi % MB) * GRP;
        const uint32_t bytes = lane - first < CH ? (uint32_t)s_cnt[gb + lane] * 4u : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
        if (lane == 0) mbar_arrive_expect_tx(bar_full + 8 * buf, total);
        __syncwarp();
        if (bytes)
            bulk_load(sbase + (uint32_t)slots_off + (((buf * CH + lane - first) * slot_stride) << 2), s_src[gb + lane],
                      bytes, bar_full + 8 * buf);
    };

    f32x2_t accp[KV / 2], dlp[LB][KV / 2];
    float ksum[KV], kcomp[KV];
#pragma unroll
    for (int j = 0; j < KV / 2; ++j) accp[j] = 0ull;
#pragma unroll
    for (int k = 0; k < KV; ++k) ksum[k] = kcomp[k] = 0.f;
#pragma unroll
    for (int li = 0; li < LB; ++li)
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) dlp[li][j] = 0ull;
    uint32_t cur_l = 0xFFFFFFFFu;
    const f32x2_t rdp = pack2(rcp_dt, rcp_dt), t0p = pack2(p.t0, p.t0);

    // Distances of a point with the given x differences.
    auto point_dist = [&](float gy, float gz, auto&& dx, f32x2_t (&d)[KV / 2]) {
        const float ddy = sub_rn(py, gy), ddz = sub_rn(pz, gz);
        const float ddy2 = mul_rn(ddy, ddy);
        const f32x2_t ddzp = pack2(ddz, ddz), ddy2p = pack2(ddy2, ddy2);
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) {
            const f32x2_t x = dx(j);
            float q0, q1;
            unpack2(fma_rn2(ddzp, ddzp, fma_rn2(x, x, ddy2p)), q0, q1);
            d[j] = pack2(sqrt_approx(q0), sqrt_approx(q1));
        }
    };
    auto laser_dist = [&](uint32_t l, f32x2_t (&d)[KV / 2]) {
        const float4 g = p.lscan[min(l, p.L - 1)];
        point_dist(g.y, g.z, [&](int j) {
            return pack2(sub_rn(p.xs[min(tx0 + 2 * j, p.Vx - 1)], g.x), sub_rn(p.xs[min(tx0 + 2 * j + 1, p.Vx - 1)], g.x));
        }, d);
    };
    auto spad_dist = [&](uint32_t o, f32x2_t (&d)[KV / 2]) {
        const float4 g = s_geo[o];
        f32x2_t dx[KV / 2];
#pragma unroll
        for (int j = 0; j < KV / 4; ++j) {
            const ulonglong2 v = s_dx[o * (KV / 4) + j];
            dx[2 * j] = v.x;
            dx[2 * j + 1] = v.y;
        }
        point_dist(g.y, g.z, [&](int j) { return dx[j]; }, d);
    };

    // Triples of pair o with the laser distances dl and the SPAD distances ds
    // (transient_reconstruction.cuh:155-162).
    auto pair_terms = [&](uint32_t o, const f32x2_t (&dl)[KV / 2], const f32x2_t (&ds)[KV / 2]) {
        const int4 m = s_meta[o];
        const f32x2_t biasp = pack2(__int_as_float(m.x), __int_as_float(m.y));
        const f32x2_t bncp = pack2(__int_as_float(m.w), __int_as_float(m.w));
#pragma unroll
        for (int j0 = 0; j0 < KV / 2; j0 += 2) {
            f32x2_t sq[2], Iq[2];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
                f32x2_t dist = add_rn2(dl[j0 + jj], ds[j0 + jj]);
                if (MODE != EX_T0ZERO) dist = sub_rn2(dist, t0p);
                if (BOUNCE) dist = add_rn2(dist, bncp);
                float b0, b1;
                unpack2(add_rz2(mul_rn2(dist, rdp), biasp), b0, b1);
                Iq[jj] = pack2(read_bin<CLAMP>(b0, m.z, p.slot_w), read_bin<CLAMP>(b1, m.z, p.slot_w));
                sq[jj] = mul_rn2(dist, dist);
            }
            float m0, m1;
            // Weights of two pairs from one reciprocal per lane: 1 / s0 = s1 / (s0 s1).
            unpack2(mul_rn2(sq[0], sq[1]), m0, m1);
            const f32x2_t r = pack2(rcp_approx(m0), rcp_approx(m1));
            accp[j0] = fmaf2(Iq[0], mul_rn2(r, sq[1]), accp[j0]);
            accp[j0 + 1] = fmaf2(Iq[1], mul_rn2(r, sq[0]), accp[j0 + 1]);
        }
    };
    // The same, guarded: the reference's own weight per triple, clamped bins
    // (by conversion where negative paths are possible).
    auto pair_terms_guarded = [&](uint32_t o, const f32x2_t (&dl)[KV / 2], const f32x2_t (&ds)[KV / 2]) {
        const int4 m = s_meta[o];
        const float bias = __int_as_float(m.x), bnc = __int_as_float(m.w);
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) {
            float dl2[2], ds2[2], ac[2];
            unpack2(dl[j], dl2[0], dl2[1]);
            unpack2(ds[j], ds2[0], ds2[1]);
            unpack2(accp[j], ac[0], ac[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float dist = sub_rn(add_rn(dl2[h], ds2[h]), p.t0);
                if (BOUNCE) dist = add_rn(dist, bnc);
                const float x = ref_bin_ratio(dist, rcp_dt);
                const uint32_t rel = MODE == EX_EXACT ? (uint32_t)(__float2int_rz(x) - m.x)
                                                      : __float_as_uint(add_rz(x, bias)) - 0x4B000000u;
                const float I = lds_f32((uint32_t)m.z + (min(rel, p.slot_w) << 2));
                ac[h] = fmaf(I, ref_safe_rcp(mul_rn(dist, dist)), ac[h]);
            }
            accp[j] = pack2(ac[0], ac[1]);
        }
    };

    // A previous kernel's writes to this memory before the bulk copies' writes.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // barriers initialised, sentinels written
    if (warp < 2 && (uint32_t)warp < mine) plan_group(warp);
    if (warp == 0 && nstages > 0) produce(0);
    for (uint32_t gi = 0; gi < mine; ++gi) {
        const uint32_t gb = (gi % MB) * GRP;
        for (uint32_t h = 0; h < sub; ++h) {
            const uint64_t st = (uint64_t)gi * sub + h;
            const uint32_t buf = st % NB;
            wait(bar_full + 8 * buf, (uint32_t)(st / NB) & 1);
            if (st + 1 < nstages && warp == (int)((st + 1) % NW)) produce(st + 1);
            if (h == 0 && gi + 2 < mine && !dead && warp == (int)((st + NW / 2) % NW)) plan_group(gi + 2);
            const int2 grp = s_group[gi % MB];
            const uint32_t i1 = min((h + 1) * CH, (uint32_t)grp.x);
            if (warp_ok && !dead) {
                auto walk = [&](auto&& terms) {
                    for (uint32_t i = h * CH; i < i1; i += LB) {
                        const uint32_t l = __float_as_uint(s_geo[gb + i].w);
                        if (l != cur_l) {  // a new laser, or block of LB of them (uniform across the CTA)
                            cur_l = l;
#pragma unroll
                            for (int li = 0; li < LB; ++li) laser_dist(l + li, dlp[li]);
                        }
                        f32x2_t ds[KV / 2];
                        spad_dist(gb + i, ds);
#pragma unroll
                        for (int li = 0; li < LB; ++li) terms(gb + i + li, dlp[li], ds);
                    }
                };
                if (!grp.y) walk(pair_terms);
                else walk(pair_terms_guarded);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * buf);
        }
#pragma unroll
        for (int j = 0; j < KV / 2; ++j) {
            float a0, a1;
            unpack2(accp[j], a0, a1);
            kahan_add(a0, ksum[2 * j], kcomp[2 * j]);
            kahan_add(a1, ksum[2 * j + 1], kcomp[2 * j + 1]);
            accp[j] = 0ull;
        }
    }

    if (!row_ok) return;
    const size_t at = ((size_t)vz * p.Vy + vy) * p.Vx + tx0, n = (size_t)p.Vx * p.Vy * p.Vz;
    float* out = p.chains == 1 ? p.volume + at : p.chain_sums + (size_t)rank * 2 * n + at;
#pragma unroll
    for (int k = 0; k < KV; ++k)
        if (tx0 + k < p.Vx) {
            out[k] = ksum[k];
            if (p.chains > 1) out[n + k] = kcomp[k];
        }
}

namespace {

constexpr int kKV = 8, kWY = 2, kWZ = 4;
constexpr int kExhaustiveCtasPerSm = 2;  // 256 threads of up to 128 registers

template <int MODE, bool BOUNCE, bool CLAMP, int LB, uint32_t NB = ExhaustiveGatherParams::kWindowBufs>
fbp_status go_exhaustive(fbp_context* ctx, ExhaustiveGatherParams p, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kernel = exhaustive_gather_kernel<kKV, kWY, kWZ, MODE, BOUNCE, CLAMP, LB, NB>;
    FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t n = (uint64_t)p.Vx * p.Vy * p.Vz;
    grid.x *= p.chains;
    kernel<<<grid, 32 * kWY * kWZ, smem, stream>>>(p);
    FBP_CHECK_LAUNCH(ctx, "exhaustive_gather_kernel");
    return p.chains > 1 ? fold_chains(ctx, p.chain_sums, p.chains, n, p.volume, stream) : FBP_OK;
}

template <int MODE, int LB>
fbp_status go_exhaustive(fbp_context* ctx, const ExhaustiveGatherParams& p, dim3 grid, size_t smem, cudaStream_t s,
                         bool bounce, bool capped) {
    if (bounce) {
        if (capped) return go_exhaustive<MODE, true, true, LB>(ctx, p, grid, smem, s);
        return go_exhaustive<MODE, true, false, LB>(ctx, p, grid, smem, s);
    }
    if (capped) return go_exhaustive<MODE, false, true, LB>(ctx, p, grid, smem, s);
    return go_exhaustive<MODE, false, false, LB>(ctx, p, grid, smem, s);
}

template <int LB>
fbp_status dispatch_exhaustive(fbp_context* ctx, const ExhaustiveGatherParams& p, dim3 grid, size_t smem,
                               cudaStream_t s, bool bounce, float t0, bool capped) {
    if (t0 > 0.f) return go_exhaustive<EX_EXACT, LB>(ctx, p, grid, smem, s, bounce, capped);
    if (t0 == 0.f) return go_exhaustive<EX_T0ZERO, LB>(ctx, p, grid, smem, s, bounce, capped);
    return go_exhaustive<EX_FAST, LB>(ctx, p, grid, smem, s, bounce, capped);
}

// Windows with room for two only (one pair to a stage).  EX_EXACT's results are
// those of the other two where no path is negative.
fbp_status dispatch_widest(fbp_context* ctx, const ExhaustiveGatherParams& p, dim3 grid, size_t smem, cudaStream_t s,
                           bool bounce, bool capped) {
    if (bounce) {
        if (capped) return go_exhaustive<EX_EXACT, true, true, 1, 2>(ctx, p, grid, smem, s);
        return go_exhaustive<EX_EXACT, true, false, 1, 2>(ctx, p, grid, smem, s);
    }
    if (capped) return go_exhaustive<EX_EXACT, false, true, 1, 2>(ctx, p, grid, smem, s);
    return go_exhaustive<EX_EXACT, false, false, 1, 2>(ctx, p, grid, smem, s);
}

fbp_status launch_exhaustive(fbp_context* ctx, const fbp_recon_info& in, const void* cube, int dtype, const float* laser_xyz,
                             const float* sensor_xyz, float* volume, cudaStream_t stream) {
    const uint32_t L = in.num_laser_targets, Sn = in.num_sensor_targets, T = in.num_time_bins;
    const uint32_t Vx = in.voxel_res[0], Vy = in.voxel_res[1], Vz = in.voxel_res[2];
    constexpr int ALIGN = 4;  // FP32 rows
    const double ex = (double)std::min<uint32_t>(kKV, Vx) * std::fabs(in.voxel_size[0]);
    const double ey = (double)std::min<uint32_t>(4 * kWZ, Vz) * std::fabs(in.voxel_size[1]);
    const double ez = (double)std::min<uint32_t>(8 * kWY, Vy) * std::fabs(in.voxel_size[2]);
    WindowPlan wp;
    auto plan = [&](int bufs) {
        return plan_window(ctx, ex, ey, ez, in.time_step, T, ALIGN, sizeof(float), ExhaustiveGatherParams::meta_bytes(kKV),
                           &wp, "fbp_backproject_exhaustive", 0.0, kExhaustiveCtasPerSm, bufs);
    };
    // Three windows to a CTA up to some 17,700 bins, two up to 26,600.
    const bool widest = plan(ExhaustiveGatherParams::kWindowBufs) == FBP_ERR_UNSUPPORTED;
    if (widest) {
        clear_error();
        FBP_TRY(plan(2));
    }
    const uint32_t slot_w = wp.slot_w, pitch = wp.pitch;
    const uint64_t npairs = (uint64_t)L * Sn;

    // Laser blocks of 4 where padding the lasers to whole blocks costs no more
    // than a SPAD distance per pair would (about 8 of 21 issue cycles).
    const bool blocks = !widest && wp.ch % 4 == 0 && (L + 3) / 4 * 4 * 3 <= L * 4;
    const uint64_t groups = ((uint64_t)(blocks ? (L + 3) / 4 * 4 : L) * Sn + ExhaustiveGatherParams::kGroup - 1) /
                            ExhaustiveGatherParams::kGroup;
    ExhaustiveGatherParams p{};
    p.chains = split_chains(ctx, (uint64_t)cdiv(Vx, kKV) * cdiv(Vy, 8 * kWY) * cdiv(Vz, 4 * kWZ),
                            busy_warps(in.voxel_res), groups,
                            resident_ctas(wp.smem, kExhaustiveCtasPerSm), 3.2, (uint64_t)Vx * Vy * Vz);
    float* rows = nullptr;
    FBP_TRY(gather_scratch(ctx, npairs * pitch * sizeof(float), &p.chains, (uint64_t)Vx * Vy * Vz, stream, &rows,
                           &p.chain_sums));
    PrepTables tables{};
    FBP_TRY(table_buffers(ctx, in, laser_xyz, sensor_xyz, true, stream, &tables));
    FBP_TRY(prepare_gather(ctx, dtype, PrepRows{cube, rows, npairs, T, pitch, 0}, tables, stream));

    p.lscan = tables.lasers;
    p.sscan = tables.sensors;
    p.xs = tables.axes;
    p.ys = p.xs + Vx;
    p.zs = p.ys + Vz;
    p.volume = volume;
    p.status = ctx->status_dev;
    p.rows = rows;
    p.Vx = Vx; p.Vy = Vy; p.Vz = Vz; p.L = L; p.S = Sn; p.T = T;
    p.t0 = in.time_offset;
    p.dt = in.time_step;
    p.row_pitch = pitch;
    p.slot_w = slot_w;
    p.ch = wp.ch;
    p.exact_weights = ctx->weight_mode == FBP_WEIGHTS_REFERENCE;
    dim3 grid(cdiv(Vx, kKV), cdiv(Vy, 8 * kWY), cdiv(Vz, 4 * kWZ));
    const bool bounce = in.discard_first_last_bounces == 0;
    if (widest) return dispatch_widest(ctx, p, grid, wp.smem, stream, bounce, wp.capped);
    if (blocks) return dispatch_exhaustive<4>(ctx, p, grid, wp.smem, stream, bounce, in.time_offset, wp.capped);
    return dispatch_exhaustive<1>(ctx, p, grid, wp.smem, stream, bounce, in.time_offset, wp.capped);
}

}  // namespace
}  // namespace fbp

using namespace fbp;

extern "C" fbp_status fbp_backproject_exhaustive(fbp_context* ctx, const fbp_recon_info* info, const void* cube,
                                                 int dtype, const float* laser_xyz, const float* sensor_xyz,
                                                 float* volume, void* stream) {
    return guarded("fbp_backproject_exhaustive", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        FBP_TRY(validate_info(info, true, "fbp_backproject_exhaustive"));
        if (!cube || !laser_xyz || !sensor_xyz || !volume)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_exhaustive: null buffer");
        cudaStream_t s = (cudaStream_t)stream;
        if (dtype != FBP_F32 && dtype != FBP_BF16 && dtype != FBP_F16)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_backproject_exhaustive: unknown dtype");
        return launch_exhaustive(ctx, *info, cube, dtype, laser_xyz, sensor_xyz, volume, s);
    });
}
