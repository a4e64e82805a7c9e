// Post-processing of the reconstructed volume: min-max normalisation and the
// LoG / Laplacian 3-D filters.
//
// Replaces Laser::normalizeMatrix (Laser.cu:317-339: two CUB reductions and
// normalizeReconstruction, transient_postprocessing.cuh:10-17) and
// PostprocessingFilters::compute (PostprocessingFilters.h:5-39,
// PostprocessingFilters.cu:12-98).  The convolutions keep the reference's tap
// order and FMA sequence, so FP32 outputs can match the reference kernels bit
// for bit; neighbourhoods come from a shared-memory tile instead of 125 (or
// k^3) global loads per voxel.
#include "fbp_internal.cuh"

#include <cmath>
#include <cstring>
#include <vector>

namespace fbp {

// ------------------------------------------------------- min-max reduction --

constexpr int kReduceThreads = 512;

__device__ __forceinline__ void block_minmax(float& mn, float& mx) {
    __shared__ float smn[32], smx[32];
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { smn[w] = mn; smx[w] = mx; }
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    if (w == 0) {
        mn = l < nw ? smn[l] : INFINITY;
        mx = l < nw ? smx[l] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
    }
}

// Pass 1: per-block min/max into partials[2*b], partials[2*b+1].
__global__ void minmax_partial_kernel(const float* __restrict__ v, uint64_t n, float* __restrict__ partials) {
    float mn = INFINITY, mx = -INFINITY;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    // Vectorised body when the pointer is 16-byte aligned.
    if ((reinterpret_cast<uintptr_t>(v) & 15) == 0) {
        const float4* v4 = reinterpret_cast<const float4*>(v);
        const uint64_t n4 = n / 4;
        for (uint64_t j = i; j < n4; j += stride) {
            const float4 a = v4[j];
            mn = fminf(mn, fminf(fminf(a.x, a.y), fminf(a.z, a.w)));
            mx = fmaxf(mx, fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)));
        }
        for (uint64_t j = n4 * 4 + i; j < n; j += stride) {
            mn = fminf(mn, v[j]);
            mx = fmaxf(mx, v[j]);
        }
    } else {
        for (uint64_t j = i; j < n; j += stride) {
            mn = fminf(mn, v[j]);
            mx = fmaxf(mx, v[j]);
        }
    }
    block_minmax(mn, mx);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = mn;
        partials[2 * blockIdx.x + 1] = mx;
    }
}

// Pass 2: normalizeReconstruction, v = (v - min) * safeRCP(max - min), every
// block folding the partials by itself (a launch less than a fold of its own).
__global__ void normalize_apply_kernel(float* __restrict__ v, uint64_t n, const float* __restrict__ partials, int nparts) {
    __shared__ float s_mm[2];
    {
        float mn = INFINITY, mx = -INFINITY;
        for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
            const float2 p = reinterpret_cast<const float2*>(partials)[i];
            mn = fminf(mn, p.x);
            mx = fmaxf(mx, p.y);
        }
        block_minmax(mn, mx);
        if (threadIdx.x == 0) {
            s_mm[0] = mn;
            s_mm[1] = mx;
        }
        __syncthreads();
    }
    const float mn = s_mm[0];
    const float r = ref_safe_rcp(sub_rn(s_mm[1], mn));
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint64_t tail = 0;
    if ((reinterpret_cast<uintptr_t>(v) & 15) == 0) {
        float4* v4 = reinterpret_cast<float4*>(v);
        const uint64_t n4 = n / 4;
        for (uint64_t j = i; j < n4; j += stride) {
            float4 a = v4[j];
            a.x = mul_rn(sub_rn(a.x, mn), r);
            a.y = mul_rn(sub_rn(a.y, mn), r);
            a.z = mul_rn(sub_rn(a.z, mn), r);
            a.w = mul_rn(sub_rn(a.w, mn), r);
            v4[j] = a;
        }
        tail = n4 * 4;
    }
    for (uint64_t j = tail + i; j < n; j += stride) v[j] = mul_rn(sub_rn(v[j], mn), r);
}

int minmax_blocks(const fbp_context* ctx, uint64_t n) {
    const uint64_t want = (n + 4ull * kReduceThreads - 1) / (4ull * kReduceThreads);
    const uint64_t cap = (uint64_t)ctx->sm_count * 4;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(want, cap));
}

fbp_status normalize_device(fbp_context* ctx, float* v, uint64_t n, cudaStream_t stream) {
    const int nb = minmax_blocks(ctx, n);
    void* ws = nullptr;
    FBP_TRY(workspace(ctx, WS_PARTIALS, (size_t)2 * nb * sizeof(float), stream, &ws));
    float* partials = static_cast<float*>(ws);
    minmax_partial_kernel<<<nb, kReduceThreads, 0, stream>>>(v, n, partials);
    FBP_CHECK_LAUNCH(ctx, "minmax_partial_kernel");
    const unsigned ab = (unsigned)std::min<uint64_t>(cdiv(n, 4 * 256), (uint64_t)ctx->sm_count * 8);
    normalize_apply_kernel<<<ab, 256, 0, stream>>>(v, n, partials, nb);
    FBP_CHECK_LAUNCH(ctx, "normalize_apply_kernel");
    return FBP_OK;
}

// ------------------------------------------------------------- LoG filter --

constexpr int kLogMaxK = 15;

// LoG taps passed by value (kernel parameters, so concurrent calls with
// different kernels do not share state): ksize^3 weights, ksize = 2H+1 or 2H+2.
template <int H>
struct LogTaps {
    float w[(2 * H + 2) * (2 * H + 2) * (2 * H + 2)];
};

// Output tile 8x8x8 per CTA, halo tile (8 + 2h)^3 in shared memory.
// Taps in the reference's order (kz, ky, kx innermost), sum = fma(v, w, sum)
// (LoGFilter, transient_postprocessing.cuh:52-83).
template <int H>
__global__ void __launch_bounds__(512) log_filter_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                         uint32_t nx, uint32_t ny, uint32_t nz, int ksize,
                                                         const __grid_constant__ LogTaps<H> taps) {
    constexpr int E = 8 + 2 * H;
    extern __shared__ float tile[];  // [E][E][E]
    const int x0 = blockIdx.x * 8, y0 = blockIdx.y * 8, z0 = blockIdx.z * 8;
    const int tid = threadIdx.x + 8 * (threadIdx.y + 8 * threadIdx.z);
    constexpr int NE = E * E * E, B = 4;
    for (int i0 = tid; i0 < NE; i0 += B * 512) {
        float v[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int i = i0 + u * 512;
            if (i < NE) {
                const int lx = i % E, ly = (i / E) % E, lz = i / (E * E);
                const int gx = min(max(x0 + lx - H, 0), (int)nx - 1);
                const int gy = min(max(y0 + ly - H, 0), (int)ny - 1);
                const int gz = min(max(z0 + lz - H, 0), (int)nz - 1);
                v[u] = in[((size_t)gz * ny + gy) * nx + gx];
            }
        }
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (i0 + u * 512 < NE) tile[i0 + u * 512] = v[u];
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y, z = z0 + threadIdx.z;
    if (x >= (int)nx || y >= (int)ny || z >= (int)nz) return;
    float sum = 0.f;
    for (int kz = -H; kz <= H; ++kz)
        for (int ky = -H; ky <= H; ++ky) {
            const float* row = tile + ((threadIdx.z + H + kz) * E + (threadIdx.y + H + ky)) * E + threadIdx.x + H;
            const float* wrow = taps.w + ((kz + H) * ksize + (ky + H)) * ksize + H;
#pragma unroll
            for (int kx = -H; kx <= H; ++kx) sum = fma_rn(row[kx], wrow[kx], sum);
        }
    out[((size_t)z * ny + y) * nx + x] = sum;
}


// The same filter for odd ksize = 2H+1 with H <= 2, streaming along z: a thread
// walks the input planes of its columns once, keeping the K = 2H+1 outputs a
// plane reaches in a rotating window of accumulators (plane pl adds tap
// kz = 2H - k to output pl - 2H + k; the loop is unrolled over K planes, so the
// rotation is in the register names).  Each thread owns two columns, x and
// x + 16, as the halves of packed FP32 pairs: one fma.rn.f32x2 applies a tap to
// both outputs with the scalar rounding on each half, and every output receives
// its terms in the reference's order (plane = kz ascending, then ky, then kx),
// so the result is bitwise that of log_filter_kernel.
// The taps of a LoG depend on kx^2 + ky^2 + kz^2 alone (4 values for K = 3, 10
// for K = 5; the host checks their bits), so they stay in registers.  The
// planes pass through a ring in shared memory, asynchronous copies three ahead.
// Bound by the FMA issue (a packed instruction holds the port two cycles): 125
// FMAs per voxel are 52 us at 256^3.  89 us there; one plane ahead
// through registers 97, and with the whole tile in shared memory first, slabs of
// 16 planes and taps from the constant bank 125.
template <int H>
struct LogTaps2 {
    unsigned long long w2[3 * H * H + 1];  // (w, w) by squared distance
};

constexpr int kLogTX = 32, kLogTY = 8;

// Four bytes from global to shared memory, asynchronously.
__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <int H>
__global__ void __launch_bounds__(128, 7) log_filter_stream_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                                   uint32_t nx, uint32_t ny, uint32_t nz, uint32_t tz,
                                                                   const LogTaps2<H> taps) {
    constexpr int K = 2 * H + 1, HX = kLogTX / 2, TY = kLogTY, EX = HX + 2 * H, EY = TY + 2 * H, NT = HX * TY;
    constexpr int NE = EX * EY, PER = (NE + NT - 1) / NT;
    constexpr int RING = 4;
    __shared__ f32x2_t tile[RING][EY][EX];
    const int x0 = blockIdx.x * kLogTX, y0 = blockIdx.y * TY, z0 = blockIdx.z * tz;
    const int z1 = min(z0 + (int)tz, (int)nz);
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + HX * ty;
    f32x2_t w[3 * H * H + 1];
#pragma unroll
    for (int i = 0; i <= 3 * H * H; ++i) w[i] = taps.w2[i];
    // This thread's samples of a plane (borders clamped).  Samples that only
    // outputs beyond the volume would use are left out: lanes that copy one
    // clamped address into many places take a pass each.
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t oa[PER], ob[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int e = tid + u * NT, gx = x0 + e % EX - H, gy = y0 + e / EX - H;
        const uint32_t row = (uint32_t)min(max(gy, 0), (int)ny - 1) * nx;
        const bool used = e < NE && gy < (int)ny + H;
        oa[u] = used && gx < (int)nx + H ? row + min(max(gx, 0), (int)nx - 1) : kNone;
        ob[u] = used && gx + HX < (int)nx + H ? row + min(max(gx + HX, 0), (int)nx - 1) : kNone;
    }
    const size_t plane = (size_t)nx * ny;
    const int planes = z1 - z0 + 2 * H;
    auto load = [&](int pl) {  // input plane z0 - H + pl into its place in the ring (a group even past the last)
        if (pl < planes) {
            const float* src = in + (size_t)min(max(z0 + pl - H, 0), (int)nz - 1) * plane;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                float* dst = reinterpret_cast<float*>(&tile[pl % RING][0][0] + tid + u * NT);
                if (oa[u] != kNone) copy_async4(dst, src + oa[u]);
                if (ob[u] != kNone) copy_async4(dst + 1, src + ob[u]);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int xa = x0 + tx, xb = xa + HX, y = y0 + ty;
    const bool ok_a = xa < (int)nx && y < (int)ny, ok_b = xb < (int)nx && y < (int)ny;
    const size_t row = (size_t)y * nx;
    f32x2_t acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0ull;
    for (int pl = 0; pl < RING - 1; ++pl) load(pl);
#pragma unroll 1
    for (int p0 = 0; p0 < planes; p0 += K) {
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const int pl = p0 + u;
            if (pl >= planes) break;
            asm volatile("cp.async.wait_group %0;" ::"n"(RING - 2) : "memory");  // this thread's part of plane pl
            __syncthreads();  // everyone's; and all are through with plane pl - 1
            load(pl + RING - 1);
            const f32x2_t(*t)[EX] = tile[pl % RING];
#pragma unroll
            for (int ky = 0; ky < K; ++ky) {
                f32x2_t r[K];
#pragma unroll
                for (int kx = 0; kx < K; ++kx) r[kx] = t[ty + ky][tx + kx];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int dz = H - k, dy = ky - H;  // kz = 2H - k
                    f32x2_t& a = acc[(u + 1 + k) % K];
#pragma unroll
                    for (int kx = 0; kx < K; ++kx) a = fma_rn2(r[kx], w[dz * dz + dy * dy + (kx - H) * (kx - H)], a);
                }
            }
            f32x2_t& done = acc[(u + 1) % K];  // output plane pl - 2H
            if (pl >= 2 * H) {
                float a, b;
                unpack2(done, a, b);
                float* o = out + (size_t)(z0 + pl - 2 * H) * plane + row;
                if (ok_a) o[xa] = a;
                if (ok_b) o[xb] = b;
            }
            done = 0ull;
        }
    }
}

// ------------------------------------------------------- Laplacian filter --

// laplacianFilter (transient_postprocessing.cuh:21-50): k^3 * v - (sum of the
// k^3 box, zero outside the volume), box summed with x outermost, z innermost.
template <int H>
__global__ void __launch_bounds__(512) laplacian_filter_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                               uint32_t nx, uint32_t ny, uint32_t nz, float k3) {
    constexpr int E = 8 + 2 * H;
    extern __shared__ float tile[];
    const int x0 = blockIdx.x * 8, y0 = blockIdx.y * 8, z0 = blockIdx.z * 8;
    const int tid = threadIdx.x + 8 * (threadIdx.y + 8 * threadIdx.z);
    for (int i = tid; i < E * E * E; i += 512) {
        const int lx = i % E, ly = (i / E) % E, lz = i / (E * E);
        const int gx = x0 + lx - H, gy = y0 + ly - H, gz = z0 + lz - H;
        float v = 0.f;
        if (gx >= 0 && gx < (int)nx && gy >= 0 && gy < (int)ny && gz >= 0 && gz < (int)nz)
            v = in[((size_t)gz * ny + gy) * nx + gx];
        tile[i] = v;
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y, z = z0 + threadIdx.z;
    if (x >= (int)nx || y >= (int)ny || z >= (int)nz) return;
    float lap = 0.f;
    for (int dx = -H; dx <= H; ++dx)
        for (int dy = -H; dy <= H; ++dy)
#pragma unroll
            for (int dz = -H; dz <= H; ++dz)
                lap = add_rn(lap, tile[((threadIdx.z + H + dz) * E + (threadIdx.y + H + dy)) * E + threadIdx.x + H + dx]);
    const float c = tile[((threadIdx.z + H) * E + (threadIdx.y + H)) * E + threadIdx.x + H];
    out[((size_t)z * ny + y) * nx + x] = fma_rn(k3, c, -lap);
}


// laplacianFilter (transient_postprocessing.cuh:21-50) register-blocked along
// z: a thread owns one (x, y) column of 32 outputs and adds the K^3
// neighbours of each in the reference's order (dx, dy, dz; zero outside the
// volume), then centre * K^3 - sum.  The outputs z and z + 16 are the halves
// of packed FP32 pairs: the tile holds (v[z], v[z + 16]) pairs along z, and
// one add.rn.f32x2 adds a neighbour to both sums, so the result is bitwise
// that of the scalar sum at half the add instructions.
template <int H>
__global__ void __launch_bounds__(128) laplacian_zpair_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                              uint32_t nx, uint32_t ny, uint32_t nz, float k3) {
    constexpr int K = 2 * H + 1, TX = 32, TY = 4, TZ = 32, HZ = 16;
    constexpr int EX = TX + 2 * H, EY = TY + 2 * H, EZ2 = HZ + 2 * H;  // pairs (z, z + 16), z < EZ2
    __shared__ f32x2_t tile[EZ2][EY][EX];
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * TZ;
    const int tid = threadIdx.x + TX * threadIdx.y;
    constexpr int NT = TX * TY, NE = EX * EY * EZ2, B = 8;
    for (int i0 = tid; i0 < NE; i0 += B * NT) {
        float va[B], vb[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int i = i0 + u * NT;
            va[u] = vb[u] = 0.f;  // zero outside the volume
            if (i < NE) {
                const int lx = i % EX, ly = (i / EX) % EY, lz = i / (EX * EY);
                const int gx = x0 + lx - H, gy = y0 + ly - H, ga = z0 + lz - H, gb = ga + HZ;
                if (gx >= 0 && gx < (int)nx && gy >= 0 && gy < (int)ny) {
                    const size_t col = (size_t)gy * nx + gx, plane = (size_t)nx * ny;
                    if (ga >= 0 && ga < (int)nz) va[u] = in[ga * plane + col];
                    if (gb >= 0 && gb < (int)nz) vb[u] = in[gb * plane + col];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (i0 + u * NT < NE) (&tile[0][0][0])[i0 + u * NT] = pack2(va[u], vb[u]);
    }
    __syncthreads();
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x = x0 + tx, y = y0 + ty;
    if (x >= (int)nx || y >= (int)ny) return;
    f32x2_t lap[HZ];  // (sum of output z, sum of output z + 16)
#pragma unroll
    for (int z = 0; z < HZ; ++z) lap[z] = 0ull;
#pragma unroll 1
    for (int dx = 0; dx < K; ++dx) {
#pragma unroll 1
        for (int dy = 0; dy < K; ++dy) {
            f32x2_t c[EZ2];
#pragma unroll
            for (int z = 0; z < EZ2; ++z) c[z] = tile[z][ty + dy][tx + dx];
#pragma unroll
            for (int z = 0; z < HZ; ++z)
#pragma unroll
                for (int dz = 0; dz < K; ++dz) lap[z] = add_rn2(lap[z], c[z + dz]);
        }
    }
#pragma unroll
    for (int z = 0; z < HZ; ++z) {
        float la, lb, ca, cb;
        unpack2(lap[z], la, lb);
        unpack2(tile[z + H][ty + H][tx + H], ca, cb);  // (v[z + H], v[z + 16 + H]) of this column
        const size_t col = (size_t)y * nx + x, plane = (size_t)nx * ny;
        if (z0 + z < (int)nz) out[(z0 + z) * plane + col] = fma_rn(k3, ca, -la);
        if (z0 + z + HZ < (int)nz) out[(z0 + z + HZ) * plane + col] = fma_rn(k3, cb, -lb);
    }
}

fbp_status launch_log(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz, int ksize,
                      float sigma, cudaStream_t stream);
fbp_status launch_laplacian(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz,
                            int ksize, cudaStream_t stream);
fbp_status launch_log_fft(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz,
                          float sigma, cudaStream_t stream);

// Host-side LoG weights: PostprocessingFilters.cu:102-175 in float, same step order.
fbp_status log_weights_host(int size, float sigma, float* taps) {
    if (size <= 0 || !taps) return set_error(FBP_ERR_INVALID_ARG, "LoG weights: size must be > 0");
    const int half = (size - 1) / 2;
    const float var = sigma * sigma;
    const int n = size * size * size;
    std::vector<float> g(n), rr(n);
    float gmax = 0.0f;
    for (int kz = 0; kz < size; ++kz)
        for (int ky = 0; ky < size; ++ky)
            for (int kx = 0; kx < size; ++kx) {
                const float x = (float)(kx - half), y = (float)(ky - half), z = (float)(kz - half);
                const int i = kz * size * size + ky * size + kx;
                rr[i] = x * x + y * y + z * z;
                g[i] = std::exp(-(x * x + y * y + z * z) / (2.0f * var));
                gmax = std::max(g[i], gmax);
            }
    const float cutoff = 1.19209290e-07f * gmax;  // FLT_EPSILON * max
    float gsum = 0.0f;
    for (float& v : g) {
        if (v < cutoff) v = 0.0f;
        gsum += v;
    }
    if (gsum != 0.0f)
        for (float& v : g) v /= gsum;
    float lsum = 0.0f;
    for (int i = 0; i < n; ++i) {
        g[i] = g[i] * (rr[i] - 3.0f * var) / (var * var);
        lsum += g[i];
    }
    const float mean = lsum / (float)n;  // subtracted so the taps sum to zero
    for (int i = 0; i < n; ++i) taps[i] = g[i] - mean;
    return FBP_OK;
}

template <int H>
static fbp_status log_h(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz, int ksize,
                        const float* w, cudaStream_t stream) {
    LogTaps<H> taps{};
    for (int i = 0; i < ksize * ksize * ksize; ++i) taps.w[i] = w[i];
    if constexpr (H >= 1 && H <= 2) {
        if (ksize == 2 * H + 1) {
            // The taps by squared distance, if they depend on nothing else.
            LogTaps2<H> taps2{};
            bool radial = (uint64_t)nx * ny < (1ull << 32), seen[3 * H * H + 1] = {};
            for (int i = 0; i < ksize * ksize * ksize; ++i) {
                const int x = i % ksize - H, y = i / ksize % ksize - H, z = i / (ksize * ksize) - H;
                uint32_t b;
                std::memcpy(&b, &w[i], 4);
                const int d = x * x + y * y + z * z;
                const unsigned long long v = ((unsigned long long)b << 32) | b;  // (w, w)
                radial = radial && (!seen[d] || taps2.w2[d] == v);
                seen[d] = true;
                taps2.w2[d] = v;
            }
            if (radial) {
                // Planes per CTA: the fewest plane steps on the busiest SM
                // (seven CTAs resident; two steps' worth of set-up), where
                // fewer than five CTAs take as long as five (a step's latency):
                // K = 3 at 128^3 7.8 us so, 12.1 by the steps alone.
                uint32_t tz = 8;
                uint64_t least = ~0ull;
                const uint64_t columns = (uint64_t)cdiv(nx, kLogTX) * cdiv(ny, kLogTY);
                for (uint32_t c = 8; c <= 256; c *= 2) {
                    const uint32_t slabs = cdiv(nz, c), planes = cdiv(nz, slabs);
                    const uint64_t rounds = cdiv(columns * slabs, (uint64_t)ctx->sm_count);
                    const uint64_t steps = std::max<uint64_t>(rounds, 5) * (planes + 2 * H + 2);
                    if (steps < least) {
                        least = steps;
                        tz = planes;
                    }
                }
                dim3 grid(cdiv(nx, kLogTX), cdiv(ny, kLogTY), cdiv(nz, tz));
                log_filter_stream_kernel<H><<<grid, dim3(kLogTX / 2, kLogTY), 0, stream>>>(in, out, nx, ny, nz, tz, taps2);
                FBP_CHECK_LAUNCH(ctx, "log_filter_stream_kernel");
                return FBP_OK;
            }
        }
    }
    constexpr int E = 8 + 2 * H;
    const size_t smem = sizeof(float) * E * E * E;
    FBP_TRY_CUDA(cudaFuncSetAttribute(log_filter_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(cdiv(nx, 8), cdiv(ny, 8), cdiv(nz, 8));
    log_filter_kernel<H><<<grid, dim3(8, 8, 8), smem, stream>>>(in, out, nx, ny, nz, ksize, taps);
    FBP_CHECK_LAUNCH(ctx, "log_filter_kernel");
    return FBP_OK;
}

template <int H>
static fbp_status lap_h(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz, float k3,
                        cudaStream_t stream) {
    if constexpr (H <= 2) {
        const dim3 grid(cdiv(nx, 32), cdiv(ny, 4), cdiv(nz, 32));
        laplacian_zpair_kernel<H><<<grid, dim3(32, 4), 0, stream>>>(in, out, nx, ny, nz, k3);
        FBP_CHECK_LAUNCH(ctx, "laplacian_zpair_kernel");
        return FBP_OK;
    }
    constexpr int E = 8 + 2 * H;
    const size_t smem = sizeof(float) * E * E * E;
    FBP_TRY_CUDA(cudaFuncSetAttribute(laplacian_filter_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(cdiv(nx, 8), cdiv(ny, 8), cdiv(nz, 8));
    laplacian_filter_kernel<H><<<grid, dim3(8, 8, 8), smem, stream>>>(in, out, nx, ny, nz, k3);
    FBP_CHECK_LAUNCH(ctx, "laplacian_filter_kernel");
    return FBP_OK;
}

fbp_status launch_log(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz, int ksize,
                      float sigma, cudaStream_t stream) {
    if (ksize < 1 || ksize > kLogMaxK)
        return set_error(FBP_ERR_UNSUPPORTED, "LoG filter: kernel size must be in [1, 15]");
    std::vector<float> w((size_t)ksize * ksize * ksize);
    FBP_TRY(log_weights_host(ksize, sigma, w.data()));
    // The reference's kernelHalf = (k - 1) / 2 (PostprocessingFilters.cu:25).
    switch ((ksize - 1) / 2) {
        case 0: return log_h<0>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 1: return log_h<1>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 2: return log_h<2>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 3: return log_h<3>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 4: return log_h<4>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 5: return log_h<5>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        case 6: return log_h<6>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
        default: return log_h<7>(ctx, in, out, nx, ny, nz, ksize, w.data(), stream);
    }
}

fbp_status launch_laplacian(fbp_context* ctx, const float* in, float* out, uint32_t nx, uint32_t ny, uint32_t nz,
                            int ksize, cudaStream_t stream) {
    if (ksize < 1 || ksize > kLogMaxK)
        return set_error(FBP_ERR_UNSUPPORTED, "Laplacian filter: kernel size must be in [1, 15]");
    // laplacianFilter receives the size as a float and uses floor(size / 2)
    // for the half width and size^3 (as float products) for the centre weight.
    const float fs = (float)ksize;
    const float k3 = fs * fs * fs;
    switch ((int)std::floor(fs / 2.0f)) {
        case 0: return lap_h<0>(ctx, in, out, nx, ny, nz, k3, stream);
        case 1: return lap_h<1>(ctx, in, out, nx, ny, nz, k3, stream);
        case 2: return lap_h<2>(ctx, in, out, nx, ny, nz, k3, stream);
        case 3: return lap_h<3>(ctx, in, out, nx, ny, nz, k3, stream);
        case 4: return lap_h<4>(ctx, in, out, nx, ny, nz, k3, stream);
        case 5: return lap_h<5>(ctx, in, out, nx, ny, nz, k3, stream);
        case 6: return lap_h<6>(ctx, in, out, nx, ny, nz, k3, stream);
        default: return lap_h<7>(ctx, in, out, nx, ny, nz, k3, stream);
    }
}

}  // namespace fbp

using namespace fbp;

extern "C" fbp_status fbp_log_weights(int size, float sigma, float* w) {
    return guarded("fbp_log_weights", [&]() -> fbp_status {
        clear_error();
        return log_weights_host(size, sigma, w);
    });
}

extern "C" fbp_status fbp_normalize_minmax(fbp_context* ctx, float* v, uint64_t n, void* stream) {
    return guarded("fbp_normalize_minmax", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        if (!v || n == 0) return set_error(FBP_ERR_INVALID_ARG, "fbp_normalize_minmax: null buffer or n == 0");
        return normalize_device(ctx, v, n, (cudaStream_t)stream);
    });
}

// ------------------------------------------ allocation-free normalisation --
//
// fbp_normalize_minmax_noalloc: the same two passes as fbp_normalize_minmax,
// but its scratch (one min/max pair per reduction block) lives in this
// file-scope array instead of context workspace, so the call allocates nothing
// and needs no fbp_context.  Every device that loads the library holds the array
// (8 KiB) until the process exits.  The partial pass
// strides over the input with up to 1024 blocks (4 per SM, like the context
// entry point), one partial slot each; inputs are limited to 2^30 elements.
// All calls on a device share the array: each call overwrites every slot it
// reads before reading it, and two calls that overlap on the GPU (different
// streams, no ordering between them) race on it.
namespace fbp {
constexpr int kNoAllocMaxBlocks = 1024;
constexpr uint64_t kNoAllocMaxElems = 1ull << 30;
static __device__ __align__(256) float g_noalloc_scratch[2 * kNoAllocMaxBlocks];

// Device address of g_noalloc_scratch on the current device, looked up on
// every call (the first call on a device loads the module; later lookups are
// cheap, and a module reloaded after a device reset gets its new address).
// Host code must not pass the symbol itself to a kernel: on the host it only
// names a stand-in object.
static fbp_status noalloc_scratch(float** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_error(e, "fbp_normalize_minmax_noalloc: cudaGetSymbolAddress");
    *out = static_cast<float*>(p);
    return FBP_OK;
}
}  // namespace fbp

extern "C" fbp_status fbp_normalize_minmax_noalloc(float* v, uint64_t n, void* stream) {
    return guarded("fbp_normalize_minmax_noalloc", [&]() -> fbp_status {
        clear_error();
        if (!v || n == 0) return set_error(FBP_ERR_INVALID_ARG, "fbp_normalize_minmax_noalloc: null buffer or n == 0");
        if (n > kNoAllocMaxElems)
            return set_error(FBP_ERR_UNSUPPORTED,
                             "fbp_normalize_minmax_noalloc: n exceeds 2^30 elements (the static scratch holds 1024 "
                             "partial min/max pairs); use fbp_normalize_minmax");
        // An error left pending by earlier work is reported as such, not as
        // this call's launch failure (and left for the caller to clear).
        const cudaError_t pending = cudaPeekAtLastError();
        if (pending != cudaSuccess)
            return cuda_error(pending, "fbp_normalize_minmax_noalloc: a CUDA error was pending before the call");
        int dev = -1;
        FBP_TRY_CUDA(cudaGetDevice(&dev));
        cudaPointerAttributes attr{};
        FBP_TRY_CUDA(cudaPointerGetAttributes(&attr, v));
        if ((attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged) || attr.device != dev)
            return set_error(FBP_ERR_INVALID_ARG,
                             "fbp_normalize_minmax_noalloc: v is not device memory of the current device");
        float* scratch = nullptr;
        FBP_TRY(noalloc_scratch(&scratch));
        int sms = 0;
        FBP_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        cudaStream_t s = (cudaStream_t)stream;
        const uint64_t want = (n + 4ull * kReduceThreads - 1) / (4ull * kReduceThreads);
        const uint64_t cap = std::min<uint64_t>(kNoAllocMaxBlocks, 4ull * (uint64_t)std::max(sms, 1));
        const int nb = (int)std::max<uint64_t>(1, std::min(want, cap));
        minmax_partial_kernel<<<nb, kReduceThreads, 0, s>>>(v, n, scratch);
        FBP_TRY_CUDA(cudaGetLastError());
        const unsigned ab = (unsigned)std::min<uint64_t>(cdiv(n, 4 * 256), 1216);
        normalize_apply_kernel<<<ab, 256, 0, s>>>(v, n, scratch, nb);
        FBP_TRY_CUDA(cudaGetLastError());
        return FBP_OK;
    });
}

extern "C" fbp_status fbp_postfilter(fbp_context* ctx, int kind, int kernel_size, float sigma, const float* in,
                                     float* out, uint32_t nx, uint32_t ny, uint32_t nz, void* stream) {
    return guarded("fbp_postfilter", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        if (!in || !out) return set_error(FBP_ERR_INVALID_ARG, "fbp_postfilter: null buffer");
        if (nx == 0 || ny == 0 || nz == 0) return set_error(FBP_ERR_INVALID_ARG, "fbp_postfilter: empty volume");
        const size_t n = (size_t)nx * ny * nz;
        if (in == out && kind != FBP_FILTER_NONE)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_postfilter: in and out must be different buffers");
        cudaStream_t s = (cudaStream_t)stream;
        switch (kind) {
            case FBP_FILTER_NONE:
                if (in != out) FBP_TRY_CUDA(cudaMemcpyAsync(out, in, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
                return FBP_OK;
            case FBP_FILTER_LAPLACIAN: return launch_laplacian(ctx, in, out, nx, ny, nz, kernel_size, s);
            case FBP_FILTER_LOG: return launch_log(ctx, in, out, nx, ny, nz, kernel_size, sigma, s);
            case FBP_FILTER_LOG_FFT: return launch_log_fft(ctx, in, out, nx, ny, nz, sigma, s);
            default: return set_error(FBP_ERR_INVALID_ARG, "fbp_postfilter: unknown filter kind");
        }
    });
}
