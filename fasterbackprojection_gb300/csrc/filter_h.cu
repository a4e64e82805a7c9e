// Temporal band-pass filter of every scan point's histogram.
//
// Replaces Laser::filter_H_cuda (Laser.cu:128-240), padIntensity (:80-126)
// and multiplyHK (fourier.cuh:17-31).  The reference pads each histogram by
// t6sigma - 1 bins on both sides, runs a batched complex FFT of length
// n = T + 2(t6sigma - 1), multiplies by the FFT of an ifft-shifted complex
// Gaussian-windowed wave K, inverse-transforms without the 1/n factor and
// keeps the real part of the unpadded bins.  For a real input that equals
//     out[t] = n * sum_u h_ext[u] * Re(K_shift[(t - u) mod n])
// with h_ext the padded signal, so the filter here is a direct real
// correlation with n * Re(K_shift) taps, truncated where the taps fall below
// 1e-12 of the largest (the Gaussian envelope makes the rest negligible).
// No FFT, no host round trip, the filter runs in place on device data.
#include "fbp_internal.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

namespace fbp {

constexpr int kMaxTaps = 2048;
// Taps by value (kernel parameters, no longer than the kernel needs): concurrent
// calls share no state.
template <int N>
struct FilterTaps {
    float w[N];
};

// One CTA filters one series at a time (grid-stride over series).  Shared
// memory holds the padded period P[k] = h_ext[k - pad], k < n, extended
// circularly by R on both sides: S[i] = P[(i - R) mod n], i < n + 2R, so
//     out[t] = sum_{j=0}^{2R} taps[j] * S[t + pad + 2R - j]
// is the circular correlation the padded FFTs compute.
// Every thread produces Q = 8 consecutive outputs.  It keeps two windows of
// Q values of S in registers (ping-pong: the window that served the high half
// of one block of Q taps serves the low half of the next) and adds tap J + s
// to output q from window slot Q + q - s: one 32-byte row of S per Q taps for
// Q * Q FMAs.  Each output still sums its taps in order j = 0..2R; the taps
// are zero-padded to a multiple of 2Q (zero terms), and S is preceded by F
// zero slots (3Q <= F < 4Q, making S-index + F of every window start a
// multiple of Q) so the last, unused window loads stay in bounds.
// Rows of S are 8 floats, ROW apart.  ROW = 12: the 16-byte loads of 8
// consecutive threads (8 consecutive rows) fall in 8 different bank groups and
// every load of a thread is an immediate offset from its first row.  ROW = 8, two
// thirds of the shared memory, for long series: the halves of row k trade places
// when bit 2 of k is set, which keeps the bank groups apart and costs 12
// integer instructions per bin.
constexpr int kFilterQ = 8, kRowPadded = 12, kRowDense = 8;

template <int ROW>
__device__ __forceinline__ int srow_addr(int k, int half) {
    return ROW == kRowDense ? (8 * k + (k & 4)) ^ (4 * half) : k * ROW + 4 * half;
}

template <int ROW>
__device__ __forceinline__ void srow_load(const float* sh, int k, float (&v)[kFilterQ]) {
    const float4 a = *reinterpret_cast<const float4*>(sh + srow_addr<ROW>(k, 0));
    const float4 b = *reinterpret_cast<const float4*>(sh + srow_addr<ROW>(k, 1));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// acc[q] += t[st] * window slot (Q + q - st), slots [0, Q) in lo, [Q, 2Q) in hi.
__device__ __forceinline__ void filter_block(const float* t, const float (&lo)[kFilterQ], const float (&hi)[kFilterQ],
                                             float (&acc)[kFilterQ]) {
    constexpr int Q = kFilterQ;
#pragma unroll
    for (int st = 0; st < Q; ++st)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int m = Q + q - st;
            acc[q] = fmaf(m < Q ? lo[m] : hi[m - Q], t[st], acc[q]);
        }
}

// Taps J .. J + Q - 1 from the shared copy (two 16-byte loads).
__device__ __forceinline__ void filter_block_shared(const float* s_taps, int J, const float (&lo)[kFilterQ],
                                                    const float (&hi)[kFilterQ], float (&acc)[kFilterQ]) {
    const float4 ta = *reinterpret_cast<const float4*>(s_taps + J);
    const float4 tb = *reinterpret_cast<const float4*>(s_taps + J + 4);
    const float t[kFilterQ] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
    filter_block(t, lo, hi, acc);
}

// NJ > 0: exactly NJ blocks of 2Q taps, unrolled, each FMA reading its tap
// from the kernel parameters (constant bank; zero past the last tap).
// NJ == 0: any tap count, taps from the shared copy.
// Bound by the FMA issue: 112 taps per bin.  The fill used to take a fifth of
// the instructions (circular index, clamp and border per sample); now a thread
// works out the slots of its first kPrefetch half rows once, and loads the next
// series' samples before this one is filtered.
// 65536 x 1024: 371 -> 298 us (FMA pipe 69 %, issue
// 85 %).
// (With many taps, NJ == 0, and 128 threads or more the fill is a small part:
// nothing is kept or loaded ahead.)
constexpr int prefetch_rows(int nj, int nt) { return nj > 0 || nt <= 64 ? 3 : 0; }
constexpr int filter_taps(int nj) { return nj > 0 ? 2 * kFilterQ * nj : kMaxTaps; }

template <int NJ, int nt, int ROW>
__global__ void __launch_bounds__(nt, 1024 / nt) filter_h_kernel(float* __restrict__ data, uint64_t nseries, uint32_t T, int n,
                                                       int R, int pad, int edge, int F, int ntp, int rows,
                                                       const __grid_constant__ FilterTaps<filter_taps(NJ)> taps) {
    constexpr int Q = kFilterQ;
    extern __shared__ __align__(16) float sh[];  // taps (ntp, zero-padded), then `rows` rows of S
    const int E = n + 2 * R;
    float* s_taps = sh;
    float* sser = sh + ntp;
    if (NJ == 0)
        for (int j = threadIdx.x; j < ntp; j += nt) s_taps[j] = taps.w[j];
    // Slot i of S (S index): the sample it takes and whether it does.  Slots
    // before S[0] and past S[E - 1] are zero; a slot whose signal index falls
    // outside [0, T) takes the clamped border sample (edge) or zero.
    auto slot = [&](int i, bool& keep) -> uint32_t {
        int k = i - R;  // circular index: -R <= k < n + R for i in [0, E), R < n
        k += k < 0 ? n : 0;
        k -= k >= n ? n : 0;
        const int u = k - pad;  // signal index
        keep = i >= 0 && i < E && (edge || (u >= 0 && u < (int)T));
        return (uint32_t)min(max(u, 0), (int)T - 1);
    };
    // The slots of this thread's first kPrefetch half rows (the same for every
    // series): half row g holds slots 4 g - F and on.
    constexpr int kPrefetch = prefetch_rows(NJ, nt);
    uint32_t from[kPrefetch + 1][4], kept = 0;
#pragma unroll
    for (int u = 0; u < kPrefetch; ++u)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            bool keep;
            from[u][b] = slot(4 * ((int)threadIdx.x + u * nt) + b - F, keep);
            kept |= (uint32_t)keep << (4 * u + b);
        }
    auto store_half = [&](int g, const float (&v)[4]) {
        *reinterpret_cast<float4*>(sser + srow_addr<ROW>(g >> 1, g & 1)) = make_float4(v[0], v[1], v[2], v[3]);
    };
    float pre[kPrefetch + 1][4];
    auto prefetch = [&](const float* h) {
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u)
#pragma unroll
            for (int b = 0; b < 4; ++b) pre[u][b] = h[from[u][b]];
    };
    if (blockIdx.x < nseries) prefetch(data + (uint64_t)blockIdx.x * T);
    for (uint64_t s = blockIdx.x; s < nseries; s += gridDim.x) {
        float* h = data + s * T;
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u) {
            const int g = threadIdx.x + u * nt;
            float v[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) v[b] = kept >> (4 * u + b) & 1 ? pre[u][b] : 0.f;
            if (g < 2 * rows) store_half(g, v);
        }
        for (int g = threadIdx.x + kPrefetch * nt; g < 2 * rows; g += nt) {
            float v[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                bool keep;
                const uint32_t u = slot(4 * g + b - F, keep);
                v[b] = keep ? h[u] : 0.f;
            }
            store_half(g, v);
        }
        if (s + gridDim.x < nseries) prefetch(data + (s + gridDim.x) * T);
        __syncthreads();
        for (int t0 = threadIdx.x * Q; t0 < (int)T; t0 += nt * Q) {
            // out[t0 + q] = sum_j taps[j] * S[b0 - j + q], b0 = t0 + pad + 2R; in slots
            // b = b0 + F (a multiple of Q), window of block J: slots b - J - Q .. b - J + Q.
            const int kb = (t0 + pad + 2 * R + F) >> 3;  // row of slot b
            float A[Q], B[Q], acc[Q];
            srow_load<ROW>(sser, kb - 1, A);
            srow_load<ROW>(sser, kb, B);
#pragma unroll
            for (int q = 0; q < Q; ++q) acc[q] = 0.f;
            if constexpr (NJ > 0) {
#pragma unroll
                for (int jj = 0; jj < NJ; ++jj) {
                    const int k = kb - 2 * jj;  // kb - J / Q with J = 2Q jj
                    filter_block(taps.w + 2 * Q * jj, A, B, acc);
                    srow_load<ROW>(sser, k - 2, B);  // low window of block J + Q
                    filter_block(taps.w + 2 * Q * jj + Q, B, A, acc);
                    srow_load<ROW>(sser, k - 3, A);  // low window of block J + 2Q
                }
            } else {
                for (int J = 0; J < ntp; J += 2 * Q) {
                    const int k = kb - (J >> 3);
                    filter_block_shared(s_taps, J, A, B, acc);
                    srow_load<ROW>(sser, k - 2, B);  // low window of block J + Q
                    filter_block_shared(s_taps, J + Q, B, A, acc);
                    srow_load<ROW>(sser, k - 3, A);  // low window of block J + 2Q
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (t0 + q < (int)T) h[t0 + q] = acc[q];
        }
        __syncthreads();
    }
}

// Host: the taps of filter_H (Laser.cu:131-172) in double precision.
// Returns R (taps cover lags -R..R), the padding, and n.
fbp_status filter_h_taps(uint32_t nt, float delta_t, float wl_mean, float wl_sigma, std::vector<float>& taps, int& R,
                         int& pad, int& n_out) {
    // Laser.cu:131-139, in float like the reference.
    float sig_f = wl_sigma;
    if (std::fabs(wl_sigma - 0.0f) < 1.19209290e-07f) sig_f = wl_mean / std::sqrt(2.0f);
    const double sigma = sig_f;
    int t6 = (int)std::round(6.0f * sig_f / delta_t);
    if (t6 % 2 == 1) t6 += 1;
    if (t6 < 1) return set_error(FBP_ERR_INVALID_ARG, "filter_H: wavelength too short for the bin width");
    const int n = (int)nt + 2 * (t6 - 1);
    pad = t6 - 1;
    n_out = n;
    const double dt = delta_t;
    const double tmax = dt * (n - 1);
    std::vector<double> env(n);
    double envsum = 0.0;
    for (int i = 0; i < n; ++i) {
        const double v = (i * dt - tmax * 0.5) / sigma;
        env[i] = std::exp(-(v * v) * 0.5);
        envsum += env[i];
    }
    // Re(K_shift[m]) = Re(K[(m + n/2) % n]); lag delta uses index delta mod n.
    // env[src] / envsum bounds |kr|, so a cosine is worked out only where it
    // can matter (5104 series of 1767 bins, bound by this: 89 -> 48 us a call).
    auto src = [&](int m) { return ((m + n) % n + n / 2) % n; };  // -n <= m
    auto kr = [&](int m) {
        const double phase = 2.0 * M_PI * ((long)src(m) * dt) / (double)wl_mean;
        return env[src(m)] * std::cos(phase) / envsum;
    };
    auto above = [&](int m, double bound) { return env[src(m)] / envsum > bound && std::fabs(kr(m)) > bound; };
    // Lags are circular over the padded period: |lag| <= n/2 covers them all.
    double kmax = 0.0;
    for (int m = 0; m <= n / 2; ++m) {  // from the centre outwards
        if (above(m, kmax)) kmax = std::fabs(kr(m));
        if (above(-m, kmax)) kmax = std::fabs(kr(-m));
    }
    int r = n / 2;
    while (r > 0 && !above(r, 1e-12 * kmax) && !above(-r, 1e-12 * kmax)) --r;
    if (2 * r + 1 > kMaxTaps) return set_error(FBP_ERR_UNSUPPORTED, "filter_H: filter longer than 2047 taps");
    R = r;
    taps.assign(2 * r + 1, 0.f);
    for (int j = 0; j <= 2 * r; ++j) taps[j] = (float)((double)n * kr(j - r));
    return FBP_OK;
}

fbp_status filter_h_device(fbp_context* ctx, float* data, uint64_t nseries, uint32_t T, float delta_t, float wl_mean,
                           float wl_sigma, int border, cudaStream_t stream) {
    std::vector<float> taps;
    int R = 0, pad = 0, n = 0;
    FBP_TRY(filter_h_taps(T, delta_t, wl_mean, wl_sigma, taps, R, pad, n));
    constexpr int Q = kFilterQ;
    const int ntp = (2 * R + 1 + 2 * Q - 1) / (2 * Q) * (2 * Q);
    if (ntp > kMaxTaps) return set_error(FBP_ERR_UNSUPPORTED, "filter_H: filter longer than the tap table");
    // F zero slots before S: 3Q <= F < 4Q with (pad + 2R + F) % Q == 0.
    const int F = 3 * Q + (Q - (pad + 2 * R + 3 * Q) % Q) % Q;
    // Highest slot read: t0 + pad + 2R + F + Q - 1 with t0 <= T - 1 (< E + F + Q).
    const int rows = (n + 2 * R + F + Q) / Q + 1;
    auto smem_of = [&](int row) { return ((size_t)ntp + (size_t)row * rows) * sizeof(float); };
    if (smem_of(kRowDense) > (size_t)ctx->smem_optin)
        return set_error(FBP_ERR_UNSUPPORTED, "filter_H: series too long for one CTA");
    taps.resize((size_t)ntp, 0.f);
    auto fit = [&](int row) { return kSmSharedBytes / (smem_of(row) + kCtaReservedShared); };  // CTAs to an SM, by shared memory
    auto launch = [&](auto nj, auto nt, auto row) -> fbp_status {
        constexpr int NJ = decltype(nj)::value, threads = decltype(nt)::value, ROW = decltype(row)::value;
        auto kernel = filter_h_kernel<NJ, threads, ROW>;
        const size_t smem = smem_of(ROW);
        FilterTaps<filter_taps(NJ)> tp;
        std::copy(taps.begin(), taps.end(), tp.w);
        FBP_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        // One CTA per resident slot (64 registers a thread), or twice as many
        // where that leaves each only a few series; long series, whose setup is
        // nothing beside them, 16 to an SM.
        const size_t resident = std::max<size_t>(1, std::min<size_t>(std::min<size_t>(32, 1024 / threads), fit(ROW)));
        const uint64_t slots = (uint64_t)ctx->sm_count * resident;
        const uint64_t most = ROW == kRowDense ? (uint64_t)ctx->sm_count * 16 : nseries < 8 * slots ? 2 * slots : slots;
        kernel<<<(unsigned)std::min<uint64_t>(nseries, most), threads, smem, stream>>>(
            data, nseries, T, n, R, pad, border == FBP_BORDER_EDGE, F, ntp, rows, tp);
        FBP_CHECK_LAUNCH(ctx, "filter_h_kernel");
        return FBP_OK;
    };
    // Threads for one pass over a series (8 bins each): 65536 x 128 with 128
    // threads 65.7 us, with 32 38.7 us.  Padded rows while six series fit an SM
    // (some 6,000 bins), or four (9,000) with taps enough to pay for it; then dense
    // ones (1000 x 8192: 4-bin waves 40 us padded and 37 dense, 10-bin waves 50 and
    // 55; 4096 x 10000, 4-bin waves 243 and 193), from where four of them fit (some
    // 11,000 bins) with 256 threads (4096 x 20000, 10-bin waves: 1043 us padded,
    // 583 so).  Waves of more than 20 bins (NJ == 0) have borders and taps that
    // outweigh the bins of a short series: 32 or 64 threads only where there are
    // series enough to fill the GPU with them (150-bin waves: 2000 x 128 63 us with
    // 32 threads, 53 with 128; 60-bin waves: 20000 x 128 152 and 185).
    auto go = [&](auto nj) -> fbp_status {
        constexpr int NJ = decltype(nj)::value;
        constexpr std::integral_constant<int, kRowPadded> padded{};
        constexpr std::integral_constant<int, kRowDense> dense{};
        if (fit(kRowDense) <= (NJ > 0 ? 4 : 2)) return launch(nj, std::integral_constant<int, 256>{}, dense);
        if constexpr (NJ > 0) {
            // (few series: threads enough to load each in one go, too)
            auto enough = [&](uint32_t nt) {
                return T <= nt * Q && (nseries > 2ull * ctx->sm_count || 2 * (uint32_t)rows <= prefetch_rows(NJ, 32) * nt);
            };
            if (enough(32)) return launch(nj, std::integral_constant<int, 32>{}, padded);
            if (enough(64)) return launch(nj, std::integral_constant<int, 64>{}, padded);
            if (fit(kRowPadded) >= (NJ >= 5 ? 4 : 6)) return launch(nj, std::integral_constant<int, 128>{}, padded);
        } else if (T <= 64 * Q && fit(kRowPadded) >= 6) {
            if (T <= 32 * Q && nseries > 50ull * ctx->sm_count) return launch(nj, std::integral_constant<int, 32>{}, padded);
            if (T > 32 * Q && nseries > 4ull * ctx->sm_count) return launch(nj, std::integral_constant<int, 64>{}, padded);
        }
        return launch(nj, std::integral_constant<int, 128>{}, dense);
    };
    // Unrolled forms for 2 .. 12 blocks of 16 taps (wavelengths of about 2
    // to 20 bins; 10 bins, the reference's default, gives 107 taps = 7 blocks).
    switch (ntp / (2 * Q)) {
        case 2: return go(std::integral_constant<int, 2>{});
        case 3: return go(std::integral_constant<int, 3>{});
        case 4: return go(std::integral_constant<int, 4>{});
        case 5: return go(std::integral_constant<int, 5>{});
        case 6: return go(std::integral_constant<int, 6>{});
        case 7: return go(std::integral_constant<int, 7>{});
        case 8: return go(std::integral_constant<int, 8>{});
        case 9: return go(std::integral_constant<int, 9>{});
        case 10: return go(std::integral_constant<int, 10>{});
        case 11: return go(std::integral_constant<int, 11>{});
        case 12: return go(std::integral_constant<int, 12>{});
        default: return go(std::integral_constant<int, 0>{});
    }
}

}  // namespace fbp

using namespace fbp;

extern "C" fbp_status fbp_filter_h(fbp_context* ctx, float* data, uint64_t num_series, uint32_t num_bins, float delta_t,
                                   float wl_mean, float wl_sigma, int border, void* stream) {
    return guarded("fbp_filter_h", [&]() -> fbp_status {
        clear_error();
        FBP_TRY(check_ctx(ctx));
        if (!data || num_series == 0 || num_bins == 0) return set_error(FBP_ERR_INVALID_ARG, "fbp_filter_h: empty input");
        if (!(delta_t > 0.f) || !(wl_mean > 0.f)) return set_error(FBP_ERR_INVALID_ARG, "fbp_filter_h: delta_t and wl_mean must be > 0");
        if (border != FBP_BORDER_ZERO && border != FBP_BORDER_EDGE)
            return set_error(FBP_ERR_INVALID_ARG, "fbp_filter_h: unknown border mode");
        return filter_h_device(ctx, data, num_series, num_bins, delta_t, wl_mean, wl_sigma, border, (cudaStream_t)stream);
    });
}
