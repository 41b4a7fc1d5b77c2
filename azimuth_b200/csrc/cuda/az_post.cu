// Film post-processing on the GPU: OutputPixelsToFile's normalisation,
// photographic tone mapping and gamma correction (src/azimuth_main.cpp:
// 1620-1760) and the writers' 8-bit conversion (:1473-1475), for a device
// film that stays untouched.
//
//   k_post_luminance  colour / TotalWeight, luminance 0.27 R + 0.67 G + 0.06 B
//                     (src/azimuth_math.cpp:1866-1880), sum of log(L + 1e-5) in
//                     double (azimuth accumulates it serially in float), and the
//                     first histogram of the selection below
//   k_post_histogram, k_post_pick
//                     the burn-out luminance at index round((1 - burnout / 100)
//                     (N - 1)) of the sorted luminances (azimuth: qsort), by a
//                     radix selection of 11, 11 and 10 bits
//   k_post_map        Ld = Ls (1 + Ls / Lwhite^2) / (1 + Ls), (C / L)^saturation
//                     Ld clamped, then sRGB or 1/gamma, then (u8)(clamp01(C) 255)
//
// Full HD takes 2.7 ms with a full radix sort, an intermediate colour image and
// five cudaMalloc / cudaFree pairs; the selection reads 4 bytes a pixel twice,
// the map reads the film again (both from L2), and the scratch comes from the
// pool.  What is left is bound by the wait for the host between selection and map
// (40 us of 122) and, on the device, by the powf of the map: three a pixel at a
// saturation of 1, else six.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>

#include "az_internal.h"
#include "az_pool.h"

namespace az {
namespace {

__device__ __forceinline__ float lum3(float r, float g, float b) { return r * 0.27f + g * 0.67f + b * 0.06f; }
__device__ __forceinline__ float clamp01(float v) { return fminf(1.0f, fmaxf(0.0f, v)); }

constexpr uint32_t kBins = 2048;   // of the first two passes; the last has 1024
constexpr int kPostBlock = 256;

struct PostScratch {
    double logsum;
    float white;
    alignas(16) uint32_t hist[3][kBins];
};

// Keys whose unsigned order is the luminances' order (a radix sort's: negative
// values below, NaN by its sign at either end, the two zeros equal).
__device__ __forceinline__ uint32_t sort_key(float l) {
    const uint32_t u = l == 0.0f ? 0u : __float_as_uint(l);
    return u ^ (u >> 31 ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
    return __uint_as_float(k ^ (k >> 31 ? 0x80000000u : 0xFFFFFFFFu));
}

__device__ __forceinline__ void colour_of(const float4 p, float c[3]) {
    c[0] = p.x / p.w;
    c[1] = p.y / p.w;
    c[2] = p.z / p.w;
}

// Adds a block's histogram in shared memory to the global one.
__device__ __forceinline__ void add_histogram(const uint32_t *block, uint32_t *global) {
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kBins; b += kPostBlock)
        if (block[b]) atomicAdd(&global[b], block[b]);
}

__global__ void __launch_bounds__(kPostBlock) k_post_luminance(const float4 *film, uint32_t n, uint32_t *keys,
                                                               PostScratch *S) {
    __shared__ uint32_t bins[kBins];
    __shared__ double sums[kPostBlock / 32];
    for (uint32_t b = threadIdx.x; b < kBins; b += kPostBlock) bins[b] = 0u;
    __syncthreads();
    double part = 0.0;
#pragma unroll 4
    for (uint32_t i = blockIdx.x * kPostBlock + threadIdx.x; i < n; i += gridDim.x * kPostBlock) {
        float c[3];
        colour_of(film[i], c);
        const float l = lum3(c[0], c[1], c[2]);
        part += (double)logf(l + 0.00001f);
        const uint32_t k = sort_key(l);
        keys[i] = k;
        atomicAdd(&bins[k >> 21], 1u);
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
    if ((threadIdx.x & 31u) == 0) sums[threadIdx.x >> 5] = part;
    add_histogram(bins, S->hist[0]);
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kPostBlock / 32; w++) t += sums[w];
        atomicAdd(&S->logsum, t);
    }
}

// The bin of `hist` that holds element `rank` (0-based) and the element's rank
// within it; called by the whole block.
__device__ __forceinline__ uint32_t pick_bin(const uint32_t *hist, uint32_t rank, uint32_t &rest) {
    constexpr uint32_t kPer = kBins / kPostBlock;
    static_assert(kPer == 8, "two 16-byte loads a thread");
    __shared__ uint32_t warps[kPostBlock / 32];
    __shared__ uint32_t found[2];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint4 *src = reinterpret_cast<const uint4 *>(hist) + 2u * threadIdx.x;
    const uint4 h0 = src[0], h1 = src[1];
    const uint32_t h[kPer] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    uint32_t own = 0;
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++) own += h[k];
    uint32_t before = own;   // inclusive within the warp
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, before, d);
        if (lane >= d) before += v;
    }
    if (lane == 31) warps[warp] = before;
    __syncthreads();
    before -= own;
    for (uint32_t w = 0; w < warp; w++) before += warps[w];
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++) {
        if (rank >= before && rank - before < h[k]) {
            found[0] = threadIdx.x * kPer + k;
            found[1] = rank - before;
        }
        before += h[k];
    }
    __syncthreads();
    rest = found[1];
    const uint32_t bin = found[0];
    __syncthreads();
    return bin;
}

// PASS 1 and 2: the next bits of the keys that share the selected prefix.
// Four keys a load: with one, a thread waited for memory 14 times.
template <int PASS>
__global__ void __launch_bounds__(kPostBlock) k_post_histogram(const uint32_t *keys, uint32_t n, uint32_t rank,
                                                               PostScratch *S) {
    __shared__ uint32_t bins[kBins];
    for (uint32_t b = threadIdx.x; b < kBins; b += kPostBlock) bins[b] = 0u;
    uint32_t rest;
    uint32_t prefix = pick_bin(S->hist[0], rank, rest);
    if (PASS == 2) prefix = prefix << 11 | pick_bin(S->hist[1], rest, rest);
    auto count = [&](uint32_t k) {
        if (k >> (PASS == 1 ? 21 : 10) == prefix) atomicAdd(&bins[PASS == 1 ? (k >> 10) & 2047u : k & 1023u], 1u);
    };
    const uint32_t first = blockIdx.x * kPostBlock + threadIdx.x, step = gridDim.x * kPostBlock;
#pragma unroll 2
    for (uint32_t i = first; i < n / 4u; i += step) {
        const uint4 k = reinterpret_cast<const uint4 *>(keys)[i];
        count(k.x);
        count(k.y);
        count(k.z);
        count(k.w);
    }
    if (first < (n & 3u)) count(keys[(n & ~3u) + first]);
    add_histogram(bins, S->hist[PASS]);
}

__global__ void __launch_bounds__(kPostBlock) k_post_pick(uint32_t rank, PostScratch *S) {
    uint32_t rest;
    const uint32_t a = pick_bin(S->hist[0], rank, rest), b = pick_bin(S->hist[1], rest, rest);
    const uint32_t c = pick_bin(S->hist[2], rest, rest);
    if (threadIdx.x == 0) S->white = key_value(a << 21 | b << 10 | c);
}

struct MapParams {
    uint32_t n;
    int tonemapped;
    float factor, lw2, saturation;
    float inv_gamma;
    uint32_t srgb, linear;
};

// powf(q, 1) is q for every q, NaN and infinities among them (all 2^32 were
// tried), so the default saturation of 1 needs three powf a pixel instead of six.
__device__ __forceinline__ void map_colour(float c[3], const MapParams &P) {
    if (P.tonemapped) {
        const float l = lum3(c[0], c[1], c[2]);
        if (l != 0.0f) {
            const float ls = l * P.factor;
            const float ld = (ls * (1.0f + (ls / P.lw2))) / (1.0f + ls);
            for (int k = 0; k < 3; k++) {
                const float q = c[k] / l;
                c[k] = clamp01((P.saturation == 1.0f ? q : powf(q, P.saturation)) * ld);
            }
        }
    }
    if (P.linear) return;
    for (int k = 0; k < 3; k++) {
        if (P.srgb) c[k] = c[k] > 0.0031308f ? 1.055f * powf(c[k], P.inv_gamma) - 0.055f : c[k] * 12.92f;
        else c[k] = powf(c[k], P.inv_gamma);
    }
}

// Four pixels a thread, so that a thread's bytes are three whole words (WIDE:
// outputs aligned for it); the last pixels, and unaligned outputs, one by one.
template <bool WIDE>
__global__ void k_post_map(const float4 *film, float *rgb, uint8_t *rgb8, MapParams P) {
    const uint32_t quads = (P.n + 3u) / 4u;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < quads; q += gridDim.x * blockDim.x) {
        const uint32_t i = 4u * q, m = min(4u, P.n - i);
        float c[12];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            if (k < m) {
                colour_of(film[i + k], c + 3 * k);
                map_colour(c + 3 * k, P);
            }
        if (WIDE && m == 4u) {
            if (rgb) {
                float4 *o = reinterpret_cast<float4 *>(rgb + 3 * (size_t)i);
                for (int k = 0; k < 3; k++) o[k] = make_float4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
            }
            if (rgb8) {
                uint32_t *o = reinterpret_cast<uint32_t *>(rgb8 + 3 * (size_t)i);
                for (int k = 0; k < 3; k++) {
                    uint32_t w = 0;
                    for (int b = 0; b < 4; b++) w |= (uint32_t)(uint8_t)(clamp01(c[4 * k + b]) * 255.0f) << (8 * b);
                    o[k] = w;
                }
            }
            continue;
        }
#pragma unroll
        for (uint32_t k = 0; k < 12; k++)
            if (k < 3u * m) {
                if (rgb) rgb[3 * (size_t)i + k] = c[k];
                if (rgb8) rgb8[3 * (size_t)i + k] = (uint8_t)(clamp01(c[k]) * 255.0f);
            }
    }
}

}  // namespace

int PostProcess(const az_pixel *film, uint32_t w, uint32_t h, const az_tonemap *tm, float inv_gamma, uint32_t srgb,
                uint32_t linear, float *rgb_out, uint8_t *rgb8_out, cudaStream_t st) {
    const uint32_t n = w * h;
    if (n == 0) return AZ_OK;
    const bool tonemapped = !linear && tm && tm->Operator != AZ_Tonemap_None;
    if (tm && tm->Operator > AZ_Tonemap_Photographic) return SetError(AZ_ERR_INVALID_ARGUMENT, "unknown tone-mapping operator");
    const float4 *pix = reinterpret_cast<const float4 *>(film);
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    MapParams P;
    memset(&P, 0, sizeof(P));
    P.n = n;
    P.inv_gamma = inv_gamma;
    P.srgb = srgb;
    P.linear = linear;
    PoolBuf<uint32_t> keys;
    PoolBuf<PostScratch> scratch;
    if (tonemapped) {
        AZ_CUDA_TRY(keys.alloc(n, st));
        AZ_CUDA_TRY(scratch.alloc(1, st));
        AZ_CUDA_TRY(cudaMemsetAsync(scratch.p, 0, sizeof(PostScratch), st));
        const uint32_t li = (uint32_t)((1.0f - tm->BurnoutPercentage * 0.01f) * (float)(n - 1) + 0.5f);
        const uint32_t rank = std::min(li, n - 1);
        // a block sums and counts at least 8 pixels a thread before it adds to the global sums
        const int grid = std::max(1, std::min(sms * 4, (int)((n + 8 * kPostBlock - 1) / (8 * kPostBlock))));
        k_post_luminance<<<grid, kPostBlock, 0, st>>>(pix, n, keys.p, scratch.p);
        k_post_histogram<1><<<grid, kPostBlock, 0, st>>>(keys.p, n, rank, scratch.p);
        k_post_histogram<2><<<grid, kPostBlock, 0, st>>>(keys.p, n, rank, scratch.p);
        k_post_pick<<<1, kPostBlock, 0, st>>>(rank, scratch.p);
        AZ_CUDA_TRY(cudaGetLastError());
        PostScratch head;   // its first two fields
        AZ_CUDA_TRY(cudaMemcpyAsync(&head, scratch.p, offsetof(PostScratch, hist), cudaMemcpyDeviceToHost, st));
        AZ_CUDA_TRY(cudaStreamSynchronize(st));
        // in float on the host, like azimuth
        const float logavg = expf((float)head.logsum / (float)n);
        P.tonemapped = 1;
        P.factor = tm->KeyValue / logavg;
        P.lw2 = head.white * P.factor;
        P.lw2 = P.lw2 * P.lw2;
        P.saturation = tm->Saturation;
    }
    const int grid = (int)std::min<uint64_t>((uint64_t)sms * 16, ((uint64_t)n + 4 * 128 - 1) / (4 * 128));
    if ((uintptr_t)rgb_out % 16 == 0 && (uintptr_t)rgb8_out % 4 == 0)
        k_post_map<true><<<grid, 128, 0, st>>>(pix, rgb_out, rgb8_out, P);
    else
        k_post_map<false><<<grid, 128, 0, st>>>(pix, rgb_out, rgb8_out, P);
    AZ_CUDA_TRY(cudaGetLastError());
    AZ_CUDA_TRY(cudaStreamSynchronize(st));
    return AZ_OK;
}

}  // namespace az
