// weftk_quadtree.cu — quadtree tiling (variance rule) and tile extraction on the device
// (include/weftk_quadtree.h).
//
// Tiling: one CTA per macro tile.  The macro tile's luminance (float64, the host's expression
// 0.2126 R + 0.7152 G + 0.0722 B on u8 values, left to right) goes to shared memory; one warp per
// candidate square takes its variance (mean, then mean of squared deviations, float64).  The
// reference's depth-first order is the Morton order of the tiles' corners, so one thread per
// smallest square finds the tile it lies in, and a ballot ranks the tiles.  They are staged per
// macro tile; placement CTAs each sum the counts before their own macro tiles and copy.
// Extraction: one CTA per tile, pixels through the host's 256-entry sRGB-decode table, float4 per
// pixel.
// Bound: latency.  1024 x 1024 (256 macro tiles, 7435 tiles): tiling 11 us, placement 3, extraction
// 12; they took 34, 32 and 27 with divisions by the square's side in every step, one thread walking
// the tree, one CTA copying all tiles and a large tile's pixels waited for one by one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/weftk_quadtree.h"
#include "weftk_common.cuh"

namespace weftk {

extern __device__ int g_device_status;

namespace {

constexpr int QT_MAX = 64;                       // largest macro tile side
constexpr int QT_MAX_TILES = (QT_MAX / 8) * (QT_MAX / 8);  // tiles per macro tile, bound
constexpr int QT_PLACE_THREADS = 256, QT_PLACE_CTAS = 512;  // threads of a placement CTA, most CTAs

__device__ __forceinline__ double lum_u8(const uint8_t* p) {
    return __dadd_rn(__dadd_rn(__dmul_rn(0.2126, (double)p[0]), __dmul_rn(0.7152, (double)p[1])),
                     __dmul_rn(0.0722, (double)p[2]));
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// squares of side s > min_tile at every level, level l of side MT >> l, row-major inside a level
__global__ void __launch_bounds__(256) qt_split_kernel(const uint8_t* __restrict__ img, int h, int w, int MT, int mt,
                                                       double thr, int n_mx, int32_t* __restrict__ stage,
                                                       int32_t* __restrict__ counts) {
    __shared__ double lum[QT_MAX * QT_MAX];
    __shared__ unsigned char split[1 + 4 + 16 + 64];
    __shared__ int first_half;
    const int mb = blockIdx.x, my = mb / n_mx, mx = mb - my * n_mx;
    const int x0 = mx * MT, y0 = my * MT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lm = 31 - __clz(MT), depth = lm - (31 - __clz(mt));
#pragma unroll 4
    for (int i = tid; i < MT * MT; i += 256) {
        const int yy = min(y0 + (i >> lm), h - 1), xx = min(x0 + (i & (MT - 1)), w - 1);  // edge padding
        lum[i] = lum_u8(img + ((size_t)yy * w + xx) * 3);
    }
    __syncthreads();
    const int n_sq = ((1 << (2 * depth)) - 1) / 3;  // 1 + 4 + ... squares that may split
    for (int q = warp; q < n_sq; q += 8) {
        int l = 0, base = 0;
        while (q >= base + (1 << (2 * l))) {
            base += 1 << (2 * l);
            ++l;
        }
        const int ls = lm - l, s = 1 << ls, k = q - base;
        const double* sq0 = lum + (((k >> l) << ls) << lm) + ((k & ((1 << l) - 1)) << ls);
        const int n = s * s;
        // (s >= 16, so n is a multiple of 256)
        double sum = 0.0;
#pragma unroll 8
        for (int i = lane; i < n; i += 32) sum += sq0[((i >> ls) << lm) + (i & (s - 1))];
        const double mean = warp_sum_d(sum) / (double)n;
        double sq = 0.0;
#pragma unroll 8
        for (int i = lane; i < n; i += 32) {
            const double d = sq0[((i >> ls) << lm) + (i & (s - 1))] - mean;
            sq += d * d;
        }
        const double var = warp_sum_d(sq) / (double)n;
        if (lane == 0) split[q] = var > thr;
    }
    if (tid == 0) first_half = 0;
    __syncthreads();
    // one thread per smallest square, in Morton order (top-left, top-right, bottom-left, bottom-right)
    if (tid < 64) {
        int x = 0, y = 0, l = 0;  // the square's place in units of mt, the level of its tile
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            x |= ((tid >> (2 * b)) & 1) << b;
            y |= ((tid >> (2 * b + 1)) & 1) << b;
        }
        const bool real = tid < 1 << (2 * depth);
        for (int base = 0; real && l < depth; base += 1 << (2 * l), ++l)
            if (!split[base + ((y >> (depth - l)) << l) + (x >> (depth - l))]) break;
        const int s = MT >> l;
        const bool starts = real && (tid & ((1 << (2 * (depth - l))) - 1)) == 0;
        const unsigned who = __ballot_sync(0xffffffffu, starts);
        if (tid == 0) first_half = __popc(who);
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const int at = __popc(who & ((1u << lane) - 1u)) + (warp ? first_half : 0);
        if (starts) {
            int32_t* o = stage + ((size_t)mb * QT_MAX_TILES + at) * 3;
            o[0] = x0 + x * mt;
            o[1] = y0 + y * mt;
            o[2] = s;
        }
        if (tid == 32) counts[mb] = first_half + __popc(who);
    }
}

// Every CTA takes `per` macro tiles: it sums the counts before them, then each warp copies its macro
// tiles' staged tiles to their place.
__global__ void __launch_bounds__(QT_PLACE_THREADS) qt_place_kernel(const int32_t* __restrict__ stage,
                                                                    const int32_t* __restrict__ counts, int n_macro,
                                                                    int per, int32_t* __restrict__ tiles, int max_tiles,
                                                                    int32_t* __restrict__ n_out) {
    constexpr int NW = QT_PLACE_THREADS / 32;
    __shared__ int wtot[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = blockIdx.x * per, hi = min(n_macro, lo + per);
    auto warp_sum_i = [](int v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    int s = 0;
#pragma unroll 4
    for (int i = tid; i < lo; i += QT_PLACE_THREADS) s += counts[i];
    s = warp_sum_i(s);
    if (lane == 0) wtot[warp] = s;
    __syncthreads();
    int off = 0;
    for (int k = 0; k < NW; ++k) off += wtot[k];
    for (int i0 = lo; i0 < hi; i0 += 32) {  // 32 macro tiles at a time: every warp scans them, then copies its own
        const int c = i0 + lane < hi ? counts[i0 + lane] : 0;
        int v = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        for (int j = warp; j < 32 && i0 + j < hi; j += NW) {
            const int first = off + __shfl_sync(0xffffffffu, v - c, j), n = __shfl_sync(0xffffffffu, c, j);
            const int32_t* src = stage + (size_t)(i0 + j) * QT_MAX_TILES * 3;
            const long long fit = min((long long)n, (long long)max_tiles - first);
            for (long long k = lane; k < 3 * fit; k += 32) tiles[(long long)first * 3 + k] = src[k];
        }
        off += __shfl_sync(0xffffffffu, v, 31);
    }
    if (tid == 0 && hi == n_macro) {
        *n_out = min(off, max_tiles);
        if (off > max_tiles) atomicCAS(&g_device_status, 0, WEFTK_E_RANGE);
    }
}

// one CTA of EX_THREADS per tile (most tiles are 8 px: 64 pixels); the 1 KB sRGB table is read
// through the read-only cache
constexpr int EX_THREADS = 64;

__global__ void __launch_bounds__(EX_THREADS) extract_tiles_kernel(const uint8_t* __restrict__ img, int h, int w,
                                                                   const float* __restrict__ tab,
                                                                   const int32_t* __restrict__ tiles, int n_tiles,
                                                                   const int32_t* __restrict__ px_off,
                                                                   float4* __restrict__ out) {
    const int t = blockIdx.x;
    const int tx = tiles[t * 3], ty = tiles[t * 3 + 1], s = tiles[t * 3 + 2];
    if (s < 1 || s > 64) {
        if (threadIdx.x == 0) atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
        return;
    }
    float4* dst = out + px_off[t];
    const float inv = 1.0f / (float)s;
#pragma unroll 8
    for (int i = threadIdx.x; i < s * s; i += EX_THREADS) {
        const int y = (int)(((float)i + 0.5f) * inv);  // i / s: exact, for i < 4096 and s <= 64
        const int yy = min(ty + y, h - 1), xx = min(tx + i - y * s, w - 1);
        const uint8_t* p = img + ((size_t)yy * w + xx) * 3;
        dst[i] = make_float4(__ldg(tab + p[0]), __ldg(tab + p[1]), __ldg(tab + p[2]), 0.0f);
    }
}

bool pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

}  // namespace
}  // namespace weftk

using namespace weftk;

extern "C" int weftk_quadtree_work_bytes(int h, int w, int max_tile, int min_tile, int64_t* bytes) {
    WEFTK_REQUIRE(bytes && h > 0 && w > 0 && pow2(max_tile) && pow2(min_tile) && min_tile >= 8 &&
                      min_tile <= max_tile && max_tile <= QT_MAX,
                  "quadtree_work_bytes: bad size");
    const int64_t n_macro = (int64_t)((h + max_tile - 1) / max_tile) * ((w + max_tile - 1) / max_tile);
    *bytes = n_macro * (QT_MAX_TILES * 3 + 1) * (int64_t)sizeof(int32_t);
    return WEFTK_OK;
}

extern "C" int weftk_quadtree_variance(const uint8_t* d_img, int h, int w, double threshold, int max_tile,
                                       int min_tile, int32_t* d_tiles, int max_tiles, int32_t* d_n_tiles,
                                       void* d_work, void* stream) {
    int64_t need = 0;
    int rc = weftk_quadtree_work_bytes(h, w, max_tile, min_tile, &need);
    if (rc) return rc;
    WEFTK_REQUIRE(d_img && d_tiles && d_n_tiles && d_work && max_tiles >= 0, "quadtree_variance: null pointer");
    const int n_mx = (w + max_tile - 1) / max_tile, n_my = (h + max_tile - 1) / max_tile;
    const long long n_macro = (long long)n_mx * n_my;
    WEFTK_REQUIRE(n_macro < (1ll << 30), "quadtree_variance: image too large");
    int32_t* stage = static_cast<int32_t*>(d_work);
    int32_t* counts = stage + n_macro * QT_MAX_TILES * 3;
    cudaStream_t s = (cudaStream_t)stream;
    qt_split_kernel<<<(unsigned)n_macro, 256, 0, s>>>(d_img, h, w, max_tile, min_tile, threshold, n_mx, stage, counts);
    WEFTK_CUDA(cudaGetLastError());
    const int per = std::max(8, ceil_div(n_macro, QT_PLACE_CTAS));
    qt_place_kernel<<<ceil_div(n_macro, per), QT_PLACE_THREADS, 0, s>>>(stage, counts, (int)n_macro, per, d_tiles,
                                                                        max_tiles, d_n_tiles);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_extract_tiles(const uint8_t* d_img, int h, int w, const float* d_lut, const int32_t* d_tiles,
                                   int n_tiles, const int32_t* d_px_off, float* d_src4, void* stream) {
    WEFTK_REQUIRE(h > 0 && w > 0 && n_tiles >= 0, "extract_tiles: bad size");
    if (n_tiles == 0) return WEFTK_OK;
    WEFTK_REQUIRE(d_img && d_lut && d_tiles && d_px_off && d_src4, "extract_tiles: null pointer");
    extract_tiles_kernel<<<n_tiles, EX_THREADS, 0, (cudaStream_t)stream>>>(d_img, h, w, d_lut, d_tiles, n_tiles, d_px_off,
                                                                     reinterpret_cast<float4*>(d_src4));
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}
