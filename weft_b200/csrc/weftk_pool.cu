// weftk_pool.cu — initial constant / linear candidate pools generated on the device
// (include/weftk_pool.h).
//
// One CTA per tile, launched per tile side so that shared memory is sized for it.  The
// stages follow the reference's per-tile worker (src/weft/encoder.py:2490-2517):
//   1. pixels into shared memory as three channel planes; float32 luminance;
//   2. the reference's Sobel (src/weft/edge_analysis.py:17-41: every tap of its offset slices
//      reads lum[y-1][x-1], summed tap by tap in float32), magnitude, angle in [0, pi); all but
//      the pixels of two columns lie on an axis, whose bins are taken once, so the float64 arctan2
//      runs over a compacted list of the others;
//   3. orientation histogram: pixels counting-sorted by bin (stable, raster order inside a
//      bin), then numpy's pairwise float32 sum per bin; the dominant orientations;
//   4. luminance sorted by (value, pixel index) for the palette runs and the 25th / 75th
//      percentiles (64-bit keys in registers, exchanged by shuffles, through shared memory only
//      across warps); the np.gradient magnitude and its 75th percentile by rank selection;
//   5. every mean the two generators take, as numpy computes it: a sequential float32 sum per
//      channel in the reference's pixel order (raster, or luminance order for palette runs),
//      divided by the count in float32 — one thread per region or split line (both of its
//      sides in one pass over the pixels, the side test read from a table built once per
//      quality) and one to three channels; four pixels per shared-memory read and one predicated
//      addition per pixel, side and channel;
//   6. the palettes (the colours' pairwise near tests in parallel, the keep walk on one
//      thread);
//   7. de-duplication by the reference's coarse key.  A colour or line enters the list with a fixed set
//      of alphas, and sets that share an alpha are one group, so whole units (a colour, a line) are
//      repeats, not single candidates: each unit is compared with the earlier ones of its group on a
//      packed key; the surviving records are staged per warp and written in whole words.
//
// Bound: instruction issue and latency at 8 px (11 thousand warp instructions a tile, two warps, so the
// scratch is kept small for 16 CTAs a SM), one CTA's latency at 64 px (the sequential sums: 4096 dependent
// additions are 9 us).  A 1024 x 1024 picture's 6122 / 1048 / 227 / 38 tiles of 8 / 16 / 32 / 64 px take
// 100 / 44 / 50 / 78 us launched alone, and took 125 / 58 / 77 / 173 with arctan2 at every pixel, a sort
// through shared memory, gathered palette sums and every candidate its own key and hash-table entry.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <set>

#include "../../include/weftk_pool.h"
#include "weftk_common.cuh"

static_assert(sizeof(WeftPoolTables) == 64, "WeftPoolTables layout is part of the C ABI");

namespace weftk {

extern __device__ int g_device_status;

namespace {

constexpr int NB = 12;                           // orientation histogram bins
constexpr int MAXC = WEFTK_POOL_MAX_CONST_LINEAR;
constexpr int NSPL = WEFTK_POOL_SPLITS;          // split rows per tile side in the side-bit table
constexpr int NFIX = 33;                         // fixed regions (below)
constexpr int MAXPAL = 16;
constexpr int NCOL = 13;                         // palette colours tested: tile mean + regions 21..32

// Fixed regions whose means are taken: 0 the tile, 1..4 its quadrants, 5..20 its 4x4 blocks
// (row-major), 21..29 the palette runs of the luminance order (2, 3 and 4 equal runs), 30
// luminance above its 75th percentile, 31 below its 25th, 32 np.gradient magnitude at or above
// its 75th.  Split lines (both sides) are kept apart: the dominant orientations' centre lines,
// then the template lines.

// A unit of the candidate list: a colour or a split line, listed with each alpha of its group.
constexpr int MAXU = MAXPAL + 4 + 3 * NB + 16 + WEFTK_POOL_MAX_SPECS;
static_assert(MAXU < 256, "a unit's index fits a byte");

// per-tile scratch besides the pixel planes (static part of the shared memory)
template <int N>
struct Scratch {
    float rmean[NFIX][3];     // sum / count in float32 (0 for an empty region)
    int rcnt[NFIX];
    float smean[NSPL][2][3];  // per split line in use: side a, side b (0 for an empty side)
    int scnt[NSPL];           // pixels on side a
    double edges[NB + 1];
    float hist[NB];
    int bin_start[NB + 1];
    int peaks[NB];
    int axis_bin[3];          // bins of the angles of (+-x, 0), (0, +y), (0, -y)
    int n_peaks, n_split, n_pend;
    float p25, p75, pm75;
    unsigned tmask[3][N / 32];  // pixels above the 75th / below the 25th luminance percentile, gradient >= its 75th
    // palettes (the template palette extends the edge palette) and the candidate list's segments
    float cpal[NCOL][3];
    unsigned near_mask[NCOL];
    float pal[MAXPAL][3];
    int npal_e, npal_t;
    ulonglong2 key[MAXU];     // x: line, colour 0's low 20 bits; y: its rest, colour 1, group, BAD_KEY
    int bad;                  // some unit's key does not pack
    int place[MAXU], wtot[(MAXU + 31) / 32 + 16];
    unsigned short rec_of[MAXC];
    int n_out;
    int wcnt[16][NB];
    int sel[N <= 64 ? 64 : 260];  // rank selection: histogram, bin, count before, count (or N sorted values)
};

__device__ __forceinline__ float clamp01(float v) { return fmaxf(0.0f, fminf(1.0f, v)); }

// numpy's pairwise float32 summation of x[0..n) (the contiguous add-reduce loop: fewer than 8
// sequentially, up to 128 with 8 accumulators combined pairwise, larger halves split at a
// multiple of 8), each addition rounded on its own.  pairwise_block is a leaf, or all of n <= 128.
// x[i] stands at word i + i / 128, so that lanes on leaves 128 elements apart read different banks.
__device__ __forceinline__ int spread(int i) { return i + (i >> 7); }

__device__ float pairwise_block(const float* x, int at, int n) {
    auto get = [&](int i) { return x[spread(at + i)]; };
    if (n < 8) {
        float r = -0.0f;
        for (int i = 0; i < n; ++i) r = __fadd_rn(r, get(i));
        return r;
    }
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = get(j);
    int i = 8;
    for (; i < n - (n % 8); i += 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) r[j] = __fadd_rn(r[j], get(i + j));
    }
    float res = __fadd_rn(__fadd_rn(__fadd_rn(r[0], r[1]), __fadd_rn(r[2], r[3])),
                          __fadd_rn(__fadd_rn(r[4], r[5]), __fadd_rn(r[6], r[7])));
    for (; i < n; ++i) res = __fadd_rn(res, get(i));
    return res;
}

// The same sum by a whole warp (every lane gets it), n <= 8192: numpy splits n > 128 elements at half,
// rounded down to a multiple of 8, and adds the halves' sums.  A lane walks down to two of the 64
// depth-6 positions, sums the leaf there if its path is the leaf's first, and the halves meet level by
// level.
__device__ float warp_pairwise_sum(const float* x, int at, int n, int lane) {
    float v[2];
    unsigned inner = 0;  // levels at which the lane's (first) path is still an inner node
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int path = 2 * lane + h;
        int off = at, len = n, d = 0;
        for (; d < 6 && len > 128; ++d) {
            if (h == 0) inner |= 1u << d;
            int half = len / 2;
            half -= half % 8;
            if ((path >> (5 - d)) & 1) {
                off += half;
                len -= half;
            } else {
                len = half;
            }
        }
        const bool first = (path & ((1 << (6 - d)) - 1)) == 0;  // of the paths below this leaf
        v[h] = first ? pairwise_block(x, off, len) : 0.0f;
    }
    if ((inner >> 5) & 1u) v[0] = __fadd_rn(v[0], v[1]);
#pragma unroll
    for (int d = 4; d >= 0; --d) {
        const float right = __shfl_down_sync(0xffffffffu, v[0], 1 << (4 - d));
        if ((inner >> d) & 1u) v[0] = __fadd_rn(v[0], right);
    }
    return __shfl_sync(0xffffffffu, v[0], 0);
}

// side test of the reference's split: (x - x0) * (y1 - y0) - (y - y0) * (x1 - x0) >= 0 in float32
__device__ __forceinline__ bool side_a(float4 c, int x, int y) {
    const float t = __fsub_rn(__fmul_rn(__fsub_rn((float)x, c.x), c.z), __fmul_rn(__fsub_rn((float)y, c.y), c.w));
    return t >= 0.0f;
}

// sum over (a - b)^2 < 0.002 in float64, as the reference's palette test (Python floats)
__device__ bool near_pair(const float* c, const float* p) {
    double s = 0.0;
    for (int k = 0; k < 3; ++k) {
        const double d = __dsub_rn((double)c[k], (double)p[k]);
        s = __dadd_rn(s, __dmul_rn(d, d));
    }
    return s < 0.002;
}

__device__ __forceinline__ int qkey(double v, double s) { return (int)(long long)__dadd_rn(__dmul_rn(v, s), 0.5); }

// Dynamic shared memory of one tile of N pixels: seven float planes (r, g, b, luminance, the
// np.gradient magnitude, the Sobel magnitude, a sort key), the sorted pixel indices, the bins.
constexpr size_t POOL_FLOAT_PLANES = 7;
// At the end the records are staged there, 32 per warp.
__host__ __device__ constexpr size_t pool_smem_bytes(int n, int warps) {
    const size_t planes = (size_t)n * (POOL_FLOAT_PLANES * sizeof(float) + sizeof(int) + sizeof(uint8_t));
    const size_t stage = (size_t)warps * 32 * sizeof(WeftPrim);
    return planes > stage ? planes : stage;
}

// words of the side-bit table before tile side TS (8, 16, 32, 64), per split row
template <int TS>
__host__ __device__ constexpr int side_words_before() {
    return TS == 8 ? 0 : TS == 16 ? 2 : TS == 32 ? 10 : 42;
}

// run [a, b) of the luminance order behind palette region r (21..29: 2, 3 and 4 equal runs)
__device__ __forceinline__ void run_bounds(const int32_t* cuts, int si, int r, int& a, int& b) {
    const int j = r - 21;
    const int k = j < 2 ? 0 : j < 5 ? 1 : 2;
    const int jj = j - (k == 0 ? 0 : k == 1 ? 2 : 5);
    const int32_t* cut = cuts + (si * 3 + k) * 5;
    a = cut[jj];
    b = cut[jj + 1];
}

// A key's geometry and colour fields are packed (11 and 12 bits each, signed by offset) when each lies in
// its field's range; BAD_KEY marks one that does not pack, whose equality is then decided on the
// unpacked fields.
constexpr unsigned long long BAD_KEY = 1ull << 63;

// int(v * 64 + 0.5) of a colour: the product is exact in float32, so the sum is compared instead of
// rounded where the value is an ordinary one.
__device__ __forceinline__ int colour_key(float v) {
    if (v >= 0.0f && v < 30.0f) {
        const float t = v * 64.0f;
        const int k = (int)t;
        return k + (t - (float)k >= 0.5f);
    }
    return qkey((double)v, 64.0);
}

__device__ __forceinline__ unsigned long long pack_field(int v, int bits, bool& ok) {
    const int off = 1 << (bits - 1);
    ok = ok && v >= -off && v < off;
    return (unsigned long long)(unsigned)(v + off) & ((1ull << bits) - 1ull);
}

__device__ __forceinline__ unsigned long long pack_colour(float r, float g, float b) {
    bool ok = true;
    const unsigned long long k = pack_field(colour_key(r), 12, ok) | (pack_field(colour_key(g), 12, ok) << 12) |
                                 (pack_field(colour_key(b), 12, ok) << 24);
    return ok ? k : BAD_KEY;
}

__device__ __forceinline__ unsigned long long pack_line(const double* g) {
    bool ok = true;
    unsigned long long k = 0;
    for (int j = 0; j < 4; ++j) k |= pack_field(qkey(g[j], 4.0), 11, ok) << (11 * j);
    return ok ? k : BAD_KEY;
}

// Adds v to the sums of the side that bit `bit` of `word` names (predicated: a side's sum is left
// alone, not added zero to; the same value).
__device__ __forceinline__ void add_side(float (&a)[3], float (&b)[3], float v0, float v1, float v2, unsigned word,
                                         unsigned bit) {
    asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %6, %7;\n\tsetp.ne.b32 p, t, 0;\n\t"
        "@p add.rn.f32 %0, %0, %8;\n\t@p add.rn.f32 %1, %1, %9;\n\t@p add.rn.f32 %2, %2, %10;\n\t"
        "@!p add.rn.f32 %3, %3, %8;\n\t@!p add.rn.f32 %4, %4, %9;\n\t@!p add.rn.f32 %5, %5, %10;\n\t}"
        : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(b[0]), "+f"(b[1]), "+f"(b[2])
        : "r"(word), "r"(bit), "f"(v0), "f"(v1), "f"(v2));
}
__device__ __forceinline__ void add_side(float (&a)[1], float (&b)[1], float v, unsigned word, unsigned bit) {
    asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %2, %3;\n\tsetp.ne.b32 p, t, 0;\n\t"
        "@p add.rn.f32 %0, %0, %4;\n\t@!p add.rn.f32 %1, %1, %4;\n\t}"
        : "+f"(a[0]), "+f"(b[0])
        : "r"(word), "r"(bit), "f"(v));
}
__device__ __forceinline__ void add_in(float& a, float v, unsigned word, unsigned bit) {
    asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.b32 p, t, 0;\n\t"
        "@p add.rn.f32 %0, %0, %3;\n\t}"
        : "+f"(a)
        : "r"(word), "r"(bit), "f"(v));
}

// A float's bits in an order unsigned integers have (zeros alike); NaN past the infinities.
__device__ __forceinline__ unsigned ordered_bits(float v) {
    const unsigned u = __float_as_uint(v == 0.0f ? 0.0f : v);
    return u ^ ((unsigned)((int)u >> 31) | 0x80000000u);
}

// Bitonic sort of N 64-bit keys by NT threads, E = N / NT consecutive ones in each thread's registers:
// strides inside a thread by compare, inside a warp by shuffle, across warps through ex[N].
// One warp (NT = 32, tid = lane) needs no ex.
template <int N, int NT, class K>
__device__ void block_sort(K (&v)[N / NT], K* ex, int tid) {
    constexpr int E = N / NT;
    for (int k = 2; k <= N; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (NT > 32 && j >= 32 * E) {
                __syncthreads();  // the last reads of ex
#pragma unroll
                for (int e = 0; e < E; ++e) ex[e * NT + tid] = v[e];
                __syncthreads();
                const int other = tid ^ (j / E);
                const bool low = ((tid * E) & j) == 0, up = ((tid * E) & k) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const K o = ex[e * NT + other];
                    v[e] = (low == up) == (v[e] < o) ? v[e] : o;
                }
            } else if (j >= E) {
                const bool low = ((tid * E) & j) == 0, up = ((tid * E) & k) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const K o = __shfl_xor_sync(0xffffffffu, v[e], j / E);
                    v[e] = (low == up) == (v[e] < o) ? v[e] : o;
                }
            } else {
#pragma unroll
                for (int jj = E / 2; jj > 0; jj >>= 1) {
                    if (jj != j) continue;
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        if (e & jj) continue;
                        const bool up = ((tid * E + e) & k) == 0;
                        const K a = v[e], b = v[e | jj];
                        const bool swap = (a > b) == up;
                        v[e] = swap ? b : a;
                        v[e | jj] = swap ? a : b;
                    }
                }
            }
        }
    }
}

// Values of ranks r and r + 1 (ascending) among x[0..n), all >= 0 (NaN past the infinities), by the
// whole CTA: the bits are found eight at a time from a histogram of the values that share the bits
// found so far.  h: 256 + 3 words of scratch.
template <int NT>
__device__ void rank_pair(const float* x, int n, int r, int* h, float& lo, float& hi) {
    const int tid = threadIdx.x;
    unsigned prefix = 0, mask = 0;
    int rank = r, count = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        __syncthreads();
        for (int i = tid; i < 256; i += NT) h[i] = 0;
        __syncthreads();
        for (int p = tid; p < n; p += NT) {
            const unsigned u = __float_as_uint(x[p]);
            const bool in = (u & mask) == prefix;
            const unsigned b = (u >> shift) & 255u;
            // the first digits are shared by almost every value: one addition per distinct digit
            const unsigned peers = __match_any_sync(__activemask(), in ? b : 256u);
            if (in && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[b], __popc(peers));
        }
        __syncthreads();
        if (tid < 32) {
            int c[8], run = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                c[k] = h[tid * 8 + k];
                run += c[k];
            }
            int incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            int before = incl - run;
            if (rank >= before && rank < incl) {
                int k = 0;
#pragma unroll
                for (int q = 0; q < 7; ++q)
                    if (k == q && rank >= before + c[q]) {
                        before += c[q];
                        k = q + 1;
                    }
                h[256] = tid * 8 + k;
                h[257] = before;
                h[258] = h[tid * 8 + k];
            }
        }
        __syncthreads();
        prefix |= (unsigned)h[256] << shift;
        mask |= 255u << shift;
        rank -= h[257];
        count = h[258];
    }
    lo = __uint_as_float(prefix);
    hi = lo;
    if (rank + 1 < count || r + 1 >= n) return;  // the next rank holds the same value (uniform)
    unsigned next = 0xffffffffu;
    for (int p = tid; p < n; p += NT) {
        const unsigned u = __float_as_uint(x[p]);
        if (u > prefix) next = min(next, u);
    }
    next = __reduce_min_sync(0xffffffffu, next);
    __syncthreads();
    if ((tid & 31) == 0) h[tid >> 5] = (int)next;
    __syncthreads();
    next = (unsigned)h[0];
    for (int w = 1; w < NT / 32; ++w) next = min(next, (unsigned)h[w]);
    hi = __uint_as_float(next);
}

// numpy's linear percentile between the values a, b of ranks floor(vi), floor(vi) + 1 (float32)
__device__ __forceinline__ float percentile_rank(int n, int q, int& lo, float& g) {
    const float vi = __fmul_rn((float)(n - 1), __fdiv_rn((float)q, 100.0f));
    lo = (int)floorf(vi);
    g = __fsub_rn(vi, (float)lo);
    return vi;
}
__device__ __forceinline__ float percentile_lerp(float a, float b, float g) {
    const float d = __fsub_rn(b, a);
    return g >= 0.5f ? __fsub_rn(b, __fmul_rn(d, __fsub_rn(1.0f, g))) : __fadd_rn(a, __fmul_rn(d, g));
}

// the reference's Sobel at pixel p: gx[y][x] = sum over the taps (dy, dx) whose slices reach (y, x) of
// k[dy][dx] * lum[y-1][x-1]; rows reached: dy 0 -> 1..TS-2, 1 -> 1..TS-1, 2 -> 2..TS-1 (columns alike)
template <int TS>
__device__ __forceinline__ void sobel(const float* lum, int p, float& gx, float& gy) {
    constexpr float KX[9] = {-1, 0, 1, -2, 0, 2, -1, 0, 1};
    constexpr float KY[9] = {-1, -2, -1, 0, 0, 0, 1, 2, 1};
    const int y = p / TS, x = p % TS;
    gx = 0.0f;
    gy = 0.0f;
    if (y >= 1 && x >= 1) {
        const float L = lum[(y - 1) * TS + (x - 1)];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const bool row = dy == 0 ? (y <= TS - 2) : dy == 1 ? true : (y >= 2);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const bool cl = dx == 0 ? (x <= TS - 2) : dx == 1 ? true : (x >= 2);
                if (row && cl) {
                    gx = __fadd_rn(gx, __fmul_rn(KX[dy * 3 + dx], L));
                    gy = __fadd_rn(gy, __fmul_rn(KY[dy * 3 + dx], L));
                }
            }
        }
    }
}

// histogram bin of a gradient: arctan2 rounded to float32, numpy's float32 % pi, NB for no bin (NaN)
__device__ int angle_bin(float gx, float gy, const double* edges) {
    const float PI32 = 3.14159274101257324f;  // float32(pi): numpy casts the Python float
    const float ang = (float)atan2((double)gy, (double)gx);
    float m = fmodf(ang, PI32);
    if (m != 0.0f) {
        if (m < 0.0f) m = __fadd_rn(m, PI32);
    } else {
        m = 0.0f;
    }
    const double md = (double)m;
    for (int i = 0; i < NB; ++i)
        if (md >= edges[i] && md < edges[i + 1]) return i;
    return NB;
}

template <int TS, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) gen_pool_kernel(WeftPoolTables tb, WeftPoolJob job, int si) {
    constexpr int N = TS * TS;
    constexpr int NW = NT / 32;
    constexpr int WPS = N / 32;             // side-bit words per split row
    constexpr int CH = TS <= 16 ? 3 : 1;    // channels summed by one thread
    constexpr int G = 3 / CH;
    constexpr int LOG_TS = TS == 8 ? 3 : TS == 16 ? 4 : TS == 32 ? 5 : 6;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* col = reinterpret_cast<float*>(smem_raw);  // [3][N]
    float* lum = col + 3 * N;                         // [N]
    float* magt = lum + N;                            // [N] np.gradient magnitude
    float* mags = magt + N;                           // [N] Sobel magnitude, then sorted magt
    float* skey = mags + N;                           // [N] bin-sorted magnitudes (spread, into sidx)
    int* sidx = reinterpret_cast<int*>(skey + N);     // [N] pixel of each sorted luminance
    uint8_t* bin = reinterpret_cast<uint8_t*>(sidx + N);  // [N]
    static_assert(POOL_FLOAT_PLANES == 7, "the planes above are col[3], lum, magt, mags, skey");
    static_assert(NW <= 16, "the histogram's per-warp counters hold 16 warps");
    static_assert(N % 32 == 0 && NT % 32 == 0, "whole words and warps");
    __shared__ Scratch<N> S;

    const int t = job.tiles[si][blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool want0 = job.kinds_mask & 1, want1 = job.kinds_mask & 2;

    // 1. pixels and luminance 0.2126 r + 0.7152 g + 0.0722 b (float32, left to right)
    if (tid <= NB) S.edges[tid] = tb.bin_edges[tid];
    const float4* src = reinterpret_cast<const float4*>(job.src) + job.px_off[t];
    for (int p = tid; p < N; p += NT) {
        const float4 v = src[p];
        col[p] = v.x;
        col[N + p] = v.y;
        col[2 * N + p] = v.z;
        lum[p] = __fadd_rn(__fadd_rn(__fmul_rn(0.2126f, v.x), __fmul_rn(0.7152f, v.y)), __fmul_rn(0.0722f, v.z));
    }
    __syncthreads();

    // 2. Sobel magnitude and orientation bin; np.gradient (template): central differences / 2 inside,
    //    one-sided at the edges.  gx is exactly 0 but in columns 1 and TS - 1 (the taps cancel), so
    //    nearly every angle is one of (+-x, 0), (0, +y), (0, -y); the rest goes to a list (in sidx)
    if (tid < 3) S.axis_bin[tid] = angle_bin(tid == 0 ? 1.0f : 0.0f, tid == 0 ? 0.0f : tid == 1 ? 1.0f : -1.0f, S.edges);
    if (tid == 0) S.n_pend = 0;
    __syncthreads();
    const int bin_x = S.axis_bin[0], bin_up = S.axis_bin[1], bin_down = S.axis_bin[2];
    for (int p = tid; p < N; p += NT) {
        const int y = p / TS, x = p % TS;
        float gx, gy;
        sobel<TS>(lum, p, gx, gy);
        mags[p] = __fsqrt_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)));
        // (0, 0), (+-x, 0): angle 0 or pi, 0 after % pi
        const bool pend = !(gy == 0.0f && gx == gx) && !(gx == 0.0f && gy == gy);
        bin[p] = (uint8_t)(gy == 0.0f ? bin_x : gy > 0.0f ? bin_up : bin_down);
        const unsigned who = __ballot_sync(0xffffffffu, pend);
        if (who) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&S.n_pend, __popc(who));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (pend) sidx[at + __popc(who & ((1u << lane) - 1u))] = p;
        }
        // np.gradient along rows (gy) and columns (gx)
        const float* L = lum;
        const float ty = y == 0 ? __fsub_rn(L[TS + x], L[x])
                         : y == TS - 1 ? __fsub_rn(L[p], L[p - TS])
                                       : __fmul_rn(__fsub_rn(L[p + TS], L[p - TS]), 0.5f);
        const float tx = x == 0 ? __fsub_rn(L[p + 1], L[p])
                         : x == TS - 1 ? __fsub_rn(L[p], L[p - 1])
                                       : __fmul_rn(__fsub_rn(L[p + 1], L[p - 1]), 0.5f);
        magt[p] = __fsqrt_rn(__fadd_rn(__fmul_rn(tx, tx), __fmul_rn(ty, ty)));
    }
    __syncthreads();
    for (int i = tid; i < S.n_pend; i += NT) {
        const int p = sidx[i];
        float gx, gy;
        sobel<TS>(lum, p, gx, gy);
        bin[p] = (uint8_t)angle_bin(gx, gy, S.edges);
    }
    for (int i = tid; i < 16 * NB; i += NT) (&S.wcnt[0][0])[i] = 0;
    if (tid == 0) S.n_peaks = 0;
    __syncthreads();

    // 3. histogram: stable counting sort of the Sobel magnitudes by bin into skey
    if (want1) {
        constexpr int CHUNK = N / NW;
        const int lo = warp * CHUNK;
        for (int base = lo; base < lo + CHUNK; base += 32) {
            const int b = bin[base + lane];
            const unsigned m = __match_any_sync(0xffffffffu, b);
            if (lane == __ffs(m) - 1 && b < NB) S.wcnt[warp][b] += __popc(m);
            __syncwarp();
        }
        __syncthreads();
        if (warp == 0) {  // exclusive sums in (bin, warp) order: a lane per bin, its warps in turn
            int c[NW], sum = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                c[w] = lane < NB ? S.wcnt[w][lane] : 0;
                sum += c[w];
            }
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            int at = incl - sum;
            if (lane < NB) {
                S.bin_start[lane] = at;
                if (lane == NB - 1) S.bin_start[NB] = incl;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    S.wcnt[w][lane] = at;
                    at += c[w];
                }
            }
        }
        __syncthreads();
        for (int base = lo; base < lo + CHUNK; base += 32) {
            const int b = bin[base + lane];
            const unsigned m = __match_any_sync(0xffffffffu, b);
            if (b < NB) skey[spread(S.wcnt[warp][b] + __popc(m & ((1u << lane) - 1u)))] = mags[base + lane];
            __syncwarp();
            if (lane == __ffs(m) - 1 && b < NB) S.wcnt[warp][b] += __popc(m);
            __syncwarp();
        }
        __syncthreads();
        if (N <= 128) {  // every bin is one leaf
            if (tid < NB) S.hist[tid] = pairwise_block(skey, S.bin_start[tid], S.bin_start[tid + 1] - S.bin_start[tid]);
        } else {
            for (int b = warp; b < NB; b += NW) {
                const float h = warp_pairwise_sum(skey, S.bin_start[b], S.bin_start[b + 1] - S.bin_start[b], lane);
                if (lane == 0) S.hist[b] = h;
            }
        }
        __syncthreads();
        if (tid == 0) {
            float hmax = S.hist[0];
            for (int i = 1; i < NB; ++i) hmax = fmaxf(hmax, S.hist[i]);
            int np = 0;
            if (hmax < 1e-6f) {
                for (int i = 0; i < 4; ++i) S.peaks[np++] = NB + i;
            } else {
                const float thr = __fmul_rn(hmax, 0.2f);
                for (int i = 0; i < NB; ++i)
                    if (S.hist[i] >= thr) S.peaks[np++] = i;
            }
            S.n_peaks = np;
        }
    }

    // 4. luminance sorted by (value, index), its percentiles and the gradient's; the colours in that order
    float* srt = magt;  // [3][N]: the planes magt, mags, skey, once they are done with
    {
        int lo75;
        float g75, ma = 0.0f, mb = 0.0f;
        percentile_rank(N, 75, lo75, g75);
        __syncthreads();  // skey's and mags's readers
        if constexpr (NT == 64) {  // 8 px: one warp sorts the luminance, the other the gradient
            if (warp == 0) {
                unsigned long long v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    v[e] = ((unsigned long long)ordered_bits(lum[lane * 2 + e]) << 32) | (unsigned)(lane * 2 + e);
                block_sort<N, 32>(v, static_cast<unsigned long long*>(nullptr), lane);
                sidx[lane * 2] = (int)(unsigned)v[0];
                sidx[lane * 2 + 1] = (int)(unsigned)v[1];
            } else {
                unsigned v[2] = {__float_as_uint(magt[lane * 2]), __float_as_uint(magt[lane * 2 + 1])};  // >= 0
                block_sort<N, 32>(v, static_cast<unsigned*>(nullptr), lane);
                S.sel[lane * 2] = (int)v[0];
                S.sel[lane * 2 + 1] = (int)v[1];
            }
            __syncthreads();
            ma = __int_as_float(S.sel[lo75]);
            mb = __int_as_float(S.sel[min(lo75 + 1, N - 1)]);
        } else {
            constexpr int E = N / NT;
            unsigned long long* ex = reinterpret_cast<unsigned long long*>(skey);  // skey and sidx: N words each
            unsigned long long v[E];
#pragma unroll
            for (int e = 0; e < E; ++e)
                v[e] = ((unsigned long long)ordered_bits(lum[tid * E + e]) << 32) | (unsigned)(tid * E + e);
            block_sort<N, NT>(v, ex, tid);
            __syncthreads();
#pragma unroll
            for (int e = 0; e < E; ++e) sidx[tid * E + e] = (int)(unsigned)v[e];
            rank_pair<NT>(magt, N, lo75, S.sel, ma, mb);
            __syncthreads();
        }
        if (tid < 2) {
            int lo;
            float g;
            percentile_rank(N, tid ? 75 : 25, lo, g);
            (tid ? S.p75 : S.p25) = percentile_lerp(lum[sidx[lo]], lum[sidx[min(lo + 1, N - 1)]], g);
        }
        if (tid == 0) {
            S.pm75 = percentile_lerp(ma, mb, g75);
            S.n_split = want1 ? S.n_peaks + tb.n_spec : 0;
        }
    }
    __syncthreads();
    // membership of the three percentile regions, one bit per pixel
    for (int base = warp * 32; base < N; base += NT) {
        const int p = base + lane;
        const float l = lum[p], g = magt[p];
        const unsigned gt = __ballot_sync(0xffffffffu, l > S.p75);
        const unsigned lt = __ballot_sync(0xffffffffu, l < S.p25);
        const unsigned ge = __ballot_sync(0xffffffffu, g >= S.pm75);
        if (lane == 0) {
            S.tmask[0][base >> 5] = gt;
            S.tmask[1][base >> 5] = lt;
            S.tmask[2][base >> 5] = ge;
        }
    }
    __syncthreads();
    for (int p = tid; p < N; p += NT) {
        const int from = sidx[p];
#pragma unroll
        for (int c = 0; c < 3; ++c) srt[c * N + p] = col[c * N + from];
    }
    __syncthreads();

    // 5. every mean's sum, as numpy takes it: a sequential float32 sum per channel in the
    //    reference's pixel order.  One thread per split line (both sides: the side test read from
    //    the side-bit table) or fixed region, over CH channels; split lines are the dominant
    //    orientations' centre lines, then the template lines.  Jobs come in three groups, each
    //    starting on a warp boundary so a warp runs one loop shape: split lines; whole-tile
    //    scans (the three percentile regions and the tile); index runs (palette runs of the
    //    luminance order, quadrants, 4x4 blocks).  numpy adds the pixels outside a region as +0.0,
    //    which leaves a sum that starts at +0.0 unchanged (round to nearest never makes it -0.0), so
    //    they are not added.
    {
        const int nsplit = S.n_split;
        constexpr int NSCAN = 4, NRUN = NFIX - NSCAN;
        const int la = (nsplit * G + 31) & ~31, lb = (NSCAN * G + 31) & ~31, lc = (NRUN * G + 31) & ~31;
        const uint32_t* sbits = tb.side_bits + side_words_before<TS>() * NSPL;
        for (int slot = tid; slot < la + lb + lc; slot += NT) {
            const int grp = slot < la ? 0 : slot < la + lb ? 1 : 2;
            const int j = slot - (grp == 0 ? 0 : grp == 1 ? la : la + lb);
            const int nj = grp == 0 ? nsplit : grp == 1 ? NSCAN : NRUN;
            if (j >= nj * G) continue;  // padding up to the warp boundary
            const int cg = j / nj, u = j - cg * nj, c0 = cg * CH;  // channel-major with one channel per thread
            float sa[CH], sb[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) sa[c] = sb[c] = 0.0f;
            const float4* plane = reinterpret_cast<const float4*>(col + c0 * N);
            if (grp == 0) {
                const int row = u < S.n_peaks ? S.peaks[u] : 16 + (u - S.n_peaks);
                const uint32_t* m = sbits + row * WPS;
                int ca = 0;
                uint32_t next = __ldg(m);
                for (int w = 0; w < WPS; ++w) {
                    const uint32_t word = next;
                    if (w + 1 < WPS) next = __ldg(m + w + 1);
                    ca += __popc(word);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 v0 = plane[w * 8 + q];
                        const float x0[4] = {v0.x, v0.y, v0.z, v0.w};
                        if constexpr (CH == 3) {
                            const float4 v1 = plane[N / 4 + w * 8 + q], v2 = plane[N / 2 + w * 8 + q];
                            const float x1[4] = {v1.x, v1.y, v1.z, v1.w}, x2[4] = {v2.x, v2.y, v2.z, v2.w};
#pragma unroll
                            for (int b = 0; b < 4; ++b) add_side(sa, sb, x0[b], x1[b], x2[b], word, 1u << (q * 4 + b));
                        } else {
#pragma unroll
                            for (int b = 0; b < 4; ++b) add_side(sa, sb, x0[b], word, 1u << (q * 4 + b));
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    S.smean[u][0][c0 + c] = ca > 0 ? __fdiv_rn(sa[c], (float)ca) : 0.0f;
                    S.smean[u][1][c0 + c] = ca < N ? __fdiv_rn(sb[c], (float)(N - ca)) : 0.0f;
                }
                if (c0 == 0) S.scnt[u] = ca;
            } else if (grp == 1) {  // above the 75th / below the 25th luminance percentile, gradient
                                    // at or above its 75th, the whole tile: raster order
                const int r = u < 3 ? 30 + u : 0;
                int cnt = 0;
                for (int w = 0; w < WPS; ++w) {
                    const uint32_t word = r == 0 ? 0xffffffffu : S.tmask[r - 30][w];
                    cnt += __popc(word);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
#pragma unroll
                        for (int c = 0; c < CH; ++c) {
                            const float4 v = plane[c * (N / 4) + w * 8 + q];
                            add_in(sa[c], v.x, word, 1u << (q * 4));
                            add_in(sa[c], v.y, word, 1u << (q * 4 + 1));
                            add_in(sa[c], v.z, word, 1u << (q * 4 + 2));
                            add_in(sa[c], v.w, word, 1u << (q * 4 + 3));
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < CH; ++c) S.rmean[r][c0 + c] = cnt > 0 ? __fdiv_rn(sa[c], (float)cnt) : 0.0f;
                if (c0 == 0) S.rcnt[r] = cnt;
            } else {  // palette run [a, b) of the luminance order, or a quadrant / 4x4 block row by row:
                      // `rows` runs of `len` neighbours, `pitch` apart
                const int r = u < 9 ? 21 + u : u - 8;
                int at = 0, len, rows = 1;
                const float* from = col + c0 * N;
                if (r >= 21) {
                    int b;
                    run_bounds(tb.cuts, si, r, at, b);
                    len = b > at ? b - at : 0;
                    from = srt + c0 * N;
                } else {
                    const int lg = r <= 4 ? LOG_TS - 1 : LOG_TS - 2;  // side TS/2 or TS/4
                    const int q = r <= 4 ? r - 1 : r - 5, per = r <= 4 ? 2 : 4;
                    at = ((q / per) << lg) * TS + ((q % per) << lg);
                    rows = len = 1 << lg;
                }
                const int total = rows * len;
                for (int row = 0; row < rows; ++row, at += TS) {
                    int k = at;
                    const int end = at + len, head = min((at + 3) & ~3, end);
                    for (; k < head; ++k)
#pragma unroll
                        for (int c = 0; c < CH; ++c) sa[c] = __fadd_rn(sa[c], from[c * N + k]);
#pragma unroll 2
                    for (; k + 4 <= end; k += 4)
#pragma unroll
                        for (int c = 0; c < CH; ++c) {
                            const float4 v = *reinterpret_cast<const float4*>(from + c * N + k);
                            sa[c] = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sa[c], v.x), v.y), v.z), v.w);
                        }
                    for (; k < end; ++k)
#pragma unroll
                        for (int c = 0; c < CH; ++c) sa[c] = __fadd_rn(sa[c], from[c * N + k]);
                }
#pragma unroll
                for (int c = 0; c < CH; ++c) S.rmean[r][c0 + c] = total > 0 ? __fdiv_rn(sa[c], (float)total) : 0.0f;
                if (c0 == 0) S.rcnt[r] = total;
            }
        }
    }
    __syncthreads();

    // 6. palettes: the 13 colours (tile mean, then regions 21..32 in order), their pairwise
    //    near tests in parallel, then one thread keeps each colour that is not near one kept
    //    before it
    if (tid < NCOL) {
        float m[3];
        const int r = 20 + tid;
        int a = 0, b = 1;
        if (tid >= 1 && r < 30) run_bounds(tb.cuts, si, r, a, b);
        if (tid >= 1 && r < 30 && b <= a) {
            const int p = sidx[min(a, N - 1)];
            for (int c = 0; c < 3; ++c) m[c] = col[c * N + p];
        } else if (tid >= 1 && S.rcnt[r] > 0) {
            for (int c = 0; c < 3; ++c) m[c] = S.rmean[r][c];
        } else {
            for (int c = 0; c < 3; ++c) m[c] = S.rmean[0][c];
        }
        for (int c = 0; c < 3; ++c) S.cpal[tid][c] = clamp01(m[c]);
    }
    __syncthreads();
    if (tid < NCOL) {
        unsigned near = 0;
        for (int a = 0; a < tid; ++a)
            if (near_pair(S.cpal[tid], S.cpal[a])) near |= 1u << a;
        S.near_mask[tid] = near;
    }
    __syncthreads();
    if (tid == 0) {
        unsigned kept = 1u;
        int npal = 1;
        for (int c = 0; c < 3; ++c) S.pal[0][c] = S.cpal[0][c];
        for (int i = 1; i < NCOL; ++i) {
            if (i == 10) S.npal_e = npal;  // the template palette adds bright / dark / edge colours
            if (!(S.near_mask[i] & kept) && npal < MAXPAL) {
                kept |= 1u << i;
                for (int c = 0; c < 3; ++c) S.pal[npal][c] = S.cpal[i][c];
                ++npal;
            }
        }
        S.npal_t = npal;
    }
    __syncthreads();

    // 7. The candidate list is (edge pool) palette x 4 alphas, quadrants x 2, per orientation its centre
    //    line x 3 and two offset lines, (template pool) palette x 4, quadrants x 2, blocks, template
    //    lines x 3 (through the centre) or x 1.  The template pool's quadrants and the colours it shares
    //    with the edge palette repeat the edge pool's.  Units in list order: edge palette, quadrants,
    //    per orientation three lines, the palette's extra colours, blocks, template lines.
    const int n_peaks = S.n_peaks, npal_e = want0 ? S.npal_e : 0, npal_t = want0 ? S.npal_t : 0;
    const int n_quad = want0 ? 4 : 0, n_block = want0 ? 16 : 0, n_lines = want1 ? n_peaks * 3 : 0;
    const int n_spec = want1 ? tb.n_spec : 0;
    const int u_quad = npal_e, u_orient = u_quad + n_quad, u_extra = u_orient + n_lines,
              u_block = u_extra + (npal_t - npal_e), u_spec = u_block + n_block, n_unit = u_spec + n_spec;
    // unit u: its group (kind and set of alphas), its place in its group's order, its alphas' number
    //   groups: 0 palette (1, .7, .4, .2), 1 quadrants (.5, .3), 2 blocks (.25), 3 centre lines
    //   (1, .7, .4), 4 other lines (.5)
    auto unit_group = [&](int u) {
        if (u < u_quad) return 0;
        if (u < u_orient) return 1;
        if (u < u_extra) return (u - u_orient) % 3 == 0 ? 3 : 4;
        if (u < u_block) return 0;
        if (u < u_spec) return 2;
        return u - u_spec < tb.n_centre ? 3 : 4;
    };
    auto group_alphas = [](int g) { return g == 0 ? 4 : g == 1 ? 2 : g == 3 ? 3 : 1; };
    // side means of the lines as they are listed: an empty side takes the tile mean; the edge pool clamps
    // them, the template pool does not
    for (int i = tid; i < 2 * (n_peaks + n_spec) * 3; i += NT) {
        const int line = i / 6, side = (i / 3) & 1, k = i % 3, na = S.scnt[line];
        const float v = (side ? N - na : na) > 0 ? S.smean[line][side][k] : S.rmean[0][k];
        S.smean[line][side][k] = line < n_peaks ? clamp01(v) : v;
    }
    if (tid < 20 * 3) (&S.rmean[1][0])[tid] = clamp01((&S.rmean[1][0])[tid]);  // quadrants and blocks
    if (tid == 0) S.bad = 0;
    __syncthreads();
    // unit u's colours (c1: null for a constant) and line (null for a constant)
    auto unit_at = [&](int u, const float*& c0, const float*& c1, const double*& g) {
        c1 = nullptr;
        g = nullptr;
        if (u < u_quad) {
            c0 = S.pal[u];
        } else if (u < u_orient) {
            c0 = S.rmean[1 + u - u_quad];
        } else if (u < u_extra) {
            const int line = (u - u_orient) / 3;
            c0 = S.smean[line][0];
            c1 = S.smean[line][1];
            g = tb.orient_geom + ((size_t)(si * 16 + S.peaks[line]) * 3 + (u - u_orient) % 3) * 4;
        } else if (u < u_block) {
            c0 = S.pal[npal_e + u - u_extra];
        } else if (u < u_spec) {
            c0 = S.rmean[5 + u - u_block];
        } else {
            c0 = S.smean[n_peaks + u - u_spec][0];
            c1 = S.smean[n_peaks + u - u_spec][1];
            g = tb.spec_geom + (size_t)(si * WEFTK_POOL_MAX_SPECS + u - u_spec) * 4;
        }
    };
    for (int u = tid; u < n_unit; u += NT) {
        const float *c0, *c1;
        const double* g;
        unit_at(u, c0, c1, g);
        unsigned long long k0 = pack_colour(c0[0], c0[1], c0[2]), k1 = 0, kg = 0;
        if (g != nullptr) {
            k1 = pack_colour(c1[0], c1[1], c1[2]);
            kg = pack_line(g);
        }
        ulonglong2 key;
        key.x = kg | (k0 << 44);
        key.y = ((k0 & ~BAD_KEY) >> 20) | (k1 << 16) | ((unsigned long long)unit_group(u) << 52);
        if ((k0 | k1 | kg) & BAD_KEY) {
            key.y |= BAD_KEY;
            S.bad = 1;
        }
        S.key[u] = key;
    }
    __syncthreads();
    // the reference's key, field by field, for a unit whose key does not pack
    auto full_key = [&](int u, int (&key)[10]) {
        const float *c0, *c1;
        const double* g;
        unit_at(u, c0, c1, g);
        for (int k = 0; k < 4; ++k) key[k] = g ? qkey(g[k], 4.0) : 0;
        for (int k = 0; k < 3; ++k) {
            key[4 + k] = qkey((double)c0[k], 64.0);
            key[7 + k] = c1 ? qkey((double)c1[k], 64.0) : 0;
        }
    };
    // first occurrences: a unit is a repeat when an earlier one of its group has its key
    for (int base = 0; base < n_unit; base += NT) {
        const int u = base + tid;
        int count = 0;
        if (u < n_unit) {
            const ulonglong2 key = S.key[u];
            const int gr = unit_group(u);
            bool again = false;
            // (only the template lines and the extra colours look back past their own stretch)
            const int from = gr == 1 ? u_quad : gr == 2 ? u_block : gr >= 3 ? u_orient : 0;
            if (!(key.y & BAD_KEY)) {
#pragma unroll 4
                for (int v = from; v < u; ++v) {
                    const ulonglong2 o = S.key[v];
                    again = again || (((o.x ^ key.x) | (o.y ^ key.y)) == 0);
                }
            }
            if (S.bad && (key.y & BAD_KEY)) {
                int a[10];
                full_key(u, a);
                for (int v = from; v < u && !again; ++v) {
                    if (!(S.key[v].y & BAD_KEY) || unit_group(v) != gr) continue;
                    int b[10];
                    full_key(v, b);
                    again = true;
                    for (int k = 0; k < 10; ++k) again = again && a[k] == b[k];
                }
            }
            count = again ? 0 : group_alphas(gr);
        }
        // places: exclusive sums of the counts over the units
        int incl = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) S.wtot[(base >> 5) + warp] = incl;
        if (u < n_unit) S.place[u] = count ? incl - count : -1;
    }
    __syncthreads();
    if (tid == 0) {
        int n = 0;
        for (int w = 0; w < (n_unit + 31) / 32; ++w) {
            const int c = S.wtot[w];
            S.wtot[w] = n;
            n += c;
        }
        const int listed = n_quad * 4 + (npal_e + npal_t) * 4 + n_block + n_lines / 3 * 5 + n_spec +
                           (want1 ? tb.n_centre * 2 : 0);  // with the repeats; MAXC <= pool_cap
        if (listed > MAXC) {
            atomicCAS(&g_device_status, 0, WEFTK_E_RANGE);
            n = min(n, MAXC);
        }
        S.n_out = n;
        job.pool_cnt[t] = n;
    }
    __syncthreads();
    const int n_out = S.n_out;
    for (int u = tid; u < n_unit; u += NT) {  // which unit and alpha each record is
        if (S.place[u] < 0) continue;
        const int at = S.wtot[u >> 5] + S.place[u], gr = unit_group(u);
        for (int k = 0; k < group_alphas(gr); ++k)
            if (at + k < n_out) S.rec_of[at + k] = (unsigned short)(u | (gr << 8) | (k << 12));
    }
    __syncthreads();
    // the records: 32 of a warp are staged (the planes are done with) and written together, word by word
    WeftPrim* out = job.cand + job.pool_off[t];
    WeftPrim* stage = reinterpret_cast<WeftPrim*>(smem_raw) + warp * 32;
    for (int first = warp * 32; first < n_out; first += NT) {
        const int m = min(32, n_out - first);
        if (lane < m) {
            const unsigned what = S.rec_of[first + lane];
            const float *c0, *c1;
            const double* g;
            unit_at(what & 255u, c0, c1, g);
            const int gr = (what >> 8) & 15u, k = what >> 12;
            WeftPrim p;
            p.kind = gr >= 3 ? 1 : 0;
            for (int j = 0; j < 7; ++j) p.geom[j] = j < 4 && g ? (float)g[j] : 0.0f;
            for (int j = 0; j < 3; ++j) {
                p.color0[j] = c0[j];
                p.color1[j] = c1 ? c1[j] : 0.0f;
            }
            // the reference's Python floats, rounded to float32
            p.alpha = gr == 0 || gr == 3 ? (k == 0 ? 1.0f : k == 1 ? 0.7f : k == 2 ? 0.4f : 0.2f)
                      : gr == 1         ? (k == 0 ? 0.5f : 0.3f)
                      : gr == 2         ? 0.25f
                                        : 0.5f;
            stage[lane] = p;
        }
        __syncwarp();
        int* dst = reinterpret_cast<int*>(out + first);
        const int* from = reinterpret_cast<const int*>(stage);
        for (int k = lane; k < m * (int)(sizeof(WeftPrim) / 4); k += 32) dst[k] = from[k];
        __syncwarp();
    }
}

// the side test of every split row over every tile side's pixel grid, one thread per word
__global__ void side_bits_kernel(WeftPoolTables tb, uint32_t* out) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= WEFTK_POOL_SIDE_WORDS) return;
    int si = 0;
    while (si < 3 && gid >= (si == 0 ? 2 : si == 1 ? 10 : 42) * NSPL) ++si;
    const int before = si == 0 ? 0 : si == 1 ? 2 : si == 2 ? 10 : 42;
    const int ts = 8 << si, wps = ts * ts / 32;
    const int local = gid - before * NSPL, row = local / wps, w = local - row * wps;
    const float* m = row < 16 ? tb.orient_mask + (si * 16 + row) * 4
                     : row - 16 < tb.n_spec ? tb.spec_mask + (si * WEFTK_POOL_MAX_SPECS + (row - 16)) * 4
                                            : nullptr;
    uint32_t word = 0;
    if (m) {
        const float4 c = make_float4(m[0], m[1], m[2], m[3]);
        for (int b = 0; b < 32; ++b) {
            const int p = w * 32 + b;
            if (side_a(c, p % ts, p / ts)) word |= 1u << b;
        }
    }
    out[gid] = word;
}

template <int TS, int NT>
int launch_gen(const WeftPoolTables& tb, const WeftPoolJob& job, int si, cudaStream_t stream) {
    const int n = job.n_tiles[si];
    if (n == 0) return WEFTK_OK;
    constexpr int N = TS * TS;
    const size_t dyn = (pool_smem_bytes(N, NT / 32) + 15) / 16 * 16;
    // the static scratch and the pixel planes together exceed the default 48 KB: opt in once
    // per device (under a lock, so concurrent first calls agree)
    {
        int dev = 0;
        WEFTK_CUDA(cudaGetDevice(&dev));
        static std::mutex mu;
        static std::set<int> done;
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count(dev)) {
            WEFTK_CUDA(cudaFuncSetAttribute(gen_pool_kernel<TS, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)dyn));
            done.insert(dev);
        }
    }
    gen_pool_kernel<TS, NT><<<n, NT, dyn, stream>>>(tb, job, si);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

}  // namespace
}  // namespace weftk

using namespace weftk;

// Side streams of the current device that run the larger tile classes beside the 8-px class
// (forked from and joined back into the caller's stream with events, so a captured graph gets
// parallel branches).  Created on a host thread's first call on a device and kept for the life of
// the process; per host thread, so concurrent callers never share the events.
struct SideStreams {
    cudaStream_t s[3] = {nullptr, nullptr, nullptr};
    cudaEvent_t fork = nullptr, join[3] = {nullptr, nullptr, nullptr};
};

int side_streams(SideStreams** out) {
    thread_local SideStreams per_dev[64];
    int dev = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    WEFTK_REQUIRE(dev >= 0 && dev < 64, "gen_pools: device index beyond 63");
    SideStreams& ss = per_dev[dev];
    if (!ss.fork) {
        for (int i = 0; i < 3; ++i) {
            WEFTK_CUDA(cudaStreamCreateWithFlags(&ss.s[i], cudaStreamNonBlocking));
            WEFTK_CUDA(cudaEventCreateWithFlags(&ss.join[i], cudaEventDisableTiming));
        }
        WEFTK_CUDA(cudaEventCreateWithFlags(&ss.fork, cudaEventDisableTiming));
    }
    *out = &ss;
    return WEFTK_OK;
}

extern "C" int weftk_pool_side_bits(const WeftPoolTables* tables, uint32_t* d_bits, void* stream) {
    WEFTK_REQUIRE(tables && d_bits, "pool_side_bits: null argument");
    WEFTK_REQUIRE(tables->n_spec >= 0 && tables->n_spec <= WEFTK_POOL_MAX_SPECS, "pool_side_bits: bad template table");
    WEFTK_REQUIRE(tables->orient_mask && (tables->n_spec == 0 || tables->spec_mask), "pool_side_bits: null table");
    constexpr int block = 256;
    side_bits_kernel<<<(WEFTK_POOL_SIDE_WORDS + block - 1) / block, block, 0, (cudaStream_t)stream>>>(*tables, d_bits);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_gen_pools(const WeftPoolTables* tables, const WeftPoolJob* job, void* stream) {
    WEFTK_REQUIRE(tables && job, "gen_pools: null argument");
    WEFTK_REQUIRE(tables->n_spec >= 0 && tables->n_spec <= WEFTK_POOL_MAX_SPECS &&
                      tables->n_centre >= 0 && tables->n_centre <= tables->n_spec,
                  "gen_pools: bad template table");
    WEFTK_REQUIRE(job->pool_cap >= WEFTK_POOL_MAX_CONST_LINEAR, "gen_pools: pool_cap below the per-tile bound");
    WEFTK_REQUIRE((job->kinds_mask & ~3) == 0, "gen_pools: only constant and linear patches are generated");
    int any = 0;
    for (int i = 0; i < 4; ++i) {
        WEFTK_REQUIRE(job->n_tiles[i] >= 0, "gen_pools: negative tile count");
        any |= job->n_tiles[i] > 0;
        WEFTK_REQUIRE(job->n_tiles[i] == 0 || job->tiles[i], "gen_pools: null tile list");
    }
    if (!any) return WEFTK_OK;
    WEFTK_REQUIRE(job->src && job->px_off && job->pool_off && job->cand && job->pool_cnt, "gen_pools: null pointer");
    WEFTK_REQUIRE(tables->bin_edges && tables->cuts && tables->orient_geom && tables->orient_mask &&
                      tables->side_bits && (tables->n_spec == 0 || (tables->spec_geom && tables->spec_mask)),
                  "gen_pools: null table");
    cudaStream_t s = (cudaStream_t)stream;
    SideStreams* ss = nullptr;
    int rc = side_streams(&ss);
    if (rc) return rc;
    // the 64-, 32- and 16-px classes (few CTAs, long ones) on side streams, the 8-px class here
    WEFTK_CUDA(cudaEventRecord(ss->fork, s));
    for (int i = 0; i < 3; ++i) WEFTK_CUDA(cudaStreamWaitEvent(ss->s[i], ss->fork, 0));
    if ((rc = launch_gen<64, 512>(*tables, *job, 3, ss->s[0]))) return rc;
    if ((rc = launch_gen<32, 256>(*tables, *job, 2, ss->s[1]))) return rc;
    if ((rc = launch_gen<16, 128>(*tables, *job, 1, ss->s[2]))) return rc;
    if ((rc = launch_gen<8, 64>(*tables, *job, 0, s))) return rc;
    for (int i = 0; i < 3; ++i) {
        WEFTK_CUDA(cudaEventRecord(ss->join[i], ss->s[i]));
        WEFTK_CUDA(cudaStreamWaitEvent(s, ss->join[i], 0));
    }
    return WEFTK_OK;
}
