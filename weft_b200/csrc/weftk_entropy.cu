// weftk_entropy.cu — chunked order-0 rANS decode, and a file's tiles from their wire bytes to the
// decoder walk's arrays (see include/weftk_entropy.h).
//
// rANS: one warp per chunk, one serial chain.  Bound: that chain's latency, so everything is
// taken off it that can be: one table read per symbol (frequency and offset), the coded bytes read ahead
// four at a time into a 64-bit window, the refill without a branch.  128 chunks of 2000 bytes at 6.6 bits
// take 122 us; with three tables, a byte read per refill step and each lane filling its own symbols' slots
// they took 193.
//
// Tiles: one thread per tile walks its records and writes primitives and descriptor (10 us for 8548 tiles,
// 80 KB: the latency of records that follow one another); one CTA orders the work items by cost (22 us).
// The whole call on that file, 1024 x 1024 pixels to host memory, takes 0.95 ms (0.8 of it the pixels' copy)
// and took 142 with the entropy decode and the parse in Python.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "../../include/weftk_entropy.h"
#include "weftk_common.cuh"
#include "weftk_scene.cuh"

namespace weftk {

extern __device__ int g_device_status;

constexpr int RANS_PROB_BITS = 12;
constexpr int RANS_TOT = 1 << RANS_PROB_BITS;
constexpr unsigned RANS_L = 1u << 23;

__device__ __forceinline__ unsigned rd_u32(const uint8_t* p) {
    return (unsigned)p[0] | ((unsigned)p[1] << 8) | ((unsigned)p[2] << 16) | ((unsigned)p[3] << 24);
}

__device__ __forceinline__ unsigned rd_u16(const uint8_t* p) { return (unsigned)p[0] | ((unsigned)p[1] << 8); }

// One warp per CTA and chunk; what does not parse sets *status (first error wins).
__global__ void __launch_bounds__(32) rans_decode_kernel(const uint8_t* __restrict__ payload, long long payload_len,
                                                         const WeftRansChunk* __restrict__ chunks,
                                                         uint8_t* __restrict__ out, long long out_len, int* status) {
    __shared__ uint2 lut[RANS_TOT];  // the symbol's frequency, the slot's offset among the symbol's
    __shared__ uint8_t sym[RANS_TOT];
    __shared__ unsigned key[256];       // frequency, below 1 + the place in the header that gave it
    __shared__ unsigned short start[256];
    const int lane = threadIdx.x;
    auto refuse = [&] {
        if (lane == 0) atomicCAS(status ? status : &g_device_status, 0, WEFTK_E_ARG);
    };
    const WeftRansChunk ch = chunks[blockIdx.x];
    if (ch.coded_offset < 0 || ch.coded_length < 5 || ch.coded_offset + ch.coded_length > payload_len ||
        ch.raw_offset < 0 || ch.raw_length < 0 || ch.raw_offset + ch.raw_length > out_len)
        return refuse();
    const uint8_t* p = payload + ch.coded_offset;
    const long long len = ch.coded_length;
    uint8_t* dst = out + ch.raw_offset;
    const int mode = p[0];
    const long long n = rd_u32(p + 1);
    if (n != ch.raw_length || (mode != 0 && mode != 1)) return refuse();
    if (mode == 0) {  // raw
        if (5 + n != len) return refuse();
        for (long long i = lane; i < n; i += 32) dst[i] = p[5 + i];
        return;
    }
    if (len < 7) return refuse();
    const int n_sym = (int)rd_u16(p + 5);
    const long long hdr = 7 + 3LL * n_sym;
    if (n_sym > 256 || hdr + 8 > len) return refuse();
    for (int i = lane; i < 256; i += 32) key[i] = 0;
    __syncwarp();
    // (a symbol listed twice keeps its last frequency)
    for (int k = lane; k < n_sym; k += 32) atomicMax(&key[p[7 + 3 * k]], ((unsigned)(k + 1) << 16) | rd_u16(p + 8 + 3 * k));
    __syncwarp();
    // cumulative frequencies: lane l sums symbols [8l, 8l + 8), then an exclusive warp scan
    unsigned loc[8], run = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        loc[j] = run;
        run += key[lane * 8 + j] & 0xffffu;
    }
    unsigned incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (__shfl_sync(0xffffffffu, incl, 31) != RANS_TOT) return refuse();
#pragma unroll
    for (int j = 0; j < 8; ++j) start[lane * 8 + j] = (unsigned short)(incl - run + loc[j]);
    __syncwarp();
    for (int s = 0; s < 256; ++s) {
        const unsigned f = key[s] & 0xffffu;
        for (unsigned k = lane; k < f; k += 32) {
            lut[start[s] + k] = make_uint2(f, k);
            sym[start[s] + k] = (uint8_t)s;
        }
    }
    __syncwarp();
    const unsigned x = rd_u32(p + hdr);
    const long long m = rd_u32(p + hdr + 4);
    if (hdr + 8 + m != len) return refuse();
    // the coded bytes are consumed from the last to the first: `win` holds the next `have` bits, first one
    // on top; whole aligned words follow (one may begin before the bytes, inside the chunk's header).
    // Every lane runs the chain; lane l keeps the slot of each block's symbol l and writes it
    const uint8_t* em = p + hdr + 8;
    struct State {
        unsigned x, ahead;
        int have;
        unsigned long long win;
        long long left;  // bits of the coded bytes not yet consumed
        const unsigned* word;
    } st;
    const uint8_t* end = em + m;
    st.x = x;
    st.left = 8 * m;
    st.win = 0;
    st.have = 0;
    while (((uintptr_t)end & 3u) != 0 && end > em) {
        st.win |= (unsigned long long)*--end << (56 - st.have);
        st.have += 8;
    }
    st.word = reinterpret_cast<const unsigned*>(end);
    st.ahead = end > em ? *--st.word : 0;
    auto refill = [&] {  // to 32 bits at least, as long as there are any: two symbols take 16 each at most
        if (st.have <= 32) {
            st.win |= (unsigned long long)st.ahead << (32 - st.have);
            st.have += 32;
            st.ahead = reinterpret_cast<const uint8_t*>(st.word) > em ? *--st.word : 0;
        }
    };
    unsigned mine = 0;
    for (long long i = 0; i < n; i += 32) {
        const int block = (int)min(32LL, n - i);
        const State before = st;
        bool again = block < 32 || st.left < 32 * 16;  // two bytes a symbol at most
        if (!again) {
            bool odd = false;
#pragma unroll 8
            for (int k = 0; k < 32; k += 2) {
                refill();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned slot = st.x & (RANS_TOT - 1);
                    if (lane == k + h) mine = slot;
                    const uint2 e = lut[slot];
                    const unsigned v = e.x * (st.x >> RANS_PROB_BITS) + e.y;
                    odd = odd || v - 128u >= 0x80000000u - 128u;  // (not in a stream an encoder wrote)
                    const int take = v < RANS_L ? (v < (RANS_L >> 8) ? 16 : 8) : 0;
                    st.x = __funnelshift_l((unsigned)(st.win >> 32), v, take);
                    st.win <<= take;
                    st.have -= take;
                    st.left -= take;
                }
            }
            again = odd;
            if (odd) st = before;
        }
        if (again) {  // the last symbols, or bytes that no encoder writes: byte by byte
            for (int k = 0; k < block; ++k) {
                const unsigned slot = st.x & (RANS_TOT - 1);
                if (lane == k) mine = slot;
                const uint2 e = lut[slot];
                st.x = e.x * (st.x >> RANS_PROB_BITS) + e.y;
                for (; st.x < RANS_L && st.left > 0; st.left -= 8, st.have -= 8, st.win <<= 8) {
                    refill();
                    st.x = (st.x << 8) | (unsigned)(st.win >> 56);
                }
            }
        }
        if (lane < block) dst[i + lane] = sym[mine];
    }
}

// ------------------------------------------------------------------ a file's tiles
// u32 / u16 fields stand at any byte
struct SceneFile {
    const uint8_t *toc, *res0, *res1, *qtree, *raw;
    int n_tiles, n_res1;
    long long raw_len;
    double sx, sy;
    int scaled, out_w, out_h;
    int cap_prims, cap_cp48, cap_items;
    WeftTileDecodeDesc* descs;
    WeftPrim* prims;
    float *cp48, *grids;
    int2* items;
    int* n_items;
    int* status;
};

// target rect edges: round half to even of the float64 product, as Python's round
__host__ __device__ inline int scene_edge(int v, double s) {
#ifdef __CUDA_ARCH__
    return __double2int_rn(__dmul_rn((double)v, s));
#else
    return (int)std::nearbyint((double)v * s);
#endif
}

__host__ __device__ inline void scene_rect(const uint8_t* q, bool scaled, double sx, double sy, int& x0, int& y0,
                                           int& w, int& h, int& side) {
    const int qx = q[0] | (q[1] << 8), qy = q[2] | (q[3] << 8);
    side = q[4];
    x0 = qx;
    y0 = qy;
    w = h = side;
    if (scaled) {
        x0 = scene_edge(qx, sx);
        y0 = scene_edge(qy, sy);
        w = scene_edge(qx + side, sx) - x0;
        h = scene_edge(qy + side, sy) - y0;
        w = w < 1 ? 1 : w;
        h = h < 1 ? 1 : h;
    }
}

// rows of an item and the tile's rows inside the image (weftk_render_tiles)
__host__ __device__ inline void scene_items(int x0, int y0, int w, int h, int out_w, int out_h, int& rows, int& r0,
                                            int& r1) {
    auto floor4 = [](int v) { return v >= 0 ? v / 4 : -((-v + 3) / 4); };
    const int g = floor4(x0 + w + 3) - floor4(x0);
    rows = WEFTK_DECODE_ITEM_GROUPS / g;
    rows = rows < 1 ? 1 : rows;
    r0 = y0 < 0 ? -y0 : 0;
    r1 = h < out_h - y0 ? h : out_h - y0;
    if (x0 >= out_w || x0 + w <= 0 || r1 < r0) r1 = r0;
}

// A primitive's slot is its byte offset over 7, a control grid's over 50: no primitive is shorter, so the
// slots are apart without counting the ones before.
constexpr int SCENE_MIN_PRIM = 7, SCENE_GRID_PRIM = 50;

__global__ void __launch_bounds__(64) scene_tiles_kernel(SceneFile F) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= F.n_tiles) return;
    WeftTileDecodeDesc d = {};
    bool ok = *F.status == 0;
    scene_rect(F.qtree + 5LL * t, F.scaled != 0, F.sx, F.sy, d.target_x0, d.target_y0, d.target_w, d.target_h,
               d.source_size);
    d.res1_index = t < F.n_res1 ? t : -1;
    if (F.res0) {
        const int8_t* r = reinterpret_cast<const int8_t*>(F.res0) + 3LL * t;
        d.res0_r = __fdiv_rn((float)r[0], 255.0f);
        d.res0_g = __fdiv_rn((float)r[1], 255.0f);
        d.res0_b = __fdiv_rn((float)r[2], 255.0f);
    }
    const long long a = rd_u32(F.toc + 4LL * t), b = rd_u32(F.toc + 4LL * t + 4);
    ok = ok && a < b && b <= F.raw_len;
    if (ok) {
        const int n = F.raw[a];
        const int slot0 = (int)(a / SCENE_MIN_PRIM);
        long long off = a + 1;
        ok = n <= 48 && slot0 + n <= F.cap_prims;
        for (int i = 0; i < n && ok; ++i) {
            // the kind, the payload's length, geometry words, colours, alpha
            const int kind = off + 2 <= b ? F.raw[off] : 255, len = kind < 255 ? F.raw[off + 1] : 0;
            const int words = kind == 0 ? 0 : kind == 1 ? 4 : kind == 2 ? 5 : kind == 3 ? 7 : kind == 4 ? 6 : 0;
            const int want = kind == 5 ? 48 : 2 * words + (kind == 1 ? 6 : 3) + 2;
            ok = kind <= 5 && len == want && off + 2 + len <= b;
            if (!ok) break;
            const uint8_t* p = F.raw + off + 2;
            WeftPrim rec = {};
            rec.kind = kind;
            if (kind == 5) {
                const int grid = (int)(off / SCENE_GRID_PRIM);
                ok = grid < F.cap_cp48;
                if (!ok) break;
                rec.geom[0] = (float)grid;
                rec.alpha = 1.0f;
                for (int k = 0; k < 48; ++k)
                    F.cp48[(size_t)grid * 48 + k] = __double2float_rn(__ddiv_rn((double)p[k], 255.0));
            } else {
                // kind 2's and 3's last word is a thickness in [0, 4], the rest coordinates in [0, 15]
#pragma unroll
                for (int k = 0; k < 7; ++k)
                    if (k < words) {
                        const double hi = (kind == 2 && k == 4) || (kind == 3 && k == 6) ? 4.0 : 15.0;
                        rec.geom[k] = __double2float_rn(__dmul_rn(__ddiv_rn((double)rd_u16(p + 2 * k), 65535.0), hi));
                    }
                p += 2 * words;
#pragma unroll
                for (int k = 0; k < 3; ++k) rec.color0[k] = __double2float_rn(__ddiv_rn((double)p[k], 255.0));
                p += 3;
                if (kind == 1) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) rec.color1[k] = __double2float_rn(__ddiv_rn((double)p[k], 255.0));
                    p += 3;
                }
                rec.alpha = __double2float_rn(__ddiv_rn((double)rd_u16(p), 65535.0));
            }
            F.prims[slot0 + i] = rec;
            off += 2 + len;
        }
        ok = ok && off == b;
        d.prim_offset = slot0;
        d.prim_count = n;
    }
    if (!ok) {
        atomicCAS(F.status, 0, WEFTK_E_ARG);
        d.prim_offset = d.prim_count = 0;
    }
    F.descs[t] = d;
}

__global__ void scene_grids_kernel(const uint8_t* __restrict__ res1, int n, float* __restrict__ grids) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) grids[i] = __fdiv_rn((float)(int8_t)res1[i], 255.0f);
}

// The work items, costly ones first: a counting sort by the cost's exponent and two bits below it.
__global__ void __launch_bounds__(1024) scene_items_kernel(SceneFile F) {
    __shared__ int hist[128], at[128];
    const int tid = threadIdx.x;
    if (*F.status != 0) {
        if (tid == 0) *F.n_items = 0;
        return;
    }
    auto each = [&](auto&& put) {
        for (int t = tid; t < F.n_tiles; t += 1024) {
            const WeftTileDecodeDesc d = F.descs[t];
            int rows, r0, r1;
            scene_items(d.target_x0, d.target_y0, d.target_w, d.target_h, F.out_w, F.out_h, rows, r0, r1);
            if (r1 <= r0) continue;
            const bool fill = d.res1_index < 0 && d.prim_count == 1 && F.prims[d.prim_offset].kind == 0;
            auto bucket = [&](int n_rows) {
                const float cost = (float)n_rows * (float)d.target_w * (fill ? 1.0f : 4.0f);  // >= 1
                return 127 - min(127, (__float_as_int(cost) >> 21) - (127 << 2));
            };
            const int full = (r1 - r0) / rows, rest = (r1 - r0) - full * rows;
            if (full) put(t, r0, rows, full, bucket(rows));
            if (rest) put(t, r0 + full * rows, rows, 1, bucket(rest));
        }
    };
    if (tid < 128) hist[tid] = 0;
    __syncthreads();
    each([&](int, int, int, int n, int b) { atomicAdd(&hist[b], n); });
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int b = 0; b < 128; ++b) {
            at[b] = run;
            run += hist[b];
        }
        *F.n_items = run <= F.cap_items ? run : 0;
        if (run > F.cap_items) atomicCAS(F.status, 0, WEFTK_E_ARG);
    }
    __syncthreads();
    each([&](int t, int first, int rows, int n, int b) {
        const int k = atomicAdd(&at[b], n);
        for (int i = 0; i < n; ++i)
            if (k + i < F.cap_items) F.items[k + i] = make_int2(t, first + i * rows);
    });
}

static uint32_t le32(const uint8_t* p) {
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}

// Checks a file's layout on the host and sizes its buffers; plan.ok false: not of the ordinary form.
int scene_plan(const WeftSceneFile& f, ScenePlan& plan) {
    plan.ok = false;
    const int n = f.n_tiles;
    if (n <= 0 || f.n_chunks <= 0 || f.out_w <= 0 || f.out_h <= 0 || f.enc_w <= 0 || f.enc_h <= 0) return WEFTK_OK;
    auto inside = [&](int64_t off, int64_t len) { return off >= 0 && len >= 0 && off <= f.blob_len && len <= f.blob_len - off; };
    if (!inside(f.prim, f.prim_len) || !inside(f.cidx, 24LL * f.n_chunks) || !inside(f.toc, 4LL * (n + 1)) ||
        !inside(f.qtree, 5LL * n) || (f.res0 >= 0 && !inside(f.res0, 3LL * n)) || f.n_res1 < 0 ||
        (f.n_res1 > 0 && !inside(f.res1, 48LL * f.n_res1)))
        return WEFTK_OK;
    const uint8_t* toc = f.blob + f.toc;
    uint32_t last = le32(toc);
    for (int i = 1; i <= n; ++i) {
        const uint32_t v = le32(toc + 4LL * i);
        if (v < last) return WEFTK_OK;
        last = v;
    }
    if (last == 0 || last > (1u << 24)) return WEFTK_OK;  // (the slots of 16 MiB of tiles take 210 MB)
    plan.raw_len = last;
    // a tile of one constant takes 8 bytes, an evaluated layer 9 to 21 more: about one for two tiles
    plan.layered = plan.raw_len >= 14LL * n;
    // the chunks cover the tiles' bytes in order, without a gap
    plan.chunks.resize(f.n_chunks);
    int64_t at = 0;
    for (int i = 0; i < f.n_chunks; ++i) {
        const uint8_t* e = f.blob + f.cidx + 24LL * i;
        WeftRansChunk& c = plan.chunks[i];
        c.raw_offset = le32(e + 8);
        c.raw_length = le32(e + 12);
        c.coded_offset = le32(e + 16);
        c.coded_length = le32(e + 20);
        if (c.raw_offset != at || c.coded_length < 5 || c.coded_offset + c.coded_length > f.prim_len) return WEFTK_OK;
        at += c.raw_length;
    }
    if (at != plan.raw_len) return WEFTK_OK;
    plan.scaled = !(f.out_w == f.enc_w && f.out_h == f.enc_h);
    plan.sx = (double)f.out_w / (double)f.enc_w;
    plan.sy = (double)f.out_h / (double)f.enc_h;
    if (plan.sx > 1024.0 || plan.sy > 1024.0) return WEFTK_OK;  // (rect edges stay far inside 32 bits)
    int64_t items = 0;
    for (int i = 0; i < n; ++i) {
        int x0, y0, w, h, side, rows, r0, r1;
        scene_rect(f.blob + f.qtree + 5LL * i, plan.scaled, plan.sx, plan.sy, x0, y0, w, h, side);
        if (side <= 0 || w > 8192 || h > 8192) return WEFTK_OK;
        scene_items(x0, y0, w, h, f.out_w, f.out_h, rows, r0, r1);
        items += (r1 - r0 + rows - 1) / rows;
    }
    if (items > (1 << 28)) return WEFTK_OK;
    plan.n_items = (int)items;
    plan.cap_prims = (int)(plan.raw_len / SCENE_MIN_PRIM) + 1;
    plan.cap_cp48 = (int)(plan.raw_len / SCENE_GRID_PRIM) + 1;
    plan.ok = true;
    return WEFTK_OK;
}

int scene_launch(const WeftSceneFile& f, const ScenePlan& plan, const SceneBuffers& b, cudaStream_t s) {
    SceneFile F = {};
    F.toc = b.blob + f.toc;
    F.res0 = f.res0 >= 0 ? b.blob + f.res0 : nullptr;
    F.qtree = b.blob + f.qtree;
    F.raw = b.raw;
    F.n_tiles = f.n_tiles;
    F.n_res1 = f.n_res1 < f.n_tiles ? f.n_res1 : f.n_tiles;
    F.raw_len = plan.raw_len;
    F.sx = plan.sx;
    F.sy = plan.sy;
    F.scaled = plan.scaled;
    F.out_w = f.out_w;
    F.out_h = f.out_h;
    F.cap_prims = plan.cap_prims;
    F.cap_cp48 = plan.cap_cp48;
    F.cap_items = plan.n_items;
    F.descs = b.descs;
    F.prims = b.prims;
    F.cp48 = b.cp48;
    F.grids = b.grids;
    F.items = b.items;
    F.n_items = b.ctl + 1;
    F.status = b.ctl;
    WEFTK_CUDA(cudaMemsetAsync(b.ctl, 0, 2 * sizeof(int), s));
    rans_decode_kernel<<<f.n_chunks, 32, 0, s>>>(b.blob + f.prim, f.prim_len, b.chunks, b.raw, plan.raw_len, b.ctl);
    scene_tiles_kernel<<<ceil_div(f.n_tiles, 64), 64, 0, s>>>(F);
    if (F.n_res1 > 0)
        scene_grids_kernel<<<ceil_div(48 * F.n_res1, 256), 256, 0, s>>>(b.blob + f.res1, 48 * F.n_res1, b.grids);
    scene_items_kernel<<<1, 1024, 0, s>>>(F);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

}  // namespace weftk

using namespace weftk;

extern "C" int weftk_rans_decode_chunks(const uint8_t* d_payload, int64_t payload_len, const WeftRansChunk* d_chunks,
                                        int n_chunks, uint8_t* d_out, int64_t out_len, void* stream) {
    WEFTK_REQUIRE(n_chunks >= 0 && payload_len >= 0 && out_len >= 0, "rans_decode_chunks: negative size");
    if (n_chunks == 0) return WEFTK_OK;
    WEFTK_REQUIRE(d_payload && d_chunks && d_out, "rans_decode_chunks: null pointer");
    rans_decode_kernel<<<n_chunks, 32, 0, (cudaStream_t)stream>>>(d_payload, payload_len, d_chunks, d_out, out_len,
                                                                  nullptr);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}
