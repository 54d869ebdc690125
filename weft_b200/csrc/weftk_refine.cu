// weftk_refine.cu — per-tile stack loss and its hand-written backward (see include/weftk_refine.h).
//
// One launch covers every tile.  Tiles are grouped by side; a tile is worked on by the warps of its
// group, which meet at a named barrier, and CTAs of the largest tiles come first so they start
// first.  The tile's parameter rows are prepared once per step into shared memory (and a curve's
// 31 polyline segments into a segment table).  The backward pass sweeps the layers back to front:
//     c_k = s_k a_k + c_{k-1} (1 - a_k)
//     dL/ds_k = g a_k,  dL/da_k = g . (s_k - c_{k-1}),  g <- g (1 - a_k)
// and chains dL/ds, dL/da into the layer's parameters.  Every sum (gradients over pixels, block and
// quadrant sums of the residual loss) has a single owner and a fixed order, so results are
// deterministic.
//
// Three kernels: refine_general_kernel for stacks of any kind and length, refine_tiles_kernel for
// single constant / linear layers without the residual loss (everything in registers), and
// refine_const_kernel for lone constant layers whose pixel sums are given.
//
// Residual-aware loss (WEFTK_LOSS_RESIDUAL): the file a fit becomes carries a
// per-tile 4x4 grid of block-mean errors that the decoder adds back with
// bilinear interpolation (src/weft/encoder.py:3248-3372, src/weft/render.py:474-515).
// With e = clamp(render) - src, M the 4x4 block-mean operator and B the decoder's
// bilinear upsampling, the decoded error is r = e - B M e (before the grid's
// 8-bit quantisation and clamping), and the loss is mean(r^2) with gradient
// 2 (I - M^T B^T) r / (3n).  Pixels are visited block-major, quadrant-major
// inside a block, so block sums and the per-quadrant sums of B^T r are
// segmented warp reductions over aligned lane groups.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "../../include/weftk_fit.h"
#include "../../include/weftk_refine.h"
#include "weftk_common.cuh"
#include "weftk_prim.cuh"

namespace weftk {

extern __device__ int g_device_status;

constexpr int MAXL = WEFTK_REFINE_MAX_PRIMS;
constexpr float TRI_SOFT_W = 0.5f;  // surrogate edge width in pixels

// The layers of one tile, staged in shared memory.
struct Layers {
    const Prep* prep;
    const float (*raw)[16];
    const float4 (*seg)[31][2];
    // per kind: linear D, 1 / D^2; line and curve 1 / sigma^3; triangle its three edges
    // (ax, ay, ex, ey, o / (L w), o / L^2, 1 / L, L)
    const float4 (*aux)[6];
};

__device__ __forceinline__ WeftPrim row_to_prim(const float* r, int kind) {
    WeftPrim p;
    p.kind = kind;
#pragma unroll
    for (int i = 0; i < 7; ++i) p.geom[i] = r[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        p.color0[i] = r[7 + i];
        p.color1[i] = r[10 + i];
    }
    p.alpha = r[13];
    return p;
}

__device__ __forceinline__ float sigmoid(float x) { return 1.0f / (1.0f + __expf(-x)); }
// Shared-memory carve-up of one tile group of refine_tiles_kernel (the WPT warps working on one
// tile).  Byte offsets; every region starts on a 16-byte boundary except the trailing doubles
// (8-byte aligned).
struct GroupLayout {
    int prep, raw, madam, vadam, gacc, lred, mom, bytes;
};

__host__ __device__ __forceinline__ GroupLayout group_layout(int wpt) {
    GroupLayout g;
    g.prep = 0;
    g.raw = g.prep + 64;
    g.madam = g.raw + 64;  // Adam moments of the row (RF_STEP)
    g.vadam = g.madam + 64;
    g.gacc = g.vadam + 64;
    g.lred = (g.gacc + wpt * 56 + 15) & ~15;
    g.mom = g.lred + wpt * 8;  // pixel moments of a lone constant layer's tile: per warp, then total
    g.bytes = (g.mom + (wpt + 1) * 6 * 8 + 15) & ~15;
    return g;
}

// Adam (PyTorch's update rule, FP32) for one value at step t (1-based), then the
// projection onto what the wire format carries: colours and alpha in [0, 1],
// coordinates in [0, 15], thickness in [0, 4] (src/weft/primitives.py:102-177).
// Projection of column col of a row onto its valid range (colours and alpha [0, 1], thickness
// [0, 4], other geometry [0, 15]).
__device__ __forceinline__ float adam_project(float x, int kind, int col) {
    if (col >= 7) return fminf(fmaxf(x, 0.0f), 1.0f);
    const bool thick = (kind == K_LINE && col == 4) || (kind == K_CURVE && col == 6);
    return fminf(fmaxf(x, 0.0f), thick ? 4.0f : 15.0f);
}

__device__ __forceinline__ float adam_update_bc(float p, float g, float& m, float& v, float bc1, float bc2, float lr,
                                                float b1, float b2, float eps, int kind, int col) {
    m = fmaf(b1, m, (1.0f - b1) * g);
    v = fmaf(b2, v, (1.0f - b2) * g * g);
    return adam_project(p - lr * (m / bc1) / (sqrtf(v / bc2) + eps), kind, col);
}

// Bias corrections 1 - beta^t of step t (1-based).
__device__ __forceinline__ void adam_bias(float b1, float b2, float t, float& bc1, float& bc2) {
    bc1 = 1.0f - powf(b1, t);
    bc2 = 1.0f - powf(b2, t);
}

__device__ __forceinline__ float adam_update(float p, float g, float& m, float& v, float t, float lr, float b1,
                                             float b2, float eps, int kind, int col) {
    float bc1, bc2;
    adam_bias(b1, b2, t, bc1, bc2);
    return adam_update_bc(p, g, m, v, bc1, bc2, lr, b1, b2, eps, kind, col);
}

// Optimiser state of the fused refine step; the per-row step count lives in m[row * 16 + 15].
struct AdamArgs {
    float* m;
    float* v;
    float lr, b1, b2, eps;
};

// CTA classes of one launch, in launch order: tiles of side > 32 (8 warps per
// tile), 17..32 (4 warps), 9..16 (2 warps), <= 8 (1 warp).  Every CTA has 8
// warps; a CTA of class c holds groups[c] tiles.
constexpr int RF_THREADS = 256;
constexpr int RF_CLASSES = 4;
constexpr int RF_SMEM_MAX = 227 * 1024;

struct RefinePlan {
    int cta_end[RF_CLASSES];  // exclusive prefix sums of the classes' CTA counts
    int list_off[RF_CLASSES];
    int n_list[RF_CLASSES];
    int groups[RF_CLASSES];
};

__host__ __device__ __forceinline__ int class_wpt(int c) { return 8 >> c; }

// a[c] without dynamic indexing (keeps the plan in registers, off the stack)
__device__ __forceinline__ int pick(const int (&a)[RF_CLASSES], int c) {
    return c == 0 ? a[0] : c == 1 ? a[1] : c == 2 ? a[2] : a[3];
}

// Gradient columns a constant or linear layer can produce (bit i = column i).
__device__ __forceinline__ unsigned grad_columns(int kind) {
    // 7 8 9 13; 0-3 7-13
    return kind == K_CONST ? 0x2380u : kind == K_LINEAR ? 0x3f8fu : 0u;
}

// Bilinear node pair (lo, hi) and weight of the decoder's 4x4 residual grid for a
// pixel index along one axis of a tile with gscale = 4 / side (src/weft/render.py:474-515:
// centre sampling, edge clamp).
__device__ __forceinline__ void grid_coord(int p, float gscale, int& lo, int& hi, float& w) {
    const float g = fminf(fmaxf(__fsub_rn(__fmul_rn((float)p + 0.5f, gscale), 0.5f), 0.0f), 3.0f);
    lo = (int)floorf(g);
    hi = min(lo + 1, 3);
    w = g - (float)lo;
}
// Quadrant columns (0..7: block q / 2, half q % 2) whose pixels interpolate from grid node n along
// one axis, with the slot (0: lower node, 1: upper node) they use: source a of node n as
// (column << 1) | slot, -1 for none.  Lower node n: the right half of block n, the left half of
// block n + 1, and for n = 0 the left half of block 0 (clamped).  Upper node n: the right half of
// block n - 1, the left half of block n (n >= 1), and for n = 3 the right half of block 3 (clamped,
// weight 0).  The left half of block 0 also names node 1 as its upper node, with weight 0; it is
// skipped.
__device__ __forceinline__ int node_source(int n, int a) {
    if (n == 0) return a < 3 ? a << 1 : -1;
    switch (a) {
        case 0: return (2 * n + 1) << 1;
        case 1: return n == 3 ? (7 << 1) | 1 : (2 * n + 2) << 1;
        case 2: return ((2 * n - 1) << 1) | 1;
        default: return ((2 * n) << 1) | 1;
    }
}

// Barrier over the warps of one tile group (named barrier 1 + group; one warp: __syncwarp).
__device__ __forceinline__ void group_sync(int wpt, int grp) {
    if (wpt == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(wpt * 32) : "memory");
}

// Single-layer stacks of a constant or linear primitive (the refined fit's stacks): the layer's
// source colour, alpha and the linear ramp parameter at one pixel, with the renderer's formulas
// (prim_eval), so the forward is the same float sequence; any other kind is a no-op here.
struct ClEval {
    float s[3], a, t, traw;
};

__device__ __forceinline__ ClEval eval_cl(const Prep& P, float px, float py) {
    ClEval r;
    r.s[0] = P.cr;
    r.s[1] = P.cg;
    r.s[2] = P.cb;
    r.a = (P.kind == K_CONST || P.kind == K_LINEAR) ? P.a : 0.0f;
    r.t = r.traw = 0.0f;
    if (P.kind == K_LINEAR) {
        r.traw = fmaf(px - P.q[0], P.q[2], (py - P.q[1]) * P.q[3]);
        r.t = clamp01(r.traw);
        const float u = 1.0f - r.t;
        r.s[0] = fmaf(P.q[4], r.t, P.cr * u);
        r.s[1] = fmaf(P.q[5], r.t, P.cg * u);
        r.s[2] = fmaf(P.q[6], r.t, P.cb * u);
    }
    return r;
}

// Gradient of that layer over black (c_{-1} = 0), accumulated into acc[14]; the same chain
// rule as general_backward's constant and linear cases.
__device__ __forceinline__ void grad_cl(const Prep& P, const float* r, const ClEval& v, float px, float py,
                                        const float (&g)[3], float (&acc)[14]) {
    if (P.kind != K_CONST && P.kind != K_LINEAR) return;
    const float dA = (r[13] >= 0.0f && r[13] <= 1.0f) ? 1.0f : 0.0f;
    float dLds[3], dLda = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        dLds[c] = g[c] * v.a;
        dLda = fmaf(g[c], v.s[c], dLda);
    }
    acc[13] = fmaf(dLda, dA, acc[13]);
    if (P.kind == K_CONST) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[7 + c] += dLds[c];
        return;
    }
    const float t = v.t;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        acc[7 + c] = fmaf(dLds[c], 1.0f - t, acc[7 + c]);
        acc[10 + c] = fmaf(dLds[c], t, acc[10 + c]);
    }
    if (v.traw > 0.0f && v.traw < 1.0f) {
        const float x0 = r[0], y0 = r[1], vx = r[2] - r[0], vy = r[3] - r[1];
        const float D = vx * vx + vy * vy + 1e-8f;
        const float qx = px - x0, qy = py - y0, N = qx * vx + qy * vy;
        const float dLdt = dLds[0] * (r[10] - r[7]) + dLds[1] * (r[11] - r[8]) + dLds[2] * (r[12] - r[9]);
        const float iD2 = 1.0f / (D * D);
        acc[0] += dLdt * ((-vx - qx) * D + N * 2.0f * vx) * iD2;
        acc[1] += dLdt * ((-vy - qy) * D + N * 2.0f * vy) * iD2;
        acc[2] += dLdt * (qx * D - N * 2.0f * vx) * iD2;
        acc[3] += dLdt * (qy * D - N * 2.0f * vy) * iD2;
    }
}

// Loss sum and colour / alpha gradient of a lone constant layer over black from the tile's pixel
// sums S = (S1 r, g, b, S2 r, g, b) over n pixels: the layer renders q = colour * alpha per
// channel, so sum (q - s)^2 = n q^2 - 2 q S1 + S2 and sum (q - s) = n q - S1.  g4 (may be null):
// d/dcolour0 (3) and d/dalpha, scaled by gscale.  Every float64 operation is rounded on its own,
// so both kernels that use it agree bit for bit.
__device__ __forceinline__ double const_layer_closed(const Prep& P, float alpha_raw, const double* S, int n,
                                                     float gscale, float* g4) {
    const float sv[3] = {P.cr, P.cg, P.cb};
    const double nd = (double)n;
    double tot = 0.0, galpha = 0.0;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const float c = __fmul_rn(sv[ch], P.a);  // blend over black: colour * alpha
        const double cc = (double)clamp01(c);
        const double e = __dadd_rn(__dsub_rn(__dmul_rn(__dmul_rn(nd, cc), cc), __dmul_rn(__dmul_rn(2.0, cc), S[ch])),
                                   S[3 + ch]);
        tot = __dadd_rn(tot, e);
        const float G = (c >= 0.0f && c <= 1.0f)
                            ? (float)__dmul_rn((double)gscale, __dsub_rn(__dmul_rn(nd, (double)c), S[ch]))
                            : 0.0f;
        if (g4) g4[ch] = __fmul_rn(G, P.a);
        galpha = __dadd_rn(galpha, (double)__fmul_rn(G, sv[ch]));
    }
    if (g4) g4[3] = (alpha_raw >= 0.0f && alpha_raw <= 1.0f) ? (float)galpha : 0.0f;
    return tot;
}

constexpr int RF_LOSS = 0, RF_GRAD = 1, RF_STEP = 2;

// Loss (MODE 0), loss + gradient (MODE 1), and loss + gradient + Adam step on the tile's own rows
// (MODE 2: params are updated in place; a group reads its row once at staging and writes it once at
// the end, and rows belong to one tile) of stacks of at most one layer, of kind constant or linear
// (checked per tile): the forward and backward run out of registers.
template <int MODE>
__global__ void __launch_bounds__(RF_THREADS, 3)
    refine_tiles_kernel(WeftStackSet set, float* __restrict__ params, const float* __restrict__ grad_loss,
                        float* __restrict__ grad, float* __restrict__ loss, RefinePlan plan, AdamArgs adam,
                        int n_steps) {
    constexpr bool BWD = MODE != RF_LOSS;
    extern __shared__ __align__(16) unsigned char rf_smem[];
    const int bx = blockIdx.x;
    const int cls = (bx >= plan.cta_end[0]) + (bx >= plan.cta_end[1]) + (bx >= plan.cta_end[2]);
    const int cta0 = cls ? pick(plan.cta_end, cls - 1) : 0;
    const int wpt = class_wpt(cls), G = pick(plan.groups, cls);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp / wpt, wig = warp - grp * wpt;  // group, warp inside the group
    if (grp >= G) return;
    const int li = ((int)blockIdx.x - cta0) * G + grp;
    if (li >= pick(plan.n_list, cls)) return;  // uniform over the group
    const int lo = pick(plan.list_off, cls);
    const int t = set.order ? set.order[lo + li] : lo + li;
    const GroupLayout lay = group_layout(wpt);
    unsigned char* base = rf_smem + (size_t)grp * lay.bytes;
    Prep* prep = reinterpret_cast<Prep*>(base + lay.prep);
    float* raw = reinterpret_cast<float*>(base + lay.raw);
    float* madam = reinterpret_cast<float*>(base + lay.madam);
    float* vadam = reinterpret_cast<float*>(base + lay.vadam);
    float* gacc_all = reinterpret_cast<float*>(base + lay.gacc);
    float* gacc = gacc_all + (size_t)wig * 14;
    double* lred = reinterpret_cast<double*>(base + lay.lred);
    double* mom = reinterpret_cast<double*>(base + lay.mom);

    const int ts = set.size[t];
    const int p0 = set.prim_off[t];
    const int K = set.prim_off[t + 1] - p0;
    if (!(ts >= 1 && ts <= 64 && K >= 0 && K <= 1)) {
        if (wig == 0 && lane == 0) {
            atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
            if (loss) loss[t] = __int_as_float(0x7fc00000);
        }
        return;
    }
    // a lone constant layer runs in refine_const_kernel when the tiles' pixel sums are given
    if (set.moments != nullptr && K == 1 && set.kind[p0] == K_CONST) return;
    const int gt = wig * 32 + lane, GT = wpt * 32;

    // ---- stage the layer (row, and for STEP the Adam moments, stay in shared memory across the
    //      launch's steps; everything else is re-derived every step)
    for (int i = gt; i < K * 16; i += GT) {
        raw[i] = params[(size_t)p0 * 16 + i];
        if (MODE == RF_STEP) {
            madam[i] = adam.m[(size_t)p0 * 16 + i];
            vadam[i] = adam.v[(size_t)p0 * 16 + i];
        }
    }
    const float4* src = reinterpret_cast<const float4*>(set.src) + set.px_off[t];
    const int n = ts * ts;
    const int chunks = (n + 31) >> 5;
    const int c_begin = (chunks * wig) / wpt, c_end = (chunks * (wig + 1)) / wpt;
    const int lts = (ts & (ts - 1)) == 0 ? __ffs(ts) - 1 : -1;  // log2(side) for power-of-two sides
    auto load_src = [&](int q) -> float4 { return q < n ? src[q] : make_float4(0.0f, 0.0f, 0.0f, 0.0f); };

    // A lone constant layer over black renders one colour q per channel (q = colour * alpha), so
    // its loss and gradient follow from the tile's pixel sums S1 = sum src, S2 = sum src^2:
    // sum over pixels of (q - src) = n q - S1, sum of (q - src)^2 = n q^2 - 2 q S1 + S2.  They are
    // taken once per launch (float64, a fixed order: per lane, then per warp, then per group).
    const bool cf = K == 1 && set.kind[p0] == K_CONST;
    if (cf) {
        double m6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int q = gt; q < n; q += GT) {
            const float4 v = src[q];
            m6[0] += v.x;
            m6[1] += v.y;
            m6[2] += v.z;
            m6[3] += (double)v.x * v.x;
            m6[4] += (double)v.y * v.y;
            m6[5] += (double)v.z * v.z;
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m6[i] += __shfl_xor_sync(FULL, m6[i], o);
        }
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < 6; ++i) mom[wig * 6 + i] = m6[i];
        group_sync(wpt, grp);
        if (gt < 6) {
            double tot = 0.0;
            for (int w = 0; w < wpt; ++w) tot += mom[w * 6 + gt];
            mom[wpt * 6 + gt] = tot;
        }
    }
    const double* S12 = mom + wpt * 6;

    double sse = 0.0;
    for (int step = 0; step < n_steps; ++step) {
        sse = 0.0;
        group_sync(wpt, grp);
        if (gt < K) {
            Prep P = prep_prim(row_to_prim(raw, set.kind[p0]));
            if (P.kind == K_BICUBIC) P.kind = K_SKIP;
            prep[0] = P;
        }
        if (BWD)
            for (int i = lane; i < K * 14; i += 32) gacc[i] = 0.0f;
        group_sync(wpt, grp);
        if (K == 1 && gt == 0 && prep[0].kind != K_CONST && prep[0].kind != K_LINEAR && prep[0].kind != K_SKIP)
            atomicCAS(&g_device_status, 0, WEFTK_E_ARG);  // not a constant/linear layer: treated as absent

        const float scale = BWD ? grad_loss[t] * 2.0f / (3.0f * (float)n) : 0.0f;
        float4 vn = c_begin < c_end && !cf ? load_src(c_begin * 32 + lane) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float acc[14];
#pragma unroll
        for (int i = 0; i < 14; ++i) acc[i] = 0.0f;
        if (cf && gt == 0) {
            float g4[4];
            sse = const_layer_closed(prep[0], raw[13], S12, n, scale, BWD ? g4 : nullptr);
            if (BWD) {
                gacc[7] = g4[0];
                gacc[8] = g4[1];
                gacc[9] = g4[2];
                gacc[13] = g4[3];
            }
        }
        for (int cidx = c_begin; !cf && cidx < c_end; ++cidx) {
            const int q = cidx * 32 + lane;
            const float4 v4 = vn;
            if (cidx + 1 < c_end) vn = load_src(q + 32);
            if (q >= n || (BWD && K == 0)) continue;
            const int y = lts >= 0 ? q >> lts : q / ts, x = lts >= 0 ? q & (ts - 1) : q - y * ts;
            const float px = (float)x + 0.5f, py = (float)y + 0.5f;
            ClEval v{};
            float c[3] = {0.0f, 0.0f, 0.0f}, e[3];
            if (K == 1) {
                v = eval_cl(prep[0], px, py);
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) c[ch] = blend(v.s[ch], v.a, 0.0f);
            }
            e[0] = clamp01(c[0]) - v4.x;
            e[1] = clamp01(c[1]) - v4.y;
            e[2] = clamp01(c[2]) - v4.z;
            sse += (double)fmaf(e[0], e[0], fmaf(e[1], e[1], e[2] * e[2]));
            if (BWD) {
                float g[3];
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) g[ch] = (c[ch] >= 0.0f && c[ch] <= 1.0f) ? scale * e[ch] : 0.0f;
                grad_cl(prep[0], raw, v, px, py, g, acc);
            }
        }
        if (!BWD) continue;
        if (K == 1 && !cf) {
            const unsigned cols = grad_columns(prep[0].kind);
#pragma unroll
            for (int i = 0; i < 14; ++i) {
                if (!((cols >> i) & 1u)) continue;
                float s2 = acc[i];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(FULL, s2, o);
                if (lane == 0) gacc[i] = s2;
            }
        }
        if (MODE == RF_STEP && gt < K)  // the row's bias corrections for this step (column 14 is free)
            adam_bias(adam.b1, adam.b2, madam[15] + 1.0f, madam[14], vadam[14]);
        group_sync(wpt, grp);
        for (int j = gt; j < K * 16; j += GT) {
            float s = 0.0f;
            if (j < 14)
                for (int w = 0; w < wpt; ++w) s += gacc_all[(size_t)w * 14 + j];
            if (grad && step == n_steps - 1) grad[(size_t)p0 * 16 + j] = s;
            if (MODE == RF_STEP && j < 14) {
                float m = madam[j], v = vadam[j];
                raw[j] = adam_update_bc(raw[j], s, m, v, madam[14], vadam[14], adam.lr, adam.b1, adam.b2, adam.eps,
                                        set.kind[p0], j);
                madam[j] = m;
                vadam[j] = v;
            }
        }
        if (MODE == RF_STEP) {
            group_sync(wpt, grp);  // every column of the row has read its step count
            if (gt < K) madam[15] += 1.0f;
        }
    }
    if (MODE == RF_STEP) {
        group_sync(wpt, grp);
        for (int i = gt; i < K * 16; i += GT) {
            const bool scratch = i == 14;  // bias-correction scratch, not state
            params[(size_t)p0 * 16 + i] = raw[i];
            adam.m[(size_t)p0 * 16 + i] = scratch ? 0.0f : madam[i];
            adam.v[(size_t)p0 * 16 + i] = scratch ? 0.0f : vadam[i];
        }
    }
    if (loss != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sse += __shfl_xor_sync(FULL, sse, o);
        if (lane == 0) lred[wig] = sse;
        group_sync(wpt, grp);
        if (gt == 0) {
            double tot = 0.0;
            for (int w = 0; w < wpt; ++w) tot += lred[w];
            loss[t] = (float)(tot / (3.0 * n));
        }
    }
}

// ------------------------------------------------------------------ general stacks
// Stacks of any kind and length, with or without the residual loss.
//
// A warp owns 32 * GN_P consecutive pixels of the tile's visit order at a time (GN_P per lane), so a
// layer's terms (shared-memory broadcasts, a curve's 31 segments above all) are read once for the
// lane's pixels and their dependent chains overlap.  The visit order is row-major, or in residual
// mode block-major and quadrant-major inside a block, so block and quadrant sums are sums inside a
// lane followed by a few shuffles over aligned lanes (an 8-px tile: residual8, shuffles alone).  The
// forward pass keeps every layer's composite below it, coverage and closest curve segment in
// thread-private memory, so the backward pass evaluates no layer again; the residual loss keeps each
// pixel's error in shared memory between its passes.  A layer's gradient columns are summed over
// the lane's pixels first and then reduced by one transposing butterfly (16 shuffles for up to 16
// columns instead of 5 each).  What a row needs once per step is spread over lanes: its prepared
// terms over four (one float64 division for all of them), the bias corrections of 32 steps over one
// warp.
//
// Bound: instruction issue.  On 1024 x 1024 pixels in 7,435 tiles, 1 .. 3 layers, 20 residual-aware
// Adam steps: 2.16 ms (11.6 ms for the kernel this replaces, which kept its history per 32-pixel
// chunk in shared memory, evaluated each layer three times a step and reduced every column by
// itself); ncu on a quarter of it: 1.6 instructions per cycle, instruction fetch the largest stall
// (warps of different tiles run different kinds), which is why the pixels per lane are 2 (4 per
// lane: 2.8 ms) and why more resident warps with fewer registers were slower (3 x 256 threads at 80
// registers: 4.4 ms).  Loss and gradient of 512 x 512 pixels with 1 .. 4 layers: 39 us (223 us).
constexpr int GN_THREADS = 512;
constexpr int GN_WARPS = GN_THREADS / 32;
constexpr int GN_CLASSES = 4;
constexpr int GN_P = 2;  // pixels per lane
// tiles of side > 32: 16 warps (four pixel runs each at 64 px), 17..32: 16, 9..16: 4, <= 8: 1
__host__ __device__ __forceinline__ int gn_wpt(int c) { return c < 2 ? GN_WARPS : c == 2 ? 4 : 1; }
__host__ __device__ __forceinline__ int gn_side(int c) { return 64 >> c; }
__device__ __forceinline__ int gn_class_of(int ts) { return ts > 32 ? 0 : ts > 16 ? 1 : ts > 8 ? 2 : 3; }

struct GeneralLayout {
    int prep, seg, aux, raw, madam, vadam, msum, quad, hnode, err, gacc, lred, bias, kind, bytes;
};

// msum holds up to four partial sums per block (a large tile's block spans several warps' runs);
// err the pixels' errors of a tile of the class (residual mode).
__host__ __device__ __forceinline__ GeneralLayout general_layout(int L, int c, bool resid) {
    GeneralLayout g;
    const int wpt = gn_wpt(c), n = gn_side(c) * gn_side(c);
    g.prep = 0;
    g.seg = g.prep + L * 64;
    g.aux = g.seg + L * 992;
    g.raw = g.aux + L * 96;
    g.madam = g.raw + L * 64;
    g.vadam = g.madam + L * 64;
    g.msum = g.vadam + L * 64;
    g.quad = g.msum + (resid ? 192 * 4 : 0);
    g.hnode = g.quad + (resid ? 768 * 4 : 0);
    g.err = g.hnode + (resid ? 48 * 4 : 0);
    g.gacc = g.err + (resid ? n * 12 : 0);
    g.lred = (g.gacc + wpt * L * 56 + 15) & ~15;
    g.bias = g.lred + wpt * 8;  // bias corrections of the next 32 steps
    g.kind = g.bias + 2 * 32 * 4;
    g.bytes = (g.kind + L * 4 + 15) & ~15;
    return g;
}

struct GeneralPlan {
    int cta_end[GN_CLASSES];
    int list_off[GN_CLASSES];
    int n_list[GN_CLASSES];
    int groups[GN_CLASSES];
    int filter;  // no order given: every class lists all tiles and keeps its own sides
};

// Sums 16 values over the warp: on return lane l holds in v[0] the total of value
// (bit 4, bit 3, bit 2, bit 1 of l read as an index); lanes l and l ^ 1 hold the same one.
__device__ __forceinline__ void warp_transpose_sum16(float (&v)[16], int lane) {
#pragma unroll
    for (int w = 8, o = 16; w >= 1; w >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
            v[i] = keep + __shfl_xor_sync(FULL, send, o);
        }
    }
    v[0] += __shfl_xor_sync(FULL, v[0], 1);
}

// The same for four values: lane l holds the total of value (bit 4, bit 3 of l).
__device__ __forceinline__ void warp_transpose_sum4(float (&v)[4], int lane) {
#pragma unroll
    for (int w = 2, o = 16; w >= 1; w >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
            v[i] = keep + __shfl_xor_sync(FULL, send, o);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v[0] += __shfl_xor_sync(FULL, v[0], o);
}

// Column of a kind's i-th reduced value (its gradient columns, packed).
__device__ __forceinline__ int packed_column(int kind, int i) {
    switch (kind) {
        case K_LINEAR: return i < 4 ? i : i + 3;                         // 0-3, 7-13
        case K_LINE: return i < 5 ? i : i < 8 ? i + 2 : 13;              // 0-4, 7-9, 13
        case K_CURVE: return i < 10 ? i : 13;                            // 0-9, 13
        default: return i < 6 ? i : i < 9 ? i + 1 : 13;                  // triangle: 0-5, 7-9, 13
    }
}
__device__ __forceinline__ int packed_count(int kind) {
    return kind == K_LINEAR ? 11 : kind == K_LINE ? 9 : kind == K_CURVE ? 11 : kind == K_TRI ? 10 : 0;
}

// Edge i (opposite vertex i) of a triangle's soft coverage prod sigmoid(s_i / w), with
// s_i = o C_i / L_i, C = ex (py - ay) - ey (px - ax) the signed distance to it (positive inside).
__device__ __forceinline__ void soft_edge(const float* g, int i, float4 (&out)[2]) {
    const float vx[3] = {g[0], g[2], g[4]}, vy[3] = {g[1], g[3], g[5]};
    const float o = (vx[1] - vx[0]) * (vy[2] - vy[0]) - (vy[1] - vy[0]) * (vx[2] - vx[0]) >= 0.0f ? 1.0f : -1.0f;
    const int ia = i == 2 ? 0 : i + 1, ib = i == 0 ? 2 : i - 1;
    const float ax = g[2 * ia], ay = g[2 * ia + 1];
    const float ex = g[2 * ib] - ax, ey = g[2 * ib + 1] - ay;
    const float L = sqrtf(ex * ex + ey * ey) + 1e-12f, iL = 1.0f / L;
    out[0] = make_float4(ax, ay, ex, ey);
    out[1] = make_float4(o * iL * (1.0f / TRI_SOFT_W), o * (iL * iL), iL, L);
}
// sigmoids of the three edges at a point (and C), their product
__device__ __forceinline__ float soft_cov(const float4* e, float px, float py, float (&sig)[3], float (&C)[3]) {
    float cov = 1.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float4 a = e[2 * i];
        C[i] = a.z * (py - a.y) - a.w * (px - a.x);
        sig[i] = sigmoid(C[i] * e[2 * i + 1].x);
        cov *= sig[i];
    }
    return cov;
}

// What the forward pass leaves of a layer at a pixel: the composite below it, the coverage (the
// layer's alpha is coverage * P.a) and, for a curve, the closest segment.
template <int LT, int P>
struct History {
    float4 c[LT][P];
    int seg[LT][P];
};

template <int P>
struct RunPixels {
    float x[P], y[P];
};

// Composite of the tile's K layers at the lane's P pixels, with the history when BWD.
template <int LT, int P, bool BWD>
__device__ __forceinline__ void general_forward(const Layers& S, int K, bool soft, const RunPixels<P>& px,
                                                float (&c)[P][3], History<LT, P>& h) {
#pragma unroll
    for (int j = 0; j < P; ++j) c[j][0] = c[j][1] = c[j][2] = 0.0f;
    for (int k = 0; k < K; ++k) {
        const Prep Q = S.prep[k];
        float cov[P];
        int sg[P];
#pragma unroll
        for (int j = 0; j < P; ++j) {
            cov[j] = 1.0f;
            sg[j] = 0;
        }
        float t[P];
        switch (Q.kind) {
            case K_CONST:
                break;
            case K_LINEAR:
#pragma unroll
                for (int j = 0; j < P; ++j) t[j] = clamp01(fmaf(px.x[j] - Q.q[0], Q.q[2], (px.y[j] - Q.q[1]) * Q.q[3]));
                break;
            case K_LINE:
#pragma unroll
                for (int j = 0; j < P; ++j)
                    cov[j] = expf(seg_d2(px.x[j], px.y[j], Q.q[0], Q.q[1], Q.q[2], Q.q[3], Q.q[4], Q.q[5]) * Q.q[6]);
                break;
            case K_CURVE: {
                float best[P];
#pragma unroll
                for (int j = 0; j < P; ++j) best[j] = 1e18f;
#pragma unroll 2
                for (int i = 0; i < 31; ++i) {
                    const float4 s0 = S.seg[k][i][0];
                    const float2 s1 = *reinterpret_cast<const float2*>(&S.seg[k][i][1]);
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        const float d = seg_d2(px.x[j], px.y[j], s0.x, s0.y, s0.z, s0.w, s1.x, s1.y);
                        if (BWD) {
                            if (d < best[j]) {
                                best[j] = d;
                                sg[j] = i;
                            }
                        } else {
                            best[j] = fminf(best[j], d);
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < P; ++j) cov[j] = expf(best[j] * Q.q[0]);
                break;
            }
            case K_TRI:
                if (soft) {
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        float sig[3], C[3];
                        cov[j] = soft_cov(S.aux[k], px.x[j], px.y[j], sig, C);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < P; ++j) cov[j] = tri_inside(Q, px.x[j], px.y[j]);
                }
                break;
            default:
#pragma unroll
                for (int j = 0; j < P; ++j) cov[j] = 0.0f;
        }
#pragma unroll
        for (int j = 0; j < P; ++j) {
            if (BWD) {
                h.c[k][j] = make_float4(c[j][0], c[j][1], c[j][2], cov[j]);
                if (Q.kind == K_CURVE) h.seg[k][j] = sg[j];
            }
            const float a = cov[j] * Q.a;
            float s0 = Q.cr, s1 = Q.cg, s2 = Q.cb;
            if (Q.kind == K_LINEAR) {
                const float u = 1.0f - t[j];
                s0 = fmaf(Q.q[4], t[j], s0 * u);
                s1 = fmaf(Q.q[5], t[j], s1 * u);
                s2 = fmaf(Q.q[6], t[j], s2 * u);
            }
            c[j][0] = blend(s0, a, c[j][0]);
            c[j][1] = blend(s1, a, c[j][1]);
            c[j][2] = blend(s2, a, c[j][2]);
        }
    }
}

// Gradients of the K layers from dL/dc at the lane's P pixels, added into gacc (the warp's rows).
template <int LT, int P>
__device__ __forceinline__ void general_backward(const Layers& S, int K, const RunPixels<P>& px, float (&g)[P][3],
                                                 const History<LT, P>& h, float* gacc, int lane) {
    for (int k = K - 1; k >= 0; --k) {
        const Prep Q = S.prep[k];
        if (Q.kind == K_SKIP) continue;  // coverage 0: the gradient passes through
        const float* r = S.raw[k];
        const float A = Q.a;
        const float dA = (r[13] >= 0.0f && r[13] <= 1.0f) ? 1.0f : 0.0f;
        float d[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = 0.0f;
        if (Q.kind == K_CONST) {
            float d4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const float4 cp = h.c[k][j];
                d4[0] = fmaf(g[j][0], A, d4[0]);
                d4[1] = fmaf(g[j][1], A, d4[1]);
                d4[2] = fmaf(g[j][2], A, d4[2]);
                d4[3] += fmaf(g[j][2], Q.cb - cp.z, fmaf(g[j][1], Q.cg - cp.y, g[j][0] * (Q.cr - cp.x)));
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) g[j][ch] *= (1.0f - A);
            }
            d4[3] *= dA;
            warp_transpose_sum4(d4, lane);
            if ((lane & 7) == 0) {
                const int i = lane >> 3;
                gacc[k * 14 + (i < 3 ? 7 + i : 13)] += d4[0];
            }
            continue;
        }
        if (Q.kind == K_LINEAR) {
            const float x0 = r[0], y0 = r[1], vx = r[2] - r[0], vy = r[3] - r[1];
            const float D = S.aux[k][0].x, iD2 = S.aux[k][0].y;
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const float4 cp = h.c[k][j];
                const float qx = px.x[j] - x0, qy = px.y[j] - y0, N = qx * vx + qy * vy;
                const float traw = fmaf(qx, Q.q[2], qy * Q.q[3]);
                const float t = clamp01(traw), u = 1.0f - t;
                const float s0 = fmaf(Q.q[4], t, Q.cr * u), s1 = fmaf(Q.q[5], t, Q.cg * u),
                            s2 = fmaf(Q.q[6], t, Q.cb * u);
                const float l0 = g[j][0] * A, l1 = g[j][1] * A, l2 = g[j][2] * A;
                d[4] = fmaf(l0, u, d[4]);
                d[5] = fmaf(l1, u, d[5]);
                d[6] = fmaf(l2, u, d[6]);
                d[7] = fmaf(l0, t, d[7]);
                d[8] = fmaf(l1, t, d[8]);
                d[9] = fmaf(l2, t, d[9]);
                d[10] += fmaf(g[j][2], s2 - cp.z, fmaf(g[j][1], s1 - cp.y, g[j][0] * (s0 - cp.x)));
                if (traw > 0.0f && traw < 1.0f) {
                    // dN/dp0 = -v - q, dN/dp1 = q; dD/dp0 = -2v, dD/dp1 = 2v
                    const float dLdt = l0 * (r[10] - r[7]) + l1 * (r[11] - r[8]) + l2 * (r[12] - r[9]);
                    d[0] += dLdt * ((-vx - qx) * D + N * 2.0f * vx) * iD2;
                    d[1] += dLdt * ((-vy - qy) * D + N * 2.0f * vy) * iD2;
                    d[2] += dLdt * (qx * D - N * 2.0f * vx) * iD2;
                    d[3] += dLdt * (qy * D - N * 2.0f * vy) * iD2;
                }
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) g[j][ch] *= (1.0f - A);
            }
            d[10] *= dA;
        } else if (Q.kind == K_TRI) {
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const float4 cp = h.c[k][j];
                const float cov = cp.w, a = cov * A;
                d[6] = fmaf(g[j][0], a, d[6]);
                d[7] = fmaf(g[j][1], a, d[7]);
                d[8] = fmaf(g[j][2], a, d[8]);
                const float dLda = fmaf(g[j][2], Q.cb - cp.z, fmaf(g[j][1], Q.cg - cp.y, g[j][0] * (Q.cr - cp.x)));
                d[9] = fmaf(dLda, cov, d[9]);
                float sig[3], C[3];
                const float sc = soft_cov(S.aux[k], px.x[j], px.y[j], sig, C) * (1.0f / TRI_SOFT_W) * (dLda * A);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int ia = (i + 1) % 3, ib = (i + 2) % 3;
                    const float4 e = S.aux[k][2 * i], f = S.aux[k][2 * i + 1];
                    // dC/da = (-ry + ey, rx - ex), dC/db = (ry, -rx); dL/da = -e/L, dL/db = e/L
                    const float rx = px.x[j] - e.x, ry = px.y[j] - e.y;
                    const float ci = C[i] * f.z, cx = ci * e.z, cy = ci * e.w;
                    const float w = sc * (1.0f - sig[i]) * f.y;
                    d[2 * ia] = fmaf(w, fmaf(e.w - ry, f.w, cx), d[2 * ia]);
                    d[2 * ia + 1] = fmaf(w, fmaf(rx - e.z, f.w, cy), d[2 * ia + 1]);
                    d[2 * ib] = fmaf(w, fmaf(ry, f.w, -cx), d[2 * ib]);
                    d[2 * ib + 1] = fmaf(w, fmaf(-rx, f.w, -cy), d[2 * ib + 1]);
                }
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) g[j][ch] *= (1.0f - a);
            }
            d[9] *= dA;
        } else {  // line, curve
            const bool line = Q.kind == K_LINE;
            const float thick = line ? r[4] : r[6];
            const float i3 = S.aux[k][0].x;
            const float Kf = line ? Q.q[6] : Q.q[0];
            float th = 0.0f;
            float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, al = 0.0f;
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const float4 cp = h.c[k][j];
                const float cov = cp.w, a = cov * A;
                c0 = fmaf(g[j][0], a, c0);
                c1 = fmaf(g[j][1], a, c1);
                c2 = fmaf(g[j][2], a, c2);
                const float dLda = fmaf(g[j][2], Q.cb - cp.z, fmaf(g[j][1], Q.cg - cp.y, g[j][0] * (Q.cr - cp.x)));
                al = fmaf(dLda, cov, al);
                const float dLdcov = dLda * A;
                float ax, ay, vx, vy, ux, uy;
                float te[2] = {0.0f, 0.0f};  // a curve's segment: the parameters of its ends
                if (line) {
                    ax = Q.q[0]; ay = Q.q[1]; vx = Q.q[2]; vy = Q.q[3]; ux = Q.q[4]; uy = Q.q[5];
                } else {
                    const int sg = h.seg[k][j];
                    const float4 s0 = S.seg[k][sg][0], s1 = S.seg[k][sg][1];
                    ax = s0.x; ay = s0.y; vx = s0.z; vy = s0.w; ux = s1.x; uy = s1.y; te[0] = s1.z; te[1] = s1.w;
                }
                const float dx = px.x[j] - ax, dy = px.y[j] - ay;
                const float t = clamp01(fmaf(dx, ux, dy * uy));
                const float ex = fmaf(-t, vx, dx), ey = fmaf(-t, vy, dy);
                const float d2 = fmaf(ex, ex, ey * ey);
                const float w = -2.0f * dLdcov * Kf * cov;
                // dd2/d(start) = -2e(1-t), dd2/d(end) = -2e t
                const float gsx = ex * (1.0f - t) * w, gsy = ey * (1.0f - t) * w;
                const float gex = ex * t * w, gey = ey * t * w;
                th += dLdcov * cov * d2;
                if (line) {
                    d[0] += gsx;
                    d[1] += gsy;
                    d[2] += gex;
                    d[3] += gey;
                } else {
                    // polyline points are Bezier samples q_i = u^2 P0 + 2ut C + t^2 P1, at the forward pass's t
#pragma unroll
                    for (int e2 = 0; e2 < 2; ++e2) {
                        const float ti = te[e2], ui = 1.0f - ti;
                        const float w0 = ui * ui, w1 = 2.0f * ui * ti, w2 = ti * ti;
                        const float gx = e2 ? gex : gsx, gy = e2 ? gey : gsy;
                        d[0] = fmaf(w0, gx, d[0]);
                        d[1] = fmaf(w0, gy, d[1]);
                        d[2] = fmaf(w1, gx, d[2]);
                        d[3] = fmaf(w1, gy, d[3]);
                        d[4] = fmaf(w2, gx, d[4]);
                        d[5] = fmaf(w2, gy, d[5]);
                    }
                }
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) g[j][ch] *= (1.0f - a);
            }
            th = thick > 0.5f ? th * i3 : 0.0f;
            al *= dA;
            if (line) {
                d[4] = th;
                d[5] = c0;
                d[6] = c1;
                d[7] = c2;
                d[8] = al;
            } else {
                d[6] = th;
                d[7] = c0;
                d[8] = c1;
                d[9] = c2;
                d[10] = al;
            }
        }
        warp_transpose_sum16(d, lane);
        const int i = lane >> 1;
        if (!(lane & 1) && i < packed_count(Q.kind)) gacc[k * 14 + packed_column(Q.kind, i)] += d[0];
    }
}

// A quarter of a layer's prepared terms (prep_prim's values): four lanes per layer, so that the
// float64 divisions of all layers (the two projection components and the falloff) are one division.
__device__ __forceinline__ void prep_quarter(Prep& out, float4 (&aux)[6], const float* r, int kind, int part) {
    float* q = out.q;
    const bool seg = kind == K_LINEAR || kind == K_LINE;
    const double vx = (double)r[2] - (double)r[0], vy = (double)r[3] - (double)r[1];
    const double sg = fmax(0.5, (double)(kind == K_LINE ? r[4] : r[6]));
    const double num = part == 0 ? vx : part == 1 ? vy : 1.0;
    const double den = part < 2 ? vx * vx + vy * vy + 1e-8 : 2.0 * sg * sg;
    const float v = (float)(num / den);
    if (kind == K_TRI && part < 3) {
        float4 e[2];
        soft_edge(r, part, e);
        aux[2 * part] = e[0];
        aux[2 * part + 1] = e[1];
    }
    if (part == 3) {
        const float c0 = r[7], c1 = r[8], c2 = r[9];
        int kd = kind >= K_CONST && kind <= K_TRI ? kind : K_SKIP;  // bicubic rows are inert
        if (kind == K_TRI) {
            const WeftPrim p = row_to_prim(r, kind);
            const Prep t = prep_prim(p);
            kd = t.kind;
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = t.q[i];
        } else if (kind == K_CURVE) {
#pragma unroll
            for (int i = 0; i < 6; ++i) q[1 + i] = r[i];
        } else if (seg) {
            q[0] = r[0];
            q[1] = r[1];
            if (kind == K_LINEAR) {
                const float fx = r[2] - r[0], fy = r[3] - r[1], D = fx * fx + fy * fy + 1e-8f;
                aux[0] = make_float4(D, 1.0f / (D * D), 0.0f, 0.0f);
                q[4] = r[10];
                q[5] = r[11];
                q[6] = r[12];
            } else {
                q[2] = (float)vx;
                q[3] = (float)vy;
            }
        }
        out.kind = kd;
        out.a = clamp01(r[13]);
        out.cr = c0;
        out.cg = c1;
        out.cb = c2;
    } else if (part == 2) {
        const float sf = fmaxf(0.5f, kind == K_LINE ? r[4] : r[6]);
        if (kind == K_LINE || kind == K_CURVE) aux[0] = make_float4(1.0f / (sf * sf * sf), 0.0f, 0.0f, 0.0f);
        if (kind == K_LINE) q[6] = -v;
        if (kind == K_CURVE) q[0] = -v;
    } else if (seg) {
        q[(kind == K_LINEAR ? 2 : 4) + part] = v;
    }
}

// The residual loss of an 8-px tile in one warp's registers: lane l holds row l / 4, columns
// 2 (l % 4) and the next, which are its 2 x 2 block's columns, so a block's sum is the two pixels
// plus lane l ^ 4's, and the 4 x 4 grid's bilinear upsampling B and its transpose (weights 3/4 for
// the pixel's own block and 1/4 for the neighbour its half faces, clamped at the border) are
// exchanges with the lanes one block to the side or above and below.  out: the derivative of the
// loss with respect to the clamped composite, up to its scale: r - M^T B^T r with r = e - B M e.
template <bool BWD>
__device__ __forceinline__ void residual8(const float (&c)[2][3], const float4 (&v)[2], int lane, float (&out)[2][3],
                                          double& sse, bool last) {
    const int bc = lane & 3, row = lane >> 2;
    const int left = bc > 0 ? lane - 1 : lane, right = bc < 3 ? lane + 1 : lane;
    const int facing = row & 1 ? (row < 7 ? lane + 8 : lane) : (row > 0 ? lane - 8 : lane);   // the faced block row
    const int sender = row & 1 ? (row < 7 ? lane + 4 : lane) : (row > 0 ? lane - 4 : lane);  // the row facing this block
    const float cy = row == 0 || row == 7 ? 1.0f : 0.75f, cl = bc == 0 ? 1.0f : 0.75f, cr = bc == 3 ? 1.0f : 0.75f;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const float s0 = ch == 0 ? v[0].x : ch == 1 ? v[0].y : v[0].z, s1 = ch == 0 ? v[1].x : ch == 1 ? v[1].y : v[1].z;
        const float e0 = clamp01(c[0][ch]) - s0, e1 = clamp01(c[1][ch]) - s1;
        float m = e0 + e1;
        m = 0.25f * (m + __shfl_xor_sync(FULL, m, 4));
        const float ml = __shfl_sync(FULL, m, left), mr = __shfl_sync(FULL, m, right);
        const float x0 = fmaf(0.75f, m - ml, ml), x1 = fmaf(0.25f, mr - m, m);
        const float n0 = __shfl_sync(FULL, x0, facing), n1 = __shfl_sync(FULL, x1, facing);
        const float r0 = e0 - fmaf(0.25f, n0 - x0, x0), r1 = e1 - fmaf(0.25f, n1 - x1, x1);
        if (last) sse += (double)fmaf(r0, r0, r1 * r1);
        if (BWD) {
            float h0 = fmaf(cy, r0, __shfl_sync(FULL, (1.0f - cy) * r0, sender));
            float h1 = fmaf(cy, r1, __shfl_sync(FULL, (1.0f - cy) * r1, sender));
            h0 += __shfl_xor_sync(FULL, h0, 4);
            h1 += __shfl_xor_sync(FULL, h1, 4);
            const float from_l = __shfl_sync(FULL, (1.0f - cr) * h1, left);
            const float from_r = __shfl_sync(FULL, (1.0f - cl) * h0, right);
            const float h = fmaf(cl, h0, cr * h1) + ((bc > 0 ? from_l : 0.0f) + (bc < 3 ? from_r : 0.0f));
            out[0][ch] = fmaf(-0.25f, h, r0);
            out[1][ch] = fmaf(-0.25f, h, r1);
        }
    }
}

// One tile by its group of warps: all steps of the launch.  LT: history depth (>= K).
template <int MODE, int LT, int P, bool RESID>
__device__ __forceinline__ void general_tile(const WeftStackSet& set, float* __restrict__ params,
                                             const float* __restrict__ grad_loss, float* __restrict__ grad,
                                             float* __restrict__ loss, int flags, int L, int cls, int t, int ts, int K,
                                             int p0, int grp, int wig, int lane, unsigned char* base, AdamArgs adam,
                                             int n_steps, bool cl_only) {
    constexpr bool BWD = MODE != RF_LOSS;
    const int wpt = gn_wpt(cls);
    constexpr bool resid = RESID;
    const bool soft = flags & WEFTK_SOFT_TRIANGLES;
    const GeneralLayout lay = general_layout(L, cls, resid);
    Prep* prep = reinterpret_cast<Prep*>(base + lay.prep);
    float4(*seg)[31][2] = reinterpret_cast<float4(*)[31][2]>(base + lay.seg);
    float4(*aux)[6] = reinterpret_cast<float4(*)[6]>(base + lay.aux);
    float(*raw)[16] = reinterpret_cast<float(*)[16]>(base + lay.raw);
    float* madam = reinterpret_cast<float*>(base + lay.madam);
    float* vadam = reinterpret_cast<float*>(base + lay.vadam);
    float* msum = reinterpret_cast<float*>(base + lay.msum);
    float* quad = reinterpret_cast<float*>(base + lay.quad);
    float* hnode = reinterpret_cast<float*>(base + lay.hnode);
    float* err = reinterpret_cast<float*>(base + lay.err);
    float* gacc_all = reinterpret_cast<float*>(base + lay.gacc);
    float* gacc = gacc_all + (size_t)wig * L * 14;
    double* lred = reinterpret_cast<double*>(base + lay.lred);
    float* bias = reinterpret_cast<float*>(base + lay.bias);
    int* kinds = reinterpret_cast<int*>(base + lay.kind);
    const int gt = wig * 32 + lane, GT = wpt * 32;

    for (int i = gt; i < K; i += GT) {
        int kind = set.kind[p0 + i];
        if (cl_only && kind > K_LINEAR && kind <= K_TRI) {
            atomicCAS(&g_device_status, 0, WEFTK_E_ARG);  // outside the declared kinds: treated as absent
            kind = K_SKIP;
        }
        kinds[i] = kind;
    }
    for (int i = gt; i < K * 16; i += GT) {
        raw[i >> 4][i & 15] = params[(size_t)p0 * 16 + i];
        if (MODE == RF_STEP) {
            madam[i] = adam.m[(size_t)p0 * 16 + i];
            vadam[i] = adam.v[(size_t)p0 * 16 + i];
        }
    }
    const Layers S{prep, raw, seg, aux};
    const float4* src = reinterpret_cast<const float4*>(set.src) + set.px_off[t];
    const int n = ts * ts;
    const int runs = (n + wpt * 32 * P - 1) / (wpt * 32 * P);  // 1, but for a 64-px tile's 16 warps (4)
    const int err_px = gn_side(cls) * gn_side(cls);
    const bool keep_err = n <= err_px;
    // Residual-mode geometry (side a power of two >= 8): block side b, block pixels bb,
    // quadrant side h = b / 2, quadrant pixels Q = bb / 4.
    const int lb = resid ? (__ffs(ts) - 1) - 2 : 0;  // log2(b)
    const int b = 1 << lb, lbb = 2 * lb, bb = 1 << lbb;
    const int lq = resid ? lbb - 2 : 0, Q = 1 << lq, lh = resid ? lb - 1 : 0, h = 1 << lh;
    const float gscale = resid ? 4.0f / (float)ts : 0.0f;
    const float inv_bb = resid ? 1.0f / (float)bb : 0.0f;
    const int lts = (ts & (ts - 1)) == 0 ? __ffs(ts) - 1 : -1;

    // an 8-px tile by one warp: row-major, a lane's two pixels are its block's columns, and the
    // residual loss runs on shuffles alone
    const bool r8 = resid && ts == 8 && wpt == 1;
    // pixel (x, y) of visit index q
    auto pixel_of = [&](int q, int& x, int& y) {
        if (resid && !r8) {
            const int j = q >> lbb, o = q & (bb - 1), qd = o >> lq, u = o & (Q - 1);
            x = (j & 3) * b + (qd & 1) * h + (u & (h - 1));
            y = (j >> 2) * b + (qd >> 1) * h + (u >> lh);
        } else if (lts >= 0) {
            y = q >> lts;
            x = q & (ts - 1);
        } else {
            y = q / ts;
            x = q - y * ts;
        }
    };
    // the lane's pixels of run i: P neighbours of the visit order (pixels past the tile repeat its last)
    auto first_of = [&](int i) { return ((i * wpt + wig) * 32 + lane) * P; };
    auto load_run = [&](int i, RunPixels<P>& px) {
        const int q0 = first_of(i);
#pragma unroll
        for (int j = 0; j < P; ++j) {
            int x, y;
            pixel_of(min(q0 + j, n - 1), x, y);
            px.x[j] = (float)x + 0.5f;
            px.y[j] = (float)y + 0.5f;
        }
    };
    auto load_src = [&](const RunPixels<P>& px, float4 (&v)[P]) {
#pragma unroll
        for (int j = 0; j < P; ++j) v[j] = __ldg(src + (int)px.y[j] * ts + (int)px.x[j]);
    };
    // decoded-error correction B M e at a pixel (block means in msum), and its node weights
    auto correction = [&](float px, float py, float (&v)[3], float& wx, float& wy) {
        int x0, x1, y0, y1;
        grid_coord((int)px, gscale, x0, x1, wx);
        grid_coord((int)py, gscale, y0, y1, wy);
        const float* r0 = msum + y0 * 12;
        const float* r1 = msum + y1 * 12;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const float c00 = r0[x0 * 3 + ch], c01 = r0[x1 * 3 + ch];
            const float c10 = r1[x0 * 3 + ch], c11 = r1[x1 * 3 + ch];
            const float top = fmaf(c01 - c00, wx, c00), bot = fmaf(c11 - c10, wx, c10);
            v[ch] = fmaf(bot - top, wy, top);
        }
    };

    History<LT, P> hist;
    double sse = 0.0;
    group_sync(wpt, grp);
    // the rows' step counts: where they agree (as a rule), the bias corrections come from a table of
    // the next 32 steps, one step per lane
    bool same_t = true;
    if (MODE == RF_STEP)
        for (int k = lane; k < K; k += 32) same_t = same_t && madam[k * 16 + 15] == madam[15];
    same_t = __all_sync(FULL, same_t);
    for (int step = 0; step < n_steps; ++step) {
        sse = 0.0;
        if (MODE == RF_STEP && same_t && (step & 31) == 0 && wig == wpt - 1 && K > 0)
            adam_bias(adam.b1, adam.b2, madam[15] + (float)(step + lane + 1), bias[lane], bias[32 + lane]);
        for (int i = gt; i < K * 4; i += GT) prep_quarter(prep[i >> 2], aux[i >> 2], raw[i >> 2], kinds[i >> 2], i & 3);
        for (int k = wig; k < K; k += wpt) {
            if (kinds[k] != K_CURVE) continue;
            // the polyline's points one per lane, the segments from their neighbours (lane_segment's values)
            const float* r = raw[k];
            const float tt = lane >= 31 ? 1.0f : (float)((double)lane * (1.0 / 31.0)), u = __fsub_rn(1.0f, tt);
            const float uu = __fmul_rn(u, u), ut2 = __fmul_rn(__fmul_rn(2.0f, u), tt), t2 = __fmul_rn(tt, tt);
            const float x = __fadd_rn(__fadd_rn(__fmul_rn(uu, r[0]), __fmul_rn(ut2, r[2])), __fmul_rn(t2, r[4]));
            const float y = __fadd_rn(__fadd_rn(__fmul_rn(uu, r[1]), __fmul_rn(ut2, r[3])), __fmul_rn(t2, r[5]));
            const float vx = __fsub_rn(__shfl_down_sync(FULL, x, 1), x), vy = __fsub_rn(__shfl_down_sync(FULL, y, 1), y);
            const float next = __shfl_down_sync(FULL, tt, 1);  // the ends' parameters, for the backward pass
            const float den = __fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), 1e-8f);
            if (lane < 31) {
                seg[k][lane][0] = make_float4(x, y, vx, vy);
                seg[k][lane][1] = make_float4(__fdiv_rn(vx, den), __fdiv_rn(vy, den), tt, next);
            }
        }
        if (BWD)
            for (int i = lane; i < K * 14; i += 32) gacc[i] = 0.0f;
        group_sync(wpt, grp);

        RunPixels<P> px;
        float c[P][3], r8e[P][3];
        const bool last = step == n_steps - 1;  // only the last step's loss is reported
        if (r8) {
            load_run(0, px);
            float4 v[P];
            load_src(px, v);
            general_forward<LT, P, BWD>(S, K, soft, px, c, hist);
            residual8<BWD>(c, v, lane, r8e, sse, last);
        } else if (RESID) {
            // ---- pass 1: block sums of e
            for (int i = 0; i < runs; ++i) {
                load_run(i, px);
                float4 v[P];
                load_src(px, v);
                general_forward<LT, P, BWD>(S, K, soft, px, c, hist);
                const int q0 = first_of(i);
                float s[3] = {0.0f, 0.0f, 0.0f};
                float e[P][3];
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const bool in = q0 + j < n;
                    e[j][0] = in ? clamp01(c[j][0]) - v[j].x : 0.0f;
                    e[j][1] = in ? clamp01(c[j][1]) - v[j].y : 0.0f;
                    e[j][2] = in ? clamp01(c[j][2]) - v[j].z : 0.0f;
                    if (keep_err && in) {
#pragma unroll
                        for (int ch = 0; ch < 3; ++ch) err[ch * err_px + q0 + j] = e[j][ch];
                    }
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch) s[ch] += e[j][ch];
                }
                // bb >= 4 >= P: the lane's pixels lie in one block
                const int span = min(bb / P, 32);
                for (int o = 1; o < span; o <<= 1)
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch) s[ch] += __shfl_xor_sync(FULL, s[ch], o);
                if ((lane & (span - 1)) == 0 && q0 < n) {
                    const int j = q0 >> lbb, part = (q0 & (bb - 1)) / (32 * P);
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch) msum[part * 48 + j * 3 + ch] = s[ch];
                }
            }
            group_sync(wpt, grp);
            for (int i = gt; i < 48; i += GT) {
                float s = msum[i];
                for (int part = 1; part < bb / (32 * P); ++part) s += msum[part * 48 + i];
                msum[i] = s * inv_bb;
            }
            group_sync(wpt, grp);
            // ---- pass 2: r = e - B M e; loss; per-quadrant sums of (bilinear weight x r)
            for (int i = 0; i < runs; ++i) {
                const int q0 = first_of(i);
                if (runs > 1) load_run(i, px);
                float4 v[P];
                if (!keep_err) {
                    load_src(px, v);
                    general_forward<LT, P, false>(S, K, soft, px, c, hist);
                }
                // the lane's quadrant sums: one quadrant (Q >= P) or one per pixel (Q = 1, P = 2)
                float acc[12];
#pragma unroll
                for (int u = 0; u < 12; ++u) acc[u] = 0.0f;
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const bool in = q0 + j < n;
                    float corr[3], r[3], wx, wy;
                    correction(px.x[j], px.y[j], corr, wx, wy);
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch) {
                        const float e = !in ? 0.0f
                                        : keep_err ? err[ch * err_px + q0 + j]
                                                   : clamp01(c[j][ch]) - (ch == 0 ? v[j].x : ch == 1 ? v[j].y : v[j].z);
                        r[ch] = in ? e - corr[ch] : 0.0f;
                        if (keep_err && in) err[ch * err_px + q0 + j] = r[ch];
                    }
                    if (last) sse += (double)fmaf(r[0], r[0], fmaf(r[1], r[1], r[2] * r[2]));
                    if (BWD) {
                        const float w4[4] = {(1.0f - wx) * (1.0f - wy), wx * (1.0f - wy), (1.0f - wx) * wy, wx * wy};
                        if (Q < P) {
                            if (in)
#pragma unroll
                                for (int u = 0; u < 12; ++u) quad[(q0 + j) * 12 + u] = w4[u / 3] * r[u % 3];
                        } else {
#pragma unroll
                            for (int u = 0; u < 12; ++u) acc[u] = fmaf(w4[u / 3], r[u % 3], acc[u]);
                        }
                    }
                }
                if (BWD && Q >= P) {
                    const int span = Q / P;  // <= 32 lanes (a 64-px tile's quadrants of 64 pixels)
                    for (int o = 1; o < span; o <<= 1)
#pragma unroll
                        for (int u = 0; u < 12; ++u) acc[u] += __shfl_xor_sync(FULL, acc[u], o);
                    if ((lane & (span - 1)) == 0 && q0 < n) {
#pragma unroll
                        for (int u = 0; u < 12; ++u) quad[(q0 >> lq) * 12 + u] = acc[u];
                    }
                }
            }
            if (BWD) {
                group_sync(wpt, grp);
                // B^T r per node: sum of the (column, slot) x (row, slot) quadrant entries that
                // interpolate from this node.
                for (int i = gt; i < 48; i += GT) {
                    const int node = i / 3, ch = i - node * 3;
                    float acc = 0.0f;
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const int sy = node_source(node >> 2, a), qy = sy >> 1, sly = sy & 1;
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc) {
                            const int sx = node_source(node & 3, cc), qx = sx >> 1, slx = sx & 1;
                            const int qi = (((qy >> 1) * 4 + (qx >> 1)) << 2) + ((qy & 1) << 1) + (qx & 1);
                            if (sy >= 0 && sx >= 0) acc += quad[qi * 12 + (sly * 2 + slx) * 3 + ch];
                        }
                    }
                    hnode[i] = acc * inv_bb;
                }
                group_sync(wpt, grp);
            }
        }

        if (BWD || !resid) {
            const float scale = BWD ? grad_loss[t] * 2.0f / (3.0f * (float)n) : 0.0f;
            for (int i = 0; i < runs; ++i) {
                const int q0 = first_of(i);
                if (!r8 && (!resid || runs > 1 || !keep_err)) {
                    load_run(i, px);
                    general_forward<LT, P, BWD>(S, K, soft, px, c, hist);
                }
                float4 v[P];
                if (!r8 && (!resid || !keep_err)) load_src(px, v);
                float g[P][3];
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const bool in = q0 + j < n;
                    float e[3];
                    if (!r8 && (!resid || !keep_err)) {
                        e[0] = clamp01(c[j][0]) - v[j].x;
                        e[1] = clamp01(c[j][1]) - v[j].y;
                        e[2] = clamp01(c[j][2]) - v[j].z;
                    }
                    if (r8) {
#pragma unroll
                        for (int ch = 0; ch < 3; ++ch) e[ch] = r8e[j][ch];
                    } else if (resid) {
                        const int blk = min(q0 + j, n - 1) >> lbb;
                        float corr[3] = {0.0f, 0.0f, 0.0f}, wx, wy;
                        if (!keep_err) correction(px.x[j], px.y[j], corr, wx, wy);
#pragma unroll
                        for (int ch = 0; ch < 3; ++ch)
                            e[ch] = (keep_err ? (in ? err[ch * err_px + q0 + j] : 0.0f) : e[ch] - corr[ch]) -
                                    hnode[blk * 3 + ch];
                    } else if (in && last) {
                        sse += (double)fmaf(e[0], e[0], fmaf(e[1], e[1], e[2] * e[2]));
                    }
#pragma unroll
                    for (int ch = 0; ch < 3; ++ch)
                        g[j][ch] = (in && c[j][ch] >= 0.0f && c[j][ch] <= 1.0f) ? scale * e[ch] : 0.0f;
                }
                if (BWD) general_backward<LT, P>(S, K, px, g, hist, gacc, lane);
            }
        }
        if (BWD) {
            if (MODE == RF_STEP && !same_t)  // each row's bias corrections for this step, once (column 14 is free)
                for (int k = gt; k < K; k += GT)
                    adam_bias(adam.b1, adam.b2, madam[k * 16 + 15] + (float)(step + 1), madam[k * 16 + 14],
                              vadam[k * 16 + 14]);
            group_sync(wpt, grp);
            for (int i = gt; i < K * 16; i += GT) {
                const int k = i >> 4, j = i & 15;
                float s = 0.0f;
                if (j < 14)
                    for (int w = 0; w < wpt; ++w) s += gacc_all[((size_t)w * L + k) * 14 + j];
                if (grad && step == n_steps - 1) grad[(size_t)(p0 + k) * 16 + j] = s;
                if (MODE == RF_STEP && j < 14) {
                    float m = madam[k * 16 + j], v = vadam[k * 16 + j];
                    const float bc1 = same_t ? bias[step & 31] : madam[k * 16 + 14];
                    const float bc2 = same_t ? bias[32 + (step & 31)] : vadam[k * 16 + 14];
                    raw[k][j] = adam_update_bc(raw[k][j], s, m, v, bc1, bc2, adam.lr, adam.b1, adam.b2, adam.eps,
                                               kinds[k], j);
                    madam[k * 16 + j] = m;
                    vadam[k * 16 + j] = v;
                }
            }
        }
        group_sync(wpt, grp);
    }
    if (MODE == RF_STEP) {
        for (int i = gt; i < K * 16; i += GT) {
            const bool scratch = (i & 15) == 14;  // bias-correction scratch, not state
            params[(size_t)p0 * 16 + i] = raw[i >> 4][i & 15];
            adam.m[(size_t)p0 * 16 + i] = scratch ? 0.0f : madam[i] + ((i & 15) == 15 ? (float)n_steps : 0.0f);
            adam.v[(size_t)p0 * 16 + i] = scratch ? 0.0f : vadam[i];
        }
    }
    if (loss != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sse += __shfl_xor_sync(FULL, sse, o);
        if (lane == 0) lred[wig] = sse;
        group_sync(wpt, grp);
        if (gt == 0) {
            double tot = 0.0;
            for (int w = 0; w < wpt; ++w) tot += lred[w];
            loss[t] = (float)(tot / (3.0 * n));
        }
    }
}

template <int MODE, int LT, bool RESID>
__global__ void __launch_bounds__(GN_THREADS, 1)
    refine_general_kernel(WeftStackSet set, float* __restrict__ params, const float* __restrict__ grad_loss,
                          float* __restrict__ grad, float* __restrict__ loss, int flags, GeneralPlan plan, int L,
                          AdamArgs adam, int n_steps, bool cl_only) {
    extern __shared__ __align__(16) unsigned char rf_smem[];
    const int bx = blockIdx.x;
    const int cls = (bx >= plan.cta_end[0]) + (bx >= plan.cta_end[1]) + (bx >= plan.cta_end[2]);
    const int cta0 = cls ? pick(plan.cta_end, cls - 1) : 0;
    const int wpt = gn_wpt(cls), G = pick(plan.groups, cls);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp / wpt, wig = warp - grp * wpt;
    if (grp >= G) return;
    const int li = (bx - cta0) * G + grp;
    if (li >= pick(plan.n_list, cls)) return;  // uniform over the group
    const int lo = pick(plan.list_off, cls);
    const int t = set.order ? set.order[lo + li] : li;
    constexpr bool resid = RESID;
    const int ts = set.size[t];
    if (plan.filter && gn_class_of(ts) != cls) return;
    const int p0 = set.prim_off[t];
    const int K = set.prim_off[t + 1] - p0;
    bool ok = ts >= 1 && ts <= 64 && K >= 0 && K <= L && (!cl_only || K <= 1);
    if (resid) ok = ok && (ts == 8 || ts == 16 || ts == 32 || ts == 64);
    if (!ok) {
        if (wig == 0 && lane == 0) {
            atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
            if (loss) loss[t] = __int_as_float(0x7fc00000);
        }
        return;
    }
    unsigned char* base = rf_smem + (size_t)grp * general_layout(L, cls, resid).bytes;
    general_tile<MODE, LT, GN_P, RESID>(set, params, grad_loss, grad, loss, flags, L, cls, t, ts, K, p0, grp, wig, lane, base,
                                 adam, n_steps, cl_only);
}

// One thread per tile whose stack is one constant layer (register path, primitives-only loss,
// the tiles' pixel sums given): the same arithmetic as refine_tiles_kernel's closed form for such a
// tile — loss n q^2 - 2 q S1 + S2 and gradient from n q - S1 per channel, Adam with projection on
// the row's colour and alpha (its other columns have zero gradient and stay where they are), the
// row's step count and bias corrections as the group path keeps them.
template <int MODE>
__global__ void __launch_bounds__(128) refine_const_kernel(WeftStackSet set, float* __restrict__ params,
                                                           const float* __restrict__ grad_loss,
                                                           float* __restrict__ grad, float* __restrict__ loss,
                                                           AdamArgs adam, int n_steps) {
    constexpr bool BWD = MODE != RF_LOSS;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= set.n_tiles) return;
    const int p0 = set.prim_off[t];
    if (set.prim_off[t + 1] - p0 != 1 || set.kind[p0] != K_CONST) return;
    const int ts = set.size[t];
    if (ts < 1 || ts > 64) return;  // reported by refine_tiles_kernel
    const int n = ts * ts;
    double S[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) S[i] = set.moments[(size_t)t * 6 + i];
    float* row = params + (size_t)p0 * 16;
    float r[16], m[16], v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        r[i] = row[i];
        m[i] = MODE == RF_STEP ? adam.m[(size_t)p0 * 16 + i] : 0.0f;
        v[i] = MODE == RF_STEP ? adam.v[(size_t)p0 * 16 + i] : 0.0f;
    }
    const float scale = BWD ? grad_loss[t] * 2.0f / (3.0f * (float)n) : 0.0f;
    // Columns other than the colour (7..9) and alpha (13) have zero gradient.  Where their moments
    // start at zero an Adam update leaves them at zero and moves the value by exactly 0, so such a
    // column only takes the projection, at the first step.
    unsigned idle = 0;
#pragma unroll
    for (int j = 0; j < 14; ++j)
        if (!(j >= 7 && j <= 9) && j != 13 && m[j] == 0.0f && v[j] == 0.0f) idle |= 1u << j;
    double sse = 0.0;
    float g4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int step = 0; step < n_steps; ++step) {
        const Prep P = prep_prim(row_to_prim(r, K_CONST));
        const double tot = const_layer_closed(P, r[13], S, n, scale, g4);
        sse = tot;
        if (MODE == RF_STEP) {
            adam_bias(adam.b1, adam.b2, m[15] + 1.0f, m[14], v[14]);
#pragma unroll
            for (int j = 0; j < 14; ++j) {
                if ((idle >> j) & 1u) {
                    if (step == 0) r[j] = adam_project(r[j], K_CONST, j);
                    continue;
                }
                const float gj = j >= 7 && j <= 9 ? g4[j - 7] : j == 13 ? g4[3] : 0.0f;
                r[j] = adam_update_bc(r[j], gj, m[j], v[j], m[14], v[14], adam.lr, adam.b1, adam.b2, adam.eps,
                                     K_CONST, j);
            }
            m[15] += 1.0f;
        }
    }
    if (BWD && grad) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            grad[(size_t)p0 * 16 + j] = j >= 7 && j <= 9 ? g4[j - 7] : j == 13 ? g4[3] : 0.0f;
    }
    if (MODE == RF_STEP) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            row[i] = r[i];
            adam.m[(size_t)p0 * 16 + i] = i == 14 ? 0.0f : m[i];
            adam.v[(size_t)p0 * 16 + i] = i == 14 ? 0.0f : v[i];
        }
    }
    if (loss != nullptr) loss[t] = (float)(sse / (3.0 * n));
}

// A side stream of the current device for the calling host thread, with the two events that fork
// work onto it and join it back.  Created on first use and kept for the life of the process (one
// per host thread and device, so concurrent callers never share the events).
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};

static int side_stream(SideStream** out) {
    thread_local std::map<int, SideStream> per_device;
    int dev = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    SideStream& s = per_device[dev];
    if (s.stream == nullptr) {
        WEFTK_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
        WEFTK_CUDA(cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming));
        WEFTK_CUDA(cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming));
    }
    *out = &s;
    return WEFTK_OK;
}

// The general kernel with history depth LT.  counts: tiles per class of the given order (ignored
// without one).
template <int MODE, int LT, bool RESID>
static int launch_general_depth(const WeftStackSet& set, float* params, const float* grad_loss, float* grad,
                                float* loss, int flags, const int* counts, int L, AdamArgs adam, cudaStream_t stream,
                                int n_steps, bool cl_only) {
    GeneralPlan plan{};
    plan.filter = set.order == nullptr;
    int smem = 0, ctas = 0, off = 0;
    for (int c = 0; c < GN_CLASSES; ++c) {
        const int bytes = general_layout(L, c, RESID).bytes;
        const int g = std::min(GN_WARPS / gn_wpt(c), RF_SMEM_MAX / bytes);
        plan.groups[c] = g;
        plan.list_off[c] = off;
        plan.n_list[c] = plan.filter ? set.n_tiles : counts[c];
        if (!plan.filter) off += counts[c];
        ctas += (plan.n_list[c] + g - 1) / g;
        plan.cta_end[c] = ctas;
        if (plan.n_list[c]) smem = std::max(smem, g * bytes);
    }
    // the dynamic shared-memory opt-in is per device and per kernel instance: remember the
    // largest size set on each device (under a lock, so concurrent first calls agree)
    {
        int dev = 0;
        WEFTK_CUDA(cudaGetDevice(&dev));
        static std::mutex mu;
        static std::map<int, int> granted;
        std::lock_guard<std::mutex> lock(mu);
        int& have = granted.try_emplace(dev, 48 * 1024).first->second;
        if (smem > have) {
            WEFTK_CUDA(cudaFuncSetAttribute(refine_general_kernel<MODE, LT, RESID>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            have = smem;
        }
    }
    refine_general_kernel<MODE, LT, RESID><<<ctas, GN_THREADS, smem, stream>>>(set, params, grad_loss, grad, loss, flags, plan,
                                                                        L, adam, n_steps, cl_only);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

template <int MODE>
static int launch_general(const WeftStackSet& set, float* params, const float* grad_loss, float* grad, float* loss,
                          int flags, const int* counts, int L, AdamArgs adam, cudaStream_t stream, int n_steps,
                          bool cl_only) {
    const bool resid = (flags & WEFTK_LOSS_RESIDUAL) != 0;
    // the loss alone keeps no history
    const int depth = MODE == RF_LOSS || L <= 4 ? 4 : L <= 16 ? 16 : MAXL;
    auto run = [&](auto lt) {
        constexpr int LT = decltype(lt)::value;
        return resid ? launch_general_depth<MODE, LT, true>(set, params, grad_loss, grad, loss, flags, counts, L, adam,
                                                            stream, n_steps, cl_only)
                     : launch_general_depth<MODE, LT, false>(set, params, grad_loss, grad, loss, flags, counts, L, adam,
                                                             stream, n_steps, cl_only);
    };
    if constexpr (MODE != RF_LOSS) {
        if (depth == 16) return run(std::integral_constant<int, 16>{});
        if (depth == MAXL) return run(std::integral_constant<int, MAXL>{});
    }
    return run(std::integral_constant<int, 4>{});
}

template <int MODE>
static int launch_refine(const WeftStackSet& set, float* params, const float* grad_loss, float* grad, float* loss,
                         int flags, AdamArgs adam, cudaStream_t stream, const char* what, int n_steps = 1) {
    if (n_steps < 1 || (MODE != RF_STEP && n_steps != 1)) return fail(WEFTK_E_ARG, std::string(what) + ": bad step count");
    if (set.n_tiles == 0) return WEFTK_OK;
    if (set.max_prims < 0 || set.max_prims > MAXL) return fail(WEFTK_E_RANGE, std::string(what) + ": stack too long");
    if (!params || !set.src || !set.px_off || !set.size || !set.prim_off || (set.max_prims > 0 && !set.kind))
        return fail(WEFTK_E_ARG, std::string(what) + ": null pointer in the stack set");
    const int L = set.max_prims > 0 ? set.max_prims : 1;
    int counts[RF_CLASSES] = {0, 0, 0, 0};
    if (set.order != nullptr) {
        if (set.n_big < 0 || set.n_mid < 0 || set.n_s16 < 0 ||
            (long long)set.n_big + set.n_mid + set.n_s16 > set.n_tiles)
            return fail(WEFTK_E_ARG, std::string(what) + ": bad size-class counts");
        counts[0] = set.n_big;
        counts[1] = set.n_mid;
        counts[2] = set.n_s16;
        counts[3] = set.n_tiles - set.n_big - set.n_mid - set.n_s16;
    }
    // single constant/linear layers only (declared by the caller, checked per tile)
    const bool cl1 = set.max_prims <= 1 && set.kinds_mask != 0 && (set.kinds_mask & ~0x3) == 0;
    const bool resid = (flags & WEFTK_LOSS_RESIDUAL) != 0;
    if (!cl1 || resid) return launch_general<MODE>(set, params, grad_loss, grad, loss, flags, counts, L, adam, stream, n_steps, cl1);

    // the register path
    if (set.order == nullptr) counts[1] = set.n_tiles;  // no split: four warps per tile
    RefinePlan plan{};
    int smem = 0, ctas = 0, off = 0;
    for (int c = 0; c < RF_CLASSES; ++c) {
        const int g = 8 / class_wpt(c);
        plan.groups[c] = g;
        plan.list_off[c] = off;
        plan.n_list[c] = counts[c];
        off += counts[c];
        ctas += (counts[c] + g - 1) / g;
        plan.cta_end[c] = ctas;
        if (counts[c]) smem = std::max(smem, g * group_layout(class_wpt(c)).bytes);  // a few KB
    }
    // lone constant layers (closed form, a thread per tile) run beside the other tiles' launch, on
    // this thread's side stream of the device (forked from and joined back into `stream`, which a
    // CUDA graph capture follows)
    SideStream* side = nullptr;
    if (set.moments != nullptr) {
        int rc = side_stream(&side);
        if (rc) return rc;
        WEFTK_CUDA(cudaEventRecord(side->fork, stream));
        WEFTK_CUDA(cudaStreamWaitEvent(side->stream, side->fork, 0));
        refine_const_kernel<MODE><<<(set.n_tiles + 127) / 128, 128, 0, side->stream>>>(set, params, grad_loss, grad,
                                                                                        loss, adam, n_steps);
        WEFTK_CUDA(cudaGetLastError());
        WEFTK_CUDA(cudaEventRecord(side->join, side->stream));
    }
    refine_tiles_kernel<MODE><<<ctas, RF_THREADS, smem, stream>>>(set, params, grad_loss, grad, loss, plan, adam,
                                                                  n_steps);
    WEFTK_CUDA(cudaGetLastError());
    if (side) WEFTK_CUDA(cudaStreamWaitEvent(stream, side->join, 0));
    return WEFTK_OK;
}

// Row r of a refinement started from a fit: thread per (row, column).
__global__ void refine_start_kernel(WeftFitState fit, const int* __restrict__ tiles, int n_rows,
                                    float* __restrict__ params, float* __restrict__ m, float* __restrict__ v,
                                    int* __restrict__ kind_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * 16) return;
    const int row = i >> 4, col = i & 15;
    const int t = tiles[row];
    m[i] = 0.0f;
    v[i] = 0.0f;
    float x = 0.0f;
    int kind = -1;
    if (t >= 0 && t < fit.n_tiles && fit.n_sel[t] >= 1) {
        const int sel = fit.sel[(size_t)t * fit.cap_max];
        const WeftPrim& P = fit.cand[fit.pool_off[t] + sel];
        kind = P.kind;
        if (col < 7) {
            const bool thick = (kind == K_LINE && col == 4) || (kind == K_CURVE && col == 6);
            x = fminf(fmaxf(P.geom[col], 0.0f), thick ? 4.0f : 15.0f);
        } else if (col < 14) {
            const float c = col < 10 ? P.color0[col - 7] : col < 13 ? P.color1[col - 10] : P.alpha;
            x = fminf(fmaxf(c, 0.0f), 1.0f);
        }
    } else if (t < 0 || t >= fit.n_tiles) {
        if (col == 0) atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
    }
    params[i] = x;
    if (col == 0) kind_out[row] = kind;
}

// Adam (PyTorch's rule) + projection onto the wire-representable box, one thread per value.
__global__ void adam_project_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                    float* __restrict__ v, const int* __restrict__ kind, int n_rows, float lr,
                                    float b1, float b2, float eps, const int* __restrict__ step) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * 16) return;
    const int col = i & 15, row = i >> 4;
    if (col >= 14) return;
    float mi = m[i], vi = v[i];
    p[i] = adam_update(p[i], g[i], mi, vi, (float)(*step + 1), lr, b1, b2, eps, kind[row], col);
    m[i] = mi;
    v[i] = vi;
}

__global__ void step_increment_kernel(int* step) { *step += 1; }

}  // namespace weftk

using namespace weftk;

extern "C" int weftk_stack_loss(const WeftStackSet* set, const float* d_params, float* d_loss, int flags,
                                void* stream) {
    WEFTK_REQUIRE(set && d_loss, "stack_loss: null argument");
    return launch_refine<RF_LOSS>(*set, const_cast<float*>(d_params), nullptr, nullptr, d_loss, flags, AdamArgs{},
                                  (cudaStream_t)stream, "stack_loss");
}

extern "C" int weftk_refine_start(const WeftFitState* fit, const int32_t* d_tiles, int n_rows, float* d_params,
                                  float* d_m, float* d_v, int32_t* d_kind, void* stream) {
    WEFTK_REQUIRE(fit && n_rows >= 0, "refine_start: bad arguments");
    if (n_rows == 0) return WEFTK_OK;
    WEFTK_REQUIRE(d_tiles && d_params && d_m && d_v && d_kind, "refine_start: null pointer");
    const int n = n_rows * 16;
    refine_start_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(*fit, d_tiles, n_rows, d_params, d_m, d_v,
                                                                            d_kind);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_adam_step(float* d_params, const float* d_grads, float* d_m, float* d_v, const int32_t* d_kind,
                               int n_rows, float lr, float beta1, float beta2, float eps, int32_t* d_step,
                               void* stream) {
    WEFTK_REQUIRE(n_rows >= 0 && (n_rows == 0 || (d_params && d_grads && d_m && d_v && d_kind && d_step)),
                  "adam_step: bad arguments");
    if (n_rows == 0) return WEFTK_OK;
    const int n = n_rows * 16;
    adam_project_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(d_params, d_grads, d_m, d_v, d_kind, n_rows,
                                                                            lr, beta1, beta2, eps, d_step);
    step_increment_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(d_step);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_stack_loss_backward(const WeftStackSet* set, const float* d_params, const float* d_grad_loss,
                                         float* d_grad_params, float* d_loss, int flags, void* stream) {
    WEFTK_REQUIRE(set && d_grad_loss && d_grad_params, "stack_loss_backward: null argument");
    return launch_refine<RF_GRAD>(*set, const_cast<float*>(d_params), d_grad_loss, d_grad_params, d_loss, flags,
                                  AdamArgs{}, (cudaStream_t)stream, "stack_loss_backward");
}

extern "C" int weftk_refine_step(const WeftStackSet* set, float* d_params, float* d_m, float* d_v,
                                 const float* d_grad_loss, float* d_loss, float* d_grad_params, float lr, float beta1,
                                 float beta2, float eps, int flags, void* stream) {
    WEFTK_REQUIRE(set && d_params && d_m && d_v && d_grad_loss, "refine_step: null argument");
    return launch_refine<RF_STEP>(*set, d_params, d_grad_loss, d_grad_params, d_loss, flags,
                                  AdamArgs{d_m, d_v, lr, beta1, beta2, eps}, (cudaStream_t)stream, "refine_step");
}

extern "C" int weftk_refine_steps(const WeftStackSet* set, int steps, float* d_params, float* d_m, float* d_v,
                                  const float* d_grad_loss, float* d_loss, float* d_grad_params, float lr, float beta1,
                                  float beta2, float eps, int flags, void* stream) {
    WEFTK_REQUIRE(set && d_params && d_m && d_v && d_grad_loss && steps >= 1, "refine_steps: bad argument");
    return launch_refine<RF_STEP>(*set, d_params, d_grad_loss, d_grad_params, d_loss, flags,
                                  AdamArgs{d_m, d_v, lr, beta1, beta2, eps}, (cudaStream_t)stream, "refine_steps",
                                  steps);
}
