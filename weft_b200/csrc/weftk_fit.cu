// weftk_fit.cu — device-resident greedy candidate-scoring fit (see include/weftk_fit.h).
//
// Scoring exploits the greedy's structure: every eval of a round is "the tile's
// selected stack + one candidate on top", and the over-composite is evaluated
// back to front, so the selected stack's composite (bg) is kept per pixel in
// HBM and each eval composites ONE primitive over it.  The float operations are
// the same sequence a full re-render performs, so results are identical to
// rendering the whole stack (blend() is shared with the decode walk).
//
// Most candidates are never scored: a candidate whose rate alone, or whose rate plus a cheap lower
// bound on its error, exceeds an objective the tile already has cannot be selected ("candidates that
// cannot win" below).  Plain fit of 1024^2 pixels at q = 75 (7,435 tiles, 2.08 M candidates): 3.28 ms
// scoring every candidate every round, 1.86 ms with the rate bound, 1.61 with rejected candidates
// skipped after a stall and items dealt in parts, 1.38 with one-warp tile tails and re-seeds off the
// critical path, 1.09 with the curves' error bound; 512^2 at q = 92: 3.13, 3.18, 2.34, 1.85, 1.79 ms.
//
// Work mapping (128-thread CTAs; a warp works on one candidate at a time, each lane owns PPL pixels
// held in registers):
//   8-px tiles   PPL=2, one warp covers the tile, warps pull their work one by one
//   16-px tiles  PPL=8, one warp covers the tile, warps pull their work one by one
//   32/64-px     PPL=8, four warps cover a 1024-pixel block; a CTA scores a run
//                of candidates on one block and combines the 4 warp sums in
//                shared memory in a fixed order.
// Per-candidate sums go to partial[slot*4 + block] (float32, fixed reduction
// order, so results are deterministic run to run).
#include <cuda_runtime.h>

#include <algorithm>

#include <climits>
#include <map>
#include <mutex>
#include <string>

#include "../../include/weftk_fit.h"
#include "weftk_common.cuh"
#include "weftk_prim.cuh"

namespace weftk {

extern __device__ int g_device_status;
__device__ __forceinline__ void fit_report(int code) { atomicCAS(&g_device_status, 0, code); }

__constant__ int c_prim_bytes[8] = WEFTK_PRIM_BYTES;

__device__ __forceinline__ int prim_bits(int kind) { return 8 * c_prim_bytes[(kind >= 0 && kind < 8) ? kind : 7]; }

// FP32 operations to evaluate and blend one primitive at one pixel (FMA = 2): const 10,
// linear 24, line 28, curve 31 segments x 16 + 13 = 509, triangle 26.
__constant__ int c_kind_ops[8] = {10, 24, 28, 509, 26, 0, 0, 0};
__device__ __forceinline__ int kind_ops(int kind) { return c_kind_ops[(kind >= 0 && kind < 8) ? kind : 7]; }

// ------------------------------------------------------------------ candidates that cannot win
// A candidate's objective is mse + lambda * bits with mse >= 0 (float32, rounded), so lambda * bits
// is a lower bound on it, and a candidate whose bound is above an objective the tile already has
// cannot be selected whatever its pixels say: it is neither scored nor looked at by the selection,
// and the selections are the same.  In a greedy round that objective is the tile's current one
// (acceptance is "strictly below it"); in the init round it is the best constant candidate's (they
// are the cheapest on the wire and to evaluate, and scored first, fit_const_*_kernel).  At quality 75 a
// linear patch costs 80 bits x 6.8e-5 = 5.4e-3 more than a constant, well above most tiles' error,
// so most tiles need only their constants.  (A NaN bound compares false and prunes nothing.)
constexpr int TILE_BOUNDED = 8;  // flags, inside the init round: cur_obj holds the best constant's objective
// Inside weftk_fit_run, flags >> TILE_SEEN: slots below it were scored against the tile's present
// composite and objective and rejected, so they stay rejected until a candidate is accepted.  A round
// after a stall therefore scores the re-seeded candidates alone.
constexpr int TILE_SEEN = 4;
constexpr int TILE_BITS = (1 << TILE_SEEN) - 1;
constexpr int BITS_CONST = 8 * 7, BITS_OTHER_MIN = 8 * 17;  // of WEFTK_PRIM_BYTES

__device__ __forceinline__ float rate_of(float lam, int bits) { return __fmul_rn(lam, (float)bits); }

// What a tile's candidates are measured against this round.
struct Bound {
    double obj;
    int base_bits, seen;
    bool on, init;
};

__device__ __forceinline__ Bound tile_bound(const WeftFitState& st, int t, bool init) {
    Bound b;
    b.init = init;
    b.base_bits = init ? 8 : st.sel_bits[t];
    b.on = !init || (st.flags[t] & TILE_BOUNDED);
    b.seen = st.flags[t] >> TILE_SEEN;
    b.obj = st.cur_obj[t];
    return b;
}

__device__ __forceinline__ bool pruned_bits(const Bound& b, float lam, int bits) {
    const double rate = (double)rate_of(lam, b.base_bits + bits);
    return b.on && (b.init ? rate > b.obj : rate >= b.obj);
}

// (the init round's constants are never pruned: the bound comes from them)
__device__ __forceinline__ bool pruned(const Bound& b, float lam, int kind) {
    return !(b.init && kind == K_CONST) && pruned_bits(b, lam, prim_bits(kind));
}

// Slot `local` of the tile (kind given) is to be scored and looked at this round.
__device__ __forceinline__ bool in_play(const Bound& b, float lam, int local, int kind) {
    return local >= b.seen && !pruned(b, lam, kind);
}

// No candidate of the tile that is left to score (after the constants, in the init round) can win.
__device__ __forceinline__ bool all_pruned(const Bound& b, float lam) {
    return lam >= 0.0f && pruned_bits(b, lam, b.init ? BITS_OTHER_MIN : BITS_CONST);
}

// A candidate's prepared terms, derived from its record where it is used: after the pruning above few
// candidates are evaluated at all, and a lane prepares one while the warp would wait for its loads.
// (Preparing every slot up front wrote and read 64 bytes a slot: 64 us of a 2.08 M candidate fit.)
__device__ __forceinline__ Prep load_prep(const WeftFitState& st, long long slot) {
    const float* f = reinterpret_cast<const float*>(st.cand + slot);
    WeftPrim c;
    c.kind = __ldg(reinterpret_cast<const int*>(f));
#pragma unroll
    for (int k = 0; k < 7; ++k) c.geom[k] = __ldg(f + 1 + k);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c.color0[k] = __ldg(f + 8 + k);
        c.color1[k] = __ldg(f + 11 + k);
    }
    c.alpha = __ldg(f + 14);
    // prep_prim's values with the divisions of every kind taken together (a warp's lanes hold
    // candidates of several kinds: kind by kind they would run one after another)
    const bool seg = c.kind == K_LINEAR || c.kind == K_LINE;
    const double vx = (double)c.geom[2] - (double)c.geom[0], vy = (double)c.geom[3] - (double)c.geom[1];
    const double den = vx * vx + vy * vy + 1e-8;
    const double sg = fmax(0.5, (double)(c.kind == K_LINE ? c.geom[4] : c.geom[6]));
    const float ux = (float)(vx / den), uy = (float)(vy / den), gk = -(float)(1.0 / (2.0 * sg * sg));
    if (c.kind == K_TRI) return prep_prim(c);
    Prep r;
    r.kind = c.kind >= K_CONST && c.kind <= K_CURVE ? c.kind : K_SKIP;  // bicubic grids are never fit candidates
    r.a = clamp01(c.alpha);
    r.cr = c.color0[0];
    r.cg = c.color0[1];
    r.cb = c.color0[2];
#pragma unroll
    for (int i = 0; i < 11; ++i) r.q[i] = 0.0f;
    if (seg) {
        r.q[0] = c.geom[0];
        r.q[1] = c.geom[1];
        if (c.kind == K_LINEAR) {
            r.q[2] = ux;
            r.q[3] = uy;
            r.q[4] = c.color1[0];
            r.q[5] = c.color1[1];
            r.q[6] = c.color1[2];
        } else {
            r.q[2] = (float)vx;
            r.q[3] = (float)vy;
            r.q[4] = ux;
            r.q[5] = uy;
            r.q[6] = gk;
        }
    } else if (c.kind == K_CURVE) {
        r.q[0] = gk;
#pragma unroll
        for (int i = 0; i < 6; ++i) r.q[1 + i] = c.geom[i];
    }
    return r;
}

__device__ __forceinline__ void put_prep(float4 (&dst)[4], const Prep& r) {
    dst[0] = make_float4(__int_as_float(r.kind), r.a, r.cr, r.cg);
    dst[1] = make_float4(r.cb, r.q[0], r.q[1], r.q[2]);
    dst[2] = make_float4(r.q[3], r.q[4], r.q[5], r.q[6]);
    dst[3] = make_float4(r.q[7], r.q[8], r.q[9], r.q[10]);
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// ------------------------------------------------------------------ prepare
__global__ void fit_prepare_kernel(WeftFitState st, const int* __restrict__ first_new) {
    const int t = blockIdx.x;
    if (t >= st.n_tiles) return;
    const int lo = first_new[t], hi = st.pool_cnt[t];
    const long long off = st.pool_off[t];
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const int kind = st.cand[off + i].kind;
        st.alive[off + i] = 1;
        st.kind[off + i] = (uint8_t)(kind >= 0 && kind < 8 ? kind : 7);
    }
    if (threadIdx.x == 0 && hi > lo) st.n_alive[t] += hi - lo;
}

// ------------------------------------------------------------------ round begin / end
// ctl (device-driven fit, may be NULL): [0] done, [1] stalls, [2] re-seed pending, [3] rounds.
// Whether the tile is evaluated this round.
__device__ __forceinline__ bool opens(const WeftFitState& st, int t, int mode, const int* ctl) {
    if (ctl != nullptr && ctl[0] != 0) return false;
    if (mode == WEFTK_FIT_INIT) return st.n_alive[t] > 0;
    return (st.flags[t] & WEFTK_TILE_COMPLEX) && st.n_alive[t] > 0 && st.n_sel[t] < st.cap[t];
}

__device__ __forceinline__ void begin_tile(const WeftFitState& st, int t, int mode, int* ctl) {
    if (t >= st.n_tiles) return;
    const bool ev = opens(st, t, mode, ctl);
    if (ctl != nullptr && t == 0) ctl[2] = 0;  // the pending re-seed (if any) ran before this launch
    int f = st.flags[t] & ~(WEFTK_TILE_EVAL | WEFTK_TILE_IMPROVED | TILE_BOUNDED);
    if (ctl == nullptr) f &= TILE_BITS;  // the fit's state may have changed since the last call
    if (ev) {
        f |= WEFTK_TILE_EVAL;
        atomicAdd(&st.status[0], 1);
    }
    st.flags[t] = f;
}

// The round's counters, the queue's and the fit's control block (each may be NULL): one launch, where
// a memset apiece cost a graph 4 us and its neighbours' gaps.
__global__ void fit_clear_kernel(int* status, int n_status, int* q_ctl, int* ctl) {
    const int i = threadIdx.x;
    if (i < n_status) status[i] = 0;
    if (q_ctl != nullptr && i < 8) q_ctl[i] = 0;
    if (ctl != nullptr && i < 4) ctl[i] = 0;
}

__global__ void fit_begin_kernel(WeftFitState st, int mode, int* ctl) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    begin_tile(st, t, mode, ctl);
}

// The round's end: the tiles' complexity, and (ctl given) the host loop's decisions on the device
// (src/weft/encoder.py:2745-2830): no evaluated tile ends the fit; a round without improvement is a
// stall, more than three stalls end it, otherwise a stall triggers a re-seed; an improving round
// resets the count.
__device__ __forceinline__ void fit_control(int evaluated, int improved, int* ctl) {
    if (ctl[0]) return;
    if (evaluated == 0) {
        ctl[0] = 1;
        return;
    }
    ctl[3] += 1;
    if (improved == 0) {
        ctl[1] += 1;
        if (ctl[1] > 3)
            ctl[0] = 1;
        else
            ctl[2] = 1;
    } else {
        ctl[1] = 0;
    }
}

__global__ void fit_end_kernel(WeftFitState st, int mode, double complex_threshold, int* ctl) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (st.queue_ctl != nullptr && t < 8) st.queue_ctl[t] = 0;  // for the next round
    if (t >= st.n_tiles) return;
    if (t == 0 && ctl != nullptr) fit_control(st.status[0], st.status[1], ctl);
    int f = st.flags[t] & ~TILE_BOUNDED;
    if (mode == WEFTK_FIT_INIT) {
        bool cx = st.cur_obj[t] > complex_threshold && st.n_alive[t] > 0;
        f = cx ? (f | WEFTK_TILE_COMPLEX) : (f & ~WEFTK_TILE_COMPLEX);
    } else if (*(volatile int*)&st.status[1] > 0) {
        f = (f & WEFTK_TILE_IMPROVED) ? (f | WEFTK_TILE_COMPLEX) : (f & ~WEFTK_TILE_COMPLEX);
    }
    st.flags[t] = f;
}

// The marks are meaningless to a later call.
// last: the last round's counters, moved to where a caller reads them.
__global__ void fit_unmark_kernel(WeftFitState st, const int* last) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) {
        const int a = last[0], b = last[1];
        st.status[0] = a;
        st.status[1] = b;
        st.status[2] = st.status[3] = 0;
    }
    if (t < st.n_tiles) st.flags[t] &= TILE_BITS;
}

// ------------------------------------------------------------------ scoring
// alpha (clamped) and colour of a constant slot
__device__ __forceinline__ float4 const_head(const WeftFitState& st, long long slot) {
    const float* f = reinterpret_cast<const float*>(st.cand + slot);
    return make_float4(clamp01(__ldg(f + 14)), __ldg(f + 8), __ldg(f + 9), __ldg(f + 10));
}

// Its squared error over the tile in closed form from the tile's pixel sums: it renders one colour q
// per channel, so sum over pixels and channels of (q - s)^2 = sum_ch n q^2 - 2 q S1 + S2.
__device__ __forceinline__ float const_closed_sse(const WeftFitState& st, int t, int ts, float4 h) {
    const double* mo = st.moments + (size_t)t * 6;
    const double npx = (double)(ts * ts);
    const float col[3] = {h.y, h.z, h.w};
    double e = 0.0;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const double q = (double)clamp01(blend(col[ch], h.x, 0.0f));
        e += npx * q * q - 2.0 * q * mo[ch] + mo[3 + ch];
    }
    return (float)e;
}

// A CTA first gathers the live candidates of its run into shared memory (prepared
// terms + slot), compacting out dead slots; warps then read their candidate's terms
// as warp-uniform shared-memory broadcasts.  A curve's 31 polyline segments are
// computed one per lane into the warp's segment table and read back the same way.
constexpr int MAX_ITEM = 128;

// Two float32 operations per instruction (each lane of the pair rounded on its own, so the values are
// the scalar ones): a curve's segments are the bulk of the scoring, and the kernels are bound by
// instruction issue, not by the FP32 pipe.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A curve segment with every term twice: (-ax, -ay), (-vx, -vy), (ux, uy).
struct __align__(16) Seg2 {
    f32x2 nax, nay, nvx, nvy, ux, uy;
};
__device__ __forceinline__ void put_seg2(Seg2& d, const Seg& s) {
    d.nax = pack2(-s.ax, -s.ax);
    d.nay = pack2(-s.ay, -s.ay);
    d.nvx = pack2(-s.vx, -s.vx);
    d.nvy = pack2(-s.vy, -s.vy);
    d.ux = pack2(s.ux, s.ux);
    d.uy = pack2(s.uy, s.uy);
}

// Alpha of a curve at PPL pixels (seg_d2 over the 31 segments, in their order); an odd last pixel is
// paired with itself.
template <int PPL>
__device__ __forceinline__ void curve_alpha2(const Prep& P, const Seg2* seg, const float (&fx)[PPL],
                                             const float (&fy)[PPL], float (&a)[PPL]) {
    constexpr int H = (PPL + 1) / 2;
    f32x2 x[H], y[H];
    float best[2 * H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int j1 = 2 * h + 1 < PPL ? 2 * h + 1 : 2 * h;
        x[h] = pack2(fx[2 * h], fx[j1]);
        y[h] = pack2(fy[2 * h], fy[j1]);
        best[2 * h] = best[2 * h + 1] = 1e18f;
    }
#pragma unroll(PPL <= 2 ? 4 : 1)
    for (int k = 0; k < 31; ++k) {
        const Seg2 s = seg[k];
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const f32x2 dx = add2(x[h], s.nax), dy = add2(y[h], s.nay), m = mul2(dy, s.uy);
            float d0, d1, m0, m1, u, unused;
            unpack2(dx, d0, d1);
            unpack2(m, m0, m1);
            unpack2(s.ux, u, unused);
            const f32x2 t = pack2(clamp01(fmaf(d0, u, m0)), clamp01(fmaf(d1, u, m1)));
            const f32x2 ex = fma2(t, s.nvx, dx), ey = fma2(t, s.nvy, dy);
            float q0, q1;
            unpack2(fma2(ex, ex, mul2(ey, ey)), q0, q1);
            best[2 * h] = fminf(best[2 * h], q0);
            best[2 * h + 1] = fminf(best[2 * h + 1], q1);
        }
    }
#pragma unroll
    for (int j = 0; j < PPL; ++j) a[j] = expf(best[j] * P.q[0]) * P.a;
}

// A lower bound on a curve's squared error at PPL pixels, at a seventh of the curve's cost (40
// instructions a pixel against 31 segments of 9), so that most curves, which are the bulk of the
// scoring and rarely win, need not be evaluated.  Every point of the polyline lies in one of two boxes
// (the control points' of its halves, widened for the chord that joins them and for rounding), so
// the coverage at a pixel is at most that of the distance to the nearer box, and the error at
// least that of the best blend weight up to it:
//     min over 0 <= w <= a exp(K d^2) of |v - w u|^2,  v = source - composite, u = colour - composite.
// (Clamping to [0, 1] changes nothing while colour and composite lie there, which the callers check.)
struct CurveBoxes {
    float x0, x1, y0, y1, u0, u1, w0, w1;  // first half, second half
};

__device__ __forceinline__ CurveBoxes curve_boxes(const Prep& P) {
    const float ax = P.q[1], ay = P.q[2], cx = P.q[3], cy = P.q[4], bx = P.q[5], by = P.q[6];
    const float px = 0.5f * (ax + cx), py = 0.5f * (ay + cy), rx = 0.5f * (cx + bx), ry = 0.5f * (cy + by);
    const float mx = 0.5f * (px + rx), my = 0.5f * (py + ry);
    const float e = 1e-3f + 1e-3f * (fabsf(ax - 2.0f * cx + bx) + fabsf(ay - 2.0f * cy + by));
    CurveBoxes b;
    b.x0 = fminf(fminf(ax, px), mx) - e;
    b.x1 = fmaxf(fmaxf(ax, px), mx) + e;
    b.y0 = fminf(fminf(ay, py), my) - e;
    b.y1 = fmaxf(fmaxf(ay, py), my) + e;
    b.u0 = fminf(fminf(bx, rx), mx) - e;
    b.u1 = fmaxf(fmaxf(bx, rx), mx) + e;
    b.w0 = fminf(fminf(by, ry), my) - e;
    b.w1 = fmaxf(fmaxf(by, ry), my) + e;
    return b;
}

template <int PPL>
__device__ __forceinline__ float curve_sse_bound(const Prep& P, const float (&fx)[PPL], const float (&fy)[PPL],
                                                 const float3 (&s)[PPL], const float3 (&g)[PPL]) {
    const CurveBoxes b = curve_boxes(P);
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
        const float dx = fmaxf(fmaxf(b.x0 - fx[j], fx[j] - b.x1), 0.0f);
        const float dy = fmaxf(fmaxf(b.y0 - fy[j], fy[j] - b.y1), 0.0f);
        const float du = fmaxf(fmaxf(b.u0 - fx[j], fx[j] - b.u1), 0.0f);
        const float dw = fmaxf(fmaxf(b.w0 - fy[j], fy[j] - b.w1), 0.0f);
        const float d2 = fminf(fmaf(dx, dx, dy * dy), fmaf(du, du, dw * dw));
        const float top = __expf(d2 * P.q[0]) * P.a * 1.0001f;
        const float vx = s[j].x - g[j].x, vy = s[j].y - g[j].y, vz = s[j].z - g[j].z;
        const float ux = P.cr - g[j].x, uy = P.cg - g[j].y, uz = P.cb - g[j].z;
        const float uu = fmaf(ux, ux, fmaf(uy, uy, fmaf(uz, uz, 1e-12f)));
        const float uv = fmaf(ux, vx, fmaf(uy, vy, uz * vz));
        const float w = fminf(fmaxf(__fdividef(uv, uu), 0.0f), top);
        const float ex = fmaf(-w, ux, vx), ey = fmaf(-w, uy, vy), ez = fmaf(-w, uz, vz);
        sum = fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, sum)));
    }
    return sum;
}

__device__ __forceinline__ bool in_unit(float x, float y, float z) {
    return x >= 0.0f && x <= 1.0f && y >= 0.0f && y <= 1.0f && z >= 0.0f && z <= 1.0f;
}

// An error of at least `lower` (a sum as above, over any part of the tile's n = ts^2 pixels) keeps the
// candidate from winning.  The margins cover the rounding of `lower` and of the error the kernels
// compute (1e-6 per channel of a pixel, twice its error) many times over.
__device__ __forceinline__ bool cannot_win(const Bound& b, float lam, int kind, float lower, float denom) {
    const float safe = lower * 0.9995f - 4e-6f * sqrtf(denom * lower) - 1e-9f;
    const double obj = (double)rate_of(lam, b.base_bits + prim_bits(kind)) + (double)(safe / denom);
    return b.on && obj * (obj > 0.0 ? 0.99999 : 1.00001) > b.obj;
}

__device__ __forceinline__ Prep smem_prep(const float4 (&s)[4]) {
    const float4 a = s[0], b = s[1], c = s[2], d = s[3];
    Prep P;
    P.kind = __float_as_int(a.x);
    P.a = a.y; P.cr = a.z; P.cg = a.w; P.cb = b.x;
    P.q[0] = b.y; P.q[1] = b.z; P.q[2] = b.w;
    P.q[3] = c.x; P.q[4] = c.y; P.q[5] = c.z; P.q[6] = c.w;
    P.q[7] = d.x; P.q[8] = d.y; P.q[9] = d.z; P.q[10] = d.w;
    return P;
}

template <int WPC>
struct ScoreSmem {
    float4 prep[MAX_ITEM][4];
    int slot[MAX_ITEM];
    int wcount[4];
    Seg2 seg[4][32];
    float low[MAX_ITEM][WPC];  // lower bounds on the curves' errors
    bool out[MAX_ITEM];
    float red[WPC > 1 ? MAX_ITEM : 1][WPC];
};

// What a thread's candidates cost (WeftFitState.work): those evaluated, so a curve counts once its bound
// has let it through.  Added up once per CTA: an atomic per item on the two counters serialised the
// CTAs of a launch.
struct Work {
    unsigned long long px = 0, ops = 0;
    __device__ __forceinline__ void add(int pixels, int kind) {
        px += pixels;
        ops += (unsigned long long)pixels * (unsigned long long)(kind_ops(kind) + 9);
    }
};

__device__ __forceinline__ void flush_work(const WeftFitState& st, Work w) {
    if (st.work == nullptr) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        w.px += __shfl_xor_sync(FULL, w.px, o);
        w.ops += __shfl_xor_sync(FULL, w.ops, o);
    }
    if ((threadIdx.x & 31) == 0 && w.px) {
        atomicAdd(&st.work[0], w.px);
        atomicAdd(&st.work[1], w.ops);
    }
}

// One scoring work item (tile, 1024-pixel block, run of candidate slots) by the whole CTA.
// INIT: the init round, over empty stacks: the cached composite is black, so it is not read and the
// blend over it is the product s * a (the fused form over +0 differs only in the sign of a zero
// result, which the clamp removes), the same values as the general form.
template <int PPL, int WPC, bool INIT>
__device__ __forceinline__ void score_item(const WeftFitState& st, const int* __restrict__ perm, const WeftFitItem w,
                                           int expect_min, int expect_max, float lam, ScoreSmem<WPC>& sm,
                                           Work& work) {
    constexpr int GROUPS = 4 / WPC;
    float4(&s_prep)[MAX_ITEM][4] = sm.prep;
    int(&s_slot)[MAX_ITEM] = sm.slot;
    int(&s_wcount)[4] = sm.wcount;
    Seg2(&s_seg)[4][32] = sm.seg;
    auto& red = sm.red;
    const int t = w.tile;
    if (t < 0 || t >= st.n_tiles) {
        if (threadIdx.x == 0) fit_report(WEFTK_E_ARG);
        return;
    }
    if (!(st.flags[t] & WEFTK_TILE_EVAL)) return;
    const int ts = st.size[t];
    const bool closed_form = INIT && st.moments != nullptr;
    // a slot range outside the state's slot arrays (a malformed caller-built pool table) is
    // rejected, never scored: the per-candidate scratch is indexed by slot
    if (ts < expect_min || ts > expect_max || w.count > MAX_ITEM || w.block < 0 || w.block >= (ts * ts + 1023) / 1024 ||
        w.first < 0 || w.first + w.count > st.pool_cap[t] || st.pool_off[t] < 0 ||
        (long long)st.pool_off[t] + w.first + w.count > st.n_slots) {
        if (threadIdx.x == 0) fit_report(WEFTK_E_ARG);
        return;
    }
    // items cover the tile's reserved slots; only the filled ones are scored
    const int count = min(w.count, st.pool_cnt[t] - w.first);
    if (count <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long off = st.pool_off[t];

    // stage the live candidates that can win (order-preserving compaction with warp ballots); a
    // bounded tile's constants are scored already (fit_const_*_kernel)
    const Bound bound = tile_bound(st, t, INIT);
    if (all_pruned(bound, lam)) return;
    long long my_slot = -1;
    bool live = false;
    if ((int)threadIdx.x < count) {
        my_slot = off + perm[off + w.first + threadIdx.x];
        const int kind = st.kind[my_slot];
        live = st.alive[my_slot] != 0 && !(INIT && bound.on && kind == K_CONST) &&
               in_play(bound, lam, (int)(my_slot - off), kind);
        if (closed_form && live && kind == K_CONST) {
            st.partial[my_slot * 4 + w.block] = w.block == 0 ? const_closed_sse(st, t, ts, const_head(st, my_slot)) : 0.0f;
            live = false;  // not evaluated per pixel
        }
    }
    const unsigned bal = __ballot_sync(FULL, live);
    if (lane == 0) s_wcount[warp] = __popc(bal);
    __syncthreads();
    int base = 0;
    for (int k = 0; k < warp; ++k) base += s_wcount[k];
    const int m = s_wcount[0] + s_wcount[1] + s_wcount[2] + s_wcount[3];
    int my_curve = 0;
    if (live) {
        const int pos = base + __popc(bal & ((1u << lane) - 1u));
        const Prep mine = load_prep(st, my_slot);
        my_curve = mine.kind == K_CURVE;
        if (!my_curve) work.add(WPC * 32 * PPL, mine.kind);  // the pixels the item covers
        put_prep(s_prep[pos], mine);
        s_slot[pos] = (int)(my_slot - off);
    }
    const int any_curve = __syncthreads_or(my_curve);
    if (m == 0) return;
    // The closed-form init round of 8-px tiles without curves: half a warp per candidate, 4 pixels
    // per lane, so the candidate's terms and its reduction are shared by twice the pixels per lane.
    // Its pixel sums run in another order than the full-warp form's (equal to float rounding), so
    // it serves only the fit with closed-form constants, which has no reference summation to match.
    bool half_done = false;
    if constexpr (INIT && PPL == 2 && WPC == 1) {
        if (closed_form && !any_curve && ts == 8) {
            const int half = lane >> 4, sub = lane & 15;
            const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
            float hx[4], hy[4];
            float3 hs[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = j * 16 + sub;  // an 8-px tile's 64 pixels
                hx[j] = (float)(p & 7) + 0.5f;
                hy[j] = (float)(p >> 3) + 0.5f;
                const float4 a = src[p];
                hs[j] = make_float3(a.x, a.y, a.z);
            }
            for (int c0 = warp * 2; c0 < m; c0 += 8) {
                const int c = min(c0 + half, m - 1);
                const Prep P = smem_prep(s_prep[c]);
                float a[4], sr[4], sg[4], sb[4];
                prim_eval<4>(P, hx, hy, a, sr, sg, sb, lane);  // no curve: no shuffles inside
                float e = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float dr = clamp01(__fmul_rn(sr[j], a[j])) - hs[j].x;
                    const float dg = clamp01(__fmul_rn(sg[j], a[j])) - hs[j].y;
                    const float db = clamp01(__fmul_rn(sb[j], a[j])) - hs[j].z;
                    e = fmaf(dr, dr, fmaf(dg, dg, fmaf(db, db, e)));
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) e += __shfl_xor_sync(FULL, e, o);
                if (sub == 0 && c0 + half < m) st.partial[(off + s_slot[c]) * 4] = e;
            }
            half_done = true;
        }
    }

    const int group = warp / WPC, wig = warp % WPC;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    const float4* bg = reinterpret_cast<const float4*>(st.bg) + st.px_off[t];
    const int pbase = w.block * 1024 + wig * 32 * PPL;
    const int lts = (ts & (ts - 1)) == 0 ? __ffs(ts) - 1 : -1;  // log2(side): no divisions
    float fx[PPL], fy[PPL];
    float3 s[PPL], g[PPL];
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
        const int p = pbase + j * 32 + lane;
        const int y = lts >= 0 ? p >> lts : p / ts;
        fx[j] = (float)(p - y * ts) + 0.5f;
        fy[j] = (float)y + 0.5f;
        const float4 a = src[p];
        s[j] = make_float3(a.x, a.y, a.z);
        if (INIT) {
            g[j] = make_float3(0.0f, 0.0f, 0.0f);
        } else {
            const float4 b = bg[p];
            g[j] = make_float3(b.x, b.y, b.z);
        }
    }
    // curves that cannot win: every warp bounds its own pixels, the warps of a candidate together
    bool unit = bound.on;
#pragma unroll
    for (int j = 0; j < PPL; ++j) unit = unit && in_unit(g[j].x, g[j].y, g[j].z);
    const bool try_bound = any_curve && !half_done && __syncthreads_and(unit);
    if (try_bound) {
        for (int c = group; c < m; c += GROUPS) {
            if (__float_as_int(s_prep[c][0].x) != K_CURVE) continue;
            const float e = warp_sum_f(curve_sse_bound<PPL>(smem_prep(s_prep[c]), fx, fy, s, g));
            if (lane == 0) sm.low[c][wig] = e;
        }
        __syncthreads();
        for (int c = threadIdx.x; c < m; c += blockDim.x) {
            bool out = false;
            if (__float_as_int(s_prep[c][0].x) == K_CURVE && in_unit(s_prep[c][0].z, s_prep[c][0].w, s_prep[c][1].x)) {
                float e = sm.low[c][0];
#pragma unroll
                for (int k = 1; k < WPC; ++k) e += sm.low[c][k];
                out = cannot_win(bound, lam, K_CURVE, e, (float)(3 * ts * ts));
            }
            sm.out[c] = out;
        }
        __syncthreads();
    }
    for (int c = group; !half_done && c < m; c += GROUPS) {
        if (try_bound && sm.out[c]) {
            if (lane == 0) {
                if (WPC == 1) st.partial[(off + s_slot[c]) * 4] = __int_as_float(0x7f800000);
                else red[c][wig] = __int_as_float(0x7f800000);
            }
            continue;
        }
        const Prep P = smem_prep(s_prep[c]);
        float a[PPL], sr[PPL], sg[PPL], sb[PPL];
        if (P.kind == K_CURVE) {
            if (wig == 0 && lane == 0) work.add(WPC * 32 * PPL, K_CURVE);
            put_seg2(s_seg[warp][lane], lane_segment(P, lane));
            __syncwarp();
#pragma unroll
            for (int j = 0; j < PPL; ++j) {
                sr[j] = P.cr;
                sg[j] = P.cg;
                sb[j] = P.cb;
            }
            curve_alpha2<PPL>(P, s_seg[warp], fx, fy, a);
            __syncwarp();
        } else {
            prim_eval<PPL>(P, fx, fy, a, sr, sg, sb, lane);
        }
        float e = 0.0f;
#pragma unroll
        for (int j = 0; j < PPL; ++j) {
            const float dr = clamp01(INIT ? __fmul_rn(sr[j], a[j]) : blend(sr[j], a[j], g[j].x)) - s[j].x;
            const float dg = clamp01(INIT ? __fmul_rn(sg[j], a[j]) : blend(sg[j], a[j], g[j].y)) - s[j].y;
            const float db = clamp01(INIT ? __fmul_rn(sb[j], a[j]) : blend(sb[j], a[j], g[j].z)) - s[j].z;
            e = fmaf(dr, dr, fmaf(dg, dg, fmaf(db, db, e)));
        }
        e = warp_sum_f(e);
        if (WPC == 1) {
            if (lane == 0) st.partial[(off + s_slot[c]) * 4] = e;
        } else if (lane == 0) {
            red[c][wig] = e;
        }
    }
    if (WPC > 1) {
        __syncthreads();
        for (int c = threadIdx.x; c < m; c += blockDim.x) {
            float e = red[c][0];
#pragma unroll
            for (int k = 1; k < WPC; ++k) e += red[c][k];
            st.partial[(off + s_slot[c]) * 4 + w.block] = e;
        }
    }
}

// One CTA per work item of the class (every item of the round's size class is launched; items of
// tiles that are not evaluated this round exit at once).
template <int PPL, int WPC, int MINB>
__global__ void __launch_bounds__(128, MINB) fit_score_kernel(WeftFitState st, const int* __restrict__ perm,
                                                        const WeftFitItem* __restrict__ items, int n_items,
                                                        int expect_min, int expect_max, float lam, bool mode_init) {
    __shared__ ScoreSmem<WPC> sm;
    if ((int)blockIdx.x >= n_items) return;
    Work work;
    if (mode_init)
        score_item<PPL, WPC, true>(st, perm, items[blockIdx.x], expect_min, expect_max, lam, sm, work);
    else
        score_item<PPL, WPC, false>(st, perm, items[blockIdx.x], expect_min, expect_max, lam, sm, work);
    __syncwarp();
    flush_work(st, work);
}

// Persistent form: a grid of about one wave of CTAs that pull the round's live items of the class
// from the work queue fit_queue_kernel built (q_items[0..q_len)), a part of an item per pull.  An
// item's candidates are dealt in at least kScoreParts parts because curves (sorted to the front of a
// pool) cost 20 times a line: an item of 32 curves on a 1024-pixel block kept its CTA for 80 us.  A
// round with few live items deals them finer still, down to one candidate per warp set, until there
// are two parts per CTA: such a round takes as long as its longest part.
template <int PPL, int WPC>
constexpr int kScoreParts = PPL * WPC <= 2 ? 2 : 4;
template <int WPC>
constexpr int kScorePartsMax = WPC == 4 ? 128 : 32;  // one candidate per WPC warps of the CTA

template <int PPL, int WPC, int MINB>
__global__ void __launch_bounds__(128, MINB) fit_score_queue_kernel(WeftFitState st, const int* __restrict__ perm,
                                                              const WeftFitItem* __restrict__ items,
                                                              const int32_t* __restrict__ q_items,
                                                              const int32_t* q_len, int32_t* q_next, int expect_min,
                                                              int expect_max, float lam, bool mode_init) {
    __shared__ ScoreSmem<WPC> sm;
    __shared__ int s_i;
    if (threadIdx.x == 0) s_i = atomicAdd(q_next, 1);
    __syncthreads();
    int len = *q_len, parts = kScoreParts<PPL, WPC>;
    while (parts < kScorePartsMax<WPC> && (long long)len * parts < (long long)gridDim.x) parts *= 2;
    len *= parts;
    Work work;
    for (;;) {
        const int i = s_i;
        if (i >= len) break;
        // the next pull is issued now and its result consumed only after this item, so the
        // atomic's round trip overlaps the scoring
        int next = 0;
        if (threadIdx.x == 0) next = atomicAdd(q_next, 1);
        WeftFitItem w = items[q_items[i / parts]];
        // a malformed count is not dealt in parts, which could pass where the whole is refused: the first pull
        // hands it on as it is
        const bool whole = w.count <= 0 || w.count > MAX_ITEM;
        if (!whole) {
            const int each = (w.count + parts - 1) / parts, from = (i % parts) * each;
            w.first += from;
            w.count = min(each, w.count - from);
        }
        if (whole ? i % parts == 0 : w.count > 0) {
            if (mode_init) score_item<PPL, WPC, true>(st, perm, w, expect_min, expect_max, lam, sm, work);
            else score_item<PPL, WPC, false>(st, perm, w, expect_min, expect_max, lam, sm, work);
        }
        __syncthreads();  // every thread has read s_i and the item's shared buffers are free
        if (threadIdx.x == 0) s_i = next;
        __syncthreads();
    }
    flush_work(st, work);
}

// The same for tiles that one warp covers with PPL pixels per lane (TS * TS = 32 * PPL: 8 and 16 px),
// warp by warp: every warp pulls a part of an item (at most 32 slots), stages its live candidates in
// its own shared memory and scores them, with no barrier and no other warp to wait for.  (With the
// CTA-wide staging above a late round spent 40 % of its instructions on staging and its warps a
// third of their time at barriers.)  Sums as score_item's, bit for bit.
template <int PPL>
struct WarpSmem {
    float4 prep[32][4];
    Seg2 seg[32];
    int slot[32];
};

// part p of `parts`: slots p, p + parts, p + 2 parts ... of the run, so that the expensive kinds at a
// pool's front are spread over its parts.
template <int TS, int PPL, bool INIT>
__device__ __forceinline__ void score_warp_item(const WeftFitState& st, const int* __restrict__ perm,
                                                const WeftFitItem w, int part, int parts, float lam, WarpSmem<PPL>& sm, int lane,
                                                Work& work) {
    const int t = w.tile;
    if (t < 0 || t >= st.n_tiles) {
        if (lane == 0) fit_report(WEFTK_E_ARG);
        return;
    }
    if (!(st.flags[t] & WEFTK_TILE_EVAL)) return;
    const long long off = st.pool_off[t];
    if (st.size[t] != TS || w.block != 0 || w.first < 0 || w.first + w.count > st.pool_cap[t] || off < 0 ||
        off + w.first + w.count > st.n_slots) {
        if (lane == 0) fit_report(WEFTK_E_ARG);
        return;
    }
    const int count = min(w.count, st.pool_cnt[t] - w.first);
    if (count <= 0) return;
    const bool closed_form = INIT && st.moments != nullptr;
    const Bound bound = tile_bound(st, t, INIT);
    if (all_pruned(bound, lam)) return;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    const float4* bg = reinterpret_cast<const float4*>(st.bg) + st.px_off[t];
    // live candidates that can win, compacted in order
    long long my_slot = -1;
    bool live = false;
    if (lane * parts + part < count) {
        my_slot = off + perm[off + w.first + lane * parts + part];
        const int kind = st.kind[my_slot];
        live = st.alive[my_slot] != 0 && !(INIT && bound.on && kind == K_CONST) &&
               in_play(bound, lam, (int)(my_slot - off), kind);
        if (closed_form && live && kind == K_CONST) {
            st.partial[my_slot * 4] = const_closed_sse(st, t, TS, const_head(st, my_slot));
            live = false;  // not evaluated per pixel
        }
    }
    const unsigned bal = __ballot_sync(FULL, live);
    const int m = __popc(bal);
    if (m == 0) return;
    bool curve = false;
    if (live) {
        const int pos = __popc(bal & ((1u << lane) - 1u));
        const Prep r = load_prep(st, my_slot);
        curve = r.kind == K_CURVE;
        if (!curve) work.add(TS * TS, r.kind);
        put_prep(sm.prep[pos], r);
        sm.slot[pos] = (int)(my_slot - off);
    }
    const bool any_curve = __any_sync(FULL, curve);
    __syncwarp();
    float mine = 0.0f;
    if (INIT && TS == 8 && closed_form && !any_curve) {
        // The closed-form init round without curves: half a warp per candidate, 4 pixels per lane, so
        // the candidate's terms and its reduction are shared by twice the pixels per lane.  Its pixel
        // sums run in another order than the full-warp form's (equal to float rounding), so it serves
        // only the fit with closed-form constants, which has no reference summation to match.
        const int half = lane >> 4, sub = lane & 15;
        float hx[4], hy[4];
        float3 hs[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = j * 16 + sub;  // an 8-px tile's 64 pixels
            hx[j] = (float)(p & 7) + 0.5f;
            hy[j] = (float)(p >> 3) + 0.5f;
            const float4 a = src[p];
            hs[j] = make_float3(a.x, a.y, a.z);
        }
        for (int c0 = 0; c0 < m; c0 += 2) {
            const int c = min(c0 + half, m - 1);
            const Prep P = smem_prep(sm.prep[c]);
            float a[4], sr[4], sg[4], sb[4];
            prim_eval<4>(P, hx, hy, a, sr, sg, sb, lane);  // no curve: no shuffles inside
            float e = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float dr = clamp01(__fmul_rn(sr[j], a[j])) - hs[j].x;
                const float dg = clamp01(__fmul_rn(sg[j], a[j])) - hs[j].y;
                const float db = clamp01(__fmul_rn(sb[j], a[j])) - hs[j].z;
                e = fmaf(dr, dr, fmaf(dg, dg, fmaf(db, db, e)));
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) e += __shfl_xor_sync(FULL, e, o);
            const float e1 = __shfl_sync(FULL, e, 16);  // lane 0 holds the even one's, lane 16 the odd one's
            const float e0 = __shfl_sync(FULL, e, 0);
            if (lane == c0) mine = e0;
            if (lane == c0 + 1) mine = e1;
        }
    } else {
        float fx[PPL], fy[PPL];
        float3 s[PPL], g[PPL];
#pragma unroll
        for (int j = 0; j < PPL; ++j) {
            const int p = j * 32 + lane;
            fx[j] = (float)(p % TS) + 0.5f;
            fy[j] = (float)(p / TS) + 0.5f;
            const float4 a = src[p];
            s[j] = make_float3(a.x, a.y, a.z);
            if (INIT) {
                g[j] = make_float3(0.0f, 0.0f, 0.0f);
            } else {
                const float4 b = bg[p];
                g[j] = make_float3(b.x, b.y, b.z);
            }
        }
        bool unit = bound.on;
#pragma unroll
        for (int j = 0; j < PPL; ++j) unit = unit && in_unit(g[j].x, g[j].y, g[j].z);
        unit = any_curve && __all_sync(FULL, unit);
        for (int c = 0; c < m; ++c) {
            const Prep P = smem_prep(sm.prep[c]);
            float a[PPL], sr[PPL], sg[PPL], sb[PPL];
            if (P.kind == K_CURVE) {
                if (unit && in_unit(P.cr, P.cg, P.cb) &&
                    cannot_win(bound, lam, K_CURVE, warp_sum_f(curve_sse_bound<PPL>(P, fx, fy, s, g)),
                               (float)(3 * TS * TS))) {
                    if (lane == c) mine = __int_as_float(0x7f800000);
                    continue;
                }
                if (lane == 0) work.add(TS * TS, K_CURVE);
                put_seg2(sm.seg[lane], lane_segment(P, lane));
                __syncwarp();
#pragma unroll
                for (int j = 0; j < PPL; ++j) {
                    sr[j] = P.cr;
                    sg[j] = P.cg;
                    sb[j] = P.cb;
                }
                curve_alpha2<PPL>(P, sm.seg, fx, fy, a);
                __syncwarp();
            } else {
                prim_eval<PPL>(P, fx, fy, a, sr, sg, sb, lane);
            }
            float e = 0.0f;
#pragma unroll
            for (int j = 0; j < PPL; ++j) {
                const float dr = clamp01(INIT ? __fmul_rn(sr[j], a[j]) : blend(sr[j], a[j], g[j].x)) - s[j].x;
                const float dg = clamp01(INIT ? __fmul_rn(sg[j], a[j]) : blend(sg[j], a[j], g[j].y)) - s[j].y;
                const float db = clamp01(INIT ? __fmul_rn(sb[j], a[j]) : blend(sb[j], a[j], g[j].z)) - s[j].z;
                e = fmaf(dr, dr, fmaf(dg, dg, fmaf(db, db, e)));
            }
            e = warp_sum_f(e);
            if (lane == c) mine = e;
        }
    }
    if (lane < m) st.partial[(off + sm.slot[lane]) * 4] = mine;
    __syncwarp();  // the next part's staging
}

template <int TS, int PPL, int MINB>
__global__ void __launch_bounds__(128, MINB) fit_score_warp_kernel(WeftFitState st, const int* __restrict__ perm,
                                                             const WeftFitItem* __restrict__ items,
                                                             const int32_t* __restrict__ q_items, const int32_t* q_len,
                                                             int32_t* q_next, float lam, bool mode_init) {
    static_assert(TS * TS == 32 * PPL, "one warp covers the tile");
    __shared__ WarpSmem<PPL> sm[4];
    const int lane = threadIdx.x & 31;
    int i = 0;
    if (lane == 0) i = atomicAdd(q_next, 1);
    // parts of at most 32 slots, finer while the warps outnumber them
    int len = *q_len, parts = MAX_ITEM / 32;
    while (parts < MAX_ITEM / 4 && (long long)len * parts < (long long)gridDim.x * 4) parts *= 2;
    len *= parts;
    Work work;
    for (;;) {
        i = __shfl_sync(FULL, i, 0);
        if (i >= len) break;
        int next = 0;  // the next pull's round trip overlaps this part
        if (lane == 0) next = atomicAdd(q_next, 1);
        const WeftFitItem w = items[q_items[i / parts]];
        if (w.count < 0 || w.count > MAX_ITEM) {
            if (lane == 0) fit_report(WEFTK_E_ARG);
        } else if (mode_init) {
            score_warp_item<TS, PPL, true>(st, perm, w, i % parts, parts, lam, sm[threadIdx.x >> 5], lane, work);
        } else {
            score_warp_item<TS, PPL, false>(st, perm, w, i % parts, parts, lam, sm[threadIdx.x >> 5], lane, work);
        }
        i = next;
    }
    flush_work(st, work);
}

// The round's work queue: per size class, the items with a candidate to score, in any order (items
// write disjoint scratch).  One warp per item.  ctl[c] counts class c's queue, ctl[3 + c] is its pull
// counter.  Inside weftk_fit_run (tile_blocks > 0) the first blocks open the round (a thread per tile,
// fit_begin_kernel's work) while the others, which read only what that leaves alone, list the items:
// one launch fewer per round.  spare: the counters the next round will use, cleared here.
__global__ void __launch_bounds__(256) fit_queue_kernel(WeftFitState st, const int* __restrict__ perm,
                                                        const WeftFitItem* __restrict__ items8, int n8,
                                                        const WeftFitItem* __restrict__ items16, int n16,
                                                        const WeftFitItem* __restrict__ items32, int n32, float lam,
                                                        bool mode_init, int tile_blocks, int* ctl, int* spare) {
    if ((int)blockIdx.x < tile_blocks) {
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        if (t < 2) spare[t] = 0;
        begin_tile(st, t, WEFTK_FIT_ROUND, ctl);
        return;
    }
    const int i = (int)(((blockIdx.x - tile_blocks) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= n8 + n16 + n32) return;
    const int c = i < n8 ? 0 : i < n8 + n16 ? 1 : 2;
    const int j = c == 0 ? i : c == 1 ? i - n8 : i - n8 - n16;
    const WeftFitItem w = (c == 0 ? items8 : c == 1 ? items16 : items32)[j];
    if (w.tile < 0 || w.tile >= st.n_tiles) {
        if (lane == 0) fit_report(WEFTK_E_ARG);
        return;
    }
    const int cnt = st.pool_cnt[w.tile];
    if (w.first >= cnt) return;
    if (tile_blocks ? !opens(st, w.tile, WEFTK_FIT_ROUND, ctl) : !(st.flags[w.tile] & WEFTK_TILE_EVAL)) return;
    const Bound bound = tile_bound(st, w.tile, mode_init);
    if (all_pruned(bound, lam)) return;
    const long long off = st.pool_off[w.tile];
    // a run outside the tile's slots goes to the scoring launch, which reports it
    bool any = w.first < 0 || w.count > MAX_ITEM || w.first + w.count > st.pool_cap[w.tile] || off < 0 ||
               off + w.first + w.count > st.n_slots;
    if (!any) {
        bool mine = false;
        for (int k = lane; k < min(w.count, cnt - w.first); k += 32) {
            const int local = perm[off + w.first + k];
            const int kind = st.kind[off + local];
            mine = mine || (st.alive[off + local] != 0 && !(mode_init && bound.on && kind == K_CONST) &&
                            in_play(bound, lam, local, kind));
        }
        any = __any_sync(FULL, mine);
    }
    if (!any || lane != 0) return;
    const int base = c == 0 ? 0 : c == 1 ? n8 : n8 + n16;
    st.queue[base + atomicAdd(&st.queue_ctl[c], 1)] = j;
}

// ------------------------------------------------------------------ the init round's constants
// Every live constant candidate over black, before the other kinds: its per-pixel error exactly as
// the class's scoring shape <PPL, WPC> sums it (PPL pixels of a lane in a chain, the warp's butterfly,
// WPC groups in order), or in closed form from the tile's pixel sums when the fit gives them.  The
// tile's best objective among them is left in cur_obj (flag TILE_BOUNDED) for the pruning above; the
// selection overwrites it.  A tile is taken up by its first work item.
//
// A warp walks the tile's slots 32 at a time, a lane keeping its own slot's sum.  Tiles of 8 and 16 px
// take one warp, larger ones a CTA of 16 (a warp per 256-pixel group).
__device__ __forceinline__ float const_obj(float sse, float denom, float lam) {
    return __fadd_rn(__fdiv_rn(sse, denom), rate_of(lam, 8 + BITS_CONST));
}

__device__ __forceinline__ float warp_min_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

// One group's sums: PPL x 32 pixels from pixel p0, for the constants of slots [base, base + 32).
template <int PPL>
__device__ __forceinline__ float const_group(const float4* __restrict__ src, int p0, unsigned todo, float4 head,
                                             int lane) {
    float3 s[PPL];
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
        const float4 a = src[p0 + j * 32 + lane];
        s[j] = make_float3(a.x, a.y, a.z);
    }
    float mine = 0.0f;
    while (todo) {
        const int c = __ffs(todo) - 1;
        todo &= todo - 1;
        const float a = __shfl_sync(FULL, head.x, c);
        // the blend over black, clamped: the same product for every pixel
        const float r = clamp01(__fmul_rn(__shfl_sync(FULL, head.y, c), a));
        const float g = clamp01(__fmul_rn(__shfl_sync(FULL, head.z, c), a));
        const float b = clamp01(__fmul_rn(__shfl_sync(FULL, head.w, c), a));
        float e = 0.0f;
#pragma unroll
        for (int j = 0; j < PPL; ++j) {
            const float dr = r - s[j].x, dg = g - s[j].y, db = b - s[j].z;
            e = fmaf(dr, dr, fmaf(dg, dg, fmaf(db, db, e)));
        }
        e = warp_sum_f(e);
        if (lane == c) mine = e;
    }
    return mine;
}

// The tile named by the item whose run starts the tile (first 0, block 0); false for the others.
__device__ __forceinline__ bool const_tile(const WeftFitState& st, const WeftFitItem& w, int lo, int hi, int& t,
                                           int& ts, int& cnt) {
    if (w.first != 0 || w.block != 0) return false;
    t = w.tile;
    if (t < 0 || t >= st.n_tiles || !(st.flags[t] & WEFTK_TILE_EVAL)) return false;
    ts = st.size[t];
    cnt = st.pool_cnt[t];
    // (a malformed table is reported by the scoring launch)
    return ts >= lo && ts <= hi && st.pool_off[t] >= 0 && cnt >= 0 && cnt <= st.pool_cap[t] &&
           (long long)st.pool_off[t] + cnt <= st.n_slots;
}

__device__ __forceinline__ bool live_const(const WeftFitState& st, long long slot) {
    const int alive = st.alive[slot], kind = st.kind[slot];  // both loads at once
    return alive != 0 && kind == K_CONST;
}

// The warp's share of the items that start a tile: a grid of about one wave of warps, each looking at
// 32 items a grid apart at a time (the items that start a tile lie together in the list).
template <class F>
__device__ __forceinline__ void for_first_items(const WeftFitItem* __restrict__ items, int n_items, F&& body) {
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    const int warps = (int)(gridDim.x * blockDim.x) >> 5;
    for (long long base = w; base < n_items; base += 32ll * warps) {
        const long long i = base + (long long)lane * warps;
        WeftFitItem it{-1, 0, 1, 0};
        if (i < n_items) it = items[i];
        for (unsigned todo = __ballot_sync(FULL, it.first == 0 && it.block == 0); todo; todo &= todo - 1) {
            WeftFitItem one = it;
            one.tile = __shfl_sync(FULL, it.tile, __ffs(todo) - 1);
            one.first = one.block = 0;
            body(one);
        }
    }
}

// 8- and 16-px tiles (one unit of WPC groups): a warp per tile.
template <int PPL, int WPC>
__global__ void __launch_bounds__(128) fit_const_small_kernel(WeftFitState st, const WeftFitItem* __restrict__ items,
                                                              int n_items, int ts_want, float lam) {
    const int lane = threadIdx.x & 31;
    for_first_items(items, n_items, [&](const WeftFitItem& it) {
    int t, ts, cnt;
    if (!const_tile(st, it, ts_want, ts_want, t, ts, cnt)) return;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    const long long off = st.pool_off[t];
    const float denom = (float)(3 * ts * ts);
    float best = __int_as_float(0x7f800000);
    bool any = false;
    int scored = 0;
    bool ahead = lane < cnt && live_const(st, off + lane);
    for (int base = 0; base < cnt; base += 32) {
        const long long slot = off + base + lane;
        const bool c = ahead;
        ahead = base + 32 + lane < cnt && live_const(st, slot + 32);  // the next 32's loads
        const unsigned todo = __ballot_sync(FULL, c);
        if (!todo) continue;
        const float4 head = c ? const_head(st, slot) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float sse = const_group<PPL>(src, 0, todo, head, lane);
#pragma unroll
        for (int g = 1; g < WPC; ++g) sse += const_group<PPL>(src, g * 32 * PPL, todo, head, lane);
        scored += __popc(todo);
        if (c) {
            st.partial[slot * 4] = sse;
            const float obj = const_obj(sse, denom, lam);
            any = any || obj == obj;
            best = fminf(best, obj);
        }
    }
    best = warp_min_f(best);
    any = __any_sync(FULL, any);
    if (lane == 0) {
        if (any) {
            st.cur_obj[t] = (double)best;
            st.flags[t] |= TILE_BOUNDED;
        }
        if (st.work != nullptr && scored) {
            atomicAdd(&st.work[0], (unsigned long long)scored * (unsigned long long)(ts * ts));
            atomicAdd(&st.work[1],
                      (unsigned long long)scored * (unsigned long long)(ts * ts) * (unsigned long long)(c_kind_ops[0] + 9));
        }
    }
    });
}

// 32- and 64-px tiles (one or four 1024-pixel units of four 256-pixel groups): a CTA of 16 warps per
// tile.  32 px: each set of four warps takes a quarter of the slots; 64 px: each takes a unit.
__global__ void __launch_bounds__(512) fit_const_large_kernel(WeftFitState st, const WeftFitItem* __restrict__ items,
                                                              int n_items, float lam) {
    __shared__ float part[4][4][32];  // [set][group][slot of the run]
    __shared__ float wbest[16];
    __shared__ int wany[16], wscored[16];
    __shared__ int todo_tile[512], n_todo;
    for (long long base = blockIdx.x; base < n_items; base += 512ll * gridDim.x) {
    // the CTA's items a grid apart, as for_first_items
    if (threadIdx.x == 0) n_todo = 0;
    __syncthreads();
    const long long i = base + (long long)threadIdx.x * gridDim.x;
    if (i < n_items && items[i].first == 0 && items[i].block == 0) todo_tile[atomicAdd(&n_todo, 1)] = items[i].tile;
    __syncthreads();
    for (int q = 0; q < n_todo; ++q) {
    int t, ts, cnt;
    if (!const_tile(st, WeftFitItem{todo_tile[q], 0, 0, 0}, 32, 64, t, ts, cnt) || (ts != 32 && ts != 64)) continue;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp >> 2, grp = warp & 3;
    const bool split = ts == 32;  // the sets split the slots instead of the units
    const int units = ts * ts / 1024, unit = split ? 0 : set;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    const long long off = st.pool_off[t];
    const float denom = (float)(3 * ts * ts);
    float best = __int_as_float(0x7f800000);
    bool any = false;
    int scored = 0;
    const int stride = split ? 128 : 32;
    for (int base0 = 0; base0 < cnt; base0 += stride) {  // uniform over the CTA
        const int base = base0 + (split ? set * 32 : 0);
        const long long slot = off + base + lane;
        const bool c = base + lane < cnt && live_const(st, slot);
        const unsigned todo = __ballot_sync(FULL, c);
        if (!__syncthreads_or(todo != 0)) continue;
        if (todo) {
            const float4 head = c ? const_head(st, slot) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            part[set][grp][lane] = const_group<8>(src, unit * 1024 + grp * 256, todo, head, lane);
        }
        __syncthreads();
        if (grp == 0 && c) {
            float sse = part[set][0][lane];
#pragma unroll
            for (int g = 1; g < 4; ++g) sse += part[set][g][lane];
            st.partial[slot * 4 + unit] = sse;
            if (split) {
                const float obj = const_obj(sse, denom, lam);
                any = any || obj == obj;
                best = fminf(best, obj);
            }
        }
        if (grp == 0 && (split || set == 0)) scored += __popc(todo);
        __syncthreads();  // the units' sums are written; part is free
        if (!split && warp == 0 && c) {
            volatile const float* p = st.partial + slot * 4;
            float sse = p[0];
            for (int b = 1; b < units; ++b) sse += p[b];
            const float obj = const_obj(sse, denom, lam);
            any = any || obj == obj;
            best = fminf(best, obj);
        }
    }
    best = warp_min_f(best);
    any = __any_sync(FULL, any);
    if (lane == 0) {
        wbest[warp] = best;
        wany[warp] = any;
        wscored[warp] = scored;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0, ok = 0;
        for (int w = 0; w < 16; ++w) {
            best = fminf(best, wbest[w]);
            ok |= wany[w];
            n += wscored[w];
        }
        if (ok) {
            st.cur_obj[t] = (double)best;
            st.flags[t] |= TILE_BOUNDED;
        }
        if (st.work != nullptr && n) {
            atomicAdd(&st.work[0], (unsigned long long)n * (unsigned long long)(ts * ts));
            atomicAdd(&st.work[1],
                      (unsigned long long)n * (unsigned long long)(ts * ts) * (unsigned long long)(c_kind_ops[0] + 9));
        }
    }
    __syncthreads();  // the next tile's sums
    }
    }
}

// Closed form, any tile side: a warp per tile.
__global__ void __launch_bounds__(128) fit_const_closed_kernel(WeftFitState st, const WeftFitItem* __restrict__ items,
                                                               int n_items, int lo, int hi, float lam) {
    const int lane = threadIdx.x & 31;
    for_first_items(items, n_items, [&](const WeftFitItem& it) {
    int t, ts, cnt;
    if (!const_tile(st, it, lo, hi, t, ts, cnt)) return;
    const long long off = st.pool_off[t];
    const int nb = (ts * ts + 1023) / 1024;
    const float denom = (float)(3 * ts * ts);
    float best = __int_as_float(0x7f800000);
    bool any = false;
    for (int base = lane; base < cnt; base += 32) {
        const long long slot = off + base;
        if (!live_const(st, slot)) continue;
        const float sse = const_closed_sse(st, t, ts, const_head(st, slot));
        st.partial[slot * 4] = sse;
        for (int b = 1; b < nb; ++b) st.partial[slot * 4 + b] = 0.0f;
        const float obj = const_obj(sse, denom, lam);
        any = any || obj == obj;
        best = fminf(best, obj);
    }
    best = warp_min_f(best);
    any = __any_sync(FULL, any);
    if (lane == 0 && any) {
        st.cur_obj[t] = (double)best;
        st.flags[t] |= TILE_BOUNDED;
    }
    });
}

// ------------------------------------------------------------------ select / accept
// A warp per tile: the argmin over its slots, then the accepted candidate composited into bg.  Tiles of
// more than 256 pixels are composited by the CTA's four warps together (one warp took 20 us over a
// 64-px tile's 4096 pixels with a curve, as long as the rest of a round with few live tiles).  mark:
// note the slots of a tile without an accepted candidate as seen (weftk_fit_run).
constexpr int SEL_WARPS = 4;

// Pixels [from, npix) in steps of `step` of the tile's composite under candidate P.
__device__ __forceinline__ void composite_tile(const WeftFitState& st, int t, int ts, const Prep& P, int from, int step,
                                               int lane) {
    const int npix = ts * ts;
    float4* bgp = reinterpret_cast<float4*>(st.bg) + st.px_off[t];
    constexpr int U = 4;
    for (int base = from; base < npix; base += step) {
        float fx[U], fy[U], a[U], sr[U], sg[U], sb[U];
        float4 g[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int p = min(base + j * 32 + lane, npix - 1);
            fx[j] = (float)(p % ts) + 0.5f;
            fy[j] = (float)(p / ts) + 0.5f;
            g[j] = bgp[p];
        }
        prim_eval<U>(P, fx, fy, a, sr, sg, sb, lane);
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int p = base + j * 32 + lane;
            if (p < npix)
                bgp[p] = make_float4(blend(sr[j], a[j], g[j].x), blend(sg[j], a[j], g[j].y),
                                     blend(sb[j], a[j], g[j].z), 0.0f);
        }
    }
}

// The tile's winning slot (pool-local), or -1; its state updated on acceptance.
__device__ __forceinline__ int select_tile(const WeftFitState& st, int t, int ts, int mode, float lam_f, double lam_d,
                                           bool mark, int lane) {
    const int flags = st.flags[t];
    if (!(flags & WEFTK_TILE_EVAL)) return -1;
    const int npix = ts * ts, nb = (npix + 1023) / 1024;
    const long long off = st.pool_off[t];
    const int cnt = st.pool_cnt[t];
    if (off < 0 || cnt < 0 || cnt > st.pool_cap[t] || off + cnt > st.n_slots) {
        if (lane == 0) fit_report(WEFTK_E_ARG);
        return -1;
    }
    const Bound bound = tile_bound(st, t, mode == WEFTK_FIT_INIT);
    const int base_bits = bound.base_bits;
    const float denom = (float)(3 * npix);
    float best = __int_as_float(0x7f800000);
    int bi = INT_MAX;
    const bool only_const = bound.init && all_pruned(bound, lam_f);
    if (bound.init || !all_pruned(bound, lam_f)) {
#pragma unroll 4
        for (int c = bound.seen + lane; c < cnt; c += 32) {
            const long long slot = off + c;
            const int kind = st.kind[slot];
            const bool alive = st.alive[slot] != 0;
            float sse = st.partial[slot * 4];
            if ((only_const && kind != K_CONST) || !alive || !in_play(bound, lam_f, c, kind)) continue;
            for (int b = 1; b < nb; ++b) sse += st.partial[slot * 4 + b];
            const float mse = __fdiv_rn(sse, denom);
            const float obj = __fadd_rn(mse, rate_of(lam_f, base_bits + prim_bits(kind)));
            if (obj < best || (obj == best && c < bi)) {
                best = obj;
                bi = c;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(FULL, best, o);
        const int oi = __shfl_xor_sync(FULL, bi, o);
        if (ob < best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    const bool accept = bi != INT_MAX && ((mode == WEFTK_FIT_INIT) || ((double)best < bound.obj));
    if (!accept) {
        if (lane == 0 && mark && cnt < (INT_MAX >> TILE_SEEN)) st.flags[t] = (flags & TILE_BITS) | (cnt << TILE_SEEN);
        return -1;
    }
    if (lane == 0) {
        const long long slot = off + bi;
        const int k = st.n_sel[t];
        if (k < st.cap_max) st.sel[(long long)t * st.cap_max + k] = bi;
        else fit_report(WEFTK_E_RANGE);
        st.n_sel[t] = k + 1;
        st.n_alive[t] -= 1;
        st.alive[slot] = 0;
        const int bits = base_bits + prim_bits(st.kind[slot]);
        st.sel_bits[t] = bits;
        if (mode == WEFTK_FIT_INIT) {
            float sse = st.partial[slot * 4];
            for (int b = 1; b < nb; ++b) sse += st.partial[slot * 4 + b];
            st.cur_obj[t] = (double)__fdiv_rn(sse, denom) + lam_d * (double)bits;
        } else {
            st.cur_obj[t] = (double)best;
        }
        st.flags[t] = (flags & TILE_BITS) | WEFTK_TILE_IMPROVED;  // nothing is seen any more
        atomicAdd(&st.status[1], 1);
    }
    return bi;
}

__global__ void __launch_bounds__(SEL_WARPS * 32) fit_select_kernel(WeftFitState st, int mode, float lam_f,
                                                                    double lam_d, bool mark) {
    __shared__ int s_win[SEL_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = blockIdx.x * SEL_WARPS + warp;
    int win = -1, ts = 0;
    if (t < st.n_tiles) {
        ts = st.size[t];
        win = select_tile(st, t, ts, mode, lam_f, lam_d, mark, lane);
    }
    // (a fit without a composite runs no round after its init round, so nothing would read it)
    if (st.bg == nullptr) return;
    if (win >= 0 && ts * ts <= 256) {
        composite_tile(st, t, ts, load_prep(st, st.pool_off[t] + win), 0, 128, lane);
        win = -1;
    }
    if (lane == 0) s_win[warp] = win;
    if (!__syncthreads_or(win >= 0)) return;
    for (int w = 0; w < SEL_WARPS; ++w) {
        if (s_win[w] < 0) continue;
        const int tw = blockIdx.x * SEL_WARPS + w;
        composite_tile(st, tw, st.size[tw], load_prep(st, st.pool_off[tw] + s_win[w]), warp * 128, SEL_WARPS * 128, lane);
    }
}

// Register-resident FMA loop for measuring the FP32 pipe: 8 independent chains per thread.
__global__ void __launch_bounds__(256) fp32_peak_kernel(float* out, int iters, float a, float b) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = (float)(threadIdx.x + k);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = fmaf(v[k], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += v[k];
    if (s == 12345.678f) out[threadIdx.x] = s;  // keeps the loop live; practically never taken
}

struct FitTiming {
    bool enabled = false;
    bool pending = false;
    cudaEvent_t start = nullptr, stop = nullptr;
    double ms = 0.0;
    int rounds = 0;
};
static FitTiming g_timing;

static int timing_collect() {
    if (!g_timing.pending) return WEFTK_OK;
    WEFTK_CUDA(cudaEventSynchronize(g_timing.stop));
    float ms = 0.0f;
    WEFTK_CUDA(cudaEventElapsedTime(&ms, g_timing.start, g_timing.stop));
    g_timing.ms += ms;
    g_timing.rounds += 1;
    g_timing.pending = false;
    return WEFTK_OK;
}

}  // namespace weftk

using namespace weftk;

// ---------------------------------------------------------------- allocation-free round
// Scoring scratch for weftk_fit_round_static: a fixed array in device memory, so
// that entry point never allocates.  Host code must not use the symbol as a
// pointer (it is a host-side stand-in); the device address comes from
// cudaGetSymbolAddress, looked up once per device.
static __device__ __align__(256) float g_fit_static_scratch[WEFTK_FIT_STATIC_SCRATCH_FLOATS];
static std::mutex g_static_mu;
static float* g_static_ptr[64] = {nullptr};

static int static_scratch_for_current_device(float** out) {
    int dev = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(WEFTK_E_RANGE, "fit_round_static: device index beyond 63");
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_fit_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_fit_static_scratch)");
        g_static_ptr[dev] = static_cast<float*>(p);
    }
    *out = g_static_ptr[dev];
    return WEFTK_OK;
}

extern "C" int weftk_fit_timing(int enable, double* score_ms, int* n_rounds) {
    int rc = timing_collect();
    if (rc) return rc;
    if (enable && !g_timing.start) {
        WEFTK_CUDA(cudaEventCreate(&g_timing.start));
        WEFTK_CUDA(cudaEventCreate(&g_timing.stop));
    }
    g_timing.enabled = enable != 0;
    if (score_ms) *score_ms = g_timing.ms;
    if (n_rounds) *n_rounds = g_timing.rounds;
    g_timing.ms = 0.0;
    g_timing.rounds = 0;
    return WEFTK_OK;
}

extern "C" int weftk_measure_fp32_peak(double* gflops) {
    WEFTK_REQUIRE(gflops, "measure_fp32_peak: null pointer");
    int dev = 0, sms = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    WEFTK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    float* out = nullptr;
    WEFTK_CUDA(cudaMalloc(&out, 256 * sizeof(float)));
    cudaEvent_t a, b;
    WEFTK_CUDA(cudaEventCreate(&a));
    WEFTK_CUDA(cudaEventCreate(&b));
    const int blocks = sms * 8, iters = 1 << 15;
    fp32_peak_kernel<<<blocks, 256>>>(out, 256, 1.0000001f, 1e-7f);  // warm-up
    float best = 1e30f;
    for (int r = 0; r < 5; ++r) {
        WEFTK_CUDA(cudaEventRecord(a));
        fp32_peak_kernel<<<blocks, 256>>>(out, iters, 1.0000001f, 1e-7f);
        WEFTK_CUDA(cudaEventRecord(b));
        WEFTK_CUDA(cudaEventSynchronize(b));
        float ms = 0.0f;
        WEFTK_CUDA(cudaEventElapsedTime(&ms, a, b));
        best = ms < best ? ms : best;
    }
    WEFTK_CUDA(cudaGetLastError());
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    *gflops = 2.0 * 8.0 * (double)iters * 256.0 * (double)blocks / (best * 1e-3) / 1e9;
    return WEFTK_OK;
}

// One CTA per tile: the tile's state, selection row, slots and composite pixels.
__global__ void fit_reset_kernel(WeftFitState st, const int* __restrict__ init_cnt) {
    const int t = blockIdx.x;
    if (t >= st.n_tiles) return;
    if (t == 0 && threadIdx.x == 0 && st.work != nullptr) {
        st.work[0] = 0;
        st.work[1] = 0;
    }
    if (threadIdx.x == 0) {
        st.pool_cnt[t] = init_cnt[t];
        st.n_alive[t] = 0;
        st.n_sel[t] = 0;
        st.sel_bits[t] = 8;
        st.flags[t] = 0;
        st.cur_obj[t] = 0.0;
    }
    for (int i = threadIdx.x; i < st.cap_max; i += blockDim.x) st.sel[(size_t)t * st.cap_max + i] = -1;
    const long long off = st.pool_off[t];
    for (int i = threadIdx.x; i < st.pool_cap[t]; i += blockDim.x) st.alive[off + i] = 0;
    const int ts = st.size[t];
    if (st.bg == nullptr) return;
    float4* bg = reinterpret_cast<float4*>(st.bg) + st.px_off[t];
    for (int i = threadIdx.x; i < ts * ts; i += blockDim.x) bg[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void fit_moments_kernel(WeftFitState st, double* __restrict__ out) {
    __shared__ double red[6][4];
    const int t = blockIdx.x;
    if (t >= st.n_tiles) return;
    const int ts = st.size[t], n = ts * ts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    double a[6] = {0, 0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float4 v = src[i];
        a[0] += v.x;
        a[1] += v.y;
        a[2] += v.z;
        a[3] += (double)v.x * v.x;
        a[4] += (double)v.y * v.y;
        a[5] += (double)v.z * v.z;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(FULL, a[k], o);
        if (lane == 0) red[k][warp] = a[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) out[(size_t)t * 6 + threadIdx.x] = red[threadIdx.x][0] + red[threadIdx.x][1] +
                                                             red[threadIdx.x][2] + red[threadIdx.x][3];
}

extern "C" int weftk_fit_moments(const WeftFitState* st, double* d_moments, void* stream) {
    WEFTK_REQUIRE(st && d_moments, "fit_moments: null argument");
    if (st->n_tiles == 0) return WEFTK_OK;
    fit_moments_kernel<<<st->n_tiles, 128, 0, (cudaStream_t)stream>>>(*st, d_moments);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_fit_reset(const WeftFitState* st, const int32_t* d_init_cnt, void* stream) {
    WEFTK_REQUIRE(st && d_init_cnt, "fit_reset: null argument");
    if (st->n_tiles == 0) return WEFTK_OK;
    fit_reset_kernel<<<st->n_tiles, 128, 0, (cudaStream_t)stream>>>(*st, d_init_cnt);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_fit_prepare(const WeftFitState* st, const int32_t* d_first_new, void* stream) {
    WEFTK_REQUIRE(st && d_first_new, "fit_prepare: null argument");
    if (st->n_tiles == 0) return WEFTK_OK;
    fit_prepare_kernel<<<st->n_tiles, 128, 0, (cudaStream_t)stream>>>(*st, d_first_new);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_fit_round_static(const WeftFitState* st, int mode, double lambda, double complex_threshold,
                                      const int32_t* d_perm, const WeftFitItem* d_items8, int n_items8,
                                      const WeftFitItem* d_items16, int n_items16, const WeftFitItem* d_items32,
                                      int n_items32, void* stream) {
    WEFTK_REQUIRE(st, "fit_round_static: null state");
    if (st->n_slots < 0 || st->n_slots > (long long)WEFTK_FIT_STATIC_SCRATCH_FLOATS / 4)
        return fail(WEFTK_E_RANGE, "fit_round_static: " + std::to_string((long long)st->n_slots) +
                                       " candidate slots need more than the " +
                                       std::to_string(WEFTK_FIT_STATIC_SCRATCH_FLOATS) +
                                       "-float static scratch (at most " +
                                       std::to_string(WEFTK_FIT_STATIC_SCRATCH_FLOATS / 4) + " slots)");
    float* scratch = nullptr;
    int rc = static_scratch_for_current_device(&scratch);
    if (rc) return rc;
    WeftFitState local = *st;
    local.partial = scratch;
    return weftk_fit_round(&local, mode, lambda, complex_threshold, d_perm, d_items8, n_items8, d_items16, n_items16,
                           d_items32, n_items32, stream);
}

// Scoring variants per size class.  A class's variants cover the same pixels per candidate pass
// (64 for 8-px tiles, 256 for 16-px tiles, one 1024-pixel block for 32/64-px tiles) with a
// different split over lanes and warps, or a different register budget.
static_assert(sizeof(WeftFitState) == 224, "WeftFitState layout is part of the C ABI");

struct ScoreShape {
    int ppl, wpc, minb;
};
static const ScoreShape kShapes[3][WEFTK_FIT_VARIANTS] = {
    {{2, 1, 7}, {2, 1, 8}, {1, 2, 8}},
    {{8, 1, 4}, {4, 2, 6}, {2, 4, 8}},
    {{8, 4, 4}, {8, 4, 3}, {8, 4, 5}},
};

// mode and rate weight of the round being enqueued (the class launchers' extra arguments)
static thread_local bool g_mode_init = false;
static thread_local float g_lam = 0.0f;

// queue of the class being launched (set while weftk_fit_round enqueues a queue-driven round)
static thread_local int g_queue_class = -1;
static thread_local int g_queue_base = 0;
static thread_local int g_sms = 148;

template <int PPL, int WPC, int MINB>
static void launch_score(const WeftFitState& st, const int* perm, const WeftFitItem* items, int n, int lo, int hi,
                         cudaStream_t s) {
    if (g_queue_class < 0) {
        fit_score_kernel<PPL, WPC, MINB><<<n, 128, 0, s>>>(st, perm, items, n, lo, hi, g_lam, g_mode_init);
        return;
    }
    const int c = g_queue_class;
    const int grid = (int)std::min<long long>((long long)n * kScorePartsMax<WPC>, g_sms * MINB);
    if constexpr (WPC == 1 && (PPL == 2 || PPL == 8)) {
        constexpr int TS = PPL == 2 ? 8 : 16;
        fit_score_warp_kernel<TS, PPL, MINB><<<grid, 128, 0, s>>>(st, perm, items, st.queue + g_queue_base,
                                                                   st.queue_ctl + c, st.queue_ctl + 3 + c, g_lam,
                                                                   g_mode_init);
    } else {
        fit_score_queue_kernel<PPL, WPC, MINB><<<grid, 128, 0, s>>>(st, perm, items, st.queue + g_queue_base,
                                                                     st.queue_ctl + c, st.queue_ctl + 3 + c, lo, hi,
                                                                     g_lam, g_mode_init);
    }
}

static void launch_score_class8(int v, const WeftFitState& st, const int* perm, const WeftFitItem* it, int n,
                                cudaStream_t s) {
    if (v == 1) launch_score<2, 1, 8>(st, perm, it, n, 8, 8, s);
    else if (v == 2) launch_score<1, 2, 8>(st, perm, it, n, 8, 8, s);
    else launch_score<2, 1, 7>(st, perm, it, n, 8, 8, s);
}

static void launch_score_class16(int v, const WeftFitState& st, const int* perm, const WeftFitItem* it, int n,
                                 cudaStream_t s) {
    if (v == 1) launch_score<4, 2, 6>(st, perm, it, n, 16, 16, s);
    else if (v == 2) launch_score<2, 4, 8>(st, perm, it, n, 16, 16, s);
    else launch_score<8, 1, 4>(st, perm, it, n, 16, 16, s);
}

static void launch_score_class32(int v, const WeftFitState& st, const int* perm, const WeftFitItem* it, int n,
                                 cudaStream_t s) {
    if (v == 1) launch_score<8, 4, 3>(st, perm, it, n, 32, 64, s);
    else if (v == 2) launch_score<8, 4, 5>(st, perm, it, n, 32, 64, s);
    else launch_score<8, 4, 4>(st, perm, it, n, 32, 64, s);
}

// The init round's constants of one size class (0: 8 px, 1: 16 px, 2: 32 and 64 px), in the class's
// summation order.
static void launch_const(const WeftFitState& st, int c, int v, const WeftFitItem* it, int n, float lam,
                         cudaStream_t s) {
    if (n == 0) return;
    const int lo = c == 0 ? 8 : c == 1 ? 16 : 32;
    const int warps = std::min(ceil_div(n, 4), g_sms * 16);
    if (st.moments != nullptr) fit_const_closed_kernel<<<warps, 128, 0, s>>>(st, it, n, lo, c == 2 ? 64 : lo, lam);
    else if (c == 2) fit_const_large_kernel<<<std::min(n, g_sms * 3), 512, 0, s>>>(st, it, n, lam);
    else if (c == 0 && v == 2) fit_const_small_kernel<1, 2><<<warps, 128, 0, s>>>(st, it, n, 8, lam);
    else if (c == 0) fit_const_small_kernel<2, 1><<<warps, 128, 0, s>>>(st, it, n, 8, lam);
    else if (v == 1) fit_const_small_kernel<4, 2><<<warps, 128, 0, s>>>(st, it, n, 16, lam);
    else if (v == 2) fit_const_small_kernel<2, 4><<<warps, 128, 0, s>>>(st, it, n, 16, lam);
    else fit_const_small_kernel<8, 1><<<warps, 128, 0, s>>>(st, it, n, 16, lam);
}

extern "C" int weftk_fit_variant(int size_class, int variant, int* pixels_per_lane, int* warps_per_candidate,
                                 int* ctas_per_sm) {
    const int c = size_class == 8 ? 0 : size_class == 16 ? 1 : size_class == 32 ? 2 : -1;
    WEFTK_REQUIRE(c >= 0 && variant >= 0 && variant < WEFTK_FIT_VARIANTS, "fit_variant: no such class or variant");
    if (pixels_per_lane) *pixels_per_lane = kShapes[c][variant].ppl;
    if (warps_per_candidate) *warps_per_candidate = kShapes[c][variant].wpc;
    if (ctas_per_sm) *ctas_per_sm = kShapes[c][variant].minb;
    return WEFTK_OK;
}

// Control block of the device-driven fit for the round being enqueued (host thread state:
// set only while weftk_fit_run enqueues its rounds).
static thread_local int* g_round_ctl = nullptr;
static thread_local int* g_init_ctl = nullptr;   // the control block to clear before the init round
static thread_local int* g_round_spare = nullptr;  // the counters of the next round (cleared by this one)

int launch_fit_reseed(const WeftFitState& st, const int* gate, cudaStream_t stream);

extern "C" int weftk_fit_run(const WeftFitState* st, int max_rounds, double lambda, double complex_threshold,
                             const int32_t* d_perm, const WeftFitItem* d_items8, int n_items8,
                             const WeftFitItem* d_items16, int n_items16, const WeftFitItem* d_items32,
                             int n_items32, int32_t* d_ctl, void* stream) {
    WEFTK_REQUIRE(st && d_ctl && max_rounds >= 0, "fit_run: bad arguments");
    WEFTK_REQUIRE(!g_timing.enabled, "fit_run: scoring timing is host-synchronised; disable it first");
    cudaStream_t s = (cudaStream_t)stream;
    if (st->n_tiles == 0) {
        WEFTK_CUDA(cudaMemsetAsync(d_ctl, 0, 4 * sizeof(int32_t), s));
        return WEFTK_OK;
    }
    WeftFitState run = *st;
    g_init_ctl = d_ctl;  // cleared with the counters
    int rc = weftk_fit_round(st, WEFTK_FIT_INIT, lambda, complex_threshold, d_perm, d_items8, n_items8, d_items16,
                             n_items16, d_items32, n_items32, stream);
    g_init_ctl = nullptr;
    for (int r = 0; !rc && r < max_rounds; ++r) {
        // rounds take the two halves of the counters in turn, so that each clears the other's
        run.status = st->status + 2 * ((r + 1) & 1);
        g_round_ctl = d_ctl;
        g_round_spare = st->status + 2 * (r & 1);
        rc = weftk_fit_round(&run, WEFTK_FIT_ROUND, lambda, complex_threshold, d_perm, d_items8, n_items8, d_items16,
                             n_items16, d_items32, n_items32, stream);
        g_round_ctl = nullptr;
        if (rc) break;
        rc = launch_fit_reseed(*st, d_ctl + 2, s);
    }
    if (rc) return rc;
    fit_unmark_kernel<<<ceil_div(std::max(st->n_tiles, 1), 256), 256, 0, s>>>(*st, run.status);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

// Side streams of the current device for the calling host thread: the 16-px and 32/64-px classes'
// scoring launches run beside the 8-px class's (forked from and joined back into the caller's
// stream, which a CUDA graph capture follows).  Created on first use, kept for the process.
struct ClassStreams {
    cudaStream_t s[2] = {nullptr, nullptr};
    cudaEvent_t fork = nullptr, join[2] = {nullptr, nullptr};
};

static int class_streams(ClassStreams** out) {
    thread_local std::map<int, ClassStreams> per_device;
    int dev = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    ClassStreams& cs = per_device[dev];
    if (cs.fork == nullptr) {
        for (int i = 0; i < 2; ++i) {
            WEFTK_CUDA(cudaStreamCreateWithFlags(&cs.s[i], cudaStreamNonBlocking));
            WEFTK_CUDA(cudaEventCreateWithFlags(&cs.join[i], cudaEventDisableTiming));
        }
        WEFTK_CUDA(cudaEventCreateWithFlags(&cs.fork, cudaEventDisableTiming));
    }
    *out = &cs;
    return WEFTK_OK;
}

extern "C" int weftk_fit_round(const WeftFitState* st, int mode, double lambda, double complex_threshold,
                               const int32_t* d_perm, const WeftFitItem* d_items8, int n_items8,
                               const WeftFitItem* d_items16, int n_items16, const WeftFitItem* d_items32,
                               int n_items32, void* stream) {
    WEFTK_REQUIRE(st && d_perm, "fit_round: null argument");
    WEFTK_REQUIRE(mode == WEFTK_FIT_INIT || mode == WEFTK_FIT_ROUND, "fit_round: bad mode");
    WEFTK_REQUIRE(mode == WEFTK_FIT_INIT || st->bg != nullptr, "fit_round: a greedy round needs the composite (bg)");
    WEFTK_REQUIRE(n_items8 >= 0 && n_items16 >= 0 && n_items32 >= 0, "fit_round: negative item count");
    for (int c = 0; c < 3; ++c)
        WEFTK_REQUIRE(st->variant[c] >= 0 && st->variant[c] < WEFTK_FIT_VARIANTS, "fit_round: bad scoring variant");
    if (st->n_tiles == 0) return WEFTK_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int nt = st->n_tiles, total = n_items8 + n_items16 + n_items32;
    const bool queued = st->queue != nullptr && st->queue_ctl != nullptr && total > 0;
    const bool merged = queued && g_round_ctl != nullptr;  // a round inside weftk_fit_run
    const bool init = mode == WEFTK_FIT_INIT;
    if (!merged) {
        fit_clear_kernel<<<1, 32, 0, s>>>(st->status, g_round_ctl == nullptr ? 4 : 2, queued ? st->queue_ctl : nullptr,
                                          g_init_ctl);
        fit_begin_kernel<<<ceil_div(nt, 256), 256, 0, s>>>(*st, mode, g_round_ctl);
    }
    if (g_timing.enabled) {
        int rc = timing_collect();
        if (rc) return rc;
        WEFTK_CUDA(cudaEventRecord(g_timing.start, s));
    }
    g_mode_init = init;
    g_lam = (float)lambda;
    {
        int dev = 0;
        WEFTK_CUDA(cudaGetDevice(&dev));
        WEFTK_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
    }
    ClassStreams* cs = nullptr;
    const bool side = !g_timing.enabled && (n_items16 > 0 || n_items32 > 0);
    auto fork = [&]() -> int {
        WEFTK_CUDA(cudaEventRecord(cs->fork, s));
        for (int i = 0; i < 2; ++i) WEFTK_CUDA(cudaStreamWaitEvent(cs->s[i], cs->fork, 0));
        return WEFTK_OK;
    };
    auto join = [&]() -> int {
        WEFTK_CUDA(cudaGetLastError());
        for (int i = 0; i < 2; ++i) {
            WEFTK_CUDA(cudaEventRecord(cs->join[i], cs->s[i]));
            WEFTK_CUDA(cudaStreamWaitEvent(s, cs->join[i], 0));
        }
        return WEFTK_OK;
    };
    int rc = WEFTK_OK;
    if (side && (rc = class_streams(&cs))) return rc;
    if (init && total > 0) {
        if (side && (rc = fork())) return rc;
        launch_const(*st, 0, st->variant[0], d_items8, n_items8, g_lam, s);
        launch_const(*st, 1, st->variant[1], d_items16, n_items16, g_lam, side ? cs->s[0] : s);
        launch_const(*st, 2, st->variant[2], d_items32, n_items32, g_lam, side ? cs->s[1] : s);
        if (side && (rc = join())) return rc;
    }
    if (queued) {
        const int tb = merged ? ceil_div(nt, 256) : 0;
        fit_queue_kernel<<<tb + ceil_div(total, 8), 256, 0, s>>>(*st, d_perm, d_items8, n_items8, d_items16, n_items16,
                                                                 d_items32, n_items32, g_lam, init, tb, g_round_ctl,
                                                                 g_round_spare);
    }
    // the size classes score disjoint tiles: the 16-px and 32/64-px classes run on side streams
    // beside the 8-px class (not while the scoring launches are being timed)
    if (side && (rc = fork())) return rc;
    if (n_items32) {
        g_queue_class = queued ? 2 : -1;
        g_queue_base = n_items8 + n_items16;
        launch_score_class32(st->variant[2], *st, d_perm, d_items32, n_items32, side ? cs->s[1] : s);
    }
    if (n_items16) {
        g_queue_class = queued ? 1 : -1;
        g_queue_base = n_items8;
        launch_score_class16(st->variant[1], *st, d_perm, d_items16, n_items16, side ? cs->s[0] : s);
    }
    if (n_items8) {
        g_queue_class = queued ? 0 : -1;
        g_queue_base = 0;
        launch_score_class8(st->variant[0], *st, d_perm, d_items8, n_items8, s);
    }
    g_queue_class = -1;
    if (side && (rc = join())) return rc;
    if (g_timing.enabled) {
        WEFTK_CUDA(cudaEventRecord(g_timing.stop, s));
        g_timing.pending = true;
    }
    fit_select_kernel<<<ceil_div(nt, SEL_WARPS), SEL_WARPS * 32, 0, s>>>(*st, mode, (float)lambda, lambda, g_round_ctl != nullptr);
    fit_end_kernel<<<ceil_div(nt, 256), 256, 0, s>>>(*st, mode, complex_threshold, g_round_ctl);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}
