// weftk_reseed.cu — device re-seeding of stalled tiles with residual-targeted candidates.
//
// Follows the reference's _generate_residual_candidates (src/weft/encoder.py:1255-1366):
// with err = src - clip(composite) and e = mean_channel |err|, pixels with e at or above
// the 60th percentile of e (numpy's linear interpolation) form the high-error set H;
// the candidates are constant patches in H's mean colours, two-colour linear patches
// split along the mean gradient of e, lines through H's centroid, a quadratic curve
// through H's leftmost, median-by-x and rightmost points, and triangles over H's
// extent — the same kinds, parameters and order as the reference, de-duplicated
// with the reference's coarse key.
//
// A persistent grid of 256-thread CTAs, one tile at a time (most tiles need nothing: 7,435 CTAs that
// only looked cost 4 us a launch).  A stalled round usually re-seeds a handful of tiles, so what counts
// is one tile's latency: 80 us for a 64-px tile with a bitonic sort of its 4096 errors and one thread
// assembling the 117 candidates, 25 us with the two order statistics the percentile needs taken by
// a radix selection (four histogram passes) and every candidate assembled and keyed by its own
// thread.  Means are accumulated in float64 and rounded to float32 (numpy
// accumulates these means in float32, so values agree to rounding).  Ties in the
// x-ordering of H are broken by raster order (numpy's default sort leaves that to
// the platform's sort implementation).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <set>

#include <climits>

#include "../../include/weftk_fit.h"
#include "weftk_common.cuh"
#include "weftk_prim.cuh"

namespace weftk {

extern __device__ int g_device_status;

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_MAX_CANDS = 128;
constexpr int KEY_LEN = 16;
constexpr int NV = 36;  // reduced values of the main pass

struct RsShared {
    double red[RS_WARPS][NV];
    double res[NV];
    int colcnt[64], colminy[64], colmaxy[64], rowcnt[64];
    WeftPrim cand[RS_MAX_CANDS];
    int key[RS_MAX_CANDS][KEY_LEN];
    unsigned hash[RS_MAX_CANDS];
    int keep[RS_MAX_CANDS];
    int hist[256];
    int sel_bin, sel_before, sel_count;
    int n_cand, n_quad, quad_of[4];
    float hi_col[3], corr[3];
    double curve[6], tri[2][6];
    double lines[4][4];  // x0 y0 x1 y1 of the four linear patches (float64, as the reference computes them)
    float lf[4][4];      // X0 Y0 DY DX rounded to float32 for the side test
};

// Sum NV per-thread values over the CTA (fixed order); result in s.res.
__device__ void block_sum(double (&v)[NV], RsShared& s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
        if (lane == 0) s.red[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double x = 0.0;
        for (int w = 0; w < RS_WARPS; ++w) x += s.red[w][threadIdx.x];
        s.res[threadIdx.x] = x;
    }
    __syncthreads();
}

__device__ __forceinline__ int qkey(double v, double scale) { return (int)(v * scale + 0.5); }

__device__ __forceinline__ float clip01d(double v) { return (float)fmin(1.0, fmax(0.0, v)); }

// Write candidate i with its dedup key and the key's hash.
__device__ __forceinline__ void put_cand(RsShared& s, int i, int kind, const double (&g)[7], int ng,
                                         const float* c0, const float* c1, double alpha) {
    WeftPrim& p = s.cand[i];
    p.kind = kind;
#pragma unroll
    for (int k = 0; k < 7; ++k) p.geom[k] = k < ng ? (float)g[k] : 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p.color0[k] = c0[k];
        p.color1[k] = c1 ? c1[k] : 0.0f;
    }
    p.alpha = (float)alpha;
    int* key = s.key[i];
    int n = 0;
    key[n++] = kind;
    for (int k = 0; k < ng; ++k) key[n++] = qkey(g[k], 4.0);
    for (int k = 0; k < 3; ++k) key[n++] = qkey((double)c0[k], 64.0);
    key[n++] = qkey(alpha, 32.0);
    if (c1)
        for (int k = 0; k < 3; ++k) key[n++] = qkey((double)c1[k], 64.0);
    while (n < KEY_LEN) key[n++] = INT_MIN;
    unsigned h = 2166136261u;
    for (int k = 0; k < KEY_LEN; ++k) h = (h ^ (unsigned)key[k]) * 16777619u;
    s.hash[i] = h;
}

// Values of rank r and r + 1 (0-based, ascending) among x[0..n), all >= 0 (or NaN, sorted last): the
// bits of a non-negative float order as unsigned integers, so rank r's bits are found eight at a
// time from a histogram of the values that share the bits found so far.  By the whole CTA.
__device__ void rank_pair(const float* x, int n, int r, RsShared& s, float& lo, float& hi) {
    const int tid = threadIdx.x;
    unsigned prefix = 0, mask = 0;
    int rank = r;
    for (int shift = 24; shift >= 0; shift -= 8) {
        s.hist[tid] = 0;
        __syncthreads();
        for (int p = tid; p < n; p += RS_THREADS) {
            const unsigned u = __float_as_uint(x[p]);
            if ((u & mask) == prefix) atomicAdd(&s.hist[(u >> shift) & 255u], 1);
        }
        __syncthreads();
        if (tid < 32) {  // the bin that holds the rank: lane l scans bins 8 l .. 8 l + 7
            int c[8], run = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                c[k] = s.hist[tid * 8 + k];
                run += c[k];
            }
            int incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (tid >= o) incl += v;
            }
            int before = incl - run;
            if (rank >= before && rank < incl) {
                int k = 0;
                while (k < 7 && rank >= before + c[k]) before += c[k++];
                s.sel_bin = tid * 8 + k;
                s.sel_before = before;
                s.sel_count = c[k];
            }
        }
        __syncthreads();
        prefix |= (unsigned)s.sel_bin << shift;
        mask |= 255u << shift;
        rank -= s.sel_before;
    }
    lo = __uint_as_float(prefix);
    hi = lo;
    if (rank + 1 < s.sel_count || r + 1 >= n) return;  // the next rank holds the same value
    unsigned next = 0xffffffffu;
    for (int p = tid; p < n; p += RS_THREADS) {
        const unsigned u = __float_as_uint(x[p]);
        if (u > prefix) next = min(next, u);
    }
    next = __reduce_min_sync(FULL, next);
    __syncthreads();
    if ((tid & 31) == 0) s.hist[tid >> 5] = (int)next;
    __syncthreads();
    next = (unsigned)s.hist[0];
    for (int w = 1; w < RS_WARPS; ++w) next = min(next, (unsigned)s.hist[w]);
    hi = __uint_as_float(next);
}

__global__ void __launch_bounds__(RS_THREADS) fit_reseed_kernel(WeftFitState st, const int* gate) {
    extern __shared__ float el[];  // the tile's errors
    __shared__ RsShared s;
    __shared__ int base_cnt, n_new, ok;
    if (gate != nullptr && *gate == 0) return;  // device-driven fit: no stall this round
    const int tid = threadIdx.x;
    for (int t = blockIdx.x; t < st.n_tiles; t += gridDim.x) {
    if (!(st.flags[t] & WEFTK_TILE_COMPLEX) || st.n_sel[t] >= st.cap[t]) continue;
    __syncthreads();  // the previous tile's shared state is read
    const int ts = st.size[t], n = ts * ts;
    const double wf = ts - 1, hf = ts - 1;
    const float4* src = reinterpret_cast<const float4*>(st.src) + st.px_off[t];
    const float4* bg = reinterpret_cast<const float4*>(st.bg) + st.px_off[t];

    for (int p = tid; p < n; p += RS_THREADS) {
        const float4 a = src[p], g = bg[p];
        const float e = __fdiv_rn(__fadd_rn(__fadd_rn(fabsf(a.x - clamp01(g.x)), fabsf(a.y - clamp01(g.y))),
                                            fabsf(a.z - clamp01(g.z))), 3.0f);
        el[p] = e;
    }
    if (tid < 64) {
        s.colcnt[tid] = 0;
        s.rowcnt[tid] = 0;
        s.colminy[tid] = INT_MAX;
        s.colmaxy[tid] = -1;
    }
    __syncthreads();
    // numpy percentile of a float32 array, linear method, all in float32:
    // q = 60/100, virtual index (n-1)*q, lerp from the far end when gamma >= 0.5
    const float vi = __fmul_rn((float)(n - 1), __fdiv_rn(60.0f, 100.0f));
    const int rank = (int)floorf(vi);
    float pa, pb;
    rank_pair(el, n, rank, s, pa, pb);
    const float pg = __fsub_rn(vi, (float)rank), pd = __fsub_rn(pb, pa);
    const float thr = (pg >= 0.5f) ? __fsub_rn(pb, __fmul_rn(pd, __fsub_rn(1.0f, pg))) : __fadd_rn(pa, __fmul_rn(pd, pg));
    const int qh = ts / 2;

    // main pass: counts and sums over H, quadrants, the gradient of e, the tile mean
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int p = tid; p < n; p += RS_THREADS) {
        const int x = p % ts, y = p / ts;
        const float4 a = src[p], g4 = bg[p];
        const float pr[3] = {clamp01(g4.x), clamp01(g4.y), clamp01(g4.z)};
        const float sv[3] = {a.x, a.y, a.z};
        v[33] += sv[0];
        v[34] += sv[1];
        v[35] += sv[2];
        // np.gradient: central differences inside, one-sided at the borders
        const float* row = el + y * ts;
        const float gx = (x == 0) ? __fsub_rn(row[1], row[0])
                         : (x == ts - 1) ? __fsub_rn(row[ts - 1], row[ts - 2])
                                         : __fdiv_rn(__fsub_rn(row[x + 1], row[x - 1]), 2.0f);
        const float gy = (y == 0) ? __fsub_rn(el[ts + x], el[x])
                         : (y == ts - 1) ? __fsub_rn(el[(ts - 1) * ts + x], el[(ts - 2) * ts + x])
                                         : __fdiv_rn(__fsub_rn(el[(y + 1) * ts + x], el[(y - 1) * ts + x]), 2.0f);
        v[31] += gx;
        v[32] += gy;
        if (el[p] >= thr) {
            v[0] += 1.0;
            for (int c = 0; c < 3; ++c) {
                v[1 + c] += sv[c];
                v[4 + c] += pr[c];
                v[7 + c] += __fsub_rn(sv[c], pr[c]);
            }
            v[10] += x;
            v[11] += y;
            const int q = (y >= qh ? 2 : 0) + (x >= qh ? 1 : 0);
            v[12 + q] += 1.0;
            for (int c = 0; c < 3; ++c) v[16 + 3 * q + c] += sv[c];
            atomicAdd(&s.colcnt[x], 1);
            atomicMin(&s.colminy[x], y);
            atomicMax(&s.colmaxy[x], y);
            atomicAdd(&s.rowcnt[y], 1);
        }
    }
    block_sum(v, s);
    const double m = s.res[0];
    if (m == 0.0) continue;  // uniform across the CTA

    // direction of the mean error gradient, and the four linear-patch lines
    if (tid == 0) {
        const double mx = (double)(float)(s.res[31] / (double)n), my = (double)(float)(s.res[32] / (double)n);
        const double nrm = sqrt(mx * mx + my * my) + 1e-8;
        const double vx = mx / nrm, vy = my / nrm;
        const double offs[3] = {0.5, 0.3, 0.7};
        for (int L = 0; L < 3; ++L) {
            const double cx = wf * offs[L], cy = hf * offs[L];
            s.lines[L][0] = cx - vx * wf * 0.6;
            s.lines[L][1] = cy - vy * hf * 0.6;
            s.lines[L][2] = cx + vx * wf * 0.6;
            s.lines[L][3] = cy + vy * hf * 0.6;
        }
        const double cx = wf * 0.5, cy = hf * 0.5;
        s.lines[3][0] = cx + vy * wf * 0.6;
        s.lines[3][1] = cy - vx * hf * 0.6;
        s.lines[3][2] = cx - vy * wf * 0.6;
        s.lines[3][3] = cy + vx * hf * 0.6;
        for (int L = 0; L < 4; ++L) {
            s.lf[L][0] = (float)s.lines[L][0];
            s.lf[L][1] = (float)s.lines[L][1];
            s.lf[L][2] = (float)(s.lines[L][3] - s.lines[L][1]);
            s.lf[L][3] = (float)(s.lines[L][2] - s.lines[L][0]);
        }
    }
    __syncthreads();
    // side means for the four lines (integer pixel coordinates, float32 side test)
    double w2[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) w2[k] = 0.0;
    for (int p = tid; p < n; p += RS_THREADS) {
        const float xf = (float)(p % ts), yf = (float)(p / ts);
        const float4 a = src[p];
#pragma unroll
        for (int L = 0; L < 4; ++L) {
            const float side = __fsub_rn(__fmul_rn(__fsub_rn(xf, s.lf[L][0]), s.lf[L][2]),
                                         __fmul_rn(__fsub_rn(yf, s.lf[L][1]), s.lf[L][3]));
            const int o = L * 8 + (side >= 0.0f ? 0 : 4);
            w2[o] += 1.0;
            w2[o + 1] += a.x;
            w2[o + 2] += a.y;
            w2[o + 3] += a.z;
        }
    }
    const double tile_mean[3] = {s.res[33] / n, s.res[34] / n, s.res[35] / n};
    double hs[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) hs[k] = s.res[k];
    __syncthreads();
    block_sum(w2, s);

    // what the candidates share: colours, the non-empty quadrants, H's extent and median point
    const int mi = (int)m;
    const double ecx = hs[10] / m, ecy = hs[11] / m;
    if (tid < 32) {
        // first and last column and row of H (two per lane)
        const bool c0 = 2 * tid < ts && s.colcnt[2 * tid] > 0, c1 = 2 * tid + 1 < ts && s.colcnt[2 * tid + 1] > 0;
        const bool r0 = 2 * tid < ts && s.rowcnt[2 * tid] > 0, r1 = 2 * tid + 1 < ts && s.rowcnt[2 * tid + 1] > 0;
        const int minx = __reduce_min_sync(FULL, c0 ? 2 * tid : c1 ? 2 * tid + 1 : INT_MAX);
        const int maxx = __reduce_max_sync(FULL, c1 ? 2 * tid + 1 : c0 ? 2 * tid : -1);
        const int miny = __reduce_min_sync(FULL, r0 ? 2 * tid : r1 ? 2 * tid + 1 : INT_MAX);
        const int maxy = __reduce_max_sync(FULL, r1 ? 2 * tid + 1 : r0 ? 2 * tid : -1);
        int X = minx, before = 0, Y = 0;
        if (mi >= 6) {
            // stable order by x (raster order within a column): first, middle, last
            const int r = mi / 2, a = s.colcnt[2 * tid], b = s.colcnt[2 * tid + 1];
            int incl = a + b;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (tid >= o) incl += v;
            }
            const int at = incl - a - b;
            const bool in_a = r >= at && r < at + a, in_b = r >= at + a && r < incl;
            const unsigned who = __ballot_sync(FULL, in_a || in_b);
            const int lane = who ? __ffs(who) - 1 : 0;
            X = __shfl_sync(FULL, in_a ? 2 * tid : 2 * tid + 1, lane);
            before = __shfl_sync(FULL, in_a ? at : at + a, lane);
            // the (r - before)-th row of H in column X
            int want = r - before;
            for (int y0 = 0; y0 < ts; y0 += 32) {
                const unsigned rows = __ballot_sync(FULL, y0 + tid < ts && el[min(y0 + tid, ts - 1) * ts + X] >= thr);
                const int c = __popc(rows);
                if (want < c) {
                    Y = y0 + __fns(rows, 0, want + 1);
                    break;
                }
                want -= c;
            }
        }
        if (tid == 0) {
            for (int c = 0; c < 3; ++c) {
                s.hi_col[c] = clip01d((double)(float)(hs[1 + c] / m));
                const float pm = (float)(hs[4 + c] / m), em = (float)(hs[7 + c] / m);
                s.corr[c] = clip01d((double)__fadd_rn(pm, em));
            }
            s.n_quad = 0;
            for (int q = 0; q < 4; ++q)
                if (hs[12 + q] > 0.0) s.quad_of[s.n_quad++] = q;
            s.n_cand = 15 + 3 * s.n_quad + 11 + 60 + 4 + (mi >= 6 ? 3 : 0) + (mi >= 3 ? 12 : 0);
            if (mi >= 6) {
                const double p0x = minx, p0y = s.colminy[minx], p1x = maxx, p1y = s.colmaxy[maxx];
                s.curve[0] = p0x;
                s.curve[1] = p0y;
                s.curve[2] = fmax(0.0, fmin(wf, 2.0 * X - (p0x + p1x) / 2.0));
                s.curve[3] = fmax(0.0, fmin(hf, 2.0 * Y - (p0y + p1y) / 2.0));
                s.curve[4] = p1x;
                s.curve[5] = p1y;
            }
            if (mi >= 3) {
                const double g1[6] = {(double)minx, (double)s.colminy[minx], (double)maxx, (double)s.colminy[maxx], ecx, ecy};
                const double g2[6] = {(double)minx, (double)miny, (double)maxx, (double)maxy, ecx, ecy};
                for (int k = 0; k < 6; ++k) {
                    s.tri[0][k] = g1[k];
                    s.tri[1][k] = g2[k];
                }
            }
        }
    }
    __syncthreads();
    // candidate tid of the list: constants (H's colour, the corrected colour, H's again x 5 alphas),
    // quadrant colours x 3, linear patches x 3 (the last x 2), lines through H's centroid (5
    // thicknesses x 2 repeats x 3 alphas x vertical, horizontal), two diagonals x 2, the curve x 3,
    // two triangles x 3 alphas x 2 repeats
    if (tid < s.n_cand) {
        double g[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        int i = tid;
        const int nq = 3 * s.n_quad, n_curve = mi >= 6 ? 3 : 0;
        if (i < 15) {
            const int k = i / 5, j = i % 5;
            const double a = j == 0 ? 0.6 : j == 1 ? 0.4 : j == 2 ? 0.25 : j == 3 ? 0.15 : 0.08;
            put_cand(s, tid, 0, g, 0, k == 1 ? s.corr : s.hi_col, nullptr, a);
        } else if ((i -= 15) < nq) {
            const int q = s.quad_of[i / 3], j = i % 3;
            float qc[3];
            for (int c = 0; c < 3; ++c) qc[c] = clip01d((double)(float)(hs[16 + 3 * q + c] / hs[12 + q]));
            put_cand(s, tid, 0, g, 0, qc, nullptr, j == 0 ? 0.35 : j == 1 ? 0.2 : 0.1);
        } else if ((i -= nq) < 11) {
            const int L = i / 3, j = i % 3;
            const double a = L < 3 ? (j == 0 ? 0.5 : j == 1 ? 0.3 : 0.15) : (j == 0 ? 0.4 : 0.2);
            float c0[3], c1[3];
            const double ca = s.res[L * 8], cb = s.res[L * 8 + 4];
            for (int c = 0; c < 3; ++c) {
                c0[c] = ca > 0 ? (float)(s.res[L * 8 + 1 + c] / ca) : (float)tile_mean[c];
                c1[c] = cb > 0 ? (float)(s.res[L * 8 + 5 + c] / cb) : (float)tile_mean[c];
            }
            for (int k = 0; k < 4; ++k) g[k] = s.lines[L][k];
            put_cand(s, tid, 1, g, 4, c0, c1, a);
        } else if ((i -= 11) < 60) {
            const int th = i / 12, j = (i % 6) / 2;
            g[4] = th == 0 ? 0.3 : th == 1 ? 0.6 : th == 2 ? 1.0 : th == 3 ? 1.5 : 2.5;
            if (i & 1) {
                g[1] = g[3] = ecy;
                g[2] = wf;
            } else {
                g[0] = g[2] = ecx;
                g[3] = hf;
            }
            put_cand(s, tid, 2, g, 5, s.hi_col, nullptr, j == 0 ? 0.5 : j == 1 ? 0.3 : 0.15);
        } else if ((i -= 60) < 4) {
            g[2] = wf;
            g[i & 1 ? 1 : 3] = hf;
            g[4] = i < 2 ? 0.5 : 1.0;
            put_cand(s, tid, 2, g, 5, s.hi_col, nullptr, 0.25);
        } else if ((i -= 4) < n_curve) {
            for (int k = 0; k < 6; ++k) g[k] = s.curve[k];
            g[6] = i == 0 ? 0.5 : i == 1 ? 1.0 : 2.0;
            put_cand(s, tid, 3, g, 7, s.hi_col, nullptr, 0.3);
        } else {
            i -= n_curve;
            const int j = (i % 6) / 2;
            for (int k = 0; k < 6; ++k) g[k] = s.tri[i / 6][k];
            put_cand(s, tid, 4, g, 6, s.hi_col, nullptr, j == 0 ? 0.4 : j == 1 ? 0.2 : 0.1);
        }
    }
    __syncthreads();
    // keep the first candidate of each key
    const int nc = s.n_cand;
    bool kept = false;
    if (tid < nc) {
        bool dup = false;
        const unsigned h = s.hash[tid];
        for (int j = 0; j < tid && !dup; ++j) {
            if (s.hash[j] != h) continue;
            bool same = true;
            for (int k = 0; k < KEY_LEN; ++k)
                if (s.key[j][k] != s.key[tid][k]) {
                    same = false;
                    break;
                }
            dup = same;
        }
        kept = !dup;
    }
    // places of the kept ones, in order
    const unsigned kb = __ballot_sync(FULL, kept);
    if ((tid & 31) == 0) s.hist[tid >> 5] = __popc(kb);
    __syncthreads();
    int place = __popc(kb & ((1u << (tid & 31)) - 1u));
    for (int w = 0; w < (tid >> 5); ++w) place += s.hist[w];
    if (tid < nc) s.keep[tid] = kept ? place : -1;
    if (tid == 0) {
        int k = 0;
        for (int w = 0; w < RS_WARPS; ++w) k += s.hist[w];
        n_new = k;
        base_cnt = st.pool_cnt[t];
        ok = base_cnt + k <= st.pool_cap[t];
        if (!ok) atomicCAS(&g_device_status, 0, WEFTK_E_RANGE);
    }
    __syncthreads();
    if (!ok) continue;
    const long long off = st.pool_off[t];
    if (tid < nc && s.keep[tid] >= 0) {
        const long long slot = off + base_cnt + s.keep[tid];
        WeftPrim* dst = const_cast<WeftPrim*>(st.cand) + slot;
        *dst = s.cand[tid];
        st.alive[slot] = 1;
        st.kind[slot] = (uint8_t)s.cand[tid].kind;
    }
    if (tid == 0) {
        st.pool_cnt[t] = base_cnt + n_new;
        st.n_alive[t] += n_new;
    }
    }
}

}  // namespace weftk

using namespace weftk;

int launch_fit_reseed(const WeftFitState& st, const int* gate, cudaStream_t stream) {
    if (st.n_tiles == 0) return WEFTK_OK;
    const int smem = 64 * 64 * (int)sizeof(float);
    int dev = 0, sms = 148;
    WEFTK_CUDA(cudaGetDevice(&dev));
    WEFTK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    {  // the dynamic shared-memory opt-in is per device: set it once per device, under a lock
        static std::mutex mu;
        static std::set<int> done;
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count(dev)) {
            WEFTK_CUDA(cudaFuncSetAttribute(fit_reseed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            done.insert(dev);
        }
    }
    fit_reseed_kernel<<<std::min(st.n_tiles, sms * 4), RS_THREADS, smem, stream>>>(st, gate);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}

extern "C" int weftk_fit_reseed(const WeftFitState* st, int quality, void* stream) {
    (void)quality;
    WEFTK_REQUIRE(st && st->bg, "fit_reseed: null state or no composite (bg)");
    return launch_fit_reseed(*st, nullptr, (cudaStream_t)stream);
}
