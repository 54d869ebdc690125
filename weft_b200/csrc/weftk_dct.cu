// weftk_dct.cu — the decoder's raster branch: per-tile DCT residual layer and the u8 BILINEAR
// resize (see include/weftk_dct.h).
//
// DCT layer: a launch per tile side, a CTA per 4096 pixels of its tiles.  Each channel's
// quantized block is gathered straight from the coefficient stream (tile-major or band-major zigzag: the
// band-to-tile permutation is only an address computation), dequantized and inverse-transformed in
// float64 as two separable passes through shared memory, rounded to float32; the three channels are then
// colour-transformed, added to the image and clipped.  The transform is the orthonormal DCT-III written
// as a matrix product with the DCT-II basis A[k][x] = c_k cos(pi (2x + 1) k / (2n)).
// Bound: latency (two CTAs a SM, a fill of the chip once: the gather, the basis and the image's pixels are
// each asked for in batches) and instruction issue; the float64 pipes are 9 % busy.  A 1024 x 1024 picture
// with its tiles of 8 to 64 px takes 41 us, 4:2:0, and took 191 with a CTA per tile, one output of a pass
// per thread, the basis read from memory and a launch per side.
//
// Resize: Pillow's ImagingResample for 8-bit images.  A sample's taps (bounds, float64 triangle
// weights normalised by their sum, rounded to 22-bit fixed point) are derived exactly as Pillow's
// precompute_coeffs / normalize_coeffs_8bpc do, then accumulated in int32 and rounded with the same clip.
// Both passes run in one kernel, the 8-bit intermediate in shared memory: 1024 x 1024 to 3840 x 2160 takes
// 36 us (99.5 MB written: 15 us) and took 98 as two kernels.  Those two (a thread per output column over 8
// rows, the intermediate in the caller's scratch) run where the window of 32 output rows does not fit
// 100 KB: a downscale by more than about 2.2 in both directions.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../../include/weftk_dct.h"
#include "weftk_common.cuh"

namespace weftk {

extern __device__ int g_device_status;

// Basis and zigzag tables for block sides n = 2, 4, ..., 64, back to back: side n = 2^L starts
// at (4^L - 4) / 3.
constexpr int kDctTab = 5460;
__device__ __align__(16) double g_dct_basis[kDctTab];  // [k * n + x] = A[k][x]; copied two at a time
__device__ short g_dct_zigzag[kDctTab];                // [u * n + v] = zigzag scan position of (u, v)

__host__ __device__ constexpr int dct_tab_off(int log2n) { return ((1 << (2 * log2n)) - 4) / 3; }
static_assert(__alignof__(g_dct_basis) >= alignof(double2), "the basis is read as double2");
static_assert(dct_tab_off(1) % 2 == 0 && dct_tab_off(2) % 2 == 0 && dct_tab_off(3) % 2 == 0 &&
                  dct_tab_off(4) % 2 == 0 && dct_tab_off(5) % 2 == 0 && dct_tab_off(6) % 2 == 0,
              "every side's basis starts on a double2");

__device__ __forceinline__ int ilog2(int n) { return 31 - __clz(n); }

__global__ void dct_tables_kernel() {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kDctTab) return;
    int L = 1;
    while (L < 6 && i >= dct_tab_off(L + 1)) ++L;
    const int n = 1 << L, r = i - dct_tab_off(L);
    const int k = r >> L, x = r & (n - 1);
    // basis: sqrt(1/n) for k = 0, else cos(((pi * (2x + 1)) * k) / (2n)) * sqrt(2/n)
    if (k == 0) {
        g_dct_basis[i] = sqrt(1.0 / (double)n);
    } else {
        const double arg = __ddiv_rn(__dmul_rn(__dmul_rn(3.141592653589793, (double)(2 * x + 1)), (double)k),
                                     (double)(2 * n));
        g_dct_basis[i] = __dmul_rn(cos(arg), sqrt(2.0 / (double)n));
    }
    // zigzag position of row-major (u, v) = (k, x): anti-diagonal s = u + v holds rows
    // lo..hi, scanned bottom-left to top-right (rows descending) when s is even, else ascending.
    const int u = k, v = x, s = u + v;
    const int before = s < n ? s * (s + 1) / 2 : n * n - (2 * n - 1 - s) * (2 * n - s) / 2;
    const int lo = s - n + 1 > 0 ? s - n + 1 : 0, hi = s < n - 1 ? s : n - 1;
    g_dct_zigzag[i] = (short)(before + ((s & 1) == 0 ? hi - u : u - lo));
}

// The layer's kernel: 256 threads take 4096 pixels' worth of tiles of one side's class (one tile of 64,
// 64 tiles of 8), so the classes of a picture are a few hundred equal CTAs, two per SM; the launches of the
// classes overlap (a launch with WEFTK_DCT_FOLLOWS may start beside the one before it).  A thread owns a 4 x 4 set of a block's outputs, rows and columns n / 4 apart, so that
// neighbouring lanes read and write neighbouring columns; per step of a pass it reads 4 + 4 values for 16
// float64 multiply-adds.  Cb and Cr of 4:2:0 go together, a quarter of the threads each.  Quantisation
// steps depend on u + v only and are tabulated per CTA.
constexpr int DC_THREADS = 256, DC_PIXELS = 4096;
constexpr int kDctBlockWords = 4640;  // doubles of one staged block set: the largest of the classes
constexpr int kDctSteps = 252;        // steps of all block sides: side 2^L has 2^(L+1) at 2^(L+1) - 4
__host__ __device__ constexpr int dct_pitch(int n) { return n >= 16 ? n + 2 : n; }
__host__ __device__ constexpr int dct_slot_words(int s) { return s * dct_pitch(s) + 2; }
static_assert(dct_pitch(2) % 2 == 0 && dct_pitch(4) % 2 == 0 && dct_pitch(8) % 2 == 0 && dct_pitch(16) % 2 == 0 &&
                  dct_pitch(32) % 2 == 0 && dct_pitch(64) % 2 == 0 && kDctBlockWords % 2 == 0 && kDctSteps % 2 == 0,
              "rows of a staged block, the blocks and the staged basis start on a double2");
static_assert(256 * dct_slot_words(4) <= kDctBlockWords && 64 * dct_slot_words(8) <= kDctBlockWords &&
                  16 * dct_slot_words(16) <= kDctBlockWords && 4 * dct_slot_words(32) <= kDctBlockWords &&
                  dct_slot_words(64) <= kDctBlockWords,
              "every class's blocks fit");
constexpr size_t kDctSmem = (2 * kDctBlockWords + 2 * kDctSteps) * sizeof(double) + 2 * DC_PIXELS * sizeof(float);

struct DctLayer {
    const WeftDctTile* tiles;
    int n_tiles, log_side;  // the class: no tile is larger
    const int16_t* coeffs;
    long long n_coeffs;
    int chroma, band;
    double step_luma, step_chroma, alpha;
    float* image;
    int width, height;
};

// 16 outputs (4 of a 2 x 2 block) of the pass along v of one block of side 2^LN: rows ub + nb i, columns
// xb + nb j, each a sum over k ascending; then of the pass along u.
template <int LN>
__device__ __forceinline__ void dct_rows(const double* __restrict__ A, const double* X, double* T, int ub, int xb) {
    constexpr int n = 1 << LN, R = n < 4 ? n : 4, nb = n / R, P = dct_pitch(n);
    double acc[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = 0.0;
    const double* a = A + xb;
    const double* x = X + ub * P;
#pragma unroll 2
    for (int k = 0; k < n; k += 2) {
        double2 v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = *reinterpret_cast<const double2*>(x + nb * i * P + k);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double w[R];
#pragma unroll
            for (int j = 0; j < R; ++j) w[j] = a[(k + h) * n + nb * j];
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < R; ++j) acc[i][j] = fma(w[j], h ? v[i].y : v[i].x, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) T[(ub + nb * i) * P + xb + nb * j] = acc[i][j];
}

template <int LN>
__device__ __forceinline__ void dct_cols(const double* __restrict__ A, const double* T, int yb, int xb,
                                         float (&out)[4][4]) {
    constexpr int n = 1 << LN, R = n < 4 ? n : 4, nb = n / R, P = dct_pitch(n);
    double acc[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = 0.0;
    const double* a = A + yb;
    const double* t = T + xb;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        double w[R], v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = a[k * n + nb * i];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = t[k * P + nb * j];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < R; ++j) acc[i][j] = fma(w[i], v[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) out[i][j] = __double2float_rn(acc[i][j]);
}

// HALF: 4:2:0 (chroma mode 2)
template <bool HALF>
__global__ void __launch_bounds__(DC_THREADS, 2) dct_layer_kernel(DctLayer L) {
    extern __shared__ __align__(16) double dct_smem[];
    double* X = dct_smem;                     // dequantized blocks [slot][u * pitch + v]
    double* T = X + kDctBlockWords;           // after the pass along v: [slot][u * pitch + x]
    double* steps = T + kDctBlockWords;       // luma, chroma
    float* R = reinterpret_cast<float*>(steps + 2 * kDctSteps);  // float32 results of channels 1, 2
    // 4:2:0 leaves room there for the phase's basis: luma's before there are results, chroma's beside them
    double* basis = reinterpret_cast<double*>(R);
    constexpr int R_PLANE = HALF ? DC_PIXELS / 4 : DC_PIXELS;
    const int tid = threadIdx.x;
    // the launch that follows may be the layer's next class (WEFTK_DCT_FOLLOWS): it can start beside this
    // one, and does its transforms, but waits for this one (below) before it touches the image.  Its
    // descriptors and coefficients are complete, since the layer's first launch started after all work
    // before it
    asm volatile("griddepcontrol.launch_dependents;");
    const int LS = L.log_side;
    const int log_slots = 12 - 2 * LS, log_tpt = 2 * LS - 4;  // slots * threads per tile = 256
    const int slot_words = dct_slot_words(1 << LS);
    const int tile0 = (int)blockIdx.x << log_slots;
    const WeftDctTile* tiles = L.tiles + tile0;
    const int n_slots = min(1 << log_slots, L.n_tiles - tile0);

    auto side_ok = [&](int S) { return S >= 4 && S <= (1 << LS) && (S & (S - 1)) == 0; };
    for (int i = tid; i < 2 * kDctSteps; i += DC_THREADS) {
        const int r = i % kDctSteps, ll = ilog2(r + 4) - 1, d = r + 4 - (2 << ll);
        const double step = i < kDctSteps ? L.step_luma : L.step_chroma;
        if (ll > LS) continue;
        steps[i] = L.alpha > 0.0
                       ? __dmul_rn(step, __dadd_rn(1.0, __dmul_rn(L.alpha, __ddiv_rn((double)d,
                                                                                     2.0 * (double)((1 << ll) - 1)))))
                       : step;
    }
    const int slot = tid >> log_tpt, lt = tid & ((1 << log_tpt) - 1);
    int S = 0;
    if (slot < n_slots) {
        S = tiles[slot].size;
        if (!side_ok(S)) {
            if (lt == 0) atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
            S = 0;
        }
    }
    // every tile of the class's side, its coefficients inside the stream (a block's positions 0 .. n n - 1
    // are all read, so its first and last bound them)
    bool ok = true;
    for (int i = tid; i < n_slots; i += DC_THREADS) {
        ok = ok && tiles[i].size == (1 << LS);
        for (int c = 0; c < 3; ++c) {
            const long long first = tiles[i].coef_base[c];
            const long long last = first + ((1LL << (HALF && c ? 2 * LS - 2 : 2 * LS)) - 1) * tiles[i].coef_stride[c];
            ok = ok && first >= 0 && first < L.n_coeffs && last >= 0 && last < L.n_coeffs;
        }
    }
    const bool plain = __syncthreads_and(ok);
    float luma[4][4];
    constexpr int n_phases = HALF ? 2 : 3;
    for (int ph = 0; ph < n_phases; ++ph) {
        const bool half = HALF && ph > 0;  // channels 1 and 2, half the side
        const int log_per = half ? 2 * LS - 1 : 2 * LS;
        __syncthreads();  // the steps; the last phase's readers of X
        // gather and dequantize: band-major streams hold neighbouring tiles' coefficients side by side,
        // tile-major ones a tile's own.  When every tile is of the class's side and inside the stream,
        // only the tile differs between a thread's coefficients
        const int lc = half ? LS - 1 : LS, nc = 1 << lc, pc = dct_pitch(nc);
        double* phase_basis = basis + (half ? 2 * R_PLANE / 2 : 0);
        if (HALF && plain) {
            const double2* from = reinterpret_cast<const double2*>(g_dct_basis + dct_tab_off(lc));
            double2* to = reinterpret_cast<double2*>(phase_basis);
#pragma unroll 8
            for (int i = tid; i < nc * nc / 2; i += DC_THREADS) to[i] = from[i];
        }
        if (plain) {
            const int chroma = L.chroma != 0 && ph > 0 ? kDctSteps : 0;
            const double* st = steps + chroma + (2 << lc) - 4;
            const short* Z = g_dct_zigzag + dct_tab_off(lc);
#pragma unroll 8
            for (int e = tid; e < (1 << (log_per + log_slots)); e += DC_THREADS) {
                const int sl = L.band ? e & ((1 << log_slots) - 1) : e >> log_per;
                const int k = L.band ? e >> log_slots : e & ((1 << log_per) - 1);
                const WeftDctTile* tp = tiles + min(sl, n_slots - 1);  // (a slot past the end: not used)
                const int q = k >> (2 * lc), idx = k & (nc * nc - 1), u = idx >> lc, v = idx & (nc - 1);
                const int c = half ? 1 + q : ph, pos = L.band ? Z[idx] : idx;
                const int coef = L.coeffs[tp->coef_base[c] + (long long)pos * tp->coef_stride[c]];
                X[sl * slot_words + (q * nc + u) * pc + v] = __dmul_rn((double)coef, __dmul_rn(st[u + v], tp->step_scale));
            }
        } else
        // (the 16 or 8 coefficients of a thread are asked for eight at a time, without a branch between)
        for (int e0 = tid; e0 < (1 << (log_per + log_slots)); e0 += 8 * DC_THREADS) {
            int v[8], at[8];
            double step[8];
            bool bad = false;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = e0 + i * DC_THREADS;
                const int sl = L.band ? e & ((1 << log_slots) - 1) : e >> log_per;
                const int k = L.band ? e >> log_slots : e & ((1 << log_per) - 1);
                const WeftDctTile* tp = tiles + min(sl, n_slots - 1);
                const int St = tp->size, l = max(half ? ilog2(St | 1) - 1 : ilog2(St | 1), 1), n = 1 << l;
                const int q = k >> (2 * l), c = half ? 1 + (q & 1) : ph, idx = k & (n * n - 1);
                const bool mine = sl < n_slots && side_ok(St) && q < (half ? 2 : 1);
                const long long pos = L.band ? (long long)g_dct_zigzag[mine ? dct_tab_off(l) + idx : 0] : (long long)idx;
                const long long a = tp->coef_base[c] + pos * tp->coef_stride[c];
                const bool in = mine && a >= 0 && a < L.n_coeffs;
                bad = bad || (mine && !in);
                v[i] = in ? (int)L.coeffs[a] : 0;
                at[i] = mine ? sl * slot_words + q * n * dct_pitch(n) + (idx >> l) * dct_pitch(n) + (idx & (n - 1)) : -1;
                const int diag = (idx >> l) + (idx & (n - 1));
                step[i] = __dmul_rn(mine ? steps[(L.chroma != 0 && c > 0 ? kDctSteps : 0) + (2 << l) - 4 + diag] : 0.0,
                                    tp->step_scale);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (at[i] >= 0) X[at[i]] = __dmul_rn((double)v[i], step[i]);
            if (bad) atomicCAS(&g_device_status, 0, WEFTK_E_ARG);
        }
        __syncthreads();
        const int n = half ? S >> 1 : S, l = S == 0 ? 0 : ilog2(n), lb = max(l - 2, 0);
        const int jobs = S == 0 ? 0 : (half ? 2 : 1) << (2 * lb);
        auto rows = [&](const double* A) {
            for (int w = lt; w < jobs; w += 1 << log_tpt) {
                const int at = slot * slot_words + (w >> (2 * lb)) * n * dct_pitch(n);
                const int ub = (w >> lb) & ((1 << lb) - 1), xb = w & ((1 << lb) - 1);
                switch (l) {
                    case 1: dct_rows<1>(A, X + at, T + at, ub, xb); break;
                    case 2: dct_rows<2>(A, X + at, T + at, ub, xb); break;
                    case 3: dct_rows<3>(A, X + at, T + at, ub, xb); break;
                    case 4: dct_rows<4>(A, X + at, T + at, ub, xb); break;
                    case 5: dct_rows<5>(A, X + at, T + at, ub, xb); break;
                    default: dct_rows<6>(A, X + at, T + at, ub, xb);
                }
            }
        };
        auto cols = [&](const double* A) {
            for (int w = lt; w < jobs; w += 1 << log_tpt) {
                const int q = w >> (2 * lb), at = slot * slot_words + q * n * dct_pitch(n);
                const int yb = (w >> lb) & ((1 << lb) - 1), xb = w & ((1 << lb) - 1);
                float r[4][4] = {};
                switch (l) {
                    case 1: dct_cols<1>(A, T + at, yb, xb, r); break;
                    case 2: dct_cols<2>(A, T + at, yb, xb, r); break;
                    case 3: dct_cols<3>(A, T + at, yb, xb, r); break;
                    case 4: dct_cols<4>(A, T + at, yb, xb, r); break;
                    case 5: dct_cols<5>(A, T + at, yb, xb, r); break;
                    default: dct_cols<6>(A, T + at, yb, xb, r);
                }
                float* Rc = R + (half ? q : ph - 1) * R_PLANE + (slot << (HALF ? 2 * LS - 2 : 2 * LS));
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (ph == 0) {
                            luma[i][j] = r[i][j];
                        } else if (l > 1 || (i < 2 && j < 2)) {
                            Rc[(yb + (i << lb)) * n + xb + (j << lb)] = r[i][j];
                        }
                    }
            }
        };
        const double* table = g_dct_basis + (S == 0 ? 0 : dct_tab_off(l));
        if (HALF && plain) rows(phase_basis);
        else rows(table);
        __syncthreads();
        if (HALF && plain) cols(phase_basis);
        else cols(table);
    }
    __syncthreads();

    asm volatile("griddepcontrol.wait;" ::: "memory");  // the image as the launches before leave it
    const int nb = S >> 2;
    if (S == 0 || lt >= nb * nb) return;
    const WeftDctTile* tp = tiles + slot;
    const int tx0 = tp->x, ty0 = tp->y, yb = lt / nb, xb = lt % nb;
    const float* R1 = R + (slot << (HALF ? 2 * LS - 2 : 2 * LS));
    const float* R2 = R1 + R_PLANE;
    // two rows' pixels are read before the first is written
#pragma unroll
    for (int i0 = 0; i0 < 4; i0 += 2) {
        float px[2][4][3];
        bool in[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const long long gy = (long long)ty0 + yb + nb * (i0 + i);
            const float* row = L.image + (gy * L.width + tx0) * 3;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const long long gx = (long long)tx0 + xb + nb * j;
                in[i][j] = gy >= 0 && gy < L.height && gx >= 0 && gx < L.width;
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) px[i][j][ch] = in[i][j] ? row[(xb + nb * j) * 3 + ch] : 0.0f;
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int y = yb + nb * (i0 + i);
            float* row = L.image + (((long long)ty0 + y) * L.width + tx0) * 3;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int x = xb + nb * j;
                const int ci = HALF ? (y >> 1) * (S >> 1) + (x >> 1) : y * S + x;
                float res[3] = {luma[i0 + i][j], R1[ci], R2[ci]};
                if (HALF || L.chroma != 0) {
                    const double Y = res[0], Cb = res[1], Cr = res[2];
                    // rows of the BT.601 YCbCr -> RGB residual matrix, each a left-to-right dot product
                    // (without its zero terms, which leave a sum as it is)
                    res[0] = __double2float_rn(__dadd_rn(Y, __dmul_rn(Cr, 1.402)));
                    res[1] = __double2float_rn(
                        __dadd_rn(__dadd_rn(Y, __dmul_rn(Cb, -0.344136)), __dmul_rn(Cr, -0.714136)));
                    res[2] = __double2float_rn(__dadd_rn(Y, __dmul_rn(Cb, 1.772)));
                }
                if (!in[i][j]) continue;
#pragma unroll
                for (int ch = 0; ch < 3; ++ch)
                    row[x * 3 + ch] = fminf(fmaxf(__fadd_rn(px[i][j][ch], res[ch]), 0.0f), 1.0f);
            }
        }
    }
}

__global__ void clip01_kernel(float* __restrict__ image, long long n) {
    const long long at = blockIdx.x * (long long)blockDim.x + threadIdx.x, all = (long long)gridDim.x * blockDim.x;
    const long long n4 = ((uintptr_t)image & 15u) == 0 ? n / 4 : 0;  // four at a time where the image allows it
    auto clip = [](float v) { return fminf(fmaxf(v, 0.0f), 1.0f); };
    float4* image4 = reinterpret_cast<float4*>(image);
    for (long long i = at; i < n4; i += all) {
        const float4 v = image4[i];
        image4[i] = make_float4(clip(v.x), clip(v.y), clip(v.z), clip(v.w));
    }
    for (long long i = 4 * n4 + at; i < n; i += all) image[i] = clip(image[i]);
}

// ---------------------------------------------------------------------------------- resize
constexpr int kResampleBits = 22;

__device__ __forceinline__ double triangle(double d) {
    if (d < 0.0) d = -d;
    return d < 1.0 ? __dsub_rn(1.0, d) : 0.0;
}

// Taps of output sample o of an in_size -> out_size BILINEAR resample (Pillow precompute_coeffs).
struct Taps {
    int first, count;
    double center, inv_fs, ww;
};

__device__ __forceinline__ Taps resample_taps(int in_size, int out_size, int o) {
    Taps t;
    const double scale = __ddiv_rn((double)in_size, (double)out_size);
    const double fs = scale < 1.0 ? 1.0 : scale;
    const double support = fs;  // triangle support 1.0 x filter scale
    t.center = __dmul_rn(__dadd_rn((double)o, 0.5), scale);
    t.inv_fs = __ddiv_rn(1.0, fs);
    int lo = (int)__dadd_rn(__dsub_rn(t.center, support), 0.5);
    if (lo < 0) lo = 0;
    int hi = (int)__dadd_rn(__dadd_rn(t.center, support), 0.5);
    if (hi > in_size) hi = in_size;
    t.first = lo;
    t.count = hi - lo;
    double ww = 0.0;
    for (int x = 0; x < t.count; ++x)
        ww = __dadd_rn(ww, triangle(__dmul_rn(__dadd_rn(__dsub_rn((double)(x + lo), t.center), 0.5), t.inv_fs)));
    t.ww = ww;
    return t;
}

__device__ __forceinline__ int tap_weight(const Taps& t, int x) {
    double w = triangle(__dmul_rn(__dadd_rn(__dsub_rn((double)(x + t.first), t.center), 0.5), t.inv_fs));
    if (t.ww != 0.0) w = __ddiv_rn(w, t.ww);
    const double s = __dmul_rn(w, (double)(1 << kResampleBits));
    return w < 0.0 ? (int)__dadd_rn(-0.5, s) : (int)__dadd_rn(0.5, s);
}

__device__ __forceinline__ int clip8(int acc) {
    const int v = acc >> kResampleBits;
    return v < 0 ? 0 : (v > 255 ? 255 : v);
}

__device__ __forceinline__ int to_u8(float v) {
    const float p = fminf(fmaxf(__fmul_rn(v, 255.0f), 0.0f), 255.0f);
    return (int)p;  // truncation, as numpy's astype(uint8)
}

// The two-kernel form: a CTA covers RS_COLS output columns x RS_ROWS rows.  A sample's taps (Pillow's
// bounds and 22-bit integer weights) depend on its output column (row pass) or output row (column
// pass) only, so they are derived once per CTA column or row and reused, not once per pixel; a
// sample with more than RS_MAXT taps (a downscale by more than about 3.5) derives each weight where
// it is used.  The weights are the same integers either way.
constexpr int RS_COLS = 128, RS_ROWS = 8, RS_MAXT = 8;

__global__ void __launch_bounds__(RS_COLS) resize_rows_kernel(const float* __restrict__ src, int src_w, int src_h,
                                                              uint8_t* __restrict__ tmp, int dst_w) {
    const int xx = blockIdx.x * RS_COLS + threadIdx.x;
    const int y0 = blockIdx.y * RS_ROWS;
    if (xx >= dst_w) return;
    const Taps t = resample_taps(src_w, dst_w, xx);
    const bool cached = t.count <= RS_MAXT;
    int k[RS_MAXT], sx[RS_MAXT];
#pragma unroll
    for (int j = 0; j < RS_MAXT; ++j) {
        k[j] = cached && j < t.count ? tap_weight(t, j) : 0;
        sx[j] = min(t.first + j, src_w - 1);
    }
    for (int r = 0; r < RS_ROWS; ++r) {
        const int y = y0 + r;
        if (y >= src_h) break;
        int a0 = 1 << (kResampleBits - 1), a1 = a0, a2 = a0;
        const float* row = src + (long long)y * src_w * 3;
        if (cached) {
#pragma unroll
            for (int j = 0; j < RS_MAXT; ++j) {
                if (j < t.count) {
                    const float* q = row + sx[j] * 3;
                    a0 += to_u8(q[0]) * k[j];
                    a1 += to_u8(q[1]) * k[j];
                    a2 += to_u8(q[2]) * k[j];
                }
            }
        } else {
            for (int x = 0; x < t.count; ++x) {
                const int s = min(t.first + x, src_w - 1);
                const int w = tap_weight(t, x);
                a0 += to_u8(row[s * 3 + 0]) * w;
                a1 += to_u8(row[s * 3 + 1]) * w;
                a2 += to_u8(row[s * 3 + 2]) * w;
            }
        }
        uint8_t* o = tmp + ((long long)y * dst_w + xx) * 3;
        o[0] = (uint8_t)clip8(a0);
        o[1] = (uint8_t)clip8(a1);
        o[2] = (uint8_t)clip8(a2);
    }
}

__global__ void __launch_bounds__(RS_COLS) resize_cols_kernel(const uint8_t* __restrict__ tmp, int src_h, int dst_w,
                                                              float* __restrict__ dst, int dst_h) {
    __shared__ int s_first[RS_ROWS], s_count[RS_ROWS], s_k[RS_ROWS][RS_MAXT];
    __shared__ Taps s_taps[RS_ROWS];
    const int xx = blockIdx.x * RS_COLS + threadIdx.x;
    const int y0 = blockIdx.y * RS_ROWS;
    // the CTA's output rows' taps, once
    if (threadIdx.x < RS_ROWS && y0 + (int)threadIdx.x < dst_h) {
        const int r = threadIdx.x;
        const Taps t = resample_taps(src_h, dst_h, y0 + r);
        s_taps[r] = t;
        s_first[r] = t.first;
        s_count[r] = t.count;
        for (int j = 0; j < RS_MAXT; ++j) s_k[r][j] = t.count <= RS_MAXT && j < t.count ? tap_weight(t, j) : 0;
    }
    __syncthreads();
    if (xx >= dst_w) return;
    for (int r = 0; r < RS_ROWS; ++r) {
        const int yy = y0 + r;
        if (yy >= dst_h) break;
        const int first = s_first[r], count = s_count[r];
        int a0 = 1 << (kResampleBits - 1), a1 = a0, a2 = a0;
        for (int y = 0; y < count; ++y) {
            const int sy = min(first + y, src_h - 1);
            const int k = count <= RS_MAXT ? s_k[r][y] : tap_weight(s_taps[r], y);
            const uint8_t* p = tmp + ((long long)sy * dst_w + xx) * 3;
            a0 += (int)p[0] * k;
            a1 += (int)p[1] * k;
            a2 += (int)p[2] * k;
        }
        float* o = dst + ((long long)yy * dst_w + xx) * 3;
        o[0] = __fdiv_rn((float)clip8(a0), 255.0f);
        o[1] = __fdiv_rn((float)clip8(a1), 255.0f);
        o[2] = __fdiv_rn((float)clip8(a2), 255.0f);
    }
}

// Both passes in one CTA of FR_COLS output columns x `ry` output rows: the source window is converted to
// bytes in shared memory once, the row pass's bytes stay there (a CTA's rows of them), and only the result
// is written.  Same integers as the two kernels above, which stay for downscales whose window is too large.
constexpr int FR_COLS = 128, FR_THREADS = 256, FR_ROW = FR_COLS * 3;
constexpr size_t FR_SMEM = 100 * 1024;

struct FusedResize {
    int ry, tx, ty;   // output rows of a CTA, most taps of a column, of a row
    int sw, sh;       // most source columns and rows of a CTA
    __host__ __device__ int src_pitch() const { return (sw * 3 + 3) & ~3; }
    __host__ __device__ size_t smem() const {
        return (size_t)(tx * FR_COLS + FR_COLS + ry * ty + 2 * ry) * 4 + (size_t)sh * (src_pitch() + FR_ROW);
    }
};

// v / 255 of a byte: 1 / 255 in two floats (the product of the low part corrects the last bit)
__device__ __forceinline__ float unit_of_byte(int v) {
    constexpr float hi = (float)(1.0 / 255.0), lo = (float)(1.0 / 255.0 - (double)hi);
    const float f = (float)v;
    return __fmaf_rn(f, hi, __fmul_rn(f, lo));
}

template <bool VEC>
__global__ void __launch_bounds__(FR_THREADS) resize_fused_kernel(const float* __restrict__ src, int src_w, int src_h,
                                                                  float* __restrict__ dst, int dst_w, int dst_h,
                                                                  FusedResize F) {
    extern __shared__ __align__(16) int rs_smem[];
    int* kx = rs_smem;                   // [tx][FR_COLS]
    int* fx = kx + F.tx * FR_COLS;       // first source column | taps << 16, relative to the window
    int* ky = fx + FR_COLS;              // [ry][ty]
    int* fy = ky + F.ry * F.ty;
    int* cy = fy + F.ry;
    uint8_t* h8 = reinterpret_cast<uint8_t*>(cy + F.ry);  // [sh][FR_ROW]
    uint8_t* s8 = h8 + F.sh * FR_ROW;                     // [sh][src_pitch]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = FR_THREADS / 32;
    const int x0 = blockIdx.x * FR_COLS, y0 = blockIdx.y * F.ry;
    const int cols = min(FR_COLS, dst_w - x0), rows = min(F.ry, dst_h - y0);
    const int sx0 = resample_taps(src_w, dst_w, x0).first, sy0 = resample_taps(src_h, dst_h, y0).first;
    if (tid < cols) {
        const Taps t = resample_taps(src_w, dst_w, x0 + tid);
        const int count = min(t.count, F.tx);
        fx[tid] = (t.first - sx0) | (count << 16);
        for (int j = 0; j < count; ++j) kx[j * FR_COLS + tid] = tap_weight(t, j);
    } else if (tid >= FR_COLS && tid - FR_COLS < rows) {
        const int r = tid - FR_COLS;
        const Taps t = resample_taps(src_h, dst_h, y0 + r);
        fy[r] = t.first - sy0;
        cy[r] = min(t.count, F.ty);
        for (int j = 0; j < cy[r]; ++j) ky[r * F.ty + j] = tap_weight(t, j);
    }
    __syncthreads();
    const int sw = min(F.sw, (fx[cols - 1] & 0xffff) + (fx[cols - 1] >> 16)), sh = min(F.sh, fy[rows - 1] + cy[rows - 1]);
    const int pitch = F.src_pitch();
    for (int r = warp; r < sh; r += NW) {
        const float* row = src + ((long long)min(sy0 + r, src_h - 1) * src_w + sx0) * 3;
        for (int i = lane; i < sw * 3; i += 32)
            s8[r * pitch + i] = (uint8_t)(sx0 * 3 + i < src_w * 3 ? to_u8(row[i]) : 0);
    }
    __syncthreads();
    // row pass: a thread per column, every other source row
    {
        const int col = tid & (FR_COLS - 1);
        if (col < cols) {
            const int first = (fx[col] & 0xffff) * 3, count = fx[col] >> 16;
            int k[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) k[j] = j < count ? kx[j * FR_COLS + col] : 0;
            for (int r = tid / FR_COLS; r < sh; r += FR_THREADS / FR_COLS) {
                int a0 = 1 << (kResampleBits - 1), a1 = a0, a2 = a0;
                const uint8_t* q = s8 + r * pitch + first;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < count) {
                        a0 += (int)q[j * 3] * k[j];
                        a1 += (int)q[j * 3 + 1] * k[j];
                        a2 += (int)q[j * 3 + 2] * k[j];
                    }
                for (int j = 4; j < count; ++j) {
                    const int w = kx[j * FR_COLS + col];
                    a0 += (int)q[j * 3] * w;
                    a1 += (int)q[j * 3 + 1] * w;
                    a2 += (int)q[j * 3 + 2] * w;
                }
                uint8_t* o = h8 + r * FR_ROW + col * 3;
                o[0] = (uint8_t)clip8(a0);
                o[1] = (uint8_t)clip8(a1);
                o[2] = (uint8_t)clip8(a2);
            }
        }
    }
    __syncthreads();
    // column pass: a warp per output row, four neighbouring bytes (VEC) or every 32nd byte per lane
    for (int r = warp; r < rows; r += NW) {
        const int first = fy[r], count = cy[r];
        const int* k = ky + r * F.ty;
        float* out = dst + ((long long)(y0 + r) * dst_w + x0) * 3;
        if constexpr (VEC) {
            int a[3][4];
#pragma unroll
            for (int w = 0; w < 3; ++w)
#pragma unroll
                for (int b = 0; b < 4; ++b) a[w][b] = 1 << (kResampleBits - 1);
            for (int y = 0; y < count; ++y) {
                const unsigned* p = reinterpret_cast<const unsigned*>(h8 + (first + y) * FR_ROW);
                const int ky1 = k[y];
#pragma unroll
                for (int w = 0; w < 3; ++w) {
                    const unsigned v = p[lane + 32 * w];
#pragma unroll
                    for (int b = 0; b < 4; ++b) a[w][b] += (int)((v >> (8 * b)) & 255u) * ky1;
                }
            }
#pragma unroll
            for (int w = 0; w < 3; ++w)
                if ((lane + 32 * w) * 4 < cols * 3)
                    reinterpret_cast<float4*>(out)[lane + 32 * w] =
                        make_float4(unit_of_byte(clip8(a[w][0])), unit_of_byte(clip8(a[w][1])),
                                    unit_of_byte(clip8(a[w][2])), unit_of_byte(clip8(a[w][3])));
        } else {
            for (int i = lane; i < cols * 3; i += 32) {
                int a = 1 << (kResampleBits - 1);
                for (int y = 0; y < count; ++y) a += (int)h8[(first + y) * FR_ROW + i] * k[y];
                out[i] = unit_of_byte(clip8(a));
            }
        }
    }
}

namespace {
std::mutex g_tab_mu;
bool g_tab_ready[64] = {};

int ensure_tables(cudaStream_t stream) {
    int dev = 0;
    WEFTK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(WEFTK_E_RANGE, "dct: device index beyond 63");
    std::lock_guard<std::mutex> lock(g_tab_mu);
    if (!g_tab_ready[dev]) {
        dct_tables_kernel<<<ceil_div(kDctTab, 256), 256, 0, stream>>>();
        WEFTK_CUDA(cudaGetLastError());
        WEFTK_CUDA(cudaStreamSynchronize(stream));  // later calls may come on other streams
        g_tab_ready[dev] = true;
    }
    return WEFTK_OK;
}

int grid_for(long long total) {
    const long long blocks = (total + 255) / 256;
    return (int)(blocks < 148LL * 64 ? (blocks > 0 ? blocks : 1) : 148LL * 64);
}
}  // namespace

}  // namespace weftk

using namespace weftk;

extern "C" int weftk_dct_apply(const WeftDctTile* d_tiles, int n_tiles, const int16_t* d_coeffs, int64_t n_coeffs,
                               int chroma_mode, int band_layout, float quant_step, float freq_alpha, int max_size,
                               float* d_image, int width, int height, int clip_all, void* stream) {
    static_assert(sizeof(WeftDctTile) == 64, "WeftDctTile must be 64 bytes");
    WEFTK_REQUIRE(n_tiles >= 0 && n_coeffs >= 0, "dct_apply: negative count");
    WEFTK_REQUIRE(chroma_mode >= 0 && chroma_mode <= 2, "dct_apply: chroma_mode must be 0, 1 or 2");
    const bool follows = (band_layout & WEFTK_DCT_FOLLOWS) != 0;
    band_layout &= ~WEFTK_DCT_FOLLOWS;
    WEFTK_REQUIRE(band_layout == 0 || band_layout == 1, "dct_apply: layout must be 0 or 1");
    WEFTK_REQUIRE(width > 0 && height > 0 && d_image, "dct_apply: bad image");
    WEFTK_REQUIRE(max_size >= 4 && max_size <= WEFTK_DCT_MAX_TILE && (max_size & (max_size - 1)) == 0,
                  "dct_apply: max_size must be a power of two in 4..64");
    WEFTK_REQUIRE(!(freq_alpha < 0.0f), "dct_apply: freq_alpha must be >= 0");
    cudaStream_t s = (cudaStream_t)stream;
    if (n_tiles > 0) {
        WEFTK_REQUIRE(d_tiles && (d_coeffs || n_coeffs == 0), "dct_apply: null pointer");
        int rc = ensure_tables(s);
        if (rc != WEFTK_OK) return rc;
        auto kernel = chroma_mode == 2 ? dct_layer_kernel<true> : dct_layer_kernel<false>;
        WEFTK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDctSmem));
        const double step = (double)quant_step;
        int log_side = 2;
        while ((1 << log_side) < max_size) ++log_side;
        const DctLayer L = {d_tiles, n_tiles, log_side, d_coeffs, (long long)n_coeffs, chroma_mode, band_layout,
                            step, step * 1.5, (double)freq_alpha, d_image, width, height};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ceil_div(n_tiles, DC_PIXELS / (max_size * max_size)));
        cfg.blockDim = dim3(DC_THREADS);
        cfg.dynamicSmemBytes = kDctSmem;
        cfg.stream = s;
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        // without the flag an ordinary launch: it reads its inputs before griddepcontrol.wait, so whatever
        // wrote them on the stream has to be complete when it starts
        cfg.attrs = &attr;
        cfg.numAttrs = follows ? 1 : 0;
        WEFTK_CUDA(cudaLaunchKernelEx(&cfg, kernel, L));
    }
    if (clip_all) {
        const long long n = (long long)width * height * 3;
        clip01_kernel<<<grid_for((n + 3) / 4), 256, 0, s>>>(d_image, n);
        WEFTK_CUDA(cudaGetLastError());
    }
    return WEFTK_OK;
}

extern "C" int weftk_raster_resize(const float* d_src, int src_w, int src_h, float* d_dst, int dst_w, int dst_h,
                                   uint8_t* d_tmp, void* stream) {
    WEFTK_REQUIRE(d_src && d_dst && d_tmp, "raster_resize: null pointer");
    WEFTK_REQUIRE(src_w > 0 && src_h > 0 && dst_w > 0 && dst_h > 0 && src_w <= 65535 && src_h <= 65535 &&
                      dst_w <= 65535 && dst_h <= 65535,
                  "raster_resize: sizes must be in 1..65535");
    cudaStream_t s = (cudaStream_t)stream;
    {
        const double scale_x = (double)src_w / (double)dst_w, scale_y = (double)src_h / (double)dst_h;
        const double fsx = std::max(scale_x, 1.0), fsy = std::max(scale_y, 1.0);
        FusedResize F;
        F.tx = std::min(src_w, (int)(2.0 * fsx) + 2);
        F.ty = std::min(src_h, (int)(2.0 * fsy) + 2);
        F.sw = std::min(src_w, (int)((FR_COLS - 1) * scale_x + 2.0 * fsx) + 3);
        // 64 output rows, or 32 where their window is too large.  Fewer lose to the two kernels, since the
        // source rows that two CTAs both filter grow against those they keep: 2048^2 to 1024^2 takes 29 us
        // (32 rows) and 40 in two kernels, 3000^2 to 1000^2 would take 98 (16 rows) and takes 84,
        // 4096^2 to 1024^2 172 (8 rows) and 113
        for (F.ry = 64; F.ry >= 32; F.ry >>= 1) {
            F.sh = std::min(src_h, (int)((F.ry - 1) * scale_y + 2.0 * fsy) + 3);
            if (F.smem() <= FR_SMEM) break;
        }
        if (F.ry >= 32 && ceil_div(dst_h, F.ry) <= 65535) {
            const dim3 grid(ceil_div(dst_w, FR_COLS), ceil_div(dst_h, F.ry));
            const bool vec = dst_w % 4 == 0 && ((uintptr_t)d_dst & 15u) == 0;
            auto kernel = vec ? resize_fused_kernel<true> : resize_fused_kernel<false>;
            WEFTK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FR_SMEM));
            kernel<<<grid, FR_THREADS, F.smem(), s>>>(d_src, src_w, src_h, d_dst, dst_w, dst_h, F);
            WEFTK_CUDA(cudaGetLastError());
            return WEFTK_OK;
        }
    }
    const dim3 grid_r(ceil_div(dst_w, RS_COLS), ceil_div(src_h, RS_ROWS));
    const dim3 grid_c(ceil_div(dst_w, RS_COLS), ceil_div(dst_h, RS_ROWS));
    WEFTK_REQUIRE(grid_r.y <= 65535 && grid_c.y <= 65535, "raster_resize: image too tall");
    resize_rows_kernel<<<grid_r, RS_COLS, 0, s>>>(d_src, src_w, src_h, d_tmp, dst_w);
    WEFTK_CUDA(cudaGetLastError());
    resize_cols_kernel<<<grid_c, RS_COLS, 0, s>>>(d_tmp, src_h, dst_w, d_dst, dst_h);
    WEFTK_CUDA(cudaGetLastError());
    return WEFTK_OK;
}
