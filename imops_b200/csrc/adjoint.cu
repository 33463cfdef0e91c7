// adjoint.cu -- hand-written adjoints of the colour + film stages for
// parameter fitting (the reference has no gradients; this is new).
//
// Differentiable forward per pixel, from demosaiced camera RGB x (demosaic is
// upstream of every parameter, so its decisions are simply held fixed):
//   y   = 2^ev * (wb (.) x)                     WB + exposure
//   a   = C y                                   camera -> ACEScg matrix (9)
//   w   = max(0, Minv a);  e_l = sum_k w_k A[k][l]     spectral exposure
//   h   = max(0, a_R - thr);  B = G_sigma * h   halation (fixed tap radius)
//   E_l = e_l + s bleed_l B
//   D_l = Dmax_l / (1 + exp(-k_l (log10 max(E_l,1e-6) - x0_l)))
//   T(l)= 2^(-sum_l D_l eps'_l(lambda));  out_c = sum_lambda Cscan[lambda][c] T
// with the baseline preset's tables (film_host.cpp), grain off.
//
// Backward: a per-pixel kernel recomputes the forward, takes the upstream
// gradient (or 2/N (out - target) for an MSE loss), and produces the curve,
// halation-strength and colour partials and the gradient w.r.t. B (a plane).
// The halation blur is recomputed instead of stored; the gradient of its sigma
// comes from inner products with blurs by derivative taps, and the gradient
// w.r.t. h is the exact transpose of the mirror-reflect blur.  Parameter
// partials are summed per block in f64 and reduced by one block in a fixed
// order (deterministic).
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "blur.cuh"
#include "film.cuh"

namespace imops {
namespace adj {

using film::HAL_R;
using film::NB81;

constexpr int NPAR = 24;  // wb3 C9 ev1 dmax3 k3 x03 s1 sigma1
constexpr int BLK = 256;

constexpr int NP = NB81 / 2;  // 40 bin pairs + bin 80

struct Const {
    float wb[3], C[9], ev2, ev;
    float dmax[3], k[3], x0[3], s, thr;
    float minv[9];
    float A[3][3];
    float bleed[3];
    // the forward's tables as pairs of bins (2l, 2l+1) for the packed f32x2
    // FMA, bin 80 alone: ne2 = -eps (the sum is -d), Cs2 per channel
    float2 ne2[3][NP];
    float2 Cs2[3][NP];
    float ne_l[3], Cs_l[3];
};

// The backward's products Q[l][e][c] = -ln2 eps[e] Cs[c] of bin pair l: dL/dD_e
// = sum_c go_c sum_l Q[l][e][c] T_l, so the backward needs only the forward's
// T_l, weighted before go is known.
struct BackTable {
    float2 Q[NP][3][3];
    float Q_l[3][3];  // bin 80
};

__device__ __forceinline__ void color_fwd(const Const& c, const float* x, float y[3], float a[3]) {
    for (int i = 0; i < 3; i++) y[i] = c.ev2 * (c.wb[i] * x[i]);
    for (int i = 0; i < 3; i++) a[i] = c.C[3 * i] * y[0] + c.C[3 * i + 1] * y[1] + c.C[3 * i + 2] * y[2];
}

__global__ void prep_kernel(const float* __restrict__ x, size_t n, const __grid_constant__ Const c,
                            float* __restrict__ h) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float y[3], a[3];
        color_fwd(c, x + 3 * p, y, a);
        h[p] = fmaxf(0.0f, a[0] - c.thr);
    }
}

// Sums over a block: each thread's N f32 sums go through a warp reduction in
// f64 to red (flush, which clears them; a thread with many terms calls it now
// and then, so that no f32 sum grows long), and the warps' sums, added in a
// fixed order, to partial[i * blocks + block] (one row a sum, so the last
// reduction reads rows).
template <int N, int THREADS>
__device__ __forceinline__ void flush(float (&acc)[N], double (&red)[N][THREADS / 32], bool first) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; i++) {
        double v = (double)acc[i];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[i][wid] = first ? v : red[i][wid] + v;
        acc[i] = 0.0f;
    }
}
template <int N, int THREADS>
__device__ __forceinline__ void store_partials(const double (&red)[N][THREADS / 32], double* __restrict__ partial) {
    __syncthreads();
    if (threadIdx.x < N) {
        double v = 0.0;
        for (int k = 0; k < THREADS / 32; k++) v += red[threadIdx.x][k];
        partial[(size_t)threadIdx.x * (gridDim.x * gridDim.y) + blockIdx.y * gridDim.x + blockIdx.x] = v;
    }
}
template <int N, int THREADS = BLK>
__device__ __forceinline__ void block_partials(float (&acc)[N], double* __restrict__ partial) {
    __shared__ double red[N][THREADS / 32];
    flush<N, THREADS>(acc, red, true);
    store_partials<N, THREADS>(red, partial);
}

// Layer exposures, log10 exposures, curve values and densities of a pixel.
struct Curve {
    float w[3], E[3], le[3], sg[3], D[3];
};
__device__ __forceinline__ Curve curve_px(const Const& c, const float (&a)[3], float b) {
    Curve v;
#pragma unroll
    for (int k = 0; k < 3; k++)
        v.w[k] = c.minv[3 * k] * a[0] + c.minv[3 * k + 1] * a[1] + c.minv[3 * k + 2] * a[2];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        float e = fmaxf(v.w[0], 0.0f) * c.A[0][l] + fmaxf(v.w[1], 0.0f) * c.A[1][l] + fmaxf(v.w[2], 0.0f) * c.A[2][l];
        v.E[l] = e + c.s * c.bleed[l] * b;
        v.le[l] = log10f(fmaxf(v.E[l], 1e-6f));
        v.sg[l] = 1.0f / (1.0f + expf(-c.k[l] * (v.le[l] - c.x0[l])));
        v.D[l] = c.dmax[l] * v.sg[l];
    }
    return v;
}

// Per-pixel forward: film RGB.  The next pixel's inputs are loaded while this
// one is scanned, so the global-load latency hides behind the 81-bin loop;
// bound by the MUFU (90 operations a pixel).
__global__ void __launch_bounds__(BLK) pixel_forward_kernel(const float* __restrict__ x, const float* __restrict__ B,
                                                            size_t n, const __grid_constant__ Const c,
                                                            float* __restrict__ out) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    float nx[3] = {0.f, 0.f, 0.f}, nb = 0.f;
    size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p < n) {
        nx[0] = x[3 * p];
        nx[1] = x[3 * p + 1];
        nx[2] = x[3 * p + 2];
        nb = B[p];
    }
    for (; p < n; p += stride) {
        const float xp[3] = {nx[0], nx[1], nx[2]};
        const float b = nb;
        if (p + stride < n) {
            nx[0] = x[3 * (p + stride)];
            nx[1] = x[3 * (p + stride) + 1];
            nx[2] = x[3 * (p + stride) + 2];
            nb = B[p + stride];
        }
        float y[3], a[3];
        color_fwd(c, xp, y, a);
        const Curve v = curve_px(c, a, b);
        // bins in pairs on the packed f32x2 FMA
        const float2 d0 = make_float2(v.D[0], v.D[0]), d1 = make_float2(v.D[1], v.D[1]),
                     d2 = make_float2(v.D[2], v.D[2]);
        float2 oo[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int l = 0; l < NP; l++) {
            float2 xd = __fmul2_rn(d0, c.ne2[0][l]);
            xd = __ffma2_rn(d1, c.ne2[1][l], xd);
            xd = __ffma2_rn(d2, c.ne2[2][l], xd);
            const float2 t = make_float2(film::ex2_fast(xd.x), film::ex2_fast(xd.y));
#pragma unroll
            for (int j = 0; j < 3; j++) oo[j] = __ffma2_rn(c.Cs2[j][l], t, oo[j]);
        }
        float xl = v.D[0] * c.ne_l[0];
        xl = fmaf(v.D[1], c.ne_l[1], xl);
        xl = fmaf(v.D[2], c.ne_l[2], xl);
        const float tl = film::ex2_fast(xl);
#pragma unroll
        for (int j = 0; j < 3; j++) out[3 * p + j] = fmaf(c.Cs_l[j], tl, oo[j].x + oo[j].y);
    }
}

// Per-pixel backward with g_out or target: writes gB (plane) and the block
// partials of dmax (0..2), k (3..5), x0 (6..8), s (9), the loss (10) and
// S[i][j] = sum over the pixels of ga_i x_j (11 + 3 i + j), ga the gradient of
// the ACEScg pixel but for its halation path: the gradients of the matrix, the
// white balance and the exposure are all combinations of S (finish_kernel), so
// ga needs no planes and the colour step no pass of its own.
//
// The scan takes 15 multiply-adds a bin, two bins a packed FMA, and 4.8 KB of
// tables a pixel: warps that read them at different places evict one another's
// constants, so one block of 20 warps an SM steps through the pixels together
// (24 MP, the barrier kept: 1.26 ms; two blocks of 8 warps 1.30, four of 4
// 1.43).  Bound by the FMA pipe (0.97 ms with the curves; busy 0.76 of the time).  One bin an FMA,
// bound by issue: 1.42 ms.  18 multiply-adds from the six forward tables alone
// (1.9 KB): 1.30 ms.
constexpr int NP1 = 20;
constexpr int PB_THREADS = 640, PB_BLOCKS = 1;
__global__ void __launch_bounds__(PB_THREADS, PB_BLOCKS) pixel_backward_kernel(
    const float* __restrict__ x, const float* __restrict__ B, const float* __restrict__ g_out,
    const float* __restrict__ target, float loss_scale, size_t n, const __grid_constant__ Const c,
    const __grid_constant__ BackTable bt, float* __restrict__ gB, double* __restrict__ partial) {
    __shared__ double red[NP1][PB_THREADS / 32];
    float acc[NP1];
#pragma unroll
    for (int i = 0; i < NP1; i++) acc[i] = 0.0f;
    int terms = 0;
    bool first_flush = true;
    const size_t stride = (size_t)gridDim.x * PB_THREADS;
    const float* gsrc = g_out ? g_out : target;
    // the next pixel's inputs are loaded while this one is scanned, so the
    // global-load latency hides behind the 81-bin loop
    float nx[3] = {0.f, 0.f, 0.f}, nb = 0.f;
    // pixels past the end are the last one with no upstream gradient
    const size_t first = blockIdx.x * (size_t)PB_THREADS;
    auto fetch = [&](size_t q) {
        q = min(q + threadIdx.x, n - 1);
#pragma unroll
        for (int k = 0; k < 3; k++) nx[k] = __ldg(x + 3 * q + k);
        nb = __ldg(B + q);
    };
    fetch(first);
    for (size_t base = first; base < n; base += stride) {
        __syncthreads();
        const bool in = base + threadIdx.x < n;
        const size_t p = min(base + threadIdx.x, n - 1);
        const float xp[3] = {nx[0], nx[1], nx[2]}, b = nb;
        // the upstream inputs, loaded before the scan that hides their latency
        const float gin[3] = {__ldg(gsrc + 3 * p), __ldg(gsrc + 3 * p + 1), __ldg(gsrc + 3 * p + 2)};
        fetch(base + stride);
        float y[3], a[3];
        color_fwd(c, xp, y, a);
        const Curve v = curve_px(c, a, b);
        float2 D[3], o[3], M[3][3];
#pragma unroll
        for (int e = 0; e < 3; e++) {
            D[e] = make_float2(v.D[e], v.D[e]);
            o[e] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int j = 0; j < 3; j++) M[e][j] = make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int l = 0; l < NP; l++) {
            float2 xd = __fmul2_rn(D[0], c.ne2[0][l]);
            xd = __ffma2_rn(D[1], c.ne2[1][l], xd);
            xd = __ffma2_rn(D[2], c.ne2[2][l], xd);
            const float2 t = make_float2(film::ex2_fast(xd.x), film::ex2_fast(xd.y));
#pragma unroll
            for (int j = 0; j < 3; j++) o[j] = __ffma2_rn(c.Cs2[j][l], t, o[j]);
#pragma unroll
            for (int e = 0; e < 3; e++) {
#pragma unroll
                for (int j = 0; j < 3; j++) M[e][j] = __ffma2_rn(bt.Q[l][e][j], t, M[e][j]);
            }
        }
        // the last bin, and the pairs' halves
        float xl = v.D[0] * c.ne_l[0];
        xl = fmaf(v.D[1], c.ne_l[1], xl);
        xl = fmaf(v.D[2], c.ne_l[2], xl);
        const float tl = film::ex2_fast(xl);
        float go[3];
        if (g_out) {
#pragma unroll
            for (int j = 0; j < 3; j++) go[j] = in ? gin[j] : 0.0f;
        } else {
            float r[3];
#pragma unroll
            for (int j = 0; j < 3; j++) r[j] = in ? fmaf(c.Cs_l[j], tl, o[j].x + o[j].y) - gin[j] : 0.0f;
            acc[10] += loss_scale * (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
#pragma unroll
            for (int j = 0; j < 3; j++) go[j] = 2.0f * loss_scale * r[j];
        }
        float gE[3];
#pragma unroll
        for (int l = 0; l < 3; l++) {
            float gD = 0.0f;
#pragma unroll
            for (int j = 0; j < 3; j++) gD = fmaf(fmaf(bt.Q_l[l][j], tl, M[l][j].x + M[l][j].y), go[j], gD);
            const float sg = v.sg[l], ds = sg * (1.0f - sg);
            acc[l] += gD * sg;
            acc[3 + l] += gD * c.dmax[l] * ds * (v.le[l] - c.x0[l]);
            acc[6 + l] += -gD * c.dmax[l] * ds * c.k[l];
            gE[l] = v.E[l] > 1e-6f ? gD * c.dmax[l] * ds * c.k[l] / (v.E[l] * 2.302585092994046f) : 0.0f;
        }
        const float gbl = c.bleed[0] * gE[0] + c.bleed[1] * gE[1] + c.bleed[2] * gE[2];
        acc[9] += gbl * b;
        if (in) gB[p] = c.s * gbl;
        float gw[3];
#pragma unroll
        for (int k = 0; k < 3; k++)
            gw[k] = v.w[k] > 0.0f ? c.A[k][0] * gE[0] + c.A[k][1] * gE[1] + c.A[k][2] * gE[2] : 0.0f;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float ga = c.minv[i] * gw[0] + c.minv[3 + i] * gw[1] + c.minv[6 + i] * gw[2];
#pragma unroll
            for (int j = 0; j < 3; j++) acc[11 + 3 * i + j] = fmaf(ga, xp[j], acc[11 + 3 * i + j]);
        }
        if (++terms == 64) {
            flush<NP1, PB_THREADS>(acc, red, first_flush);
            first_flush = false;
            terms = 0;
        }
    }
    flush<NP1, PB_THREADS>(acc, red, first_flush);
    store_partials<NP1, PB_THREADS>(red, partial);
}

// The halation path's part of S: sum of gh x_j over the pixels whose red is
// above the threshold (gh a plane; the radius-64 row pass does this itself).
constexpr int NPH = 3;
__global__ void __launch_bounds__(BLK) color_back_kernel(const float* __restrict__ x, const float* __restrict__ gh,
                                                         size_t n, const __grid_constant__ Const c,
                                                         double* __restrict__ partial) {
    float acc[NPH] = {0.0f, 0.0f, 0.0f};
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float y[3], a[3];
        const float* xp = x + 3 * p;
        color_fwd(c, xp, y, a);
        if (a[0] - c.thr > 0.0f)
            for (int j = 0; j < 3; j++) acc[j] = fmaf(gh[p], xp[j], acc[j]);
    }
    block_partials(acc, partial);
}

// The colour parameters, for the gradients from S.
struct ColorParams {
    double ev2, wb[3], C[9];
};

// One block, a warp a sum: the lanes add every 32nd partial, FIN_LOADS of them
// in flight (a row of 2368: 5.9 us; eight in flight 7.6), the warp their sums
// (fixed order).  Then a thread a parameter adds its gradient into
// grad[25] (24 parameters + loss) in the order of ImopsFilmGradParams.  With
// S_ij = sum ga_i x_j and a_i = sum_j C_ij ev2 wb_j x_j:
//   dC_ij = ev2 wb_j S_ij, dwb_j = ev2 sum_i C_ij S_ij, dev = ln2 sum_j wb_j dwb_j.
constexpr int FIN_SUMS = NP1 + NPH + 1, FIN_LOADS = 32;
__global__ void __launch_bounds__(32 * FIN_SUMS) finish_kernel(const double* __restrict__ p1, int nb1,
                                                               const double* __restrict__ ph, int nbh,
                                                               const double* __restrict__ ps, int nbs,
                                                               const __grid_constant__ ColorParams c,
                                                               double* __restrict__ grad) {
    __shared__ double sum[FIN_SUMS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* src = ps;
    int n = nbs;
    if (w < NP1) {
        src = p1 + (size_t)w * nb1;
        n = nb1;
    } else if (w < NP1 + NPH) {
        src = ph + (size_t)(w - NP1) * nbh;
        n = nbh;
    }
    double v = 0.0;
    for (int i = lane; i < n; i += 32 * FIN_LOADS) {
        double u[FIN_LOADS];
#pragma unroll
        for (int k = 0; k < FIN_LOADS; k++) u[k] = i + 32 * k < n ? src[i + 32 * k] : 0.0;
#pragma unroll
        for (int k = 0; k < FIN_LOADS; k++) v += u[k];
    }
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sum[w] = v;
    __syncthreads();
    const int t = threadIdx.x;
    auto S = [&](int i, int j) { return sum[11 + 3 * i + j] + (i == 0 ? sum[NP1 + j] : 0.0); };
    auto dwb = [&](int j) { return c.ev2 * (c.C[j] * S(0, j) + c.C[3 + j] * S(1, j) + c.C[6 + j] * S(2, j)); };
    if (t < 3) grad[t] += dwb(t);
    else if (t < 12) grad[t] += c.ev2 * c.wb[(t - 3) % 3] * S((t - 3) / 3, (t - 3) % 3);
    else if (t == 12) grad[t] += 0.69314718055994531 * (c.wb[0] * dwb(0) + c.wb[1] * dwb(1) + c.wb[2] * dwb(2));
    else if (t < 23) grad[t] += sum[t - 13];
    else if (t == 23) grad[t] += sum[NP1 + NPH];
    else if (t == 24) grad[t] += sum[10];
}

// ---- halation blurs of the adjoint ---------------------------------------------
// With B = cols_G(rows_G(h)), the gradient of sigma is <gB, dB/dsigma> =
// <gB, cols_G(rows_dG h) + cols_dG(rows_G h)> = <cols_G^T gB, rows_dG h> +
// <cols_dG^T gB, rows_G h>: both row passes of h come from one kernel, both
// transposed column passes of gB from another, which takes the two inner
// products as it goes, and dB/dsigma is never formed.
//
// Both kernels form two blurs of one input, by G and dG, both symmetric: the
// two samples at tap k and 128 - k are added once and multiplied by both
// taps, 3 operations for 4 products.

struct DualTaps {
    float t[film::R64 + 1], d[film::R64 + 1];  // taps 0 .. 64 of G and dG
};

// Row pass source: the halation source of camera RGB, max(0, a_R - threshold).
struct CamSource {
    const float* __restrict__ x;
    float m[3], thr;  // a_R = m . x
    __device__ float above(const float (&v)[3]) const {
        return __fsub_rn(fmaf(m[2], v[2], fmaf(m[1], v[1], __fmul_rn(m[0], v[0]))), thr);
    }
    __device__ float operator()(size_t i) const {
        const float* p = x + 3 * i;
        const float v[3] = {__ldg(p), __ldg(p + 1), __ldg(p + 2)};
        return fmaxf(0.0f, above(v));
    }
};

// t1 = rows_G(h), t2 = rows_dG(h); four outputs of a row a thread.  Bound by
// instruction issue (0.72 of its rate, the FMA pipe at 0.53): 24 MP 264 us for
// both, one pass by packed pairs from the same source 148.
__global__ void __launch_bounds__(film::R64_ROW_THREADS) rows_dual_kernel(const CamSource in, float* __restrict__ t1,
                                                                          float* __restrict__ t2, int W,
                                                                          const __grid_constant__ DualTaps tp) {
    using film::R64;
    constexpr int TILE = 4 * film::R64_ROW_THREADS;
    __shared__ __align__(16) float s[TILE + 2 * R64];
    const int y = blockIdx.y, x0 = blockIdx.x * TILE;
    const size_t row = (size_t)y * W;
    for (int j = threadIdx.x; j < TILE + 2 * R64; j += blockDim.x) s[j] = in(row + film::reflect(x0 - R64 + j, W));
    __syncthreads();
    const float* p = s + 4 * threadIdx.x;
    float g[4], d[4];
    // lo: samples 4q .. 4q+7 of the window, hi: 124-4q .. 131-4q
    float lo[8], hi[8];
    auto ld = [](float* v, const float* q) {
        const float4 f = *reinterpret_cast<const float4*>(q);
        v[0] = f.x;
        v[1] = f.y;
        v[2] = f.z;
        v[3] = f.w;
    };
    ld(lo, p);
    ld(hi + 4, p + 2 * R64);
#pragma unroll
    for (int j = 0; j < 4; j++) g[j] = d[j] = 0.0f;
#pragma unroll
    for (int q = 0; q < R64 / 4; q++) {
        ld(lo + 4, p + 4 * q + 4);
        ld(hi, p + 2 * R64 - 4 - 4 * q);
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float v = lo[u + j] + hi[4 - u + j];
                g[j] = fmaf(v, tp.t[4 * q + u], g[j]);
                d[j] = fmaf(v, tp.d[4 * q + u], d[j]);
            }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            lo[i] = lo[i + 4];
            hi[i + 4] = hi[i];
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {  // the centre sample
        g[j] = fmaf(lo[j], tp.t[R64], g[j]);
        d[j] = fmaf(lo[j], tp.d[R64], d[j]);
        const int x = x0 + 4 * threadIdx.x + j;
        if (x < W) {
            t1[row + x] = g[j];
            t2[row + x] = d[j];
        }
    }
}

// t3 = cols_G(g), and the block's part of <t3, t2> + <cols_dG(g), t1> into
// partial[block]; cols_ends_kernel makes both the transposes.  A block walks a
// 32-column strip over a ring of three 128-row slabs as
// blur_cols_r64_stream_kernel does; a thread forms eight outputs of a chunk from
// two windows that slide towards each other.  Bound by instruction issue (0.76
// of its rate, the FMA pipe at 0.55).  24 MP: 0.26 ms, where the three column
// passes of G(gB) and dB/dsigma took 0.53.  (The end terms in this kernel's
// epilogue cost registers: 0.32-0.45 ms.)
constexpr int CD_OUT = 8, CD_GROUPS = film::SC_SLAB / CD_OUT, CD_PER = film::SC_SLAB / CD_GROUPS;
constexpr int CD_THREADS = film::R64_COL_TW * CD_GROUPS;

__global__ void __launch_bounds__(CD_THREADS, 2) cols_dual_t_kernel(const float* __restrict__ g, int W, int H,
                                                                    int chunks, const __grid_constant__ DualTaps tp,
                                                                    const float* __restrict__ t1,
                                                                    const float* __restrict__ t2,
                                                                    float* __restrict__ t3,
                                                                    double* __restrict__ partial) {
    using film::R64;
    using film::SC_SLAB;
    constexpr int TW = film::R64_COL_TW;
    __shared__ __align__(16) float ring[3 * SC_SLAB * TW];
    const int tx = threadIdx.x % TW, ty = threadIdx.x / TW;
    const int x = blockIdx.x * TW + tx;
    const bool xin = x < W;
    const int ybase = blockIdx.y * chunks * SC_SLAB;
    const int nch = min((H - ybase + SC_SLAB - 1) / SC_SLAB, chunks);
    float v[CD_PER], dot[1] = {0.0f};
    // slab s: rows ybase - 64 + 128 s .. + 127 (mirrored at the edges)
    auto load = [&](int sl) {
        const int r0 = ybase - R64 + SC_SLAB * sl + ty;
        const bool inner = r0 - ty >= 0 && r0 - ty + SC_SLAB <= H;
#pragma unroll
        for (int q = 0; q < CD_PER; q++) {
            const int r = r0 + q * CD_GROUPS;
            v[q] = xin ? __ldg(g + (size_t)(inner ? r : film::reflect(r, H)) * W + x) : 0.0f;
        }
    };
    auto store = [&](int sl) {
        float* slab = ring + (sl % 3) * SC_SLAB * TW;
#pragma unroll
        for (int q = 0; q < CD_PER; q++) slab[(ty + q * CD_GROUPS) * TW + tx] = v[q];
    };
    load(0);
    store(0);
    load(1);
    store(1);
    __syncthreads();
    const int rb = ty * CD_OUT;
    for (int j = 0; j < nch; j++) {
        if (j + 1 < nch) load(j + 2);  // in flight during this chunk
        const float* A = ring + (j % 3) * SC_SLAB * TW + tx;
        const float* B = ring + ((j + 1) % 3) * SC_SLAB * TW - SC_SLAB * TW + tx;
        // eight window rows 8 q .. 8 q + 7 (one slab: rb and the groups are multiples of 8)
        auto rows8 = [&](float* w, int q) {
            const float* p = (rb + 8 * q < SC_SLAB ? A : B) + (rb + 8 * q) * TW;
#pragma unroll
            for (int i = 0; i < 8; i++) w[i] = p[i * TW];
        };
        float a[CD_OUT], d[CD_OUT], lo[16], hi[16];
#pragma unroll
        for (int i = 0; i < CD_OUT; i++) a[i] = d[i] = 0.0f;
        rows8(lo, 0);
        rows8(hi + 8, 2 * R64 / 8);
#pragma unroll
        for (int q = 0; q < R64 / 8; q++) {
            // lo: window rows 8q .. 8q+15, hi: 120-8q .. 135-8q
            rows8(lo + 8, q + 1);
            rows8(hi, 2 * R64 / 8 - 1 - q);
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int i = 0; i < CD_OUT; i++) {
                    const float s = lo[u + i] + hi[8 - u + i];
                    a[i] = fmaf(s, tp.t[8 * q + u], a[i]);
                    d[i] = fmaf(s, tp.d[8 * q + u], d[i]);
                }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                lo[i] = lo[i + 8];
                hi[i + 8] = hi[i];
            }
        }
        if (xin) {
            const int y0 = ybase + j * SC_SLAB + rb;
#pragma unroll
            for (int i = 0; i < CD_OUT; i++) {
                a[i] = fmaf(lo[i], tp.t[R64], a[i]);  // the centre row
                d[i] = fmaf(lo[i], tp.d[R64], d[i]);
                if (y0 + i < H) {
                    const size_t p = (size_t)(y0 + i) * W + x;
                    t3[p] = a[i];
                    dot[0] = fmaf(a[i], __ldg(t2 + p), fmaf(d[i], __ldg(t1 + p), dot[0]));
                }
            }
        }
        if (j + 1 < nch) store(j + 2);  // into the slot of slab j-1, read last in chunk j-1
        __syncthreads();
    }
    // this block's sum of the inner products
    double* red = reinterpret_cast<double*>(ring);
    double w = (double)dot[0];
    for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < CD_THREADS / 32; k++) sum += red[k];
        partial[blockIdx.y * gridDim.x + blockIdx.x] = sum;
    }
}

// The transposes' end terms (film::transpose_end) of the two radius-64 column
// blurs of g: G's added to t3 and, as the products are linear, both to the
// inner products, in partial[block].  A block has 32 columns of an end; a warp
// takes eight of the 64 distances, each sample once for both blurs and for its
// own row's term and the end row's sum.  Bound by latency: every load is in
// flight at once.  2.8 MP: 3.5 us (24 MP: 5.6), where a thread a row, the end
// rows' 64 samples one thread's, took 11.4 us (16.4).  With H <= 129 rows the
// ends share rows and one block takes both, one after the other.
__global__ void __launch_bounds__(BLK) cols_ends_kernel(const float* __restrict__ g, int W, int H,
                                                        const __grid_constant__ DualTaps tp,
                                                        const float* __restrict__ t1, const float* __restrict__ t2,
                                                        float* __restrict__ t3, double* __restrict__ partial) {
    using film::R64;
    constexpr int WARPS = BLK / 32, PER = R64 / WARPS;
    static_assert(WARPS * PER == R64, "the warps share the distances evenly");
    __shared__ float2 red[WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, x = blockIdx.x * 32 + lane;
    float acc[1] = {0.0f};
    for (int end = blockIdx.y; end < 2; end += gridDim.y) {
        const int y0 = end ? H - 1 : 0, dir = end ? -W : W;
        const size_t p0 = (size_t)y0 * W + x;
        float sa = 0.0f, sd = 0.0f;
        if (x < W) {
            const float ge = __ldg(g + p0);
            float v[PER], u1[PER], u2[PER], u3[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const ptrdiff_t p = (ptrdiff_t)p0 + (ptrdiff_t)(1 + w * PER + i) * dir;
                v[i] = __ldg(g + p);
                u1[i] = __ldg(t1 + p);
                u2[i] = __ldg(t2 + p);
                u3[i] = t3[p];
            }
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int k = 1 + w * PER + i;
                const float ta = tp.t[R64 - k], td = tp.d[R64 - k], ea = ta * ge, ed = td * ge;
                sa = fmaf(ta, v[i], sa);
                sd = fmaf(td, v[i], sd);
                t3[(ptrdiff_t)p0 + (ptrdiff_t)k * dir] = u3[i] + ea;
                acc[0] = fmaf(ea, u2[i], fmaf(ed, u1[i], acc[0]));
            }
        }
        red[w][lane] = make_float2(sa, sd);
        __syncthreads();
        if (w == 0 && x < W) {
            sa = sd = 0.0f;
#pragma unroll
            for (int i = 0; i < WARPS; i++) {
                sa += red[i][lane].x;
                sd += red[i][lane].y;
            }
            t3[p0] -= sa;
            acc[0] -= fmaf(sa, t2[p0], sd * t1[p0]);
        }
        __syncthreads();
    }
    block_partials(acc, partial);
}

// gh = rows_G^T(t3) and at once its part of S, sum of gh x_j over the pixels
// whose red is above the threshold, as block partials: gh is not stored.
// A block takes every gridDim.y-th row of its 1024 columns.  24 MP: 0.18
// ms, where the row pass, its end terms and the colour pass took 0.34.
__global__ void __launch_bounds__(film::R64_ROW_THREADS) rows_t_color_kernel(const float* __restrict__ t3,
                                                                             const float* __restrict__ x, int W, int H,
                                                                             const __grid_constant__ film::Taps2 tp,
                                                                             const CamSource src,
                                                                             double* __restrict__ partial) {
    using film::R64;
    constexpr int OUT = film::R64_ROW_OUT;
    __shared__ __align__(16) float s[film::R64_ROW_TILE + 2 * R64];
    const int x0 = blockIdx.x * film::R64_ROW_TILE, xb = OUT * threadIdx.x;
    float acc[NPH] = {0.0f, 0.0f, 0.0f};
    constexpr int SPAN = film::R64_ROW_TILE + 2 * R64, PER = (SPAN + film::R64_ROW_THREADS - 1) / film::R64_ROW_THREADS;
    // the next row is loaded while this one is blurred
    float nx[PER];
    int col[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) col[q] = film::reflect(x0 - R64 + (int)threadIdx.x + q * film::R64_ROW_THREADS, W);
    auto load = [&](int y) {
#pragma unroll
        for (int q = 0; q < PER; q++) nx[q] = __ldg(t3 + (size_t)y * W + col[q]);
    };
    load(blockIdx.y);
    for (int y = blockIdx.y; y < H; y += gridDim.y) {
        __syncthreads();  // the row before is done with s
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int j = threadIdx.x + q * film::R64_ROW_THREADS;
            if (j < SPAN) s[j] = nx[q];
        }
        __syncthreads();
        if (y + (int)gridDim.y < H) load(y + gridDim.y);
        float gh[OUT], v[OUT][3];
#pragma unroll
        for (int j = 0; j < OUT; j++)
#pragma unroll
            for (int k = 0; k < 3; k++) v[j][k] = __ldg(x + 3 * ((size_t)y * W + min(x0 + xb + j, W - 1)) + k);
        film::row_r64(s + xb, tp, gh);
        if (x0 + xb <= R64 || x0 + xb + OUT - 1 >= W - 1 - R64) {
            auto g = [&](int i) { return s[i - x0 + R64]; };
            auto w = [&](int k) { return tp.t2[k].x; };
#pragma unroll
            for (int j = 0; j < OUT; j++)
                if (x0 + xb + j < W) gh[j] += film::transpose_end(x0 + xb + j, W, R64, 0.0f, g, w);
        }
#pragma unroll
        for (int j = 0; j < OUT; j++)
            if (x0 + xb + j < W && src.above(v[j]) > 0.0f)
#pragma unroll
                for (int k = 0; k < 3; k++) acc[k] = fmaf(gh[j], v[j][k], acc[k]);
    }
    block_partials<NPH, film::R64_ROW_THREADS>(acc, partial);
}

// The same steps for a halation radius below 64: the end terms of the
// transpose added to a blur of g, and the inner products of two plane pairs.
__global__ void blurT_edges_kernel(const float* __restrict__ g, float* __restrict__ out, int W, int H,
                                   const __grid_constant__ film::Taps tp, int along_cols) {
    const int n = along_cols ? H : W, R = tp.R;   // length of a line
    const int lines = along_cols ? W : H;
    const size_t step = along_cols ? (size_t)W : 1;   // along a line
    const size_t lstep = along_cols ? 1 : (size_t)W;  // between lines
    const size_t total = (size_t)lines * (2 * R + 2);
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int line = (int)(t % lines), r = (int)(t / lines);
        const int pos = r <= R ? r : n - 1 - (r - R - 1);
        if (r > R && pos <= R) continue;  // the first-end thread of this position adds both ends' terms
        const float* gl = g + line * lstep;
        out[line * lstep + pos * step] += film::transpose_end(pos, n, R, 0.0f, [&](int i) { return gl[i * step]; },
                                                              [&](int k) { return tp.t[k]; });
    }
}

__global__ void __launch_bounds__(BLK) dot2_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                   const float* __restrict__ c, const float* __restrict__ d, size_t n,
                                                   double* __restrict__ partial) {
    float acc[1] = {0.0f};
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
        acc[0] = fmaf(a[p], b[p], fmaf(c[p], d[p], acc[0]));
    block_partials(acc, partial);
}

// ---- host ---------------------------------------------------------------------

StreamCache g_ws("adjoint workspace");

int workspace(cudaStream_t s, size_t bytes, void** out) { return g_ws.get(s, bytes, out); }

struct Arena {
    char* base;
    size_t off;
    template <class T>
    T* take(size_t count) {
        size_t a = (off + 255) & ~(size_t)255;
        T* p = reinterpret_cast<T*>(base + a);
        off = a + count * sizeof(T);
        return p;
    }
};

// Halation taps and their sigma-derivative for the fixed radius R:
// w_i = g_i / S, g_i = exp(-x_i^2 / (2 s^2)); dw_i/ds = w_i (x_i^2 - sum_j w_j x_j^2) / s^3.
void halation_taps(float sigma, int R, float* t, float* dt) {
    double sum = 0.0, m2 = 0.0;
    std::vector<double> g(2 * R + 1);
    for (int i = 0; i <= 2 * R; i++) {
        double x = i - R;
        g[i] = std::exp(-x * x / (2.0 * sigma * sigma));
        sum += g[i];
    }
    for (int i = 0; i <= 2 * R; i++) {
        double x = i - R;
        m2 += g[i] / sum * x * x;
    }
    double s3 = (double)sigma * sigma * sigma;
    for (int i = 0; i <= 2 * R; i++) {
        double x = i - R, w = g[i] / sum;
        t[i] = (float)w;
        dt[i] = (float)(w * (x * x - m2) / s3);
    }
}

// bt: the backward's table, or NULL
int build_const(const ImopsFilmGradParams& P, const ImopsBaselineFilm& F, Const* c, BackTable* bt, float* taps,
                float* dtaps) {
    film::Stock st;
    float pitch;
    ImopsBaselineFilm f2 = F;
    f2.grain_on = 0;
    int rc = film::build_stock(IMOPS_STOCK_BASELINE81, 0, 1, -1.0f, &f2, &st, &pitch);
    if (rc) return rc;
    for (int i = 0; i < 3; i++) c->wb[i] = P.wb[i];
    for (int i = 0; i < 9; i++) c->C[i] = P.matrix[i];
    c->ev = P.ev;
    c->ev2 = std::exp2(P.ev);
    for (int l = 0; l < 3; l++) {
        c->dmax[l] = P.dmax[l];
        c->k[l] = P.k[l];
        c->x0[l] = P.x0[l];
        c->bleed[l] = st.base.bleed[l];
    }
    c->s = P.hal_strength;
    c->thr = F.hal_threshold;
    for (int i = 0; i < 9; i++) c->minv[i] = st.expose.minv[i];
    for (int k = 0; k < 3; k++)
        for (int l = 0; l < 3; l++) c->A[k][l] = st.expose.A[k][l];
    const film::ScanSpec81& S = st.scan81;
    if (bt)
        for (int i = 0; i < NB81; i++)
            for (int e = 0; e < 3; e++)
                for (int j = 0; j < 3; j++) {
                    const float q = (float)(-0.69314718055994531 * (double)S.eps[e][i] * (double)S.C[i][j]);
                    if (i == NB81 - 1) bt->Q_l[e][j] = q;
                    else if (i & 1) bt->Q[i / 2][e][j].y = q;
                    else bt->Q[i / 2][e][j].x = q;
                }
    for (int l = 0; l < NP; l++)
        for (int e = 0; e < 3; e++) {
            c->ne2[e][l] = make_float2(-S.eps[e][2 * l], -S.eps[e][2 * l + 1]);
            c->Cs2[e][l] = make_float2(S.C[2 * l][e], S.C[2 * l + 1][e]);
        }
    for (int e = 0; e < 3; e++) {
        c->ne_l[e] = -S.eps[e][NB81 - 1];
        c->Cs_l[e] = S.C[NB81 - 1][e];
    }
    if (F.hal_radius < 1 || F.hal_radius > HAL_R) return fail(IMOPS_ERR_INVALID_ARGUMENT, "hal_radius must be 1..64");
    if (!(P.hal_sigma > 0.0f)) return fail(IMOPS_ERR_INVALID_ARGUMENT, "hal_sigma must be > 0");
    halation_taps(P.hal_sigma, F.hal_radius, taps, dtaps);
    return IMOPS_OK;
}

struct Bufs {
    Const c;  // passed to the kernels by value
    BackTable bt;
    CamSource src;
    film::Taps tp, dtp;  // halation taps and their sigma-derivative
    // the halation's row blurs t1, t2, its blur B, the gradient gB of B and its
    // column blur t3; h shares t3, u and gh share B (free after the pixels)
    float *t1, *t2, *t3, *B, *gB;
    double *p1, *ph, *ps;
    int nb, nb1, R;  // blocks of the per-pixel kernels and of pixel_backward_kernel
    int chunks;     // of the radius-64 column kernels
    dim3 cols_grid;
    dim3 rows_grid;  // of rows_t_color_kernel
};

DualTaps dual_taps(const Bufs& b) {
    DualTaps t;
    for (int k = 0; k <= film::R64; k++) {
        t.t[k] = b.tp.t[k];
        t.d[k] = b.dtp.t[k];
    }
    return t;
}

// The working set, and the halation: B, and for the backward t1 and t2.
int prepare(const float* x, int W, int H, const ImopsFilmGradParams* P, const ImopsBaselineFilm* F, bool backward,
            cudaStream_t s, Bufs* b) {
    if (!x || !P) return fail(IMOPS_ERR_INVALID_ARGUMENT, "param film: NULL argument");
    if (W <= 0 || H <= 0) return fail(IMOPS_ERR_INVALID_DIMENSIONS, "invalid image dimensions");
    ImopsBaselineFilm Fd;
    if (F) Fd = *F;
    else imops_baseline_film_defaults(&Fd);
    if (backward && (W <= Fd.hal_radius + 1 || H <= Fd.hal_radius + 1))
        return fail(IMOPS_ERR_UNSUPPORTED_SIZE, "param film backward: image sides must exceed the halation radius + 1");
    const size_t n = (size_t)W * H;
    b->nb = film::grid_for_n(n);
    b->nb1 = (int)std::min((n + PB_THREADS - 1) / PB_THREADS, (size_t)sm_count() * PB_BLOCKS);
    // two waves of the eight blocks an SM holds, each with as many rows as that leaves
    const int tiles = (W + film::R64_ROW_TILE - 1) / film::R64_ROW_TILE;
    b->rows_grid = dim3(tiles, std::max(1, std::min(H, 16 * sm_count() / tiles)));
    b->chunks = film::stream_chunks(W, H, sm_count());
    b->cols_grid = dim3((W + film::R64_COL_TW - 1) / film::R64_COL_TW,
                        (H + b->chunks * film::SC_SLAB - 1) / (b->chunks * film::SC_SLAB));
    const size_t ns = std::max((size_t)b->cols_grid.x * (b->cols_grid.y + 2), (size_t)b->nb);
    const size_t nh = std::max((size_t)b->rows_grid.x * b->rows_grid.y, (size_t)b->nb);
    const size_t bytes = (backward ? 5 : 3) * (n * 4 + 256) + (b->nb1 * NP1 + nh * NPH + ns) * 8 + 8192;
    void* ws = nullptr;
    int rc = workspace(s, bytes, &ws);
    if (rc) return rc;
    Arena A{static_cast<char*>(ws), 0};
    b->t1 = A.take<float>(n);
    b->B = A.take<float>(n);
    b->t3 = A.take<float>(n);
    if (backward) {
        b->t2 = A.take<float>(n);
        b->gB = A.take<float>(n);
        b->p1 = A.take<double>((size_t)b->nb1 * NP1);
        b->ph = A.take<double>(nh * NPH);
        b->ps = A.take<double>(ns);
    }
    b->tp.R = b->dtp.R = 0;
    if ((rc = build_const(*P, Fd, &b->c, backward ? &b->bt : nullptr, b->tp.t, b->dtp.t))) return rc;
    const int R = b->R = b->tp.R = b->dtp.R = Fd.hal_radius;
    if (R == film::R64) {
        CamSource& src = b->src;
        src.x = x;
        src.thr = b->c.thr;
        for (int i = 0; i < 3; i++) src.m[i] = b->c.C[i] * b->c.ev2 * b->c.wb[i];
        const dim3 rg((W + film::R64_ROW_TILE - 1) / film::R64_ROW_TILE, H);
        if (backward) rows_dual_kernel<<<rg, film::R64_ROW_THREADS, 0, s>>>(src, b->t1, b->t2, W, dual_taps(*b));
        else film::blur_rows_r64_kernel<<<rg, film::R64_ROW_THREADS, 0, s>>>(src, b->t1, W, H, film::pair_taps(b->tp));
        note_launch();
        IMOPS_CUDA_TRY(cudaGetLastError(), "param film rows");
    } else {
        float* h = b->t3;
        prep_kernel<<<b->nb, BLK, 0, s>>>(x, n, b->c, h);
        note_launch();
        if ((rc = film::blur_rows(h, b->t1, W, H, b->tp.t, R, s))) return rc;
        if (backward && (rc = film::blur_rows(h, b->t2, W, H, b->dtp.t, R, s))) return rc;
    }
    return film::blur_cols(b->t1, b->B, W, H, b->tp.t, R, s);
}

// After pixel_backward_kernel: gh = rows^T(cols^T(gB)), the partial sums of its
// part of S (*nbh of each) into ph and those of sigma's gradient (*nbs) into ps.
int backward_halation(Bufs& b, const float* x, int W, int H, int* nbh, int* nbs, cudaStream_t s) {
    const size_t n = (size_t)W * H;
    int rc;
    if (b.R == film::R64) {
        cols_dual_t_kernel<<<b.cols_grid, CD_THREADS, 0, s>>>(b.gB, W, H, b.chunks, dual_taps(b), b.t1, b.t2, b.t3,
                                                              b.ps);
        const int nb = (int)(b.cols_grid.x * b.cols_grid.y);
        const int ends = H > 2 * film::R64 + 1 ? 2 : 1;
        cols_ends_kernel<<<dim3(b.cols_grid.x, ends), BLK, 0, s>>>(b.gB, W, H, dual_taps(b), b.t1, b.t2, b.t3,
                                                                   b.ps + nb);
        *nbs = nb + (int)b.cols_grid.x * ends;
        rows_t_color_kernel<<<b.rows_grid, film::R64_ROW_THREADS, 0, s>>>(b.t3, x, W, H, film::pair_taps(b.tp), b.src,
                                                                          b.ph);
        *nbh = (int)(b.rows_grid.x * b.rows_grid.y);
        note_launch(3);
        return IMOPS_OK;
    }
    const int gc = film::grid_for_n((size_t)W * (2 * b.R + 2)), gr = film::grid_for_n((size_t)H * (2 * b.R + 2));
    float* u = b.B;
    if ((rc = film::blur_cols(b.gB, b.t3, W, H, b.tp.t, b.R, s))) return rc;
    blurT_edges_kernel<<<gc, BLK, 0, s>>>(b.gB, b.t3, W, H, b.tp, 1);
    if ((rc = film::blur_cols(b.gB, u, W, H, b.dtp.t, b.R, s))) return rc;
    blurT_edges_kernel<<<gc, BLK, 0, s>>>(b.gB, u, W, H, b.dtp, 1);
    dot2_kernel<<<b.nb, BLK, 0, s>>>(b.t3, b.t2, u, b.t1, n, b.ps);
    *nbs = b.nb;
    if ((rc = film::blur_rows(b.t3, b.B, W, H, b.tp.t, b.R, s))) return rc;
    blurT_edges_kernel<<<gr, BLK, 0, s>>>(b.t3, b.B, W, H, b.tp, 0);
    color_back_kernel<<<b.nb, BLK, 0, s>>>(x, b.B, n, b.c, b.ph);
    *nbh = b.nb;
    note_launch(5);
    return IMOPS_OK;
}

}  // namespace adj
}  // namespace imops

using namespace imops;

extern "C" int imops_param_forward(const float* cam_rgb, int w, int h, const ImopsFilmGradParams* params,
                                   const ImopsBaselineFilm* fixed, float* out, imops_stream_t stream) {
    clear_error();
    if (!out) return fail(IMOPS_ERR_INVALID_ARGUMENT, "param forward: NULL output");
    cudaStream_t s = as_stream(stream);
    adj::Bufs b;
    int rc = adj::prepare(cam_rgb, w, h, params, fixed, false, s, &b);
    if (rc) return rc;
    adj::pixel_forward_kernel<<<b.nb, adj::BLK, 0, s>>>(cam_rgb, b.B, (size_t)w * h, b.c, out);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "param forward");
    return IMOPS_OK;
}

extern "C" int imops_param_backward(const float* cam_rgb, const float* g_out, const float* target, float loss_scale,
                                    int w, int h, const ImopsFilmGradParams* params, const ImopsBaselineFilm* fixed,
                                    double* grad, imops_stream_t stream) {
    clear_error();
    if (!grad) return fail(IMOPS_ERR_INVALID_ARGUMENT, "param backward: NULL gradient buffer");
    if (!g_out && !target) return fail(IMOPS_ERR_INVALID_ARGUMENT, "param backward: need g_out or target");
    cudaStream_t s = as_stream(stream);
    adj::Bufs b;
    int rc = adj::prepare(cam_rgb, w, h, params, fixed, true, s, &b);
    if (rc) return rc;
    const size_t n = (size_t)w * h;
    adj::pixel_backward_kernel<<<b.nb1, adj::PB_THREADS, 0, s>>>(cam_rgb, b.B, g_out, target, loss_scale, n, b.c, b.bt,
                                                                 b.gB, b.p1);
    note_launch();
    int nbh = 0, nbs = 0;
    if ((rc = adj::backward_halation(b, cam_rgb, w, h, &nbh, &nbs, s))) return rc;
    adj::ColorParams cp;
    cp.ev2 = b.c.ev2;
    for (int i = 0; i < 3; i++) cp.wb[i] = b.c.wb[i];
    for (int i = 0; i < 9; i++) cp.C[i] = b.c.C[i];
    adj::finish_kernel<<<1, 32 * adj::FIN_SUMS, 0, s>>>(b.p1, b.nb1, b.ph, nbh, b.ps, nbs, cp, grad);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "param backward");
    return IMOPS_OK;
}
