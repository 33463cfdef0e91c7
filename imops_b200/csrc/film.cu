// film.cu -- spectral film simulation kernels and imops_film_process.
//
// Reference model (film::process, pichromatic/src/film/mod.rs:77-129) as a
// chain of planar kernels, in brackets what one kernel does:
//   [expose (rank-3 spectral collapse) -> local scatter] -> blur of the
//   support's plane -> [bounce -> capture LUT -> reduce] -> [DIR blur and
//   inhibition] -> grain fields -> [adjacency -> grain -> 16-bin scan ->
//   invert].
// Blurs too wide for the tiles (film_tiles.cuh) run as passes of their own.
// Baseline preset (81 bins): halation row pass (its source formed from the
// RGB) beside the grain fields -> one fused kernel doing the exposure, the
// halation column pass, the logistic curves, grain and the 81-bin scan.
//
// Layout: per-layer planes (row-major f32), so every pass is a coalesced
// stream; RGB stays interleaved as in Image.rgb_data.
#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "blur.cuh"
#include "film.cuh"

namespace imops {
namespace film {

// The baseline preset's logistic density curve D = dmax / (1 + e^(-k (log10 E
// - x0))) from the hardware base-2 logarithm and exponential (lg2 / ex2
// .approx.ftz, about 2^-22 relative) and a fast reciprocal: log10 E =
// log2 E * log10(2), e^x = 2^(x log2 e).  Within 1e-6 relative of the
// library functions' result; the film's tolerance is 1e-4.
__device__ __forceinline__ float curve_density(float E, float dmax, float k, float x0) {
    float l2;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l2) : "f"(fmaxf(E, 1e-6f)));
    const float le = l2 * 0.30102999566398120f;
    const float t = ex2_fast(-k * (le - x0) * 1.4426950408889634f);
    return __fdividef(dmax, 1.0f + t);
}

// ---------------------------------------------------------------------------
// exposure

// The basis weights of one pixel: w = max(0, Minv * rgb).  Explicit
// multiply-adds: a kernel of its own and a fused one give the same bits.
__device__ __forceinline__ float dot3(float a0, float x0, float a1, float x1, float a2, float x2) {
    return fmaf(a2, x2, fmaf(a1, x1, __fmul_rn(a0, x0)));
}
__device__ __forceinline__ void basis_weights(const ExposeSpec& X, float r, float g, float b, float (&w)[3]) {
    w[0] = fmaxf(0.0f, dot3(X.minv[0], r, X.minv[1], g, X.minv[2], b));
    w[1] = fmaxf(0.0f, dot3(X.minv[3], r, X.minv[4], g, X.minv[5], b));
    w[2] = fmaxf(0.0f, dot3(X.minv[6], r, X.minv[7], g, X.minv[8], b));
}

// Layer e's absorbed band-mean fluence from the basis weights.
__device__ __forceinline__ float layer_exposure(const ExposeSpec& X, const float (&w)[3], int e) {
    return dot3(X.A[0][e], w[0], X.A[1][e], w[1], X.A[2][e], w[2]);
}

// rgb (interleaved) -> E planes of absorbed band-mean fluence.
__global__ void expose_kernel(const float* __restrict__ rgb, size_t n, ExposeSpec X, float* __restrict__ planes) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float r = rgb[3 * p], g = rgb[3 * p + 1], b = rgb[3 * p + 2];
        float w[3];
        basis_weights(X, r, g, b, w);
        for (int e = 0; e < X.E; e++) planes[e * n + p] = layer_exposure(X, w, e);
    }
}

// local scatter: p = keep*p + mix*blur(p) (halation.rs:164-181)
__device__ __forceinline__ float mix_px(float p, float v, float keep, float mix) {
    return fmaf(mix, v, __fmul_rn(keep, p));
}
struct EpiMix {
    float* plane;
    float keep, mix;
    __device__ __forceinline__ void operator()(size_t i, float v) const { plane[i] = mix_px(plane[i], v, keep, mix); }
};
// adjacency: d += beta * (d - blur(d)) (diffusion.rs:11-28)
__device__ __forceinline__ float adjacency_px(float d, float v, float beta) { return fmaf(beta, __fsub_rn(d, v), d); }
struct EpiAdjacency {
    float* plane;
    float beta;
    __device__ __forceinline__ void operator()(size_t i, float v) const { plane[i] = adjacency_px(plane[i], v, beta); }
};

int blur_rows(const float* in, float* out, int W, int H, const float* taps, int R, cudaStream_t s) {
    if (R < 0 || R > MAXR) return fail(IMOPS_ERR_INVALID_ARGUMENT, "blur radius above 64");
    Taps tp;
    tp.R = R;
    for (int i = 0; i < 2 * R + 1; i++) tp.t[i] = taps[i];
    if (R == R64) {
        dim3 rg((W + R64_ROW_TILE - 1) / R64_ROW_TILE, H);
        blur_rows_r64_kernel<<<rg, R64_ROW_THREADS, 0, s>>>(PlaneSource{in}, out, W, H, pair_taps(tp));
    } else {
        dim3 rg((W + ROW_TILE - 1) / ROW_TILE, H);
        blur_rows_kernel<<<rg, ROW_THREADS, 0, s>>>(in, out, W, H, tp);
    }
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "blur rows");
    return IMOPS_OK;
}

// The baseline preset's halation row pass straight from interleaved RGB: the
// radius-64 row blur of max(0, R - threshold), the source formed as it is
// read instead of as a plane of its own.
static int blur_rows_halation(const float* rgb, float threshold, float* out, int W, int H, const float* taps,
                              cudaStream_t s) {
    Taps tp;
    tp.R = R64;
    for (int i = 0; i < 2 * R64 + 1; i++) tp.t[i] = taps[i];
    dim3 rg((W + R64_ROW_TILE - 1) / R64_ROW_TILE, H);
    blur_rows_r64_kernel<<<rg, R64_ROW_THREADS, 0, s>>>(HalationSource{rgb, threshold}, out, W, H, pair_taps(tp));
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "halation row pass");
    return IMOPS_OK;
}

int blur_cols(const float* in, float* out, int W, int H, const float* taps, int R, cudaStream_t s) {
    if (R < 0 || R > MAXR) return fail(IMOPS_ERR_INVALID_ARGUMENT, "blur radius above 64");
    Taps tp;
    tp.R = R;
    for (int i = 0; i < 2 * R + 1; i++) tp.t[i] = taps[i];
    if (R == R64) {
        const int ch = stream_chunks(W, H, sm_count());
        dim3 cb(R64_COL_TW, R64_COL_GROUPS),
            cg((W + R64_COL_TW - 1) / R64_COL_TW, (H + ch * SC_SLAB - 1) / (ch * SC_SLAB));
        blur_cols_r64_stream_kernel<<<cg, cb, 0, s>>>(in, W, H, ch, pair_taps(tp), EpiStore{out});
    } else {
        dim3 cb(COL_TW, COL_GROUPS), cg((W + COL_TW - 1) / COL_TW, (H + COL_TH - 1) / COL_TH);
        blur_cols_kernel<<<cg, cb, 0, s>>>(in, W, H, tp, EpiStore{out});
    }
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "blur cols");
    return IMOPS_OK;
}

int taps_for(float sigma, Taps* tp) {
    int r = gaussian_taps(sigma, tp->t, 2 * MAXR + 1);
    if (r < 0) return fail(IMOPS_ERR_UNSUPPORTED_SIZE, "film: blur radius above 64 px (pixel pitch too small)");
    tp->R = r;
    return IMOPS_OK;
}

template <class Epi>
int blur(const float* in, float* tmp, int W, int H, const Taps& tp, Epi epi, cudaStream_t s) {
    dim3 rg((W + ROW_TILE - 1) / ROW_TILE, H);
    blur_rows_kernel<<<rg, ROW_THREADS, 0, s>>>(in, tmp, W, H, tp);
    note_launch();
    dim3 cb(COL_TW, COL_GROUPS), cg((W + COL_TW - 1) / COL_TW, (H + COL_TH - 1) / COL_TH);
    blur_cols_kernel<<<cg, cb, 0, s>>>(tmp, W, H, tp, epi);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "film blur launch");
    return IMOPS_OK;
}

}  // namespace film
}  // namespace imops

#include "film_tiles.cuh"

namespace imops {
namespace film {

// ---------------------------------------------------------------------------
// support bounce, capture LUT, reduce (halation.rs:80-92, capture.rs:61-88,
// reduction.rs:16-68)

// support bounce: plane_e += gain_e * blur(deep)
struct Bounce {
    float gain[MAXE];
};
__device__ __forceinline__ float bounce_px(float p, float gain, float v) { return gain > 0.0f ? fmaf(gain, v, p) : p; }

__global__ void bounce_kernel(float* __restrict__ planes, const float* __restrict__ deep, size_t n, int E,
                              const __grid_constant__ Bounce bn) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        const float v = deep[p];
        for (int e = 0; e < E; e++)
            if (bn.gain[e] > 0.0f) planes[e * n + p] = bounce_px(planes[e * n + p], bn.gain[e], v);
    }
}

// Layer constants of the capture LUT and the reduction.
template <int E>
struct Reduce {
    float eta[E], dmax[E], inv_gamma[E], mask_scale[E];  // mask_scale 0: no mask
    int reversal[E];
};

// Developable fraction of a layer's fluence phi: linear interpolation in
// log10 phi over LUTN entries at -4 .. 8 in equal steps, so the cell is found
// by arithmetic (a search over the knots before).  With phi = 2^k m, m in
// [1, 2), the place in cells is SCALE k + SCALE log2 m + ZERO; the first
// term is exact but for the low part of SCALE (k times its upper 12 bits), and
// log2 m is at most 1, where a logarithm of phi itself, up to 27, rounds at
// 1e-6.  (The hardware logarithm for log2 m: 0.44 ms instead of 0.55 for the
// reduction, but Portra400's error against 64 bits rose from 1.2e-7 to 1.3e-7.)
// lut[i] = (entry i, entry i+1 - entry i).
__device__ __forceinline__ float lut_sample(const float2* lut, float phi) {
    constexpr double SCALE = (LUTN - 1) / 12.0 * 0.30102999566398119521;  // cells an octave
    constexpr float HI = (float)((int)(SCALE * 2048.0)) / 2048.0f, LO = (float)(SCALE - (double)HI);
    constexpr float ZERO = (float)((LUTN - 1) / 3);  // cell of phi = 1
    static_assert((LUTN - 1) % 3 == 0, "phi = 1 is a knot");
    if (!(phi > 1.0e-5f)) return lut[0].x;  // below the first knot at 1e-4 (and NaN)
    if (phi > 1.0e9f) return lut[LUTN - 1].x;
    const uint32_t b = __float_as_uint(phi);
    const float k = (float)((int)(b >> 23) - 127);
    const float lm = log2f(__uint_as_float((b & 0x007FFFFFu) | 0x3F800000u));
    const float frac = fmaf(lm, (float)SCALE, k * LO);
    const float pos = fminf(fmaxf(fmaf(k, HI, ZERO) + frac, 0.0f), (float)(LUTN - 1));
    const int i = min((int)pos, LUTN - 2);
    const float t = fminf(fmaxf(fmaf(k, HI, ZERO - (float)i) + frac, 0.0f), 1.0f);
    const float2 c = lut[i];
    return fmaf(t, c.y, c.x);
}

// f^g for f in [0, 1], g > 0, to about an ulp (1.4e-7 at g = 2.9): with
// f = 2^k (1 + t), 1 + t in [0.71, 1.41), the product g log2 f is g k +
// g log2(1 + t).  Its nearest integer n leaves g k by one fused operation, and
// log2(1 + t), at most 1/2, is good to 4e-8 as t (log2 e + t Q(t)), Q a
// polynomial of degree 7 fitted here for least error; a logarithm of f itself
// rounds at 5e-7 for f = 1e-4, an error of 10 ulp.  2^remainder is a polynomial of degree 6
// fitted here for least relative error on [-1/2, 1/2] (2e-9).  (The hardware
// exponential's 2 ulp near f = 1, where a positive print's highlights lie, were
// the largest error of the reduction.)  0 and subnormals, and results below
// 2^-125, are 0.
__device__ __forceinline__ float pow_unit(float f, float g) {
    const uint32_t up = __float_as_uint(f) - 0x3F3504F3u;  // from the bits of sqrt(1/2)
    const float k = (float)((int)up >> 23);
    const float t = __uint_as_float((up & 0x007FFFFFu) + 0x3F3504F3u) - 1.0f;
    float p = 0.12592235207557678f;
    p = fmaf(p, t, -0.20859862864017487f);
    p = fmaf(p, t, 0.21626605093479156f);
    p = fmaf(p, t, -0.23876483738422394f);
    p = fmaf(p, t, 0.2878434956073761f);
    p = fmaf(p, t, -0.36071109771728516f);
    p = fmaf(p, t, 0.48091256618499756f);
    p = fmaf(p, t, -0.7213472723960876f);
    const float lm = fmaf(t, 1.44269502f, p * (t * t));
    const float n = rintf(fmaf(g, lm, g * k));
    if (f < 1.17549435e-38f || n <= -126.0f) return 0.0f;
    const float r = fmaf(g, lm, fmaf(g, k, -n));
    float q = 0.0001535336923552677f;
    q = fmaf(q, r, 0.0013398876180872321f);
    q = fmaf(q, r, 0.00961843691766262f);
    q = fmaf(q, r, 0.055503323674201965f);
    q = fmaf(q, r, 0.24022647738456726f);
    q = fmaf(q, r, 0.6931471824645996f);
    q = fmaf(q, r, 1.0f);
    return __uint_as_float(__float_as_uint(q) + ((uint32_t)(int)n << 23));
}

// The capture LUT (capture.rs:37-58, 91-106): entry i of layer e is the
// developable fraction 1 - E[exp(-k s^2 phi)] at log10 phi = -4 + 12 i / 63 for
// log-normal grain sizes s, the expectation by the trapezoid rule over 65
// points of the normal variable, in f64: frac[e * LUTN + i].  A block a layer,
// eight lanes an entry; bound by the latency of the f64 exponentials.  3.1 us
// for six layers, where the same 8300 exponentials a layer took a host thread
// 0.14 ms a layer before the first launch of every call.
struct CaptureSpec {
    double mu[MAXE], sigma[MAXE], k[MAXE];
};
__global__ void __launch_bounds__(8 * LUTN) capture_lut_kernel(const __grid_constant__ CaptureSpec c,
                                                               float* __restrict__ frac) {
    constexpr int PTS = 65;
    __shared__ double weight[PTS], ks2[PTS];
    const int e = blockIdx.x, t = threadIdx.x;
    if (t < PTS) {
        const double z = -8.0 + 0.25 * t, s = exp(c.mu[e] + c.sigma[e] * z);
        weight[t] = (t == 0 || t == PTS - 1 ? 0.5 : 1.0) * 0.25 * 0.39894228040143267794 * exp(-0.5 * z * z);
        ks2[t] = c.k[e] * s * s;
    }
    __syncthreads();
    const int i = t >> 3;
    const double phi = exp10(-4.0 + 12.0 * ((double)i / (LUTN - 1)));
    double acc = 0.0;
    for (int j = t & 7; j < PTS; j += 8) acc += weight[j] * exp(-ks2[j] * phi);
    for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((t & 7) == 0) frac[e * LUTN + i] = (float)fmin(fmax(1.0 - acc, 0.0), 1.0);
}

// Image-dye densities over the fluences in place, and the mask densities
// (SUM: `mask` is one plane, their sum in layer order; otherwise E planes);
// BOUNCE: the support bounce `deep` is added to the fluences first.  Bound by
// instruction issue (0.84 of its rate): the interpolation and the power of each
// layer and pixel.  24 MP, six layers, with the bounce: 0.55 ms against 1.86
// (reduction and bounce epilogue apart, a binary search and powf a value).
template <int E, bool SUM, bool BOUNCE>
__global__ void __launch_bounds__(256) lut_reduce_kernel(float* __restrict__ planes, float* __restrict__ mask,
                                                         const float* __restrict__ deep, size_t n,
                                                         const float* __restrict__ frac,
                                                         const __grid_constant__ Reduce<E> c,
                                                         const __grid_constant__ Bounce bn) {
    __shared__ float2 lut[E][LUTN];
    for (int k = threadIdx.x; k < E * LUTN; k += blockDim.x) {
        const int e = k / LUTN, i = k % LUTN;
        const float a = frac[k], b = i + 1 < LUTN ? frac[k + 1] : a;
        lut[e][i] = make_float2(a, b - a);
    }
    __syncthreads();
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float x[E], v = 0.0f, M = 0.0f;
#pragma unroll
        for (int e = 0; e < E; e++) x[e] = planes[e * n + p];
        if (BOUNCE) v = __ldg(deep + p);
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (BOUNCE) x[e] = bounce_px(x[e], bn.gain[e], v);
            float f = lut_sample(lut[e], __fmul_rn(x[e], c.eta[e]));
            f = fminf(fmaxf(f, 0.0f), 1.0f);
            if (c.reversal[e]) f = 1.0f - f;
            const float q = pow_unit(f, c.inv_gamma[e]);
            planes[e * n + p] = __fmul_rn(c.dmax[e], q);
            const float m = __fmul_rn(c.mask_scale[e], 1.0f - fminf(q, 1.0f));
            if (SUM) M = __fadd_rn(M, m);
            else mask[e * n + p] = m;
        }
        if (SUM) mask[p] = M;
    }
}

// DIR inhibition: D_j *= exp(-sum_i m[i][j] * inh_i) (diffusion.rs:39-84),
// for blurs wider than dir_kernel's tiles
struct DirAny {
    float m[MAXE][MAXE];
};
__global__ void dir_apply_kernel(float* __restrict__ planes, const float* __restrict__ inh, size_t n, int E,
                                 const __grid_constant__ DirAny dir) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
        for (int j = 0; j < E; j++) {
            float tot = 0.0f;
            bool active = false;
            for (int i = 0; i < E; i++) {
                float w = dir.m[i][j];
                if (w != 0.0f) {
                    active = true;
                    tot += w * inh[i * n + p];
                }
            }
            if (active) planes[j * n + p] *= expf(-tot);
        }
}

// ---------------------------------------------------------------------------
// grain (grain.rs:20-100): SplitMix64 is counter based, so pixel x of row y
// uses draws 12x+1..12x+12 of the row stream and is generated independently.

// The blurred grain fields of LAYERS consecutive RNG layers of one tile in one
// pass: Irwin-Hall noise over the tile plus its halo, mirrored at the image
// edge; per layer the row then column passes of blur() in shared memory with
// the same taps and summation order; the fields written, and each layer's
// block sum of squares (f64) stored in partial[plane][block] for the variance.
// Plane z holds RNG layer layer0 + z.  Radius <= GR_MAXR.
//
// Layer L of row y is the SplitMix64 stream seeded seed*0xD1B54A32D192ED03 +
// L*golden + y, and pixel x takes its draws 12x+1 .. 12x+12, the sum of those
// 12 uniforms minus 6 (grain.rs:20-45, 53-66).  Draw k of layer L has the
// state seed*C + y + (L + 12x + k)*golden, which is draw L + k of layer 0's
// stream: the layers of a run of RUN pixels take 12 RUN + LAYERS - 1 draws of
// one stream, each mixed once, and every (pixel, layer) sum is a difference
// of two prefix sums.
//
// A draw enters the sums as the upper 28 bits of its 64 (modulo 2^32, which
// differences of 12 such draws cannot exceed), with the mean of what is cut
// off added back: a uniform is then good to 2^-29 and the sum exact until its
// one conversion to f32, where twelve f32 additions rounded at 2^-22 each.  The
// mixer's last xor-shift by 31 reaches only bit 32 of a draw, so it is left out.
//
// Bound by the integer ALU (11 of the 17 instructions of a draw; its pipe at 0.66
// of its rate, issue at 0.75) at 32 warps an SM.  Tiles are 128 wide and TH high, their runs a whole number of
// rounds of the 512 threads where that fits two blocks an SM: 39 rows for up
// to three layers (96 KB), 24 for six (113 KB).  Six layers in one block mix
// 13.25 draws a pixel, two blocks of three 25; with fewer than two tiles of
// 39 rows an SM the layers go three at a time, in the tile height that fills
// the SMs best (grain_rows).  24 MP: three layers 0.44 ms (0.57 with f32 sums
// of draws converted one by one), six layers 0.61 ms (2.55 one layer a launch).
constexpr int GR_TW = 128, GR_MAXR = 16, GR_RUN = 4;
constexpr int GR_THREADS = 512, GR_GROUPS = GR_THREADS / GR_TW;
constexpr int GR_TH = 39, GR_TH6 = 24;
static_assert(GR_TW == 128, "the blur loops index tile columns with & 127");
// output rows a thread, and rows of the row-blurred buffer: the last group's
// window reaches past the tile's halo where TH is not a multiple of the groups
constexpr int gr_rows(int th) { return (th + GR_GROUPS - 1) / GR_GROUPS; }
constexpr int gr_row_buffer(int th, int R) { return GR_GROUPS * gr_rows(th) + 2 * R; }

// The sums of RUN consecutive pixels x .. x+RUN-1 of row y in layers layer0 ..
// layer0+LAYERS-1, as noise values (sum minus 6).
template <int LAYERS, int RUN>
__device__ __forceinline__ void grain_noise(uint64_t seed, int layer0, int y, int x, float (&out)[RUN][LAYERS]) {
    static_assert(LAYERS <= 12, "the prefix sums kept are those of the last pixel's start");
    const uint64_t golden = 0x9E3779B97F4A7C15ull;
    // state of draw k is z0 + k * golden (mod 2^64): stepped, not multiplied
    uint64_t z0 = seed * 0xD1B54A32D192ED03ull + (uint64_t)layer0 * golden + (uint64_t)y + 12 * (uint64_t)x * golden;
    uint32_t sum = 0, start[LAYERS];  // prefix sum, and its value before each layer's draws of the pixel
    start[0] = 0;
#pragma unroll
    for (int k = 1; k <= 12 * RUN + LAYERS - 1; k++) {
        z0 += golden;
        uint64_t v = (z0 ^ (z0 >> 30)) * 0xBF58476D1CE4E5B9ull;
        v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
        sum += (uint32_t)(v >> 32) >> 4;
        const int z = k % 12, i = k / 12 - 1;
        if (z < LAYERS) {
            // 6 for the mean, 6 half units for the bits cut off
            if (i >= 0) out[i][z] = (float)(int)(sum - start[z] - 0x60000000u + 6u) * (1.0f / 268435456.0f);
            start[z] = sum;
        }
    }
}

template <int LAYERS, int TH>
__global__ void __launch_bounds__(GR_THREADS, 2) grain_field_kernel(float* __restrict__ noise, int W, int H,
                                                                    uint64_t seed, int layer0,
                                                                    const __grid_constant__ Taps tp,
                                                                    double* __restrict__ partial) {
    extern __shared__ __align__(16) float gsm[];
    __shared__ double red[GR_THREADS / 32];
    const int R = tp.R;
    const int x0 = blockIdx.x * GR_TW, y0 = blockIdx.y * TH;
    const int tid = threadIdx.x;
    // noise rows are NW samples; stored with a stride of NWP (a multiple of
    // the run, so runs and their float4 stores stay aligned)
    const int NW = GR_TW + 2 * R, NH = TH + 2 * R;
    const int NWP = (NW + GR_RUN - 1) / GR_RUN * GR_RUN;
    float* sn = gsm;                      // noise, tile + halo: LAYERS x NH x NWP
    float* sr = gsm + LAYERS * NH * NWP;  // row-blurred: gr_row_buffer rows x GR_TW (one layer at a time)
    if (x0 - R >= 0 && x0 + NWP - R <= W) {
        // runs of GR_RUN pixels over the rows (rows mirrored; the last run of
        // a row may reach past NW: those samples are generated and never
        // read); (row, run) of j stepped without a division
        const int RPR = NWP / GR_RUN, nruns = NH * RPR;
        const int dq = GR_THREADS / RPR, dr = GR_THREADS - dq * RPR;
        int r = tid / RPR, q = tid - (tid / RPR) * RPR;
        for (int j = tid; j < nruns; j += GR_THREADS) {
            float v[GR_RUN][LAYERS];
            grain_noise<LAYERS, GR_RUN>(seed, layer0, reflect(y0 - R + r, H), x0 - R + q * GR_RUN, v);
#pragma unroll
            for (int z = 0; z < LAYERS; z++) {
                static_assert(GR_RUN == 4, "one float4 store a run and layer");
                *reinterpret_cast<float4*>(sn + (z * NH + r) * NWP + q * GR_RUN) =
                    make_float4(v[0][z], v[1][z], v[2][z], v[3][z]);
            }
            r += dq;
            q += dr;
            if (q >= RPR) {
                q -= RPR;
                r++;
            }
        }
    } else {
        const int dq = GR_THREADS / NW, dr = GR_THREADS - dq * NW;
        int r = tid / NW, c = tid - (tid / NW) * NW;
        for (int idx = tid; idx < NH * NW; idx += GR_THREADS) {
            float v[1][LAYERS];
            grain_noise<LAYERS, 1>(seed, layer0, reflect(y0 - R + r, H), reflect(x0 - R + c, W), v);
#pragma unroll
            for (int z = 0; z < LAYERS; z++) sn[(z * NH + r) * NWP + c] = v[0][z];
            r += dq;
            c += dr;
            if (c >= NW) {
                c -= NW;
                r++;
            }
        }
    }
    const size_t n = (size_t)W * H;
    const int c = tid & (GR_TW - 1), x = x0 + c;
#pragma unroll 1
    for (int z = 0; z < LAYERS; z++) {
        const float* snz = sn + z * NH * NWP;
        float* out = noise + z * n + x;
        double sq = 0.0;
        __syncthreads();  // the noise is complete; sr is free again
        if (R == 3) {
            // radius 3 (a 1 px grain blur, every stock here): four outputs of
            // a row a thread, then a column of ROWS outputs, each from a
            // register window
            constexpr int ROWS = gr_rows(TH);
            for (int idx = tid; idx < NH * (GR_TW / 4); idx += GR_THREADS) {
                const int r = idx / (GR_TW / 4), g = idx % (GR_TW / 4);
                float w[12], a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int t = 0; t < 3; t++) {
                    const float4 v = *reinterpret_cast<const float4*>(snz + r * NWP + 4 * g + 4 * t);
                    w[4 * t] = v.x;
                    w[4 * t + 1] = v.y;
                    w[4 * t + 2] = v.z;
                    w[4 * t + 3] = v.w;
                }
#pragma unroll
                for (int k = 0; k <= 6; k++)
#pragma unroll
                    for (int j = 0; j < 4; j++) a[j] = fmaf(w[j + k], tp.t[k], a[j]);
                *reinterpret_cast<float4*>(sr + r * GR_TW + 4 * g) = make_float4(a[0], a[1], a[2], a[3]);
            }
            __syncthreads();
            const int rb = tid / GR_TW * ROWS;
            float a[ROWS];
#pragma unroll
            for (int j = 0; j < ROWS; j++) a[j] = 0.0f;
#pragma unroll
            for (int m = 0; m < ROWS + 6; m++) {
                const float v = sr[(rb + m) * GR_TW + c];
#pragma unroll
                for (int j = 0; j < ROWS; j++)
                    if (m - j >= 0 && m - j <= 6) a[j] = fmaf(v, tp.t[m - j], a[j]);
            }
#pragma unroll
            for (int j = 0; j < ROWS; j++) {
                const int r = rb + j;
                if (r < TH && y0 + r < H && x < W) {
                    out[(size_t)(y0 + r) * W] = a[j];
                    sq += (double)a[j] * (double)a[j];
                }
            }
        } else {
            for (int idx = tid; idx < NH * GR_TW; idx += GR_THREADS) {
                const float* s = snz + (idx >> 7) * NWP + c;
                float acc = 0.0f;
                for (int k = 0; k <= 2 * R; k++) acc = fmaf(s[k], tp.t[k], acc);
                sr[idx] = acc;
            }
            __syncthreads();
            for (int r = tid >> 7; r < TH; r += GR_GROUPS) {
                if (y0 + r >= H || x >= W) continue;
                float acc = 0.0f;
                for (int k = 0; k <= 2 * R; k++) acc = fmaf(sr[(r + k) * GR_TW + c], tp.t[k], acc);
                out[(size_t)(y0 + r) * W] = acc;
                sq += (double)acc * (double)acc;
            }
        }
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
        if ((tid & 31) == 0) red[tid >> 5] = sq;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < GR_THREADS / 32; w++) t += red[w];
            partial[(size_t)z * gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x] = t;
        }
    }
}

// sums[layer] = sum of partial[layer][0 .. nb) in a fixed order (one block
// per layer): deterministic run to run.
__global__ void __launch_bounds__(1024) sum_partials_kernel(const double* __restrict__ partial, int nb,
                                                            double* __restrict__ sums) {
    __shared__ double red[1024];
    const double* p = partial + (size_t)blockIdx.x * nb;
    double a = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) a += p[i];
    red[threadIdx.x] = a;
    __syncthreads();
    for (int w = 512; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = red[0];
}

static size_t grain_tiles(int W, int H, int th) {
    return (size_t)((W + GR_TW - 1) / GR_TW) * ((H + th - 1) / th);
}

// Fewer tiles of full height than two an SM: no six layers to a block.
static bool grain_small(int W, int H) { return grain_tiles(W, H, GR_TH) < (size_t)sm_count() * 2; }

// Tile height of the blocks of up to three layers.  A block alone on its SM
// takes 4.9 + 0.38 TH us, two at once 1.7 times that, and of more each takes
// 0.65 of it after a run-in (fitted to 13 sizes from 32x32 to 24 MP at seven
// heights): the height of the least of that.  39 from about 2 MP on; below,
// 9 against 39 rows: 324x216 8.3 us against 19.3; 640x480, 18 rows: 11.7
// against 19.9; 1200x800, 28 rows: 27.0 against 33.3; 1296x864, 34 rows: 31.6
// against 34.0.
static int grain_rows(int W, int H) {
    const int heights[] = {GR_TH, 34, 28, 18, 9};
    int best = GR_TH;
    double least = 0.0;
    for (int th : heights) {
        const double per_sm = (double)grain_tiles(W, H, th) / sm_count();
        const double cost = (4.9 + 0.38 * th) * (per_sm <= 1.0 ? 1.0 : per_sm <= 2.0 ? 1.7 : 0.6 + 0.65 * per_sm);
        if (th == GR_TH || cost < least) {
            least = cost;
            best = th;
        }
    }
    return best;
}

// Doubles of scratch that grain_fields needs for its block sums.
size_t grain_partials(int W, int H, int layers) {
    const int th = grain_rows(W, H);
    return grain_tiles(W, H, layers >= 6 && !grain_small(W, H) && GR_TH6 < th ? GR_TH6 : th) * layers;
}

template <int LAYERS, int TH>
static int grain_launch(float* noise, int W, int H, uint64_t seed, int layer0, const Taps& tp, double* partial,
                        double* sums, cudaStream_t s) {
    const int NH = TH + 2 * tp.R, NWP = (GR_TW + 2 * tp.R + GR_RUN - 1) / GR_RUN * GR_RUN;
    const size_t smem = (size_t)(LAYERS * NH * NWP + gr_row_buffer(TH, tp.R) * GR_TW) * sizeof(float);
    IMOPS_CUDA_TRY(cudaFuncSetAttribute(grain_field_kernel<LAYERS, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem),
                   "cudaFuncSetAttribute(grain)");
    const dim3 g((W + GR_TW - 1) / GR_TW, (H + TH - 1) / TH);
    grain_field_kernel<LAYERS, TH><<<g, GR_THREADS, smem, s>>>(noise, W, H, seed, layer0, tp, partial);
    sum_partials_kernel<<<LAYERS, 1024, 0, s>>>(partial, (int)(g.x * g.y), sums);
    note_launch(2);
    return IMOPS_OK;
}

template <int LAYERS>
static int grain_launch_rows(int th, float* noise, int W, int H, uint64_t seed, int layer0, const Taps& tp,
                             double* partial, double* sums, cudaStream_t s) {
    switch (th) {
        case 9: return grain_launch<LAYERS, 9>(noise, W, H, seed, layer0, tp, partial, sums, s);
        case 18: return grain_launch<LAYERS, 18>(noise, W, H, seed, layer0, tp, partial, sums, s);
        case 28: return grain_launch<LAYERS, 28>(noise, W, H, seed, layer0, tp, partial, sums, s);
        case 34: return grain_launch<LAYERS, 34>(noise, W, H, seed, layer0, tp, partial, sums, s);
        default: return grain_launch<LAYERS, GR_TH>(noise, W, H, seed, layer0, tp, partial, sums, s);
    }
}

// Blurred grain fields of RNG layers layer0 .. layer0+layers-1 (planes
// noise[z * n]) and their sums of squares sums[z].  partial: scratch of
// grain_partials(W, H, layers) doubles.
int grain_fields(float* noise, int W, int H, uint64_t seed, int layer0, int layers, const Taps& tp, double* partial,
                 double* sums, cudaStream_t s) {
    if (tp.R > GR_MAXR) return fail(IMOPS_ERR_UNSUPPORTED_SIZE, "film: grain blur radius above 16 px");
    const size_t n = (size_t)W * H;
    const bool small = grain_small(W, H);
    const int th = grain_rows(W, H);
    for (int z = 0; z < layers;) {
        int rc, take;
        float* nz = noise + z * n;
        const int left = layers - z, l0 = layer0 + z;
        if (left >= 6 && tp.R <= 3 && !small) {  // six layers and a wider halo outgrow the shared memory
            take = 6;
            rc = grain_launch<6, GR_TH6>(nz, W, H, seed, l0, tp, partial, sums + z, s);
        } else if (left >= 3) {
            take = 3;
            rc = grain_launch_rows<3>(th, nz, W, H, seed, l0, tp, partial, sums + z, s);
        } else if (left == 2) {
            take = 2;
            rc = grain_launch_rows<2>(th, nz, W, H, seed, l0, tp, partial, sums + z, s);
        } else {
            take = 1;
            rc = grain_launch_rows<1>(th, nz, W, H, seed, l0, tp, partial, sums + z, s);
        }
        if (rc) return rc;
        z += take;
    }
    IMOPS_CUDA_TRY(cudaGetLastError(), "grain fields");
    return IMOPS_OK;
}

// 1 / the RMS of a grain field from its sum of squares
__device__ __forceinline__ float grain_norm(double sumsq, size_t n) {
    const double var = sumsq / (double)n;
    return var > 1e-12 ? (float)(1.0 / sqrt(var)) : 1.0f;
}

// D <- clamp(D + kappa*taper*sqrt(D(Dmax-D))*n*norm, 0, 1.05 Dmax)
__device__ __forceinline__ float grain_px(float d, float noise, float norm, float kappa, float dmax) {
    const float dens = fminf(fmaxf(d, 0.0f), dmax);
    const float taper = fminf(__fdiv_rn(dens, fmaf(0.02f, dmax, dens)), 1.0f);
    const float sd = __fmul_rn(taper, sqrtf(fmaxf(__fmul_rn(dens, __fsub_rn(dmax, dens)), 0.0f)));
    d = fmaf(__fmul_rn(__fmul_rn(kappa, sd), noise), norm, dens);
    return fminf(fmaxf(d, 0.0f), __fmul_rn(dmax, 1.05f));
}

__global__ void grain_apply_kernel(float* __restrict__ plane, const float* __restrict__ noise, size_t n,
                                   const double* __restrict__ sumsq, float kappa, float dmax) {
    const float norm = grain_norm(*sumsq, n);
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
        plane[p] = grain_px(plane[p], noise[p], norm, kappa, dmax);
}

// ---------------------------------------------------------------------------
// scan (densitometry.rs:13-73) on the 16-bin grid
//
// A masked stock's layers share one mask curve (the stock's orange mask), so
// the mask densities enter the scan as their sum over the layers: E + 1
// products a bin instead of 2 E, and one plane where only the sum is kept.
// The tables are kernel parameters as pairs of adjacent bins (2l, 2l+1) for
// the packed f32x2 FMA, read as constant-bank operands, and the layer count
// is a template argument so the densities stay in registers.

constexpr int NP16 = NB16 / 2;
template <int E>
struct Scan16 {
    float2 ne[E][NP16];  // -eps of each layer
    float2 nm[NP16];     // -meps
    float2 C2[3][NP16];
};

template <int E>
__device__ __forceinline__ void scan16_px(const Scan16<E>& c, const float (&D)[E], float M, float* o) {
    float2 acc[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const float2 mm = make_float2(M, M);
#pragma unroll
    for (int l = 0; l < NP16; l++) {
        float2 x = __fmul2_rn(mm, c.nm[l]);
#pragma unroll
        for (int e = 0; e < E; e++) x = __ffma2_rn(make_float2(D[e], D[e]), c.ne[e][l], x);
        const float2 t = make_float2(ex2_fast(x.x), ex2_fast(x.y));
#pragma unroll
        for (int k = 0; k < 3; k++) acc[k] = __ffma2_rn(c.C2[k][l], t, acc[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) o[k] = __fadd_rn(acc[k].x, acc[k].y);
}

// The scan as a step of its own, from a plane of image and one of mask densities
// a layer; a whole image is scanned by print_kernel.  A thread a pixel: 16
// exponentials and 8 (E + 4) packed FMAs against 8 E + 12 bytes.
template <int E>
__global__ void __launch_bounds__(256) scan16_kernel(const float* __restrict__ img, const float* __restrict__ mask,
                                                     size_t n, const __grid_constant__ Scan16<E> c,
                                                     float* __restrict__ rgb) {
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float D[E], M = 0.0f, o[3];
#pragma unroll
        for (int e = 0; e < E; e++) D[e] = __ldg(img + e * n + p);
#pragma unroll
        for (int e = 0; e < E; e++) M = __fadd_rn(M, __ldg(mask + e * n + p));
        scan16_px<E>(c, D, M, o);
        rgb[3 * p] = o[0];
        rgb[3 * p + 1] = o[1];
        rgb[3 * p + 2] = o[2];
    }
}

template <int E>
static Scan16<E> scan16_pairs(const ScanSpec16& S) {
    Scan16<E> c;
    for (int l = 0; l < NP16; l++) {
        for (int e = 0; e < E; e++) c.ne[e][l] = make_float2(-S.eps[e][2 * l], -S.eps[e][2 * l + 1]);
        c.nm[l] = make_float2(-S.meps[2 * l], -S.meps[2 * l + 1]);
        for (int k = 0; k < 3; k++) c.C2[k][l] = make_float2(S.C[2 * l][k], S.C[2 * l + 1][k]);
    }
    return c;
}

// Calls f with the layer count as a compile-time constant: the stocks have
// 1 (BwStub), 2 (TriX400), 3, 6 or 7 (FujiPro400H) emulsion layers.
template <class F>
int with_layers(int E, F f) {
    switch (E) {
        case 1: return f(std::integral_constant<int, 1>{});
        case 2: return f(std::integral_constant<int, 2>{});
        case 3: return f(std::integral_constant<int, 3>{});
        case 6: return f(std::integral_constant<int, 6>{});
        case 7: return f(std::integral_constant<int, 7>{});
    }
    return fail(IMOPS_ERR_INVALID_STOCK, "film: stocks have 1, 2, 3, 6 or 7 emulsion layers");
}

// invert_negative (invert.rs:36-108): the per-channel constants from the
// mid-grey negative and Dmin (mid_dmin, device memory), and one pixel.
struct Invert {
    float dmin[3], sh[3], g[3];
};
__device__ __forceinline__ float invert_curve(float inv, float sh) { return __fdiv_rn(inv, 1.0f + __fdiv_rn(inv, sh)); }
__device__ __forceinline__ Invert invert_constants(const float* __restrict__ mid_dmin) {
    const float eps = 1e-6f, HEAD = 8.0f, MG = 0.185f;
    Invert v;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        v.dmin[c] = fmaxf(mid_dmin[3 + c], eps);
        const float mt = fminf(fmaxf(__fdiv_rn(mid_dmin[c], v.dmin[c]), eps), 1.0f - eps);
        const float im = fmaxf(__fsub_rn(__fdiv_rn(1.0f, mt), 1.0f), 0.0f);
        v.sh[c] = fmaxf(__fmul_rn(im, HEAD), eps);
        v.g[c] = __fdiv_rn(MG, fmaxf(invert_curve(im, v.sh[c]), eps));
    }
    return v;
}
__device__ __forceinline__ void invert_px(const Invert& v, float (&o)[3]) {
    const float eps = 1e-6f, KEEP = 0.55f, FADE = 0.02f;
    float raw[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float t = fminf(fmaxf(__fdiv_rn(o[c], v.dmin[c]), eps), 1.0f);
        const float inv = fmaxf(__fsub_rn(__fdiv_rn(1.0f, t), 1.0f), 0.0f);
        raw[c] = fmaxf(__fmul_rn(v.g[c], invert_curve(inv, v.sh[c])), 0.0f);
    }
    const float y = fmaxf(dot3(0.2722287168f, raw[0], 0.6740817658f, raw[1], 0.0536895174f, raw[2]), 0.0f);
    const float k = y <= 0.0f ? 0.0f : (y >= FADE ? KEEP : __fmul_rn(KEEP, __fdiv_rn(y, FADE)));
#pragma unroll
    for (int c = 0; c < 3; c++) o[c] = fmaxf(fmaf(k, __fsub_rn(raw[c], y), y), 0.0f);
}

__global__ void invert_kernel(float* __restrict__ rgb, size_t n, const float* __restrict__ mid_dmin) {
    const Invert v = invert_constants(mid_dmin);
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
        float o[3] = {rgb[3 * p], rgb[3 * p + 1], rgb[3 * p + 2]};
        invert_px(v, o);
        for (int c = 0; c < 3; c++) rgb[3 * p + c] = o[c];
    }
}

// ---- adjacency, grain, scan and inversion in one pass ------------------------
// The last four steps of the model on a 64 x 32 tile: each layer's tile comes
// in with cp.async while the layer before is blurred (adjacency), its grain
// is added, and its densities stay in shared memory (a thread's own four
// pixels); when all layers are through, the thread scans its pixels and
// inverts them.  Bound by instruction issue (0.78 of its rate; six layers).  RC: the blur radius class (taps beyond the radius are zero:
// densities are finite, so they add nothing), 0 where the densities are
// final.  Same arithmetic as the steps one by one.  24 MP, six layers, grain:
// 0.73 ms against 2.1 (12 blur launches, 6 of the grain, the scan).
constexpr int PR_THREADS = 512, PR_ROWS = ft_rpt(PR_THREADS);
template <int E>
struct Print {
    Scan16<E> scan;
    float kappa[E], dmax[E];
    float beta;
    float taps[2 * 8 + 1];  // centred in the radius class
};
template <int RC>
constexpr int print_smem_floats(int E) {
    return (RC ? 2 * ft_tile_floats(RC) + ft_row_floats(RC) : 0) + E * FT_W * FT_H;
}

template <int E, int RC>
__global__ void __launch_bounds__(PR_THREADS, 2) print_kernel(const float* __restrict__ dens,
                                                              const float* __restrict__ mask,
                                                              const float* __restrict__ noise,
                                                              const double* __restrict__ sums,
                                                              const float* __restrict__ mid_dmin, int W, int H,
                                                              const __grid_constant__ Print<E> c,
                                                              float* __restrict__ rgb) {
    extern __shared__ __align__(16) float ftsm[];
    __shared__ float norm[E];
    __shared__ Invert inv;
    constexpr int TILE = RC ? ft_tile_floats(RC) : 0;
    float* rows = ftsm + 2 * TILE;
    const int x0 = blockIdx.x * FT_W, y0 = blockIdx.y * FT_H;
    const int tx = threadIdx.x % FT_W, rb = (int)threadIdx.x / FT_W * PR_ROWS;
    float* own = ftsm + (RC ? 2 * TILE + ft_row_floats(RC) : 0) + threadIdx.x;  // [layer][row][thread]
    const size_t n = (size_t)W * H;
    const int x = x0 + tx;
    // this thread's pixels, clamped into the image (their results are not stored)
    size_t px[PR_ROWS];
#pragma unroll
    for (int r = 0; r < PR_ROWS; r++) px[r] = (size_t)min(y0 + rb + r, H - 1) * W + min(x, W - 1);
    if (noise && threadIdx.x < E) norm[threadIdx.x] = grain_norm(sums[threadIdx.x], n);
    if (mid_dmin && threadIdx.x == 32) inv = invert_constants(mid_dmin);
    FtCopy copy;
    if constexpr (RC > 0) {
        copy = ft_copy(dens, x0, y0, RC, W, H);
        ft_load<PR_THREADS>(ftsm, dens, copy, y0, RC, W, H);
        ft_commit();
    } else {
        __syncthreads();  // norm, inv
    }
#pragma unroll 1
    for (int e = 0; e < E; e++) {
        float nz[PR_ROWS], d[PR_ROWS];
#pragma unroll
        for (int r = 0; r < PR_ROWS; r++) nz[r] = noise ? __ldg(noise + e * n + px[r]) : 0.0f;
        if constexpr (RC > 0) {
            ft_wait<0>();
            __syncthreads();  // this layer's tile is complete; the row buffer and the other tile are free
            if (e + 1 < E) {
                ft_load<PR_THREADS>(ftsm + ((e + 1) & 1) * TILE, dens + (e + 1) * n, copy, y0, RC, W, H);
                ft_commit();
            }
            const float* tile = ftsm + (e & 1) * TILE;
            float v[PR_ROWS];
            ft_rows<PR_THREADS, RC>(tile, rows, c.taps);
            __syncthreads();
            ft_cols<RC>(rows, tx, rb, c.taps, v);
#pragma unroll
            for (int r = 0; r < PR_ROWS; r++)
                d[r] = adjacency_px(tile[(RC + rb + r) * ft_stride(RC) + ft_pad(RC) + RC + tx], v[r], c.beta);
        } else {
#pragma unroll
            for (int r = 0; r < PR_ROWS; r++) d[r] = __ldg(dens + e * n + px[r]);
        }
        if (noise && c.kappa[e] > 0.0f && c.dmax[e] > 0.0f) {
#pragma unroll
            for (int r = 0; r < PR_ROWS; r++) d[r] = grain_px(d[r], nz[r], norm[e], c.kappa[e], c.dmax[e]);
        }
#pragma unroll
        for (int r = 0; r < PR_ROWS; r++) own[(e * PR_ROWS + r) * PR_THREADS] = d[r];
    }
    if (x >= W) return;
#pragma unroll 1
    for (int r = 0; r < PR_ROWS; r++) {
        if (y0 + rb + r >= H) break;
        const size_t p = (size_t)(y0 + rb + r) * W + x;
        float D[E], o[3];
#pragma unroll
        for (int e = 0; e < E; e++) D[e] = own[(e * PR_ROWS + r) * PR_THREADS];
        scan16_px<E>(c.scan, D, __ldg(mask + p), o);
        if (mid_dmin) invert_px(inv, o);
        rgb[3 * p] = o[0];
        rgb[3 * p + 1] = o[1];
        rgb[3 * p + 2] = o[2];
    }
}

// Exposure of the layers and their local scatter on a 64 x 32 tile: the basis
// weights of the tile and its halo once, then each layer formed from them,
// blurred and mixed, so the layers reach memory once, scattered.  Bound by
// instruction issue (0.68 of its rate) and the barriers between its passes.
// 24 MP, six layers, radius 2: 0.56 ms against 1.5 (an exposure pass and 12 blur
// launches).
constexpr int EX_THREADS = 512, EX_ROWS = ft_rpt(EX_THREADS), EX_MAXR = 8;
__host__ __device__ constexpr int expose_smem_floats(int R) { return 5 * ft_tile_floats(R) + ft_row_floats(R); }

__global__ void __launch_bounds__(EX_THREADS, 2) expose_scatter_kernel(const float* __restrict__ rgb, int W, int H,
                                                                       const __grid_constant__ ExposeSpec X,
                                                                       const __grid_constant__ Taps tp, float keep,
                                                                       float mix, float* __restrict__ planes) {
    extern __shared__ __align__(16) float ftsm[];
    const int R = tp.R, tile = ft_tile_floats(R), SW = ft_stride(R), NH = FT_H + 2 * R;
    float* rows = ftsm + 5 * tile;
    const int x0 = blockIdx.x * FT_W, y0 = blockIdx.y * FT_H;
    const int tx = threadIdx.x % FT_W, rb = (int)threadIdx.x / FT_W * EX_ROWS, lane = threadIdx.x & 31;
    const size_t n = (size_t)W * H;
    int xs[FT_COLS];
#pragma unroll
    for (int t = 0; t < FT_COLS; t++) xs[t] = 3 * reflect(x0 - R - ft_pad(R) + lane + 32 * t, W);
    for (int r = (int)threadIdx.x >> 5; r < NH; r += EX_THREADS / 32) {
        const float* src = rgb + (size_t)reflect(y0 - R + r, H) * W * 3;
#pragma unroll
        for (int t = 0; t < FT_COLS; t++) {
            const int q = 32 * t + lane;
            if (q < SW) {
                const float* s = src + xs[t];
                float w[3];
                basis_weights(X, __ldg(s), __ldg(s + 1), __ldg(s + 2), w);
#pragma unroll
                for (int k = 0; k < 3; k++) ftsm[(2 + k) * tile + r * SW + q] = w[k];
            }
        }
    }
    __syncthreads();
    const int x = x0 + tx;
#pragma unroll 1
    for (int e = 0; e < X.E; e++) {
        float* s = ftsm + (e & 1) * tile;  // free: its readers passed the barrier in the layer between
        for (int i = threadIdx.x; i < tile; i += EX_THREADS) {
            const float w[3] = {ftsm[2 * tile + i], ftsm[3 * tile + i], ftsm[4 * tile + i]};
            s[i] = layer_exposure(X, w, e);
        }
        __syncthreads();
        float v[EX_ROWS];
        ft_blur<EX_THREADS, EX_MAXR>(s, rows, tx, rb, tp, v);
#pragma unroll
        for (int r = 0; r < EX_ROWS; r++) {
            const int y = y0 + rb + r;
            if (x < W && y < H)
                planes[e * n + (size_t)y * W + x] =
                    mix_px(s[(R + rb + r) * SW + ft_pad(R) + R + tx], v[r], keep, mix);
        }
    }
}

__global__ void fill_kernel(float* __restrict__ p, int n, float v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// mean RGB of a small buffer in f64 (invert.rs:111-125) into out[0..2], dmin into out[3..5]; one block
__global__ void mean_rgb_kernel(const float* __restrict__ rgb, int n, float dmin0, float dmin1, float dmin2,
                                float* __restrict__ out) {
    __shared__ double s[3][256];
    double a[3] = {0, 0, 0};
    for (int p = threadIdx.x; p < n; p += blockDim.x)
        for (int c = 0; c < 3; c++) a[c] += (double)rgb[3 * p + c];
    for (int c = 0; c < 3; c++) s[c][threadIdx.x] = a[c];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int c = 0; c < 3; c++) s[c][threadIdx.x] += s[c][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        for (int c = 0; c < 3; c++) out[c] = (float)(s[c][0] / (double)n);
        out[3] = dmin0;
        out[4] = dmin1;
        out[5] = dmin2;
    }
}

// ---------------------------------------------------------------------------
// baseline preset: fused halation column pass + logistic curves + grain +
// 81-bin scan.  Each block owns a 32x64 pixel tile and stages the rows of
// the halation row-pass output it needs (64 + 2*64) in shared memory.

// The 81-bin tables as pairs of adjacent bins (2l, 2l+1) for the packed f32x2
// FMA of sm_100 (FFMA2: two lanes per instruction), plus the last bin:
//   ne[e][l]  = -(eps_e(2l), eps_e(2l+1))   (negated: the sum is -d directly)
//   C2[c][l]  = (C(2l)[c], C(2l+1)[c])
// tap2[k] = (taps[k], taps[k-1]) with zero outside [0, 2R] feeds the column
// pass two outputs (rows j, j+1) per instruction; each output still sums its
// taps in ascending order.
constexpr int NP81 = NB81 / 2;  // 40 pairs + bin 80
struct Pairs81 {
    float2 ne[3][NP81];
    float2 C2[3][NP81];
    float ne_last[3], C_last[3];
};

struct Base81 {
    BaselineSpec B;
    ExposeSpec X;
    Pairs81 P;
    float2 tap2[2 * HAL_R + 2];
};

// One thread per OUT consecutive rows of a column: the halation column pass
// (register sliding window, tap pairs as parameter-bank operands, ascending
// tap order as in blur_cols), then per pixel the exposure of the three layers
// from its RGB, the logistic curves, grain and the 81-bin scan with its
// tables as parameter-bank operands; the result replaces the pixel's RGB
// (each pixel is read, a step ahead, and written by the same thread).  Four
// blocks an SM (64 registers a thread): the scan is bound by the MUFU, and
// 32 warps keep more of its exponentials in flight than 24.  Sixteen rows a
// thread; four where the blocks of sixteen would be fewer than three an SM,
// which leaves SMs short of warps and the busiest with twice the mean work:
// 640x480 29.6 -> 19.6 us, 1200x800 45.3 -> 37.8, 1536x1024 (2.6 blocks an SM)
// 58.9 -> 55.4, but 2048x1365 (4.8) 87.2 -> 90.6 and 6048x4024 626 -> 725 (the
// window's run-in, 128 rows for 32 instead of 128).
constexpr int SCAN_OUT_SMALL = 4;
template <int OUT>
__global__ void __launch_bounds__(R64_COL_TW * R64_COL_GROUPS, 4) scan81_fused_kernel(
    const float* __restrict__ hr, const float* __restrict__ noise, const double* __restrict__ sumsq, int W, int H,
    const __grid_constant__ Base81 c, float* __restrict__ rgb) {
    static_assert(HAL_R == R64, "the fused scan's column pass is the radius-64 window");
    static_assert(OUT % 2 == 0, "column outputs go in pairs");
    __shared__ float s[((R64_COL_GROUPS * OUT) + 2 * HAL_R) * R64_COL_TW];
    const int x0 = blockIdx.x * R64_COL_TW, y0 = blockIdx.y * (R64_COL_GROUPS * OUT);
    const int tx = threadIdx.x, ty = threadIdx.y, x = x0 + tx;
    if (x < W) stage_col_window<(R64_COL_GROUPS * OUT)>(s, hr, W, H, x, y0, tx, ty);
    __syncthreads();
    if (x >= W) return;
    const size_t n = (size_t)W * H;
    float norm[3] = {1.f, 1.f, 1.f};
    if (c.B.grain_sigma > 0.0f)
        for (int e = 0; e < 3; e++) {
            double var = sumsq[e] / (double)n;
            norm[e] = var > 1e-12 ? (float)(1.0 / sqrt(var)) : 1.0f;
        }
    const int rb = ty * OUT;
    // bs[q] = (output row 2q, output row 2q+1); at window row m the pair takes
    // taps m-2q and m-2q-1
    float2 bs[OUT / 2];
#pragma unroll
    for (int q = 0; q < OUT / 2; q++) bs[q] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int m = 0; m < OUT + 2 * HAL_R; m++) {
        const float v = s[(rb + m) * R64_COL_TW + tx];
        const float2 vv = make_float2(v, v);
#pragma unroll
        for (int q = 0; q < OUT / 2; q++) {
            const int k = m - 2 * q;
            if (k >= 0 && k <= 2 * HAL_R + 1) bs[q] = __ffma2_rn(vv, c.tap2[k], bs[q]);
        }
    }
    // Two pixels (rows j and j+1 of the column) a step: each table pair is
    // fetched once for both, and the next step's RGB and noise are loaded
    // while this step is scanned, so the global-load latency hides behind
    // the 81-bin loop.  Each pixel's arithmetic is unchanged.
    static_assert(OUT % 2 == 0, "pixels go in pairs");
    const bool grain = c.B.grain_sigma > 0.0f;
    float na[2][3], nz[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    auto fetch = [&](int jj) {  // rows jj, jj+1 (clamped to the image)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const size_t pp = (size_t)min(y0 + rb + jj + u, H - 1) * W + x;
#pragma unroll
            for (int e = 0; e < 3; e++) {
                na[u][e] = rgb[3 * pp + e];
                if (grain) nz[u][e] = noise[e * n + pp];
            }
        }
    };
    fetch(0);
#pragma unroll 1
    for (int j = 0; j < OUT; j += 2) {
        const int y = y0 + rb + j;
        if (y >= H) break;
        float ca[2][3], cz[2][3];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float w[3];
            basis_weights(c.X, na[u][0], na[u][1], na[u][2], w);
#pragma unroll
            for (int e = 0; e < 3; e++) {
                ca[u][e] = layer_exposure(c.X, w, e);
                cz[u][e] = nz[u][e];
            }
        }
        if (j + 2 < OUT && y + 2 < H) fetch(j + 2);
        float bsum[2] = {bs[0].x, bs[0].y};
#pragma unroll
        for (int q = 0; q < OUT / 2; q++)
            if (2 * q == j) {
                bsum[0] = bs[q].x;
                bsum[1] = bs[q].y;
            }
        float D[2][3];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int e = 0; e < 3; e++) {
                const float E = ca[u][e] + c.B.hal_strength * c.B.bleed[e] * bsum[u];
                D[u][e] = curve_density(E, c.B.dmax[e], c.B.k[e], c.B.x0[e]);
                if (grain) D[u][e] += c.B.grain_sigma * cz[u][e] * norm[e];
            }
        float2 d[2][3], o[2][3];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int e = 0; e < 3; e++) {
                d[u][e] = make_float2(D[u][e], D[u][e]);
                o[u][e] = make_float2(0.f, 0.f);
            }
#pragma unroll
        for (int l = 0; l < NP81; l++) {
            const float2 n0 = c.P.ne[0][l], n1 = c.P.ne[1][l], n2 = c.P.ne[2][l];
            const float2 c0 = c.P.C2[0][l], c1 = c.P.C2[1][l], c2 = c.P.C2[2][l];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                float2 xd = __fmul2_rn(d[u][0], n0);
                xd = __ffma2_rn(d[u][1], n1, xd);
                xd = __ffma2_rn(d[u][2], n2, xd);
                const float2 t = make_float2(ex2_fast(xd.x), ex2_fast(xd.y));
                o[u][0] = __ffma2_rn(c0, t, o[u][0]);
                o[u][1] = __ffma2_rn(c1, t, o[u][1]);
                o[u][2] = __ffma2_rn(c2, t, o[u][2]);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (y + u >= H) break;
            float xl = D[u][0] * c.P.ne_last[0];
            xl = fmaf(D[u][1], c.P.ne_last[1], xl);
            xl = fmaf(D[u][2], c.P.ne_last[2], xl);
            const float tl = ex2_fast(xl);
            const size_t p = (size_t)(y + u) * W + x;
            rgb[3 * p] = fmaf(c.P.C_last[0], tl, o[u][0].x + o[u][0].y);
            rgb[3 * p + 1] = fmaf(c.P.C_last[1], tl, o[u][1].x + o[u][1].y);
            rgb[3 * p + 2] = fmaf(c.P.C_last[2], tl, o[u][2].x + o[u][2].y);
        }
    }
}

// ---------------------------------------------------------------------------
// The 81-bin scan on the tensor cores (tcgen05, sm_100a): the same fused
// kernel (halation column pass, logistic curves, grain) with the two spectral
// contractions as BF16 MMAs with FP32 accumulation and a hi/lo split of both
// operands, per tile of 128 pixels (one warpgroup, one TMEM lane a pixel):
//   MMA1  x[128 x 96] = A1[128 x 16] . B1[96 x 16]^T      (A1, B1 in SMEM)
//         A1 row = (Dh, Dl, Dh, Dl) of the three layer densities, B1 row of
//         bin l = (eh, eh, el, el) of -eps(l) (log2 units), so
//         x = (Dh + Dl) . (eh + el) = -d(l) to f32 accuracy;
//   T = 2^x per bin (MUFU), split into bf16 T = Th + Tl, written over x in TMEM;
//   MMA2  rgb[128 x 16] += Th . Ch + Th . Cl + Tl . Ch    (A from TMEM, B in SMEM)
//         over six K-blocks of 16 bins (81 bins padded to 96 with zeros).
// Dropping Tl . Cl and bf16 rounding leave about 2^-17 relative per term.
namespace tc {

constexpr int NBP = 96;                   // bins padded to the MMA's granularity
constexpr uint32_t SBO_K16 = 256;         // K = 16 tiles: two 128-byte K-groups per 8-row group
constexpr uint32_t SBO_K96 = 1536;        // K = 96 tiles: twelve K-groups per 8-row group
constexpr int B1_WORDS = NBP * 16 / 2;    // 96 bins x 16 bf16
constexpr int B2_WORDS = 16 * NBP / 2;    // 16 channel rows (3 used) x 96 bins

// Byte offset of bf16 element (row r, k) in a K-major tile without swizzle:
// core matrices of 8 rows x 16 bytes, K-groups 128 bytes apart (LBO), 8-row
// groups `sbo` apart.
__host__ __device__ __forceinline__ uint32_t cm_off(int r, int k, uint32_t sbo) {
    return (uint32_t)(r >> 3) * sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(r & 7) * 16u + (uint32_t)(k & 7) * 2u;
}

// B operands, already in their shared-memory layout
struct Tables {
    uint32_t b1[B1_WORDS];
    uint32_t b2h[B2_WORDS];
    uint32_t b2l[B2_WORDS];
};

// dynamic shared memory (bytes)
constexpr uint32_t WIN_BYTES = (R64_COL_TH + 2 * HAL_R) * R64_COL_TW * 4;
constexpr uint32_t OFF_TAB = WIN_BYTES;
constexpr uint32_t OFF_B1 = OFF_TAB, OFF_B2H = OFF_B1 + B1_WORDS * 4, OFF_B2L = OFF_B2H + B2_WORDS * 4;
constexpr uint32_t OFF_A1 = OFF_B2L + B2_WORDS * 4;  // two warpgroups x 128 rows x 16 bf16
constexpr uint32_t OFF_BAR = OFF_A1 + 2 * 4096;      // four mbarriers
constexpr uint32_t OFF_SLOT = OFF_BAR + 32;          // TMEM base address
constexpr uint32_t SMEM_USED = OFF_SLOT + 16;
// Requested per CTA: at most two CTAs an SM, whose 2 x 256 TMEM columns fit
// the SM's 512, so no CTA waits in tcgen05.alloc for another to finish.
constexpr uint32_t SMEM_REQ = 80 * 1024;
static_assert(SMEM_USED <= SMEM_REQ && 3 * SMEM_REQ > 228 * 1024, "two CTAs an SM");

// instruction descriptors: BF16 A and B (K-major), FP32 D, M = 128
constexpr uint32_t idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
constexpr uint32_t IDESC_X = idesc(NBP), IDESC_RGB = idesc(16);

// try_wait suspends the warp until the phase completes or about SUSPEND_NS
// pass; after WAIT_LIMIT tries (about a second) the MMA is declared lost
constexpr int WAIT_LIMIT = 1 << 10;
constexpr uint32_t SUSPEND_NS = 1000000;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, no swizzle, LBO 128 bytes
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
                 ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(acc));
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
                 ::"r"(d), "r"(a), "l"(b), "r"(id), "r"(acc));
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for phase `parity` of an mbarrier: false when it gave up.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < WAIT_LIMIT; it++) {
        uint32_t ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok) : "r"(bar), "r"(parity), "r"(SUSPEND_NS) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void wg_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

__device__ __forceinline__ void ld16(uint32_t ta, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(ta));
}
__device__ __forceinline__ void ld4(uint32_t ta, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(ta));
}
__device__ __forceinline__ void st8(uint32_t ta, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(ta), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// bf16x2 of (a, b), round to nearest: a in the low half (the even K index)
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
// hi = bf16(a), bf16(b); lo = bf16 of what hi leaves out
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t& hi, uint32_t& lo) {
    hi = pack_bf16(a, b);
    lo = pack_bf16(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u));
}

}  // namespace tc

struct Base81TC {
    BaselineSpec B;
    ExposeSpec X;
    float2 tap2[2 * HAL_R + 2];
    tc::Tables T;
};

// Lost MMA completions (a bounded wait that gave up), counted across launches.
__device__ unsigned g_tc_timeouts = 0;

__global__ void __launch_bounds__(R64_COL_TW * R64_COL_GROUPS, 2) scan81_tc_kernel(
    const float* __restrict__ hr, const float* __restrict__ noise, const double* __restrict__ sumsq, int W, int H,
    const __grid_constant__ Base81TC c, float* __restrict__ rgb) {
    using namespace tc;
    static_assert(R64_COL_GROUPS == 8, "two warpgroups of four warps");
    extern __shared__ __align__(1024) uint8_t dsm[];
    float* s = reinterpret_cast<float*>(dsm);
    const int x0 = blockIdx.x * R64_COL_TW, y0 = blockIdx.y * R64_COL_TH;
    const int tx = threadIdx.x, ty = threadIdx.y, x = x0 + tx, tid = ty * 32 + tx;
    const int g = ty >> 2;     // warpgroup
    const int row = tid & 127; // this thread's MMA row (TMEM lane)
    const uint32_t sb = smem_u32(dsm);
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&c.T);
        uint32_t* dst = reinterpret_cast<uint32_t*>(dsm + OFF_TAB);
        for (int i = tid; i < (int)(sizeof(Tables) / 4); i += blockDim.x * blockDim.y) dst[i] = src[i];
    }
    if (x < W) stage_col_window<R64_COL_TH>(s, hr, W, H, x, y0, tx, ty);
    uint32_t* slot = reinterpret_cast<uint32_t*>(dsm + OFF_SLOT);
    if (tid == 0) {
        for (int i = 0; i < 4; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sb + OFF_BAR + 8 * i));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (ty == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(sb + OFF_SLOT));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tables are read by the MMAs
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tm = *slot + (uint32_t)(g * 128);                // this warpgroup's 128 columns
    const uint32_t tl = tm + (((uint32_t)(ty & 3) * 32u) << 16);    // this warp's 32 lanes
    const uint32_t bar_x = sb + OFF_BAR + 16 * g, bar_rgb = bar_x + 8;
    const uint32_t a1 = sb + OFF_A1 + 4096u * g;
    uint8_t* a1p = dsm + OFF_A1 + 4096u * g;

    const size_t n = (size_t)W * H;
    float norm[3] = {1.f, 1.f, 1.f};
    if (c.B.grain_sigma > 0.0f)
        for (int e = 0; e < 3; e++) {
            double var = sumsq[e] / (double)n;
            norm[e] = var > 1e-12 ? (float)(1.0 / sqrt(var)) : 1.0f;
        }
    const int rb = ty * R64_COL_OUT;
    float2 bs[R64_COL_OUT / 2];
#pragma unroll
    for (int q = 0; q < R64_COL_OUT / 2; q++) bs[q] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int m = 0; m < R64_COL_OUT + 2 * HAL_R; m++) {
        const float v = s[(rb + m) * R64_COL_TW + tx];
        const float2 vv = make_float2(v, v);
#pragma unroll
        for (int q = 0; q < R64_COL_OUT / 2; q++) {
            const int k = m - 2 * q;
            if (k >= 0 && k <= 2 * HAL_R + 1) bs[q] = __ffma2_rn(vv, c.tap2[k], bs[q]);
        }
    }
    const bool grain = c.B.grain_sigma > 0.0f;
    const bool xin = x < W;
    // Per step j (row y0 + rb + j of every warp: 128 pixels a warpgroup) the
    // MMAs of one step overlap the CUDA-core work of its neighbours: MMA2 of
    // step j runs while the densities of step j+1 are formed, MMA1 of step
    // j+1 while step j's pixels are stored.  RGB and noise are loaded a step
    // ahead (each pixel is read and written by the same thread).
    float la[3] = {0.f, 0.f, 0.f}, lz[3] = {0.f, 0.f, 0.f};  // inputs of the next step
    auto load_inputs = [&](int jj) {
        const int yy = y0 + rb + jj;
        if (xin && yy < H && jj < R64_COL_OUT) {
            const size_t p = (size_t)yy * W + x;
#pragma unroll
            for (int e = 0; e < 3; e++) {
                la[e] = rgb[3 * p + e];
                lz[e] = grain ? noise[e * n + p] : 0.0f;
            }
        }
    };
    // densities of step jj into A1 (k 0..11 = Dh0 Dh1 Dh2 Dl0 Dl1 Dl2 Dh0 Dh1
    // Dh2 Dl0 Dl1 Dl2, 12..15 zero), from the inputs loaded for it
    auto write_a1 = [&](int jj) {
        const int yy = y0 + rb + jj;
        float D[3] = {0.0f, 0.0f, 0.0f};
        if (xin && yy < H) {
            float bsum = bs[0].x;
#pragma unroll
            for (int q = 0; q < R64_COL_OUT / 2; q++) {
                if (2 * q == jj) bsum = bs[q].x;
                if (2 * q + 1 == jj) bsum = bs[q].y;
            }
            float w[3];
            basis_weights(c.X, la[0], la[1], la[2], w);
#pragma unroll
            for (int e = 0; e < 3; e++) {
                const float E = layer_exposure(c.X, w, e) + c.B.hal_strength * c.B.bleed[e] * bsum;
                D[e] = curve_density(E, c.B.dmax[e], c.B.k[e], c.B.x0[e]);
                if (grain) D[e] += c.B.grain_sigma * lz[e] * norm[e];
            }
        }
        uint32_t h01, l01, h2, l2;
        split_bf16(D[0], D[1], h01, l01);
        split_bf16(D[2], 0.0f, h2, l2);
        const uint32_t w0 = h01, w1 = (h2 & 0xFFFFu) | (l01 << 16), w2 = (l01 >> 16) | (l2 << 16);
        *reinterpret_cast<uint4*>(a1p + cm_off(row, 0, SBO_K16)) = make_uint4(w0, w1, w2, w0);
        *reinterpret_cast<uint4*>(a1p + cm_off(row, 8, SBO_K16)) = make_uint4(w1, w2, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    bool alive = true;
    auto wait_for = [&](uint32_t bar, uint32_t parity) {
        if (alive && !bar_wait(bar, parity)) {
            alive = false;
            atomicAdd(&g_tc_timeouts, 1u);
        }
        fence_after();
    };

    load_inputs(0);
    write_a1(0);
    load_inputs(1);
    wg_sync(1 + g);
    if (row == 0) {
        fence_after();
        mma_ss(tm, sdesc(a1, SBO_K16), sdesc(sb + OFF_B1, SBO_K16), IDESC_X, 0u);
        commit(bar_x);
    }
#pragma unroll 1
    for (int j = 0; j < R64_COL_OUT; j++) {
        const uint32_t parity = (uint32_t)j & 1u;
        wait_for(bar_x, parity);
        // T = 2^x per bin, split to bf16 hi/lo over the same columns: K-block
        // q (bins 16q .. 16q+15) keeps its hi words in columns 16q .. 16q+7
        // and its lo words in 16q+8 .. 16q+15.  Three K-blocks a batch of
        // TMEM loads, one wait each.
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[3][16];
#pragma unroll
            for (int q = 0; q < 3; q++) ld16(tl + 16u * (3 * h + q), v[q]);
            wait_ld();
#pragma unroll
            for (int q = 0; q < 3; q++) {
                uint32_t hw[8], lw[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int b0 = 16 * (3 * h + q) + 2 * i;
                    const float t0 = b0 < NB81 ? ex2_fast(__uint_as_float(v[q][2 * i])) : 0.0f;
                    const float t1 = b0 + 1 < NB81 ? ex2_fast(__uint_as_float(v[q][2 * i + 1])) : 0.0f;
                    split_bf16(t0, t1, hw[i], lw[i]);
                }
                st8(tl + 16u * (3 * h + q), hw);
                st8(tl + 16u * (3 * h + q) + 8u, lw);
            }
        }
        wait_st();
        fence_before();
        wg_sync(1 + g);
        if (row == 0 && alive) {
            fence_after();
#pragma unroll
            for (int q = 0; q < NBP / 16; q++) {
                const uint64_t bh = sdesc(sb + OFF_B2H + 256u * q, SBO_K96), bl = sdesc(sb + OFF_B2L + 256u * q, SBO_K96);
                mma_ts(tm + NBP, tm + 16u * q, bh, IDESC_RGB, q > 0 ? 1u : 0u);
                mma_ts(tm + NBP, tm + 16u * q, bl, IDESC_RGB, 1u);
                mma_ts(tm + NBP, tm + 16u * q + 8u, bh, IDESC_RGB, 1u);
            }
            commit(bar_rgb);
        }
        // next step's densities while MMA2 runs (A1 is free: MMA1 of this step is done)
        if (j + 1 < R64_COL_OUT) {
            write_a1(j + 1);
            load_inputs(j + 2);
        }
        wait_for(bar_rgb, parity);
        uint32_t o[4];
        ld4(tl + NBP, o);
        wait_ld();
        fence_before();
        wg_sync(1 + g);  // A1 of the next step written; this step's rgb read from TMEM
        if (j + 1 < R64_COL_OUT && row == 0 && alive) {
            fence_after();
            mma_ss(tm, sdesc(a1, SBO_K16), sdesc(sb + OFF_B1, SBO_K16), IDESC_X, 0u);
            commit(bar_x);
        }
        const int y = y0 + rb + j;
        if (xin && y < H) {
            const size_t p = (size_t)y * W + x;
            rgb[3 * p] = __uint_as_float(o[0]);
            rgb[3 * p + 1] = __uint_as_float(o[1]);
            rgb[3 * p + 2] = __uint_as_float(o[2]);
        }
    }
    __syncthreads();
    fence_after();
    if (ty == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(*slot));
}

// Host: bf16 of an f32, round to nearest even (finite values)
static uint16_t host_bf16(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
static float host_bf16_value(uint16_t h) {
    uint32_t u = (uint32_t)h << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

// Host: the tensor-core scan's B operands in their shared-memory layout.
static void build_base81_tc(const Stock& st, Base81TC* hp) {
    std::memset(hp, 0, sizeof(*hp));
    hp->B = st.base;
    hp->X = st.expose;
    for (int k = 0; k <= 2 * HAL_R + 1; k++)
        hp->tap2[k] = make_float2(k <= 2 * HAL_R ? st.hal_taps[k] : 0.0f, k >= 1 ? st.hal_taps[k - 1] : 0.0f);
    const ScanSpec81& S = st.scan81;
    auto put = [](uint32_t* words, uint32_t byte_off, uint16_t v) {
        reinterpret_cast<uint16_t*>(words)[byte_off / 2] = v;
    };
    for (int l = 0; l < NB81; l++)
        for (int e = 0; e < 3; e++) {
            const float ne = -S.eps[e][l];
            const uint16_t hi = host_bf16(ne), lo = host_bf16(ne - host_bf16_value(hi));
            // row l of B1 against A1's (Dh, Dl, Dh, Dl): (eh, eh, el, el)
            put(hp->T.b1, tc::cm_off(l, e, tc::SBO_K16), hi);
            put(hp->T.b1, tc::cm_off(l, 3 + e, tc::SBO_K16), hi);
            put(hp->T.b1, tc::cm_off(l, 6 + e, tc::SBO_K16), lo);
            put(hp->T.b1, tc::cm_off(l, 9 + e, tc::SBO_K16), lo);
        }
    for (int ch = 0; ch < 3; ch++)
        for (int l = 0; l < NB81; l++) {
            const float cv = S.C[l][ch];
            const uint16_t hi = host_bf16(cv), lo = host_bf16(cv - host_bf16_value(hi));
            put(hp->T.b2h, tc::cm_off(ch, l, tc::SBO_K96), hi);
            put(hp->T.b2l, tc::cm_off(ch, l, tc::SBO_K96), lo);
        }
}

// Host: the pair tables of the 81-bin scan and halation taps.
static void build_base81(const Stock& st, Base81* hp) {
    hp->B = st.base;
    hp->X = st.expose;
    const ScanSpec81& S = st.scan81;
    for (int e = 0; e < 3; e++) {
        for (int l = 0; l < NP81; l++) hp->P.ne[e][l] = make_float2(-S.eps[e][2 * l], -S.eps[e][2 * l + 1]);
        hp->P.ne_last[e] = -S.eps[e][NB81 - 1];
    }
    for (int ch = 0; ch < 3; ch++) {
        for (int l = 0; l < NP81; l++) hp->P.C2[ch][l] = make_float2(S.C[2 * l][ch], S.C[2 * l + 1][ch]);
        hp->P.C_last[ch] = S.C[NB81 - 1][ch];
    }
    for (int k = 0; k <= 2 * HAL_R + 1; k++)
        hp->tap2[k] = make_float2(k <= 2 * HAL_R ? st.hal_taps[k] : 0.0f, k >= 1 ? st.hal_taps[k - 1] : 0.0f);
}

// ---------------------------------------------------------------------------
// workspace (per device+stream, grows on demand)

StreamCache g_ws("film workspace");

int workspace(cudaStream_t s, size_t bytes, void** out) { return g_ws.get(s, bytes, out); }

int grid_for(size_t n) {
    size_t g = (n + 255) / 256, cap = (size_t)sm_count() * 8;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

int grid_for_n(size_t n) { return grid_for(n); }

// Bump allocator over the workspace.
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

size_t ref_workspace_bytes(int W, int H, int E) {
    // planes(E) + inh(E) + mask sum(1) + tmp(1) + bounce(1) + grain partials + LUT + sums
    return (size_t)(2 * E + 3) * W * H * 4 + grain_partials(W, H, E) * 8 + MAXE * LUTN * 4 + 64 * 1024;
}

// The reference model's stages (film/mod.rs:77-129), each on the stock's E
// planar layers; run_reference chains them, and the imops_film_* entry
// points expose them one by one.
//   expose: ACEScg RGB -> absorbed exposure per layer (exposure/mod.rs:45-137,
//     absorption.rs:24-108)
int stage_expose(const float* rgb, int W, int H, const Stock& st, float* planes, cudaStream_t s) {
    const size_t n = (size_t)W * H;
    expose_kernel<<<grid_for(n), 256, 0, s>>>(rgb, n, st.expose, planes);
    note_launch();
    return IMOPS_OK;
}

//   halation: local scatter in place (halation.rs:24-78); tmp: one plane
int stage_scatter(float* planes, int W, int H, const RefSpec& R, float* tmp, cudaStream_t s) {
    if (!(R.sigma_local >= 1e-3f && R.local_mix > 0.0f)) return IMOPS_OK;
    const size_t n = (size_t)W * H;
    Taps tp;
    int rc;
    if ((rc = taps_for(R.sigma_local, &tp))) return rc;
    for (int e = 0; e < R.E; e++)
        if ((rc = blur(planes + e * n, tmp, W, H, tp, EpiMix{planes + e * n, 1.0f - R.local_mix, R.local_mix}, s)))
            return rc;
    return IMOPS_OK;
}

//   expose and scatter in one pass
int expose_scatter(const float* rgb, int W, int H, const Stock& st, float* planes, float* tmp, cudaStream_t s) {
    const RefSpec& R = st.ref;
    Taps tp;
    int rc;
    const bool local = R.sigma_local >= 1e-3f && R.local_mix > 0.0f;
    if (local && (rc = taps_for(R.sigma_local, &tp))) return rc;
    if (!local || tp.R > EX_MAXR) {
        if ((rc = stage_expose(rgb, W, H, st, planes, s))) return rc;
        return stage_scatter(planes, W, H, R, tmp, s);
    }
    const size_t smem = (size_t)expose_smem_floats(tp.R) * sizeof(float);
    IMOPS_CUDA_TRY(cudaFuncSetAttribute(expose_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "cudaFuncSetAttribute(exposure)");
    const dim3 g((W + FT_W - 1) / FT_W, (H + FT_H - 1) / FT_H);
    expose_scatter_kernel<<<g, EX_THREADS, smem, s>>>(rgb, W, H, st.expose, tp, 1.0f - R.local_mix, R.local_mix,
                                                      planes);
    note_launch();
    return IMOPS_OK;
}

//   the wide bounce of the deepest layer (halation.rs:80-93): its blur in
//     *deep (NULL when the stock has none), added to the layers by
//     bounce_kernel or by the reduction; tmp, bounce: one plane each
int stage_bounce(const float* planes, int W, int H, const RefSpec& R, float* tmp, float* bounce, float** deep,
                 cudaStream_t s) {
    *deep = nullptr;
    if (!(R.sigma_wide >= 1e-3f)) return IMOPS_OK;
    Taps tp;
    int rc;
    if ((rc = taps_for(R.sigma_wide, &tp))) return rc;
    if ((rc = blur(planes + (size_t)(R.E - 1) * W * H, tmp, W, H, tp, EpiStore{bounce}, s))) return rc;
    *deep = bounce;
    return IMOPS_OK;
}

static Bounce bounce_gains(const RefSpec& R) {
    Bounce b;
    for (int e = 0; e < MAXE; e++) b.gain[e] = R.hal_gain[e];
    return b;
}

// The stock's capture LUT into lut (MAXE * LUTN floats on the device).
int launch_capture_lut(const RefSpec& R, float* lut, cudaStream_t s) {
    CaptureSpec c;
    for (int e = 0; e < MAXE; e++) {
        c.mu[e] = R.mu_ln[e];
        c.sigma[e] = R.sigma_ln[e];
        c.k[e] = R.capture_k[e];
    }
    capture_lut_kernel<<<R.E, 8 * LUTN, 0, s>>>(c, lut);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "capture LUT");
    return IMOPS_OK;
}

// The bounce (deep not NULL), the capture LUT and the reduction over the layers.
int launch_reduce(float* planes, float* mask, bool sum, const float* deep, size_t n, const RefSpec& R,
                  const float* lut, cudaStream_t s) {
    return with_layers(R.E, [&](auto e) {
        constexpr int E = decltype(e)::value;
        Reduce<E> c;
        for (int i = 0; i < E; i++) {
            c.eta[i] = R.eta[i];
            c.dmax[i] = R.dmax[i];
            c.inv_gamma[i] = R.inv_gamma[i];
            c.mask_scale[i] = R.has_mask[i] ? R.mask_scale[i] : 0.0f;
            c.reversal[i] = R.reversal[i];
        }
        const Bounce b = bounce_gains(R);
        const int g = grid_for(n);
        if (sum && deep) lut_reduce_kernel<E, true, true><<<g, 256, 0, s>>>(planes, mask, deep, n, lut, c, b);
        else if (sum) lut_reduce_kernel<E, true, false><<<g, 256, 0, s>>>(planes, mask, nullptr, n, lut, c, b);
        else lut_reduce_kernel<E, false, false><<<g, 256, 0, s>>>(planes, mask, nullptr, n, lut, c, b);
        note_launch();
        return IMOPS_OK;
    });
}

int launch_dir(const float* in, float* out, int W, int H, const Taps& tp, const RefSpec& R, cudaStream_t s) {
    return with_layers(R.E, [&](auto e) {
        constexpr int E = decltype(e)::value;
        DirMix<E> mix;
        for (int i = 0; i < E; i++)
            for (int j = 0; j < E; j++) mix.m[i][j] = R.dir[i][j];
        const size_t smem = (size_t)(2 * ft_tile_floats(tp.R) + ft_row_floats(tp.R)) * sizeof(float);
        IMOPS_CUDA_TRY(cudaFuncSetAttribute(dir_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                       "cudaFuncSetAttribute(DIR)");
        const dim3 g((W + FT_W - 1) / FT_W, (H + FT_H - 1) / FT_H);
        dir_kernel<E><<<g, DIR_THREADS, smem, s>>>(in, out, W, H, tp, mix);
        note_launch();
        return IMOPS_OK;
    });
}

static bool has_adjacency(const RefSpec& R) { return !(fabsf(R.beta) < 1e-8f || R.sigma_adj < 1e-3f); }

int stage_adjacency(float* planes, int W, int H, const RefSpec& R, float* tmp, cudaStream_t s) {
    if (!has_adjacency(R)) return IMOPS_OK;
    const size_t n = (size_t)W * H;
    Taps tp;
    int rc;
    if ((rc = taps_for(R.sigma_adj, &tp))) return rc;
    for (int e = 0; e < R.E; e++)
        if ((rc = blur(planes + e * n, tmp, W, H, tp, EpiAdjacency{planes + e * n, R.beta}, s))) return rc;
    return IMOPS_OK;
}

//   develop: capture LUT + reciprocity + reduction to image-dye and mask
//     densities, DIR inhibition, adjacency (capture.rs:61-88,
//     reduction.rs:16-68, diffusion.rs:11-84); inh: E planes, tmp: one.
//     sum: `mask` is the one plane of the layers' mask sum, and the bounce
//     `deep` (or NULL) is added first.  With result NULL the densities end
//     up in planes; otherwise in *result (planes or inh), without the
//     adjacency, which print_scan adds.
int stage_develop(float* planes, float* mask, bool sum, const float* deep, int W, int H, const Stock& st,
                  const float* lut, float* inh, float* tmp, float** result, cudaStream_t s) {
    const RefSpec& R = st.ref;
    const int E = R.E;
    const size_t n = (size_t)W * H;
    const int g = grid_for(n);
    Taps tp;
    int rc;
    if ((rc = launch_reduce(planes, mask, sum, deep, n, R, lut, s))) return rc;
    if (result) *result = planes;
    if (R.dir_any && R.sigma_dir >= 1e-3f) {
        if ((rc = taps_for(R.sigma_dir, &tp))) return rc;
        if (tp.R <= FT_MAXR) {
            float *in = planes, *out = inh;
            if (result) {
                *result = inh;
            } else {
                std::swap(in, out);
                IMOPS_CUDA_TRY(cudaMemcpyAsync(in, out, E * n * 4, cudaMemcpyDeviceToDevice, s), "copy");
            }
            if ((rc = launch_dir(in, out, W, H, tp, R, s))) return rc;
            planes = out;
        } else {
            // a blur wider than the tiles' halo: 35 mm Ektar100 images of 13715 to 13963 pixels
            // width, and wider or other ones in the sub-stage alone (a whole image's wide bounce
            // is then above 64 px)
            for (int i = 0; i < E; i++)
                if ((rc = blur(planes + i * n, tmp, W, H, tp, EpiStore{inh + i * n}, s))) return rc;
            DirAny any;
            for (int i = 0; i < MAXE; i++)
                for (int j = 0; j < MAXE; j++) any.m[i][j] = R.dir[i][j];
            dir_apply_kernel<<<g, 256, 0, s>>>(planes, inh, n, E, any);
            note_launch();
        }
    }
    return result ? IMOPS_OK : stage_adjacency(planes, W, H, R, tmp, s);
}

//   grain: seeded SplitMix64 fields, normalised and scaled per layer
//     (grain.rs:53-100); noise: E planes, partial: grain_partials(W, H, E)
//     doubles, sums: MAXE doubles
int stage_grain_fields(int W, int H, const RefSpec& R, uint64_t seed, float* noise, double* partial, double* sums,
                       cudaStream_t s) {
    Taps tp;
    int rc;
    if ((rc = taps_for(fmaxf(R.sigma_grain, 1.0f), &tp))) return rc;
    return grain_fields(noise, W, H, seed, 0, R.E, tp, partial, sums, s);
}

int stage_grain(float* planes, int W, int H, const Stock& st, uint64_t seed, float* noise, double* partial,
                double* sums, cudaStream_t s) {
    const RefSpec& R = st.ref;
    const size_t n = (size_t)W * H;
    int rc;
    if ((rc = stage_grain_fields(W, H, R, seed, noise, partial, sums, s))) return rc;
    for (int e = 0; e < R.E; e++) {
        if (R.kappa[e] <= 0.0f || R.dmax[e] <= 0.0f) continue;
        grain_apply_kernel<<<grid_for(n), 256, 0, s>>>(planes + e * n, noise + e * n, n, sums + e, R.kappa[e],
                                                      R.dmax[e]);
        note_launch();
    }
    return IMOPS_OK;
}

//   scan: densities -> ACEScg RGB of the scanned negative (scan/mod.rs:24-30,
//     densitometry.rs:13-73)
int stage_scan(const float* planes, const float* mask, int W, int H, const ScanSpec16& S, float* rgb, cudaStream_t s) {
    const size_t n = (size_t)W * H;
    return with_layers(S.E, [&](auto e) {
        constexpr int E = decltype(e)::value;
        scan16_kernel<E><<<grid_for(n), 256, 0, s>>>(planes, mask, n, scan16_pairs<E>(S), rgb);
        note_launch();
        return IMOPS_OK;
    });
}

template <int E, int RC>
int launch_print(const float* dens, const float* mask, const float* noise, const double* sums, const float* mid_dmin,
                 int W, int H, const Print<E>& c, float* rgb, cudaStream_t s) {
    const size_t smem = (size_t)print_smem_floats<RC>(E) * sizeof(float);
    IMOPS_CUDA_TRY(cudaFuncSetAttribute(print_kernel<E, RC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "cudaFuncSetAttribute(print)");
    const dim3 g((W + FT_W - 1) / FT_W, (H + FT_H - 1) / FT_H);
    print_kernel<E, RC><<<g, PR_THREADS, smem, s>>>(dens, mask, noise, sums, mid_dmin, W, H, c, rgb);
    note_launch();
    return IMOPS_OK;
}

// Adjacency, grain (noise not NULL), scan and inversion (mid_dmin not NULL)
// of the densities in one pass.  The radius classes are the stocks' at 35 mm
// up to about 25 and 50 MP; wider adjacency blurs (the stock without a wide
// bounce, BwStub, above 19200 pixels width) run as launches of their own.
int print_scan(float* dens, const float* mask, const float* noise, const double* sums, const float* mid_dmin, int W,
               int H, const Stock& st, float* tmp, float* rgb, cudaStream_t s) {
    const RefSpec& R = st.ref;
    Taps tp;
    tp.R = 0;
    int rc;
    if (has_adjacency(R) && (rc = taps_for(R.sigma_adj, &tp))) return rc;
    if (tp.R > 8) {
        if ((rc = stage_adjacency(dens, W, H, R, tmp, s))) return rc;
        tp.R = 0;
    }
    return with_layers(R.E, [&](auto e) {
        constexpr int E = decltype(e)::value;
        Print<E> c;
        c.scan = scan16_pairs<E>(st.scan16);
        for (int i = 0; i < E; i++) {
            c.kappa[i] = R.kappa[i];
            c.dmax[i] = R.dmax[i];
        }
        c.beta = R.beta;
        const int RC = tp.R == 0 ? 0 : (tp.R <= 4 ? 4 : 8);
        for (int k = 0; k < 2 * 8 + 1; k++) {
            const int j = k - RC + tp.R;
            c.taps[k] = tp.R > 0 && j >= 0 && j <= 2 * tp.R ? tp.t[j] : 0.0f;
        }
        if (RC == 0) return launch_print<E, 0>(dens, mask, noise, sums, mid_dmin, W, H, c, rgb, s);
        if (RC == 4) return launch_print<E, 4>(dens, mask, noise, sums, mid_dmin, W, H, c, rgb, s);
        return launch_print<E, 8>(dens, mask, noise, sums, mid_dmin, W, H, c, rgb, s);
    });
}

// The reference model's kernels on rgb in place, inverted with the reference
// points mid_dmin unless that is NULL; those, and the grain fields where they
// are given, are waited for on `beside` where that stream forms them.
int run_reference(float* rgb, int W, int H, const Stock& st, uint64_t seed, int grain, const float* mid_dmin, Arena& A,
                  const float* lut, cudaStream_t s, const SideStream* beside = nullptr, float* fields = nullptr,
                  double* field_sums = nullptr) {
    const int E = st.ref.E;
    const size_t n = (size_t)W * H;
    float* planes = A.take<float>(E * n);
    float* mask = A.take<float>(n);  // the layers' mask sum
    float* inh = A.take<float>(E * n);
    float* tmp = A.take<float>(n);
    float* bounce = A.take<float>(n);
    double* partial = fields ? nullptr : A.take<double>(grain_partials(W, H, E));
    double* sums = fields ? field_sums : A.take<double>(MAXE);
    int rc;
    float *deep = nullptr, *dens = nullptr;
    if ((rc = expose_scatter(rgb, W, H, st, planes, tmp, s))) return rc;
    if ((rc = stage_bounce(planes, W, H, st.ref, tmp, bounce, &deep, s))) return rc;
    if ((rc = stage_develop(planes, mask, true, deep, W, H, st, lut, inh, tmp, &dens, s))) return rc;
    // the other set of planes is free after develop: it takes the grain fields
    float* noise = fields ? fields : grain ? (dens == planes ? inh : planes) : nullptr;
    if (grain && !fields && (rc = stage_grain_fields(W, H, st.ref, seed, noise, partial, sums, s))) return rc;
    if (beside && (rc = beside->wait(s))) return rc;
    if ((rc = print_scan(dens, mask, noise, sums, mid_dmin, W, H, st, tmp, rgb, s))) return rc;
    IMOPS_CUDA_TRY(cudaGetLastError(), "film kernels");
    return IMOPS_OK;
}

// PositiveLinear's reference points (film/mod.rs:136-151): the mean RGB of
// a 32x32 mid-grey patch through the same path (seed 0) into mid_dmin[0..2]
// and the stock's normalised Dmin into mid_dmin[3..5].  Takes
// ref_workspace_bytes(32, 32, E) + 1024 * 12 bytes of A.
int mid_gray_negative(const Stock& st, int grain, Arena& A, const float* lut, float* mid_dmin, cudaStream_t s) {
    const size_t nm = 32 * 32;
    float g = relative_to_absolute_y(0.185f, st.ref.box_iso);
    float* dpatch = A.take<float>(nm * 3);
    fill_kernel<<<12, 256, 0, s>>>(dpatch, (int)nm * 3, g);
    note_launch();
    int rc;
    if ((rc = run_reference(dpatch, 32, 32, st, 0, grain, nullptr, A, lut, s))) return rc;
    mean_rgb_kernel<<<1, 256, 0, s>>>(dpatch, (int)nm, st.ref.dmin_norm[0], st.ref.dmin_norm[1], st.ref.dmin_norm[2],
                                      mid_dmin);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "film mid-grey patch");
    return IMOPS_OK;
}

// run_reference with the work that does not depend on the image on the
// caller's side stream, up to the print: a positive's mid-grey patch, whose
// dozen small kernels take 60 us, or the grain fields (grain_beside: into
// planes of their own).  Not both: the grain before the patch delays the print
// (640x480, six layers: 142 -> 177 us), and after it is late itself.  The
// stream waits for the side stream on every way out, as its scratch is the
// stream's.
int run_beside(float* rgb, int W, int H, const Stock& st, const ImopsFilmParams& P, Arena& A, const float* lut,
               float* mid_dmin, bool grain_beside, cudaStream_t s) {
    SideStream ss;
    int rc = side_stream(s, &ss);
    if (rc || (rc = ss.fork(s))) return rc;
    float* fields = nullptr;
    double* sums = nullptr;
    if (grain_beside) {
        fields = A.take<float>(st.ref.E * (size_t)W * H);
        double* partial = A.take<double>(grain_partials(W, H, st.ref.E));
        sums = A.take<double>(MAXE);
        rc = stage_grain_fields(W, H, st.ref, P.seed, fields, partial, sums, ss.side);
    }
    if (!rc && mid_dmin) rc = mid_gray_negative(st, P.grain, A, lut, mid_dmin, ss.side);
    const int joined = ss.record(s);
    if (!rc && !joined) rc = run_reference(rgb, W, H, st, P.seed, P.grain, mid_dmin, A, lut, s, &ss, fields, sums);
    if (rc && !joined) ss.wait(s);
    return rc ? rc : joined;
}

// The layer values (layers x pixels) at which the grain runs beside the other
// kernels.  Six layers: 640x480 128 -> 96 us, 1200x800 215 -> 187, 2048x1365
// 434 -> 413; three: 87 -> 71, 136 -> 122, 285 -> 269; one: 0.3 MP 45 -> 46
// (the events), 1 MP 68 -> 57.  Above, the gain falls to 1% (24 MP 3404 ->
// 3375) of the time for a fifth more memory.
constexpr size_t GRAIN_BESIDE_LEAST = (size_t)600 << 10, GRAIN_BESIDE_MOST = (size_t)32 << 20;

int process_reference(float* rgb, int W, int H, const ImopsFilmParams& P, cudaStream_t s) {
    Stock st;
    float pitch = 0;
    int rc = build_stock(P.stock, P.film_format, W, P.shutter_seconds, nullptr, &st, &pitch);
    if (rc) return rc;
    const size_t n = (size_t)W * H;
    const size_t nm = 32 * 32;
    size_t bytes = ref_workspace_bytes(W, H, st.ref.E) + ref_workspace_bytes(32, 32, st.ref.E) + nm * 12 + 4096;
    const bool positive = P.output == IMOPS_FILM_POSITIVE_LINEAR && !st.ref.any_reversal;
    const size_t values = st.ref.E * n;
    bool grain_beside = P.grain && !positive && values >= GRAIN_BESIDE_LEAST && values <= GRAIN_BESIDE_MOST;
    const size_t more = grain_beside ? values * 4 + grain_partials(W, H, st.ref.E) * 8 + 1024 : 0;
    void* ws = nullptr;
    rc = workspace(s, bytes + more, &ws);
    if (rc && more) {  // no room for planes of the grain's own
        clear_error();
        grain_beside = false;
        rc = workspace(s, bytes, &ws);
    }
    if (rc) return rc;
    Arena A{static_cast<char*>(ws), 0};
    float* lut = A.take<float>(MAXE * LUTN);
    float* mid_dmin = A.take<float>(8);
    if ((rc = launch_capture_lut(st.ref, lut, s))) return rc;
    if (positive || grain_beside)
        return run_beside(rgb, W, H, st, P, A, lut, positive ? mid_dmin : nullptr, grain_beside, s);
    return run_reference(rgb, W, H, st, P.seed, P.grain, nullptr, A, lut, s);
}

// One sub-stage call: the stock (reference model only) and, once its layers are
// known, an arena in the film workspace.
struct StageCtx {
    Stock st;
    Arena A;
    float* lut;  // the capture LUT's place (launch_capture_lut fills it)
};

// extra(E): bytes of the arena besides the LUT for a stock of E layers.
template <class Extra>
int stage_ctx(const ImopsFilmParams* P, int W, int H, Extra extra, cudaStream_t s, StageCtx* c) {
    if (!P) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film stage: NULL params");
    if (W <= 0 || H <= 0) return fail(IMOPS_ERR_INVALID_DIMENSIONS, "invalid image dimensions");
    float pitch = 0;
    int rc = build_stock(P->stock, P->film_format, W, P->shutter_seconds, nullptr, &c->st, &pitch);
    if (rc) return rc;
    if (c->st.model != MODEL_REFERENCE)
        return fail(IMOPS_ERR_INVALID_STOCK, "film stages: the baseline preset runs only whole (imops_film_process)");
    void* ws = nullptr;
    const size_t bytes = MAXE * LUTN * sizeof(float) + (size_t)extra(c->st.ref.E) + 4096;
    if ((rc = workspace(s, bytes, &ws))) return rc;
    c->A = Arena{static_cast<char*>(ws), 0};
    c->lut = c->A.take<float>(MAXE * LUTN);
    return IMOPS_OK;
}
size_t no_extra(int) { return 0; }

}  // namespace film
}  // namespace imops

namespace imops {
namespace film {

// Bytes of the baseline preset's working set for a W x H image: the
// halation row pass, three grain fields, the grain's block sums (and the
// Arena's 256-byte alignment).  The layer exposures and the halation source
// are formed from the RGB where they are read.
size_t baseline_scratch_bytes(int W, int H) {
    const size_t n = (size_t)W * H;
    return (1 + 3) * n * 4 + grain_partials(W, H, 3) * 8 + 4096;
}

int baseline_stock(int W, const ImopsBaselineFilm& P, Stock* st) {
    if (P.scan != IMOPS_SCAN_FP32 && P.scan != IMOPS_SCAN_BF16_TC)
        return fail(IMOPS_ERR_INVALID_ARGUMENT, "film: unknown scan (IMOPS_SCAN_FP32 or IMOPS_SCAN_BF16_TC)");
    float pitch;
    return build_stock(IMOPS_STOCK_BASELINE81, 0, W, -1.0f, &P, st, &pitch);
}

// Baseline preset forward on an ACEScg image in place, with the working set
// in the library's per-(device, stream) workspace.
int baseline_forward_impl(float* rgb, int W, int H, const ImopsBaselineFilm* Pp, cudaStream_t s) {
    ImopsBaselineFilm P;
    if (Pp) P = *Pp;
    else imops_baseline_film_defaults(&P);
    Stock st;
    int rc = baseline_stock(W, P, &st);
    if (rc) return rc;
    void* ws = nullptr;
    if ((rc = workspace(s, baseline_scratch_bytes(W, H), &ws))) return rc;
    return baseline_forward_in(rgb, W, H, P, st, ws, s);
}

// The baseline preset's kernels with the working set at `scratch` (256-byte
// aligned, baseline_scratch_bytes(W, H) long).  Every byte the kernels read
// there is written earlier in the same call.
int baseline_forward_in(float* rgb, int W, int H, const ImopsBaselineFilm& P, const Stock& st, void* scratch,
                        cudaStream_t s) {
    int rc;
    const size_t n = (size_t)W * H;
    if (st.expose.E != 3 || !st.expose.hal_src)
        return fail(IMOPS_ERR_INVALID_STOCK, "film: the baseline preset's exposure is three layers with halation");
    Arena A{static_cast<char*>(scratch), 0};
    double* sums = A.take<double>(4);
    float* hr = A.take<float>(n);
    float* noise = A.take<float>(3 * n);
    double* gpart = A.take<double>(grain_partials(W, H, 3));
    Base81 hp;
    build_base81(st, &hp);
    if (P.grain_on && P.grain_sigma != 0.0f) {
        // grain fields on the side stream while the halation row pass runs on
        // s; the scan waits for both
        Taps tp;
        if ((rc = taps_for(fmaxf(P.grain_blur, 1.0f), &tp))) return rc;
        SideStream ss;
        if ((rc = side_stream(s, &ss)) || (rc = ss.fork(s))) return rc;
        rc = grain_fields(noise, W, H, P.seed, 0, 3, tp, gpart, sums, ss.side);
        const int joined = ss.record(s);
        if (!rc && !joined) rc = blur_rows_halation(rgb, st.expose.hal_threshold, hr, W, H, st.hal_taps, s);
        if (!joined) {
            const int waited = ss.wait(s);
            if (!rc) rc = waited;
        }
        if (rc || (rc = joined)) return rc;
    } else {
        if ((rc = blur_rows_halation(rgb, st.expose.hal_threshold, hr, W, H, st.hal_taps, s))) return rc;
    }
    dim3 cb(R64_COL_TW, R64_COL_GROUPS), cg((W + R64_COL_TW - 1) / R64_COL_TW, (H + R64_COL_TH - 1) / R64_COL_TH);
    if (P.scan == IMOPS_SCAN_BF16_TC) {
        Base81TC tp;
        build_base81_tc(st, &tp);
        IMOPS_CUDA_TRY(cudaFuncSetAttribute(scan81_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)tc::SMEM_REQ),
                       "cudaFuncSetAttribute(tensor-core scan)");
        scan81_tc_kernel<<<cg, cb, tc::SMEM_REQ, s>>>(hr, noise, sums, W, H, tp, rgb);
    } else {
        if ((long)cg.x * cg.y < 3L * sm_count()) {
            cg.y = (H + R64_COL_GROUPS * SCAN_OUT_SMALL - 1) / (R64_COL_GROUPS * SCAN_OUT_SMALL);
            scan81_fused_kernel<SCAN_OUT_SMALL><<<cg, cb, 0, s>>>(hr, noise, sums, W, H, hp, rgb);
        } else {
            scan81_fused_kernel<R64_COL_OUT><<<cg, cb, 0, s>>>(hr, noise, sums, W, H, hp, rgb);
        }
    }
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "baseline film kernels");
    return IMOPS_OK;
}

}  // namespace film
}  // namespace imops


using namespace imops;

// ---- the reference model's sub-stages ----------------------------------------

extern "C" int imops_film_layers(const ImopsFilmParams* params, int* layers) {
    clear_error();
    if (!layers) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_layers: NULL output");
    film::StageCtx c;
    if (!params) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film stage: NULL params");
    float pitch = 0;
    int rc = film::build_stock(params->stock, params->film_format, 1024, params->shutter_seconds, nullptr, &c.st,
                               &pitch);
    if (rc) return rc;
    if (c.st.model != film::MODEL_REFERENCE)
        return fail(IMOPS_ERR_INVALID_STOCK, "film stages: the baseline preset runs only whole (imops_film_process)");
    *layers = c.st.ref.E;
    return IMOPS_OK;
}

extern "C" int imops_film_expose(const float* rgb, int w, int h, const ImopsFilmParams* params, float* planes,
                                 imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    film::StageCtx c;
    int rc = film::stage_ctx(params, w, h, film::no_extra, s, &c);
    if (rc) return rc;
    if (!rgb || !planes) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_expose: NULL buffer");
    if ((rc = film::stage_expose(rgb, w, h, c.st, planes, s))) return rc;
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_expose");
    return IMOPS_OK;
}

extern "C" int imops_film_halation(float* planes, int w, int h, const ImopsFilmParams* params,
                                   imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    const size_t n = (size_t)(w > 0 ? w : 0) * (h > 0 ? h : 0);
    film::StageCtx c;
    int rc = film::stage_ctx(params, w, h, [=](int) { return 2 * n * 4 + 512; }, s, &c);
    if (rc) return rc;
    if (!planes) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_halation: NULL buffer");
    float* tmp = c.A.take<float>(n);
    float* bounce = c.A.take<float>(n);
    float* deep = nullptr;
    if ((rc = film::stage_scatter(planes, w, h, c.st.ref, tmp, s))) return rc;
    if ((rc = film::stage_bounce(planes, w, h, c.st.ref, tmp, bounce, &deep, s))) return rc;
    if (deep) {
        film::bounce_kernel<<<film::grid_for(n), 256, 0, s>>>(planes, deep, n, c.st.ref.E,
                                                              film::bounce_gains(c.st.ref));
        note_launch();
    }
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_halation");
    return IMOPS_OK;
}

extern "C" int imops_film_develop(float* planes, float* mask, int w, int h, const ImopsFilmParams* params,
                                  imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    const size_t n = (size_t)(w > 0 ? w : 0) * (h > 0 ? h : 0);
    film::StageCtx c;
    int rc = film::stage_ctx(params, w, h, [=](int E) { return (E + 1) * n * 4 + 512; }, s, &c);
    if (rc) return rc;
    if (!planes || !mask) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_develop: NULL buffer");
    float* inh = c.A.take<float>((size_t)c.st.ref.E * n);
    float* tmp = c.A.take<float>(n);
    if ((rc = film::launch_capture_lut(c.st.ref, c.lut, s))) return rc;
    if ((rc = film::stage_develop(planes, mask, false, nullptr, w, h, c.st, c.lut, inh, tmp, nullptr, s))) return rc;
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_develop");
    return IMOPS_OK;
}

extern "C" int imops_film_grain(float* planes, int w, int h, const ImopsFilmParams* params, imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    const size_t n = (size_t)(w > 0 ? w : 0) * (h > 0 ? h : 0);
    film::StageCtx c;
    int rc = film::stage_ctx(
        params, w, h, [=](int E) { return E * n * 4 + film::grain_partials(w, h, E) * 8 + film::MAXE * 8 + 768; }, s,
        &c);
    if (rc) return rc;
    if (!planes) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_grain: NULL buffer");
    if (!params->grain) return IMOPS_OK;
    float* noise = c.A.take<float>(c.st.ref.E * n);
    double* partial = c.A.take<double>(film::grain_partials(w, h, c.st.ref.E));
    double* sums = c.A.take<double>(film::MAXE);
    if ((rc = film::stage_grain(planes, w, h, c.st, params->seed, noise, partial, sums, s))) return rc;
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_grain");
    return IMOPS_OK;
}

extern "C" int imops_film_scan(const float* planes, const float* mask, int w, int h, const ImopsFilmParams* params,
                               float* rgb, imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    film::StageCtx c;
    int rc = film::stage_ctx(params, w, h, film::no_extra, s, &c);
    if (rc) return rc;
    if (!planes || !mask || !rgb) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_scan: NULL buffer");
    if ((rc = film::stage_scan(planes, mask, w, h, c.st.scan16, rgb, s))) return rc;
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_scan");
    return IMOPS_OK;
}

extern "C" int imops_film_invert(float* rgb, int w, int h, const ImopsFilmParams* params, imops_stream_t stream) {
    clear_error();
    cudaStream_t s = as_stream(stream);
    // the mid-grey patch's path and its reference points come from the same arena
    const size_t nm = 32 * 32;
    film::StageCtx c;
    int rc = film::stage_ctx(
        params, w, h, [=](int E) { return film::ref_workspace_bytes(32, 32, E) + nm * 12 + 1024; }, s, &c);
    if (rc) return rc;
    if (!rgb) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film_invert: NULL buffer");
    if (!(params->output == IMOPS_FILM_POSITIVE_LINEAR && !c.st.ref.any_reversal)) return IMOPS_OK;
    float* mid_dmin = c.A.take<float>(8);
    if ((rc = film::launch_capture_lut(c.st.ref, c.lut, s))) return rc;
    if ((rc = film::mid_gray_negative(c.st, params->grain, c.A, c.lut, mid_dmin, s))) return rc;
    const size_t n = (size_t)w * h;
    film::invert_kernel<<<film::grid_for(n), 256, 0, s>>>(rgb, n, mid_dmin);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "film_invert");
    return IMOPS_OK;
}

extern "C" int imops_film_process(float* rgb, int w, int h, int color_space, const ImopsFilmParams* params,
                                  const ImopsBaselineFilm* baseline, imops_stream_t stream) {
    clear_error();
    if (!params) return fail(IMOPS_ERR_INVALID_ARGUMENT, "film: NULL params");
    if (color_space != IMOPS_CS_ACESCG)
        return fail(IMOPS_ERR_WRONG_COLOR_SPACE, "wrong color space: expected ACEScg");
    if (w <= 0 || h <= 0 || !rgb) return fail(IMOPS_ERR_INVALID_DIMENSIONS, "invalid image dimensions");
    cudaStream_t s = as_stream(stream);
    if (params->stock == IMOPS_STOCK_BASELINE81) {
        // without an explicit preset, the defaults with the module's grain seed
        ImopsBaselineFilm d;
        if (!baseline) {
            imops_baseline_film_defaults(&d);
            d.seed = params->seed;
            d.grain_on = params->grain;
            baseline = &d;
        }
        return film::baseline_forward_impl(rgb, w, h, baseline, s);
    }
    return film::process_reference(rgb, w, h, *params, s);
}

extern "C" int imops_tensor_timeouts(unsigned* count) {
    clear_error();
    if (!count) return fail(IMOPS_ERR_INVALID_ARGUMENT, "imops_tensor_timeouts: NULL output");
    IMOPS_CUDA_TRY(cudaMemcpyFromSymbol(count, film::g_tc_timeouts, sizeof(unsigned)), "read tensor-core timeouts");
    return IMOPS_OK;
}
