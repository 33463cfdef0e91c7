// blur.cuh -- the separable Gaussian blurs with mirror reflection shared by the
// film simulation (film.cu) and the adjoints (adjoint.cu).
#pragma once

#include "film.cuh"

namespace imops {
namespace film {

constexpr int MAXR = 64;  // largest blur radius handled (129 taps)

struct Taps {
    int R;
    float t[2 * MAXR + 1];
};

// Radius-64 taps as pairs t2[k] = (t[k], t[k-1]), zero outside [0, 128]:
// the radius-64 kernels accumulate two adjacent outputs per packed f32x2 FMA
// (output j takes tap k, output j+1 tap k-1 of the same input sample), each
// output still summing its taps in ascending order.
struct Taps2 {
    float2 t2[2 * MAXR + 2];
};

static Taps2 pair_taps(const Taps& tp) {
    Taps2 p;
    for (int k = 0; k <= 2 * MAXR + 1; k++)
        p.t2[k] = make_float2(k <= 2 * MAXR ? tp.t[k] : 0.0f, k >= 1 ? tp.t[k - 1] : 0.0f);
    return p;
}

__device__ __forceinline__ int reflect(int i, int n) {
    // blur.rs:70-89: mirror without repeating the edge sample
    if (n == 1) return 0;
    int x = i;
    for (;;) {
        if (x < 0) x = -x;
        else if (x >= n) x = 2 * n - 2 - x;
        else return x;
    }
}

// ---------------------------------------------------------------------------
// separable Gaussian blur with mirror reflection (blur.rs:10-89)

// One kernel pair for any radius up to 64 (the reference model's wide bounce,
// the adjoint with another radius than 64).  A thread slides a window over
// several outputs (4 along a row, 16 down a column), so a staged sample is
// read once for all of them instead of once per tap and output; the head and
// tail of the window test the tap range, the middle does not.  Each output
// sums its taps in ascending order.
constexpr int ROW_OUT = 4, ROW_THREADS = 256, ROW_TILE = ROW_OUT * ROW_THREADS;

static __global__ void __launch_bounds__(ROW_THREADS)
    blur_rows_kernel(const float* __restrict__ in, float* __restrict__ out, int W, int H,
                     const __grid_constant__ Taps tp) {
    __shared__ __align__(16) float s[ROW_TILE + 2 * MAXR + ROW_OUT];
    const int y = blockIdx.y, x0 = blockIdx.x * ROW_TILE, R2 = 2 * tp.R;
    const float* row = in + (size_t)y * W;
    // only the samples that outputs inside the image read
    const int span = min(ROW_TILE, W - x0) + R2;
    for (int j = threadIdx.x; j < span; j += ROW_THREADS) s[j] = __ldg(row + reflect(x0 - tp.R + j, W));
    __syncthreads();
    const int xb = ROW_OUT * threadIdx.x;
    if (x0 + xb >= W) return;
    float a[ROW_OUT] = {0.0f, 0.0f, 0.0f, 0.0f};
    // samples 4q .. 4q+3 of the window: sample 4q+u is tap 4q+u-j of output j
    auto step = [&](int q, bool lo, bool hi) {
        const float4 v4 = *reinterpret_cast<const float4*>(s + xb + 4 * q);
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int j = 0; j < ROW_OUT; j++) {
                const int k = 4 * q + u - j;
                if ((!lo || k >= 0) && (!hi || k <= R2)) a[j] = fmaf(v[u], tp.t[k], a[j]);
            }
    };
    step(0, true, true);
    int q = 1;
#pragma unroll 2
    for (; 4 * q + 3 <= R2; q++) step(q, false, false);
    for (; 4 * q - 3 <= R2; q++) step(q, false, true);
    float* o = out + (size_t)y * W + x0 + xb;
#pragma unroll
    for (int j = 0; j < ROW_OUT; j++)
        if (x0 + xb + j < W) o[j] = a[j];
}

constexpr int COL_TW = 32, COL_GROUPS = 8, COL_OUT = 16, COL_TH = COL_GROUPS * COL_OUT;  // 32x8 threads, 16 rows each

// Column pass; epi(index, blurred) writes the result.
template <class Epi>
__global__ void __launch_bounds__(COL_TW * COL_GROUPS) blur_cols_kernel(const float* __restrict__ in, int W, int H,
                                                                        const __grid_constant__ Taps tp, Epi epi) {
    __shared__ float s[(COL_TH + 2 * MAXR) * COL_TW];
    const int tx = threadIdx.x, ty = threadIdx.y, x = blockIdx.x * COL_TW + tx, y0 = blockIdx.y * COL_TH;
    const int R2 = 2 * tp.R, rb = ty * COL_OUT;
    if (x < W) {
        const int span = min(COL_TH, H - y0) + R2;
        if (y0 - tp.R >= 0 && y0 - tp.R + span <= H) {
            const float* src = in + (size_t)(y0 - tp.R) * W + x;
#pragma unroll 8
            for (int j = ty; j < span; j += COL_GROUPS) s[j * COL_TW + tx] = __ldg(src + (size_t)j * W);
        } else {
            for (int j = ty; j < span; j += COL_GROUPS)
                s[j * COL_TW + tx] = __ldg(in + (size_t)reflect(y0 - tp.R + j, H) * W + x);
        }
    }
    __syncthreads();
    if (x >= W || y0 + rb >= H) return;
    float a[COL_OUT];
#pragma unroll
    for (int j = 0; j < COL_OUT; j++) a[j] = 0.0f;
    // rows m0 .. m0+15 of the window: row m is tap m-j of output j
    auto step = [&](int m0, bool lo, bool hi) {
#pragma unroll
        for (int u = 0; u < COL_OUT; u++) {
            const int m = m0 + u;
            if (hi && m > R2 + COL_OUT - 1) break;
            const float v = s[(rb + m) * COL_TW + tx];
#pragma unroll
            for (int j = 0; j < COL_OUT; j++)
                if ((!lo || u - j >= 0) && (!hi || m - j <= R2)) a[j] = fmaf(v, tp.t[m - j], a[j]);
        }
    };
    step(0, true, true);
    int m0 = COL_OUT;
    for (; m0 + COL_OUT - 1 <= R2; m0 += COL_OUT) step(m0, false, false);
    for (; m0 <= R2 + COL_OUT - 1; m0 += COL_OUT) step(m0, false, true);
#pragma unroll
    for (int j = 0; j < COL_OUT; j++) {
        const int y = y0 + rb + j;
        if (y < H) epi((size_t)y * W + x, a[j]);
    }
}

// Radius-64 specialisations (the baseline preset's halation and the adjoint):
// the 129 taps are compile-time indexed parameter-bank operands and each
// thread slides one window of loaded samples over several outputs, so the
// loop is nearly all FMAs.  Every output still sums its taps in ascending
// order: results are bit-identical to the generic kernels.
constexpr int R64 = 64;
constexpr int R64_ROW_OUT = 4;                      // outputs per thread
constexpr int R64_ROW_THREADS = 256;
constexpr int R64_ROW_TILE = R64_ROW_OUT * R64_ROW_THREADS;  // 1024 outputs per block

// Row-pass sources: a plane, or the baseline preset's halation source
// max(0, R - threshold) formed from interleaved RGB as it is read.
struct PlaneSource {
    const float* __restrict__ p;
    __device__ float operator()(size_t i) const { return __ldg(p + i); }
};
struct HalationSource {
    const float* __restrict__ rgb;
    float threshold;
    __device__ float operator()(size_t i) const { return fmaxf(0.0f, __ldg(rgb + 3 * i) - threshold); }
};

// Transpose of the mirror-reflect blur pass (blur.rs:70-89) for symmetric
// taps w and a line of n > R + 1 samples (one reflection at most).  The blur
// reads index -j as j; its transpose sends the weight meant for -j to j.  So
// the transpose is the blur itself plus terms at the ends only: at distance
// d (1 <= d <= R) from an end, + w[R - d] * g[end]; at the end itself,
// - sum_{j=1..R} w[R - j] * g[end -+ j].  Returns the terms at position `pos`;
// g(i) is sample i of the line, w(k) tap k.
template <class T, class G, class Wt>
__device__ __forceinline__ T transpose_end(int pos, int n, int R, T d, G g, Wt w) {
    const int q = n - 1 - pos;
    if (pos == 0) {
        T acc = d - d;
#pragma unroll 8
        for (int j = 1; j <= R; j++) acc = acc + w(R - j) * g(j);
        d = d - acc;
    } else if (pos <= R) {
        d = d + w(R - pos) * g(0);
    }
    if (q == 0) {
        T acc = d - d;
#pragma unroll 8
        for (int j = 1; j <= R; j++) acc = acc + w(R - j) * g(n - 1 - j);
        d = d - acc;
    } else if (q <= R) {
        d = d + w(R - q) * g(n - 1);
    }
    return d;
}

// The R64_ROW_OUT outputs whose 129-sample windows start at s, s + 1, ...
// (s 16-byte aligned in shared memory).
__device__ __forceinline__ void row_r64(const float* s, const Taps2& tp, float (&out)[R64_ROW_OUT]) {
    static_assert(R64_ROW_OUT % 2 == 0, "outputs go in pairs");
    float2 acc[R64_ROW_OUT / 2];
#pragma unroll
    for (int j = 0; j < R64_ROW_OUT / 2; j++) acc[j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < (R64_ROW_OUT + 2 * R64) / 4; q++) {
        const float4 v4 = *reinterpret_cast<const float4*>(s + 4 * q);
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float2 vv = make_float2(v[u], v[u]);
#pragma unroll
            for (int j = 0; j < R64_ROW_OUT / 2; j++) {
                const int k = 4 * q + u - 2 * j;
                if (k >= 0 && k <= 2 * R64 + 1) acc[j] = __ffma2_rn(vv, tp.t2[k], acc[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < R64_ROW_OUT / 2; j++) {
        out[2 * j] = acc[j].x;
        out[2 * j + 1] = acc[j].y;
    }
}

template <class Src>
__global__ void __launch_bounds__(R64_ROW_THREADS) blur_rows_r64_kernel(const Src in, float* __restrict__ out, int W,
                                                                       int H, const __grid_constant__ Taps2 tp) {
    __shared__ __align__(16) float s[R64_ROW_TILE + 2 * R64];
    const int y = blockIdx.y, x0 = blockIdx.x * R64_ROW_TILE;
    const size_t row = (size_t)y * W;
    for (int j = threadIdx.x; j < R64_ROW_TILE + 2 * R64; j += blockDim.x) s[j] = in(row + reflect(x0 - R64 + j, W));
    __syncthreads();
    const int xb = R64_ROW_OUT * threadIdx.x;
    float a[R64_ROW_OUT];
    row_r64(s + xb, tp, a);
    float* o = out + (size_t)y * W;
#pragma unroll
    for (int j = 0; j < R64_ROW_OUT; j++)
        if (x0 + xb + j < W) o[x0 + xb + j] = a[j];
}

constexpr int R64_COL_TW = 32, R64_COL_GROUPS = 8, R64_COL_OUT = 16;  // 32x8 threads, 16 rows each
constexpr int R64_COL_TH = R64_COL_GROUPS * R64_COL_OUT;              // 128 output rows per block
// the plain column blur: output rows per thread
constexpr int BLUR_COL_OUT = 16;

// Stages rows y0 - 64 .. y0 + TH + 63 of column x into the block's window s
// (mirrored at the image edges).  Blocks whose rows all lie inside
// the image read them directly, the loop unrolled so a thread's 32 loads are
// in flight together; edge blocks mirror each row.
template <int TH>
__device__ __forceinline__ void stage_col_window(float* s, const float* __restrict__ in, int W, int H, int x, int y0,
                                                 int tx, int ty) {
    constexpr int ROWS = TH + 2 * R64;
    if (y0 - R64 >= 0 && y0 + TH + R64 <= H) {
        const float* src = in + (size_t)(y0 - R64) * W + x;
#pragma unroll
        for (int j = ty; j < ROWS; j += R64_COL_GROUPS) s[j * R64_COL_TW + tx] = __ldg(src + (size_t)j * W);
    } else {
        for (int j = ty; j < ROWS; j += R64_COL_GROUPS)
            s[j * R64_COL_TW + tx] = __ldg(in + (size_t)reflect(y0 - R64 + j, H) * W + x);
    }
}

// Streaming radius-64 column pass.  A CTA walks a 32-column strip down a
// segment of SC_CHUNKS chunks of 128 output rows.  Its shared window is a
// ring of three 128-row slabs: chunk j reads slabs j and j+1 while the rows
// of slab j+2 are loaded into registers (issued before the chunk's FMAs, so
// their latency hides behind them) and stored into the slot of slab j-1
// afterwards.  A segment reads (chunks + 2) slabs for its chunks' rows
// (1.5x for four chunks, against 2x for a block that stages the 256 rows of
// one chunk).  Images too small for three blocks an SM at four chunks take
// segments of fewer chunks (stream_chunks).  Each output sums its taps in
// ascending order with the pair taps (t[k], t[k-1]): the same value as the
// generic column blur.
constexpr int SC_SLAB = R64_COL_GROUPS * BLUR_COL_OUT;  // 128 rows: one chunk of outputs, one slab of inputs
constexpr int SC_CHUNKS = 4;

// Chunks of a segment for a W x H image: four, or as few as leave three
// blocks for each of `sms` SMs (2048 x 1365, 148 SMs: one chunk, 23 us against 27.5).
inline int stream_chunks(int W, int H, int sms) {
    const int strips = (W + R64_COL_TW - 1) / R64_COL_TW, chunks = (H + SC_SLAB - 1) / SC_SLAB;
    int c = SC_CHUNKS;
    while (c > 1 && strips * ((chunks + c - 1) / c) < 3 * sms) c /= 2;
    return c;
}
constexpr int SC_PER = SC_SLAB / R64_COL_GROUPS;  // slab rows loaded per thread

template <class Epi>
__global__ void __launch_bounds__(R64_COL_TW * R64_COL_GROUPS) blur_cols_r64_stream_kernel(
    const float* __restrict__ in, int W, int H, int chunks, const __grid_constant__ Taps2 tp, Epi epi) {
    static_assert(SC_SLAB == 2 * R64, "a chunk's 256-row window is two slabs");
    __shared__ float ring[3 * SC_SLAB * R64_COL_TW];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x = blockIdx.x * R64_COL_TW + tx;
    const bool xin = x < W;
    const int ybase = blockIdx.y * chunks * SC_SLAB;
    const int left = (H - ybase + SC_SLAB - 1) / SC_SLAB;
    const int nch = left < chunks ? left : chunks;
    float v[SC_PER];
    // slab s: rows ybase - 64 + 128 s .. + 127 of column x (mirrored at the edges)
    auto load = [&](int sl) {
        const int r0 = ybase - R64 + SC_SLAB * sl;
        if (r0 >= 0 && r0 + SC_SLAB <= H) {
            const float* src = in + (size_t)(r0 + ty) * W + x;
#pragma unroll
            for (int q = 0; q < SC_PER; q++) v[q] = xin ? __ldg(src + (size_t)q * R64_COL_GROUPS * W) : 0.0f;
        } else {
#pragma unroll
            for (int q = 0; q < SC_PER; q++)
                v[q] = xin ? __ldg(in + (size_t)reflect(r0 + ty + q * R64_COL_GROUPS, H) * W + x) : 0.0f;
        }
    };
    auto store = [&](int sl) {
        float* slab = ring + (sl % 3) * SC_SLAB * R64_COL_TW;
#pragma unroll
        for (int q = 0; q < SC_PER; q++) slab[(ty + q * R64_COL_GROUPS) * R64_COL_TW + tx] = v[q];
    };
    load(0);
    store(0);
    load(1);
    store(1);
    __syncthreads();
    const int rb = ty * BLUR_COL_OUT;
    for (int j = 0; j < nch; j++) {
        if (j + 1 < nch) load(j + 2);  // in flight during this chunk
        const float* A = ring + (j % 3) * SC_SLAB * R64_COL_TW;
        const float* B = ring + ((j + 1) % 3) * SC_SLAB * R64_COL_TW;
        float2 acc[BLUR_COL_OUT / 2];
#pragma unroll
        for (int q = 0; q < BLUR_COL_OUT / 2; q++) acc[q] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int m = 0; m < BLUR_COL_OUT + 2 * R64; m++) {
            const int row = rb + m;
            const float val = row < SC_SLAB ? A[row * R64_COL_TW + tx] : B[(row - SC_SLAB) * R64_COL_TW + tx];
            const float2 vv = make_float2(val, val);
#pragma unroll
            for (int q = 0; q < BLUR_COL_OUT / 2; q++) {
                const int k = m - 2 * q;
                if (k >= 0 && k <= 2 * R64 + 1) acc[q] = __ffma2_rn(vv, tp.t2[k], acc[q]);
            }
        }
        if (xin) {
            const int y0 = ybase + j * SC_SLAB + rb;
#pragma unroll
            for (int q = 0; q < BLUR_COL_OUT / 2; q++) {
                const int yy = y0 + 2 * q;
                if (yy < H) epi((size_t)yy * W + x, acc[q].x);
                if (yy + 1 < H) epi((size_t)(yy + 1) * W + x, acc[q].y);
            }
        }
        if (j + 1 < nch) store(j + 2);  // into the slot of slab j-1, read last in chunk j-1
        __syncthreads();
    }
}

struct EpiStore {
    float* out;
    __device__ __forceinline__ void operator()(size_t i, float v) const { out[i] = v; }
};
}  // namespace film
}  // namespace imops
