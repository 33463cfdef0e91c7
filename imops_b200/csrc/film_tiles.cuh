// film_tiles.cuh -- separable blurs of small radius over several layer planes
// in one kernel, for the reference film model (included by film.cu).
//
// The model's local scatter, DIR inhibition and adjacency blur every layer
// with a Gaussian of a few pixels.  As a row launch and a column launch a
// layer, each pass moved the plane through memory and read a shared sample
// per tap.  Here a block owns a 64 x 32 tile of every layer: the tile and its
// halo come in with cp.async (the next layer's while this one is blurred),
// the row pass slides a register window over four outputs a thread and the
// column pass over eight, with the taps as constant-bank operands (the radius
// a template argument).  Every output sums its taps in ascending order, rows
// first, as the separate passes do.
#pragma once

#include "blur.cuh"

namespace imops {
namespace film {

constexpr int FT_W = 64, FT_H = 32, FT_MAXR = 16;
// rows a thread of a block of T threads
constexpr int ft_rpt(int T) { return FT_W * FT_H / T; }

// A staged row starts ft_pad(R) samples left of the halo, at a column that is
// a multiple of 4 (x0 is), and its stride is a multiple of 4: the copies and
// the row pass move float4s.
__host__ __device__ constexpr int ft_pad(int R) { return (4 - R % 4) % 4; }
__host__ __device__ constexpr int ft_stride(int R) { return (ft_pad(R) + FT_W + 2 * R + 3) / 4 * 4; }
__host__ __device__ constexpr int ft_tile_floats(int R) { return (FT_H + 2 * R) * ft_stride(R); }
__host__ __device__ constexpr int ft_row_floats(int R) { return (FT_H + 2 * R) * FT_W; }

__device__ __forceinline__ void ft_cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void ft_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void ft_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ft_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// How a block copies its tiles: whole rows a warp.  Where every staged sample
// is an image sample and rows are 16-byte aligned (planes are, when W is a
// multiple of 4 and the first is), lane l copies the float4 l; elsewhere the
// samples l, l + 32, l + 64 and l + 96 one by one, its image columns (mirrored
// at the edges) the same for every row and plane.
constexpr int FT_COLS = 4;
static_assert(ft_stride(FT_MAXR) <= 128 && ft_stride(FT_MAXR - 1) <= 128, "a row is at most 32 float4s");
struct FtCopy {
    int x[FT_COLS];
    bool vec;
};
__device__ __forceinline__ FtCopy ft_copy(const float* plane, int x0, int y0, int R, int W, int H) {
    FtCopy c;
    const int xs = x0 - R - ft_pad(R);
    c.vec = (W & 3) == 0 && ((uintptr_t)plane & 15) == 0 && xs >= 0 && xs + ft_stride(R) <= W && y0 >= R &&
            y0 + FT_H + R <= H;
    const int lane = threadIdx.x & 31;
    if (c.vec) c.x[0] = xs + 4 * lane;
    else
#pragma unroll
        for (int t = 0; t < FT_COLS; t++) c.x[t] = reflect(xs + lane + 32 * t, W);
    return c;
}

// Starts the copy of one plane's tile and halo.
template <int T>
__device__ __forceinline__ void ft_load(float* s, const float* __restrict__ plane, const FtCopy& c, int y0, int R,
                                        int W, int H) {
    const int SW = ft_stride(R), NH = FT_H + 2 * R, lane = threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
    if (c.vec) {
        if (4 * lane < SW) {
            const float* src = plane + (size_t)(y0 - R + warp) * W + c.x[0];
            float* dst = s + warp * SW + 4 * lane;
            for (int r = warp; r < NH; r += T / 32) {
                ft_cp16(dst, src);
                src += (size_t)(T / 32) * W;
                dst += T / 32 * SW;
            }
        }
        return;
    }
    for (int r = warp; r < NH; r += T / 32) {
        const float* src = plane + (size_t)reflect(y0 - R + r, H) * W;
        float* dst = s + r * SW + lane;
#pragma unroll
        for (int t = 0; t < FT_COLS; t++)
            if (32 * t + lane < SW) ft_cp4(dst + 32 * t, src + c.x[t]);
    }
}

// Row pass over the tile and its row halo: s (stride ft_stride(R)) -> rows (stride FT_W).
template <int T, int R>
__device__ __forceinline__ void ft_rows(const float* s, float* rows, const float* taps) {
    constexpr int SW = ft_stride(R), A = ft_pad(R), NH = FT_H + 2 * R, NQ = (A + 4 + 2 * R + 3) / 4;
    for (int i = threadIdx.x; i < NH * (FT_W / 4); i += T) {
        const int r = i / (FT_W / 4), g = i % (FT_W / 4);
        const float* p = s + r * SW + 4 * g;
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const float4 v4 = *reinterpret_cast<const float4*>(p + 4 * q);
            const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int k = 4 * q + u - A - j;
                    if (k >= 0 && k <= 2 * R) a[j] = fmaf(v[u], taps[k], a[j]);
                }
        }
        *reinterpret_cast<float4*>(rows + r * FT_W + 4 * g) = make_float4(a[0], a[1], a[2], a[3]);
    }
}

// Column pass: the N outputs of this thread (column tx, rows rb ..).
template <int R, int N>
__device__ __forceinline__ void ft_cols(const float* rows, int tx, int rb, const float* taps, float (&out)[N]) {
#pragma unroll
    for (int j = 0; j < N; j++) out[j] = 0.0f;
#pragma unroll
    for (int m = 0; m < N + 2 * R; m++) {
        const float v = rows[(rb + m) * FT_W + tx];
#pragma unroll
        for (int j = 0; j < N; j++) {
            const int k = m - j;
            if (k >= 0 && k <= 2 * R) out[j] = fmaf(v, taps[k], out[j]);
        }
    }
}

// Row pass, barrier, column pass with the radius as a template argument.
template <int T, int RMAX, int R = 1, int N>
__device__ __forceinline__ void ft_blur(const float* s, float* rows, int tx, int rb, const Taps& tp, float (&out)[N]) {
    if constexpr (R <= RMAX) {
        if (tp.R == R) {
            ft_rows<T, R>(s, rows, tp.t);
            __syncthreads();
            ft_cols<R>(rows, tx, rb, tp.t, out);
        } else {
            ft_blur<T, RMAX, R + 1>(s, rows, tx, rb, tp, out);
        }
    }
}

// ---- DIR inhibition (diffusion.rs:39-84) -------------------------------------
// out_j = in_j exp(-sum_i m[i][j] blur(in_i)), every layer blurred and mixed in
// one kernel: the layers' inhibition of a thread's eight pixels accumulates
// in registers as the layers go by, so a layer's blur is never stored.  Bound
// by instruction issue (0.66 of the issue rate at two blocks an SM: the
// accumulators take 48 of 128 registers).  24 MP, six layers, radius 9:
// 0.66 ms against 2.8 ms as twelve blur launches and a mixing pass (0.90 with
// the halo copied sample by sample in index order).
template <int E>
struct DirMix {
    float m[E][E];
};

constexpr int DIR_THREADS = 256, DIR_ROWS = ft_rpt(DIR_THREADS);

template <int E>
__global__ void __launch_bounds__(DIR_THREADS, E <= 3 ? 3 : 2)
    dir_kernel(const float* __restrict__ in, float* __restrict__ out, int W, int H, const __grid_constant__ Taps tp,
               const __grid_constant__ DirMix<E> mix) {
    extern __shared__ __align__(16) float ftsm[];
    const int R = tp.R, tile = ft_tile_floats(R);
    float* rows = ftsm + 2 * tile;
    const int x0 = blockIdx.x * FT_W, y0 = blockIdx.y * FT_H;
    const int tx = threadIdx.x % FT_W, rb = (int)threadIdx.x / FT_W * DIR_ROWS;
    const size_t n = (size_t)W * H;
    float tot[E][DIR_ROWS];
#pragma unroll
    for (int j = 0; j < E; j++)
#pragma unroll
        for (int r = 0; r < DIR_ROWS; r++) tot[j][r] = 0.0f;
    const FtCopy cols = ft_copy(in, x0, y0, R, W, H);
    ft_load<DIR_THREADS>(ftsm, in, cols, y0, R, W, H);
    ft_commit();
#pragma unroll 1
    for (int i = 0; i < E; i++) {
        ft_wait<0>();
        __syncthreads();  // this layer's tile is complete; the row buffer and the other tile are free
        if (i + 1 < E) {
            ft_load<DIR_THREADS>(ftsm + ((i + 1) & 1) * tile, in + (i + 1) * n, cols, y0, R, W, H);
            ft_commit();
        }
        float v[DIR_ROWS];
        ft_blur<DIR_THREADS, FT_MAXR>(ftsm + (i & 1) * tile, rows, tx, rb, tp, v);
#pragma unroll
        for (int j = 0; j < E; j++) {
            const float w = mix.m[i][j];
            if (w != 0.0f)
#pragma unroll
                for (int r = 0; r < DIR_ROWS; r++) tot[j][r] = fmaf(w, v[r], tot[j][r]);
        }
    }
    const int x = x0 + tx;
    if (x >= W) return;
#pragma unroll
    for (int r = 0; r < DIR_ROWS; r++) {
        const int y = y0 + rb + r;
        if (y >= H) break;
        const size_t p = (size_t)y * W + x;
#pragma unroll
        for (int j = 0; j < E; j++) out[j * n + p] = __fmul_rn(__ldg(in + j * n + p), expf(-tot[j][r]));
    }
}

}  // namespace film
}  // namespace imops
