// demosaic_simple.cu -- the reference's 3x3 same-colour mean ("Markesteijn",
// pichromatic/src/demosaic.rs:108-186) and the quad-sampling previews
// (Fast / SuperFast / SuperSuperFast, demosaic.rs:189-356).
//
// The mean reads a mosaic (4 B a pixel, or 2 B of the sensor frame, scaled
// while it is staged) and writes 12 B.  Every Bayer CFA is a shift of RGGB and
// every X-Trans sensor's CFA a shift of one 6x6 pattern, so for those the
// kernel aligns each thread's run of pixels with the pattern: the colour of
// every site in a run's window is then a compile-time constant (per row phase,
// and a warp handles one row), the per-colour sums are plain adds and the
// counts constants.  Other CFAs take the per-pixel kernel.  Both sum each
// colour's sites in row-major order and divide once, as the reference's f32
// code does; built with --fmad=false.
#include <type_traits>

#include "cfa_canon.cuh"
#include "color.cuh"
#include "common.cuh"
#include "demosaic_simple.cuh"

namespace imops {
namespace simple {

using canon::BayerCanon;
using canon::canonical_offset;
using canon::XTransCanon;

// One output pixel: the mean of each colour's sites among the 8 neighbours
// (the window clamped at the image edges), the centre's own colour keeping
// the centre sample.  Cfa: CfaFixed<2, 2> / CfaFixed<6, 6> for Bayer and
// X-Trans, CfaDev for other periods; coordinates here are never negative.
// in(y, x): the mosaic; in.load(in.window(row, col), a, b): sample (a, b) of the
// 3x3 window about (row, col), from one address for the window (24 MP by the
// per-pixel kernel: other 6x6 CFAs 247 us, 268 with an address a sample; other
// 2x2 ones 169, 191).
template <class In, class Cfa>
__device__ __forceinline__ void mean_px(const In& in, int W, int H, const Cfa& cfa, int row, int col, float* o) {
    const int centre = cfa.at(row, col);
    if (row >= 1 && row + 1 < H && col >= 1 && col + 1 < W) {
        // interior: the whole 3x3 window, unrolled and branch-free; each
        // colour's sum takes its sites in row-major order (predicated adds)
        const float* p = in.window(row, col);
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                if (a == 1 && b == 1) continue;
                const int k = cfa.at(row + a - 1, col + b - 1);
                const float v = in.load(p, a, b);
                s0 = k == 0 ? s0 + v : s0;
                n0 = k == 0 ? n0 + 1.0f : n0;
                s1 = k == 1 ? s1 + v : s1;
                n1 = k == 1 ? n1 + 1.0f : n1;
                s2 = k == 2 ? s2 + v : s2;
                n2 = k == 2 ? n2 + 1.0f : n2;
            }
        const float self = in(row, col);
        o[0] = centre == 0 ? self : (n0 > 0.0f ? s0 / n0 : 0.0f);
        o[1] = centre == 1 ? self : (n1 > 0.0f ? s1 / n1 : 0.0f);
        o[2] = centre == 2 ? self : (n2 > 0.0f ? s2 / n2 : 0.0f);
        return;
    }
    int y0 = row > 0 ? row - 1 : 0, y1 = row + 1 < H - 1 ? row + 1 : H - 1;
    int x0 = col > 0 ? col - 1 : 0, x1 = col + 1 < W - 1 ? col + 1 : W - 1;
    // one row-major pass over the window: each colour's sum takes its sites
    // in the order of the reference's per-colour loops
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
    for (int ny = y0; ny <= y1; ny++)
        for (int nx = x0; nx <= x1; nx++) {
            if (ny == row && nx == col) continue;
            const int k = cfa.at(ny, nx);
            const float v = in(ny, nx);
            if (k == 0) {
                s0 += v;
                n0 += 1.0f;
            } else if (k == 1) {
                s1 += v;
                n1 += 1.0f;
            } else if (k == 2) {
                s2 += v;
                n2 += 1.0f;
            }
        }
    const float self = in(row, col);
    o[0] = centre == 0 ? self : (n0 > 0.0f ? s0 / n0 : 0.0f);
    o[1] = centre == 1 ? self : (n1 > 0.0f ? s1 / n1 : 0.0f);
    o[2] = centre == 2 ? self : (n2 > 0.0f ? s2 / n2 : 0.0f);
}

// An f32 mosaic.
struct SrcF32 {
    const float* __restrict__ p;
    int W;
    using Raw = float;
    __device__ __forceinline__ float operator()(int y, int x) const { return __ldg(p + (size_t)y * W + x); }
    __device__ __forceinline__ const float* window(int row, int col) const {
        return p + (size_t)(row - 1) * W + (col - 1);
    }
    __device__ __forceinline__ float load(const float* q, int a, int b) const { return __ldg(q + (size_t)a * W + b); }
};

// The mean alone.
struct NoEpilogue {
    __device__ __forceinline__ void apply(float&, float&, float&) const {}
};

// One thread per output pixel, for CFAs that are no shift of a canonical
// pattern; epi (NoEpilogue or color::Epilogue) maps each pixel's RGB before
// the store.
template <class Cfa, class Epi>
__global__ void mean3x3_kernel(const float* __restrict__ in, int W, int H, const __grid_constant__ Cfa cfa,
                               const __grid_constant__ Epi epi, float* __restrict__ out) {
    int col = blockIdx.x * blockDim.x + threadIdx.x;
    int row = blockIdx.y * blockDim.y + threadIdx.y;
    if (col >= W || row >= H) return;
    float v[3];
    mean_px(SrcF32{in, W}, W, H, cfa, row, col, v);
    epi.apply(v[0], v[1], v[2]);
    float* o = out + ((size_t)row * W + col) * 3;
    o[0] = v[0];
    o[1] = v[1];
    o[2] = v[2];
}

// Phase-aligned kernel geometry: a warp handles one image row, RUN pixels a
// lane, 32 * RUN pixels a warp; RUN is a multiple of both periods.  A block's
// eight rows share ten staged ones.
constexpr int RUN = 6;
constexpr int WARP_PX = 32 * RUN;              // 192
constexpr int IN_STRIDE = WARP_PX + 4;         // 194 staged columns, padded to a 16-byte multiple
constexpr int OUT_STRIDE = 3 * WARP_PX + 4;    // an RGB row and up to 3 floats of alignment offset
constexpr int MEAN_WARPS = 8;

// The RUN pixels of one lane at canonical row phase RP: window v = rows
// y-1..y+1, columns x0-1..x0+RUN; pixel j sits at canonical column j mod PW.
// Same adds in the same order as mean_px's interior branch, with the colour
// tests and counts folded away.
template <class P, int RP>
__device__ __forceinline__ void run_aligned(const float (&v)[3][RUN + 2], float* o) {
#pragma unroll
    for (int j = 0; j < RUN; j++) {
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                if (a == 1 && b == 1) continue;
                const int k = P::at((RP + a + P::PH - 1) % P::PH, (j + b + P::PW - 1) % P::PW);
                const float x = v[a][j + b];
                if (k == 0) {
                    s0 = s0 + x;
                    n0 = n0 + 1.0f;
                } else if (k == 1) {
                    s1 = s1 + x;
                    n1 = n1 + 1.0f;
                } else {
                    s2 = s2 + x;
                    n2 = n2 + 1.0f;
                }
            }
        const int centre = P::at(RP, j % P::PW);
        const float self = v[1][j + 1];
        o[3 * j + 0] = centre == 0 ? self : (n0 > 0.0f ? s0 / n0 : 0.0f);
        o[3 * j + 1] = centre == 1 ? self : (n1 > 0.0f ? s1 / n1 : 0.0f);
        o[3 * j + 2] = centre == 2 ? self : (n2 > 0.0f ? s2 / n2 : 0.0f);
    }
}

template <class P, int RP>
__device__ __forceinline__ void run_phase(int rp, const float (&v)[3][RUN + 2], float* o) {
    if constexpr (RP < P::PH) {
        if (rp == RP) run_aligned<P, RP>(v, o);
        else run_phase<P, RP + 1>(rp, v, o);
    }
}

// The rows a block has staged, from row y0 and column x0 of the mosaic on.
struct SrcStaged {
    const float (*s)[IN_STRIDE];
    int y0, x0;
    __device__ __forceinline__ float operator()(int y, int x) const { return s[y - y0][x - x0]; }
    __device__ __forceinline__ const float* window(int row, int col) const { return &s[row - 1 - y0][col - 1 - x0]; }
    __device__ __forceinline__ float load(const float* q, int a, int b) const { return q[a * IN_STRIDE + b]; }
};

// What the aligned kernel stages: an f32 mosaic as it is, or a u16 sensor
// frame's crop scaled as color::scale_u16_kernel does, (v - black) / (white -
// black) per cell of the level period, each sample once a block (1.29 times a
// pixel with the halo).
struct StageF32 {
    SrcF32 src;
    using Raw = float;
    __device__ __forceinline__ void init(float*) const {}
    __device__ __forceinline__ Raw fetch(int y, int x) const { return src(y, x); }
    __device__ __forceinline__ float value(Raw v, const float*, int, int) const { return v; }
    __device__ __forceinline__ int column(int) const { return 0; }
    __device__ __forceinline__ int next(int c) const { return c; }
    __device__ __forceinline__ int row(int) const { return 0; }
};
struct StageU16 {  // one level pair for all cells
    const uint16_t* __restrict__ raw;  // at the crop's origin
    int raw_w;
    color::LevelRange lv;
    using Raw = uint16_t;
    __device__ __forceinline__ void init(float*) const {}
    __device__ __forceinline__ Raw fetch(int y, int x) const { return __ldg(raw + (size_t)y * raw_w + x); }
    __device__ __forceinline__ float value(Raw v, const float*, int, int) const { return lv.scale((float)v); }
    __device__ __forceinline__ int column(int) const { return 0; }
    __device__ __forceinline__ int next(int c) const { return c; }
    __device__ __forceinline__ int row(int) const { return 0; }
};
struct StageU16Cells {
    const uint16_t* __restrict__ raw;  // at the crop's origin
    int raw_w, cx, cy, pw, ph, step;   // step = 32 % pw
    float black[144], range[144];
    using Raw = uint16_t;
    __device__ __forceinline__ void init(float* levels) const {
        for (int i = threadIdx.y * 32 + threadIdx.x; i < pw * ph; i += 32 * MEAN_WARPS) {
            levels[i] = black[i];
            levels[144 + i] = range[i];
        }
        __syncthreads();
    }
    __device__ __forceinline__ Raw fetch(int y, int x) const { return __ldg(raw + (size_t)y * raw_w + x); }
    __device__ __forceinline__ float value(Raw v, const float* levels, int row, int col) const {
        const int i = row * pw + col;
        return ((float)v - levels[i]) / levels[144 + i];
    }
    // a column's and a row's place in the level period
    __device__ __forceinline__ int column(int x) const { return (cx + x + 144 * pw) % pw; }
    __device__ __forceinline__ int next(int c) const { return c + step >= pw ? c + step - pw : c + step; }
    __device__ __forceinline__ int row(int y) const { return (cy + y + ph) % ph; }
};

// The CFA is P shifted: colour(y, x) = P::at((y - oy) mod PH, (x - ox) mod PW)
// with 0 <= ox < PW, 0 <= oy < PH.  Warp w of block (bx, by) develops row
// y = 8 by + w, pixels x_start + 192 bx .. + 191 with x_start = 0 when
// ox == 0 else ox - PW, so every lane's run starts at canonical column 0.
// The block stages its ten rows in shared memory (coalesced loads), each
// lane computes its run from there -- or, when the run or its window touches
// the image edge, each pixel with mean_px -- into a shared output row that
// the warp then stores coalesced.
//
// Bound by instruction issue with a colour epilogue, by HBM latency without.
// 24 MP: X-Trans u16 frame to ACEScg in one pass 166 us, where scaling it to an
// f32 mosaic (34) and three rows staged a warp (177) took 211; f32 mosaic to
// camera RGB 98 us (100).
template <class P, class Epi, class Stage>
__global__ void __launch_bounds__(32 * MEAN_WARPS, std::is_same<Stage, StageF32>::value ? 5 : 4) mean3x3_aligned_kernel(
    const __grid_constant__ Stage st, int W, int H, int ox, int oy, const __grid_constant__ CfaFixed<P::PW, P::PH> cfa,
    const __grid_constant__ Epi epi, float* __restrict__ out) {
    __shared__ __align__(16) float sin_[MEAN_WARPS + 2][IN_STRIDE];
    __shared__ __align__(16) float sout[MEAN_WARPS][OUT_STRIDE];
    __shared__ float levels[std::is_same<Stage, StageU16Cells>::value ? 288 : 1];
    st.init(levels);
    const int lane = threadIdx.x, w = threadIdx.y;
    const int y0 = blockIdx.y * MEAN_WARPS, y = y0 + w;
    const int xs = ox == 0 ? 0 : ox - P::PW;
    const int xw = xs + blockIdx.x * WARP_PX;  // first pixel of the warp
    // stage rows y0-1 .. y0+8, columns xw-1 .. xw+192 (zeros outside the image,
    // read by nothing that is stored): warp w row w, warps 0 and 1 also rows
    // 8 and 9.  A row's seven loads a lane are issued before its first store.
    constexpr int NQ = (WARP_PX + 2 + 31) / 32;
    const bool inner = xw >= 1 && xw + WARP_PX + 1 <= W;
    int col[NQ];
    col[0] = st.column(xw - 1 + lane);
#pragma unroll
    for (int q = 1; q < NQ; q++) col[q] = st.next(col[q - 1]);
#pragma unroll 1
    for (int a = 0; a < 2; a++) {
        const int r = w + MEAN_WARPS * a, yy = y0 - 1 + r;
        if (r >= MEAN_WARPS + 2) break;
        const bool yin = yy >= 0 && yy < H;
        typename Stage::Raw t[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int i = lane + 32 * q, x = xw - 1 + i;
            t[q] = yin && i < WARP_PX + 2 && (inner || (x >= 0 && x < W)) ? st.fetch(yy, x) : typename Stage::Raw(0);
        }
        const int rp = st.row(yy);
#pragma unroll
        for (int q = 0; q < NQ; q++)
            if (lane + 32 * q < WARP_PX + 2) sin_[r][lane + 32 * q] = st.value(t[q], levels, rp, col[q]);
    }
    __syncthreads();
    if (y >= H) return;  // whole warp: only warp-level synchronisation below
    // the warp's pixels inside the image, and the shared output row's offset
    // m: float k of the row goes to address dst0 + (k - K0), and m makes
    // shared and global 16-byte boundaries coincide
    const int p0 = xw > 0 ? xw : 0, p1 = xw + WARP_PX < W ? xw + WARP_PX : W;
    float* dst0 = out + ((size_t)y * W + p0) * 3;
    const int m = ((int)(((uintptr_t)dst0 >> 2) & 3) - 3 * (p0 - xw)) & 3;
    const int x0 = xw + RUN * lane;
    float* o = &sout[w][m + 3 * RUN * lane];
    if (y >= 1 && y + 1 < H && x0 >= 1 && x0 + RUN + 1 <= W) {
        float v[3][RUN + 2];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int c = 0; c < RUN + 2; c += 2) {
                const float2 t2 = *reinterpret_cast<const float2*>(&sin_[w + a][RUN * lane + c]);
                v[a][c] = t2.x;
                v[a][c + 1] = t2.y;
            }
        const int rp = (y + P::PH - oy) % P::PH;
        float r[3 * RUN];
        run_phase<P, 0>(rp, v, r);
        if (m & 1) {
#pragma unroll
            for (int c = 0; c < 3 * RUN; c++) o[c] = r[c];
        } else {
#pragma unroll
            for (int c = 0; c < 3 * RUN; c += 2) *reinterpret_cast<float2*>(o + c) = make_float2(r[c], r[c + 1]);
        }
    } else {
        for (int j = 0; j < RUN; j++) {
            const int x = x0 + j;
            if (x >= 0 && x < W) {
                float q[3];
                mean_px(SrcStaged{sin_, y0 - 1, xw - 1}, W, H, cfa, y, x, q);
                o[3 * j] = q[0];
                o[3 * j + 1] = q[1];
                o[3 * j + 2] = q[2];
            }
        }
    }
    __syncwarp();
    if (p1 <= p0) return;
    if constexpr (!std::is_same<Epi, NoEpilogue>::value) {
        // the colour epilogue in a loop of its own, a pixel a lane: inlined for
        // each of a run's pixels its code outgrew the instruction cache, as the
        // warps are in different row phases already
#pragma unroll 2
        for (int x = p0 + lane; x < p1; x += 32) {
            float* q = &sout[w][m + 3 * (x - xw)];
            float r = q[0], g = q[1], b = q[2];
            epi.apply(r, g, b);
            q[0] = r;
            q[1] = g;
            q[2] = b;
        }
        __syncwarp();
    }
    // shared floats K0..K1-1 -> dst0: a scalar head up to a 16-byte boundary,
    // float4 chunks, a scalar tail
    const int K0 = m + 3 * (p0 - xw), K1 = m + 3 * (p1 - xw);
    const int c0 = (K0 + 3) >> 2, c1 = K1 >> 2;
    const float* so = sout[w];
    if (c0 >= c1) {
        for (int k = K0 + lane; k < K1; k += 32) dst0[k - K0] = so[k];
        return;
    }
    if (K0 + lane < 4 * c0) dst0[lane] = so[K0 + lane];
    for (int c = c0 + lane; c < c1; c += 32)
        *reinterpret_cast<float4*>(dst0 + (4 * c - K0)) = *reinterpret_cast<const float4*>(so + 4 * c);
    if (4 * c1 + lane < K1) dst0[4 * c1 + lane - K0] = so[4 * c1 + lane];
}

template <class P, class Epi, class Stage>
void launch_aligned(const Stage& st, int w, int h, const CfaDev& c, int ox, int oy, const Epi& epi, float* rgb,
                    cudaStream_t s) {
    const int xs = ox == 0 ? 0 : ox - P::PW;
    dim3 block(32, MEAN_WARPS), grid((w - xs + WARP_PX - 1) / WARP_PX, (h + MEAN_WARPS - 1) / MEAN_WARPS);
    mean3x3_aligned_kernel<P, Epi, Stage><<<grid, block, 0, s>>>(st, w, h, ox, oy, CfaFixed<P::PW, P::PH>::from(c),
                                                                 epi, rgb);
}

// The aligned kernel where the CFA is a shift of a canonical pattern.
template <class Epi, class Stage>
bool launch_canonical(const Stage& st, int w, int h, const CfaDev& c, const Epi& epi, float* rgb, cudaStream_t s) {
    int ox, oy;
    if (canonical_offset<BayerCanon>(c, &ox, &oy)) launch_aligned<BayerCanon>(st, w, h, c, ox, oy, epi, rgb, s);
    else if (canonical_offset<XTransCanon>(c, &ox, &oy)) launch_aligned<XTransCanon>(st, w, h, c, ox, oy, epi, rgb, s);
    else return false;
    return true;
}

template <class Epi>
void launch_mean(const float* mosaic, int w, int h, const CfaDev& c, const Epi& epi, float* rgb, cudaStream_t s) {
    dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    if (launch_canonical(StageF32{{mosaic, w}}, w, h, c, epi, rgb, s)) return;
    if (c.pw == 2 && c.ph == 2)
        mean3x3_kernel<<<grid, block, 0, s>>>(mosaic, w, h, CfaFixed<2, 2>::from(c), epi, rgb);
    else if (c.pw == 6 && c.ph == 6)
        mean3x3_kernel<<<grid, block, 0, s>>>(mosaic, w, h, CfaFixed<6, 6>::from(c), epi, rgb);
    else
        mean3x3_kernel<<<grid, block, 0, s>>>(mosaic, w, h, c, epi, rgb);
}

int mean3x3(const float* mosaic, int w, int h, const CfaDev& c, const color::Epilogue* epi, float* rgb,
            cudaStream_t s) {
    if (!mosaic || !rgb) return fail(IMOPS_ERR_INVALID_ARGUMENT, "markesteijn: NULL buffer");
    if (((uintptr_t)mosaic | (uintptr_t)rgb) & 3)
        return fail(IMOPS_ERR_INVALID_ARGUMENT, "markesteijn: buffers must be 4-byte aligned float arrays");
    if (w <= 0 || h <= 0) return fail(IMOPS_ERR_INVALID_ARGUMENT, "markesteijn: empty image");
    if (fault_injected("launch")) return fail(IMOPS_ERR_CUDA, "injected launch failure (markesteijn)");
    if (epi) launch_mean(mosaic, w, h, c, *epi, rgb, s);
    else launch_mean(mosaic, w, h, c, NoEpilogue{}, rgb, s);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "markesteijn launch");
    return IMOPS_OK;
}

int mean3x3_u16(const uint16_t* raw, int raw_w, int raw_h, int cx, int cy, int w, int h, const float* black,
                const float* white, int pw, int ph, const CfaDev& c, const color::Epilogue& epi, float* rgb,
                bool* done, cudaStream_t s) {
    *done = false;
    int ox, oy;
    if (!canonical_offset<BayerCanon>(c, &ox, &oy) && !canonical_offset<XTransCanon>(c, &ox, &oy)) return IMOPS_OK;
    int rc = color::check_scale(raw, raw_w, raw_h, cx, cy, w, h, black, white, pw, ph, rgb);
    if (rc) return rc;
    if ((uintptr_t)rgb & 3)
        return fail(IMOPS_ERR_INVALID_ARGUMENT, "markesteijn: buffers must be 4-byte aligned float arrays");
    if (fault_injected("launch")) return fail(IMOPS_ERR_CUDA, "injected launch failure (markesteijn)");
    const uint16_t* origin = raw + (size_t)cy * raw_w + cx;
    color::LevelRange one;
    if (one.usable(black, white, pw * ph)) {
        launch_canonical(StageU16{origin, raw_w, one}, w, h, c, epi, rgb, s);
    } else {
        StageU16Cells st{origin, raw_w, cx, cy, pw, ph, 32 % pw, {}, {}};
        for (int i = 0; i < pw * ph; i++) {
            st.black[i] = black[i];
            st.range[i] = white[i] - black[i];
        }
        launch_canonical(st, w, h, c, epi, rgb, s);
    }
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "markesteijn launch");
    *done = true;
    return IMOPS_OK;
}

__global__ void quad_kernel(const float* __restrict__ in, int W, int nw, int nh, int factor, int4 cols,
                            float* __restrict__ out) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nw || y >= nh) return;
    size_t tl = (size_t)(y * factor) * W + (size_t)(x * factor);
    float v[3] = {0.0f, 0.0f, 0.0f};
    v[cols.x] = in[tl];
    v[cols.y] = in[tl + 1];
    v[cols.z] = in[tl + W];
    v[cols.w] = in[tl + W + 1];
    float* o = out + ((size_t)y * nw + x) * 3;
    o[0] = v[0];
    o[1] = v[1];
    o[2] = v[2];
}

}  // namespace simple
}  // namespace imops

extern "C" int imops_demosaic_markesteijn(const float* mosaic, int w, int h, const char* cfa, int shift_x,
                                          int shift_y, float* rgb, imops_stream_t stream) {
    using namespace imops;
    clear_error();
    CfaDev c;
    int rc = parse_cfa(cfa, shift_x, shift_y, &c);
    if (rc) return rc;
    return simple::mean3x3(mosaic, w, h, c, nullptr, rgb, as_stream(stream));
}

extern "C" int imops_demosaic_quad(const float* mosaic, int w, int h, const char* cfa, int shift_x, int shift_y,
                                   int factor, float* rgb, imops_stream_t stream) {
    using namespace imops;
    clear_error();
    CfaDev c;
    int rc = parse_cfa(cfa, shift_x, shift_y, &c);
    if (rc) return rc;
    if (factor != 2 && factor != 4 && factor != 8)
        return fail(IMOPS_ERR_INVALID_ARGUMENT, "quad demosaic: factor must be 2, 4 or 8");
    if (!mosaic || !rgb) return fail(IMOPS_ERR_INVALID_ARGUMENT, "quad demosaic: NULL buffer");
    int nw = w / factor, nh = h / factor;
    int4 cols = make_int4(c.at(0, 0), c.at(0, 1), c.at(1, 0), c.at(1, 1));
    if (cols.x > 2 || cols.y > 2 || cols.z > 2 || cols.w > 2)
        return fail(IMOPS_ERR_UNSUPPORTED_CFA, "quad demosaic: CFA colour outside R/G/B");
    if (nw <= 0 || nh <= 0) return IMOPS_OK;
    dim3 block(32, 8), grid((nw + 31) / 32, (nh + 7) / 8);
    simple::quad_kernel<<<grid, block, 0, as_stream(stream)>>>(mosaic, w, nw, nh, factor, cols, rgb);
    note_launch();
    IMOPS_CUDA_TRY(cudaGetLastError(), "quad demosaic launch");
    return IMOPS_OK;
}
