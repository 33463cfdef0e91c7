// color.cuh -- host-side colour constants and the per-pixel colour epilogue
// shared by the stage kernels (color.cu) and the fused pipeline.
#pragma once

#include "common.cuh"

namespace imops {
namespace color {

// camera -> XYZ(D65) matrix of camera_cst, pichromatic/src/cst.rs:12-38 and
// pseudo_inverse_matrix cst.rs:51-95, in f32 in the reference's order.
void camera_forward_matrix(const float calib[9], float fwd[9]);

// XYZ(D65) -> target 3x3 (row-major) for IMOPS_CS_{XYZD65,LINEAR_SRGB,SRGB,ACESCG};
// false for other targets.  AcesCg uses the reference's own XYZ->AP1 matrix
// (film/exposure/upsample.rs:34-38); linear sRGB the CSS Color 4 matrix.
bool xyz_to_target(int target, float m[9]);

// 2^ev in f32 as exp.rs:5 computes it (glibc powf, as Rust's f32::powf).
float exp_value(float ev);

// Absolute-luminance gain K*N^2/(t*S) (film/exposure/radiance.rs:19-31), f64 -> f32.
float luminance_gain(float shutter, float f_number, float iso);

// Per-pixel colour after demosaic, applied in the reference's module order:
// WB (cfa_coeffs.rs:4-12), exposure gain(s) (exp.rs:4-11), camera CST
// (cst.rs:39-46).  Each step is its own f32 multiply/mat-vec so the
// rounding matches the separate module passes.
struct Epilogue {
    float wb[3];
    int n_gain;       // 0..4 scalar gains applied one after another
    float gain[4];
    int do_cst;
    float fwd[9];
    float tgt[9];
    int srgb;         // apply the sRGB transfer after the target matrix
    int src_srgb;     // decode an sRGB-encoded input before the first matrix

    __device__ __forceinline__ void apply(float& r, float& g, float& b) const {
        r = r * wb[0];
        g = g * wb[1];
        b = b * wb[2];
        for (int k = 0; k < n_gain; k++) {
            r = r * gain[k];
            g = g * gain[k];
            b = b * gain[k];
        }
        if (do_cst) {
            if (src_srgb) {
                r = srgb_decode(r);
                g = srgb_decode(g);
                b = srgb_decode(b);
            }
            float x = fwd[0] * r + fwd[1] * g + fwd[2] * b;
            float y = fwd[3] * r + fwd[4] * g + fwd[5] * b;
            float z = fwd[6] * r + fwd[7] * g + fwd[8] * b;
            r = tgt[0] * x + tgt[1] * y + tgt[2] * z;
            g = tgt[3] * x + tgt[4] * y + tgt[5] * z;
            b = tgt[6] * x + tgt[7] * y + tgt[8] * z;
            if (srgb) {
                r = srgb_encode(r);
                g = srgb_encode(g);
                b = srgb_encode(b);
            }
        }
    }

    __device__ __forceinline__ static float srgb_decode(float v) {
        float a = fabsf(v);
        float l = a <= 0.04045f ? a / 12.92f : powf((a + 0.055f) / 1.055f, 2.4f);
        return v < 0.0f ? -l : l;
    }

    // sRGB transfer with odd symmetry (IEC 61966-2-1).
    __device__ __forceinline__ static float srgb_encode(float v) {
        float a = fabsf(v);
        float e = a <= 0.0031308f ? 12.92f * a : 1.055f * powf(a, 1.0f / 2.4f) - 0.055f;
        return v < 0.0f ? -e : e;
    }
};

// Colour space -> XYZ(D65) 3x3 for IMOPS_CS_{XYZD65,LINEAR_SRGB,SRGB (after
// decoding),ACESCG}; false otherwise.
bool to_xyz(int space, float m[9]);

// Division by one level range d for many samples: with y = 1/d correctly
// rounded, q = n y corrected once by the exact remainder, q + (n - q d) y, is
// the correctly rounded n / d (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990),
// three operations for the ten of a division.  Exact remainders need room
// below n: `usable` where the black level is 0 or at least 2^-20 in magnitude
// (so v - black is 0 or at least 2^-44) and the range lies in 2^-20 .. 2^20.
struct LevelRange {
    float black, range, inv;
    __device__ __forceinline__ float scale(float v) const {
        const float n = v - black, q = n * inv;
        return __fmaf_rn(__fmaf_rn(-range, q, n), inv, q);
    }
    // the n levels all the same and usable
    bool usable(const float* blacks, const float* whites, int n) {
        for (int i = 1; i < n; i++)
            if (blacks[i] != blacks[0] || whites[i] != whites[0]) return false;
        black = blacks[0];
        range = whites[0] - black;
        inv = 1.0f / range;
        const float lo = 1.0f / 1048576.0f, hi = 1048576.0f, b = black < 0.0f ? -black : black;
        return (b == 0.0f || (b >= lo && b <= hi)) && range >= lo && range <= hi;
    }
};

// The argument checks of imops_scale_u16.
int check_scale(const uint16_t* raw, int raw_w, int raw_h, int crop_x, int crop_y, int crop_w, int crop_h,
                const float* black, const float* white, int period_w, int period_h, const float* out);

// Builds an identity epilogue (no-op).
Epilogue identity_epilogue();

// Applies `e` in place to n interleaved RGB pixels on stream s.
int run_epilogue(float* rgb, size_t n, const Epilogue& e, cudaStream_t s, const char* what);

// Grid size for a grid-stride loop over n items.
int stream_grid(size_t n, int block);

// Per-pixel passes over interleaved RGB in place: a warp takes PIX_WARP
// consecutive pixels through its part of shared memory, so that global memory
// sees whole float4 rows of 512 bytes a warp instruction instead of 4-byte
// accesses 12 bytes apart (whose stores reach the L2 as three partial writes
// of every sector), and a lane's pixels lie 3 floats apart in shared memory (no
// bank conflicts).  f(r, g, b) maps a pixel.  rgb must be 16-byte aligned (VEC)
// or is accessed by 4 bytes.  Launch with pixel_grid(n) blocks of
// PIX_THREADS.  24 MP exposure gain: 86 us against 115 (89 at the copy rate).
constexpr int PIX_THREADS = 256, PIX_WARP = 128;
constexpr int PIX_BLOCK = PIX_THREADS / 32 * PIX_WARP;

inline int pixel_grid(size_t n) { return (int)((n + PIX_BLOCK - 1) / PIX_BLOCK); }

template <bool VEC, int UNROLL, class F>
__device__ __forceinline__ void map_pixels(float* __restrict__ rgb, size_t n, F f) {
    __shared__ __align__(16) float stage[PIX_THREADS / 32][3 * PIX_WARP];
    const int lane = threadIdx.x & 31;
    float* s = stage[threadIdx.x >> 5];
    const size_t p0 = blockIdx.x * (size_t)PIX_BLOCK + (threadIdx.x >> 5) * PIX_WARP;
    if (p0 >= n) return;  // whole warp: only warp-level synchronisation below
    float* g = rgb + 3 * p0;
    const int px = n - p0 < PIX_WARP ? (int)(n - p0) : PIX_WARP;
    const bool whole = VEC && px == PIX_WARP;
    if (whole) {
#pragma unroll
        for (int q = 0; q < 3; q++)
            reinterpret_cast<float4*>(s)[lane + 32 * q] = reinterpret_cast<const float4*>(g)[lane + 32 * q];
    } else {
        for (int i = lane; i < 3 * px; i += 32) s[i] = g[i];
    }
    __syncwarp();
#pragma unroll UNROLL
    for (int k = 0; k < PIX_WARP / 32; k++) {
        const int i = lane + 32 * k;
        if (i < px) {
            float r = s[3 * i], gr = s[3 * i + 1], b = s[3 * i + 2];
            f(r, gr, b);
            s[3 * i] = r;
            s[3 * i + 1] = gr;
            s[3 * i + 2] = b;
        }
    }
    __syncwarp();
    if (whole) {
#pragma unroll
        for (int q = 0; q < 3; q++)
            reinterpret_cast<float4*>(g)[lane + 32 * q] = reinterpret_cast<const float4*>(s)[lane + 32 * q];
    } else {
        for (int i = lane; i < 3 * px; i += 32) g[i] = s[i];
    }
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace color
}  // namespace imops
