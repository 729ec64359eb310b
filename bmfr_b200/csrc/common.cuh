// common.cuh — constants, geometry and exact-arithmetic helpers shared by the
// sm_100a kernels of the BMFR pipeline.
//
// The library is compiled with -fmad=false: no multiply and add is contracted
// into a fused multiply-add unless a kernel asks for it explicitly, so every
// float expression is rounded operation by operation in the order written —
// the order of the reference's expressions (opencl/bmfr.cl).  Division and
// square root are IEEE round-to-nearest (nvcc's default -prec-div/-prec-sqrt).
#pragma once

#include <cstdint>
#include <cuda_fp16.h>

namespace bmfr {

constexpr int kBlockEdge = 32;       // BLOCK_EDGE_LENGTH (bmfr.cpp:104)
constexpr int kBlockPixels = 1024;   // BLOCK_PIXELS (bmfr.cpp:105)
constexpr int kLocal = 256;          // fitter work-group (bmfr.cpp:116)
constexpr int kBuffers = 13;         // BUFFER_COUNT
constexpr int kFeatures = 10;        // BUFFER_COUNT - 3
constexpr int kNotScaled = 4;        // FEATURES_NOT_SCALED
constexpr int kScaled = 6;           // FEATURES_SCALED
constexpr int kREdge = 11;           // R_EDGE

// BLOCK_OFFSETS (bmfr.cl:267-285): per-frame jitter of the block grid.
static __constant__ int2 c_block_offsets[16] = {
    {-14, -14}, {4, -6}, {-8, 14}, {8, 0}, {-10, -8}, {2, 12}, {12, -12}, {-10, 0},
    {12, 14}, {-8, -16}, {6, 6}, {-2, -2}, {6, -14}, {-16, 12}, {14, -4}, {-6, 4}};

// Image, workset and margin sizes of one stream (bmfr.cpp:104-118).
struct Geometry {
    int W, H;          // IMAGE_WIDTH/HEIGHT
    int MW, MH;        // WORKSET_WITH_MARGINS_WIDTH/HEIGHT
    int MWb, MHb;      // margin grid in blocks
    int blocks;        // MWb * MHb
};

inline Geometry make_geometry(int W, int H) {
    Geometry g;
    g.W = W;
    g.H = H;
    const int ww = kBlockEdge * ((W + kBlockEdge - 1) / kBlockEdge);
    const int wh = kBlockEdge * ((H + kBlockEdge - 1) / kBlockEdge);
    g.MW = ww + kBlockEdge;
    g.MH = wh + kBlockEdge;
    g.MWb = g.MW / kBlockEdge;
    g.MHb = g.MH / kBlockEdge;
    g.blocks = g.MWb * g.MHb;
    return g;
}

// Per-frame scalars of accumulate_noisy_data (bmfr.cl:306-308 plus the -D
// limits and blend factor).
struct AccumArgs {
    float m[16];              // prev_frame_camera_matrix (float16 argument)
    float off_x, off_y;       // pixel_offset
    float pos_lim2, nrm_lim2; // POSITION/NORMAL_LIMIT_SQUARED
    float blend_alpha;        // BLEND_ALPHA
    int frame;
    int use_half;             // tmp_data element type
};

// NOISE_AMOUNT * 2 as an unevaluated sum of two floats (hi + lo), so that
// value + NOISE_AMOUNT * 2 * r, which the reference forms in double because
// NOISE_AMOUNT is a double literal (bmfr.cpp:58, bmfr.cl:179), is rounded
// once to float without double arithmetic on the device.
struct NoiseConst {
    float hi, lo;
    float neg_zero;   // -0.0f, known only at run time: the addend of the fitter's products (rmul2)
};

// OpenCL's fmin/fmax (and max(x, y) for the operands the kernels give it):
// y if y < x (x < y), else x; the other operand when x is NaN.  A NaN
// reaches them in taa when every bilinear weight of the history is zero
// (bmfr.cl:939: 0/0), and the clamp then returns the bound.
__device__ __forceinline__ float fmin_cl(float x, float y) { return (y < x || x != x) ? y : x; }
__device__ __forceinline__ float fmax_cl(float x, float y) { return (x < y || x != x) ? y : x; }

// Minimum and maximum of three in one operation; NaN operands are skipped.
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// mirror (bmfr.cl:209-216): valid for indices at most one size out of range.
__device__ __forceinline__ int mirror(int i, int n) {
    if (i < 0) return -i - 1;
    if (i >= n) return 2 * n - i - 1;
    return i;
}

// Programmatic dependent launch.  The pipeline's kernels are launched with
// programmatic stream serialization (launch_chained), so a kernel's launch
// is processed while the kernel before it in the stream drains; before it
// touches memory it waits here for that kernel's completion and memory
// flush, which keeps exactly the ordering of a plain stream.  Dependents
// are released implicitly as CTAs exit (no early trigger: released early,
// waiting CTAs would take the SM slots that multi-wave grids still need).
// Without the launch attribute this is a no-op.
__device__ __forceinline__ void await_previous_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// convert_int_rtn for indices that are tested against an image before use:
// saturates, and NaN maps to INT_MIN.  i and i + 1 (in unsigned arithmetic)
// lie outside every image wherever the position does.
__device__ __forceinline__ int floor_index(float v) {
    const int i = __float2int_rd(v);
    return v == v ? i : (int)0x80000000;
}

// Quotients of several numerators by one divisor, each correctly rounded: the
// divisor's correctly rounded reciprocal and Markstein's correction
// (q = a*y; r = fma(-q, d, a); q' = fma(r, y, q); negated here, so that zero
// quotients keep their sign).  That holds where the residual r is exact and
// the quotient normal: a divisor within 2^+-60 and numerators that are 0 or
// have magnitudes within [2^-64, 2^60].  `most`: the largest magnitude among
// the numerators; `least`: the smallest nonzero one, as magnitude_key gives it.
// NaN numerators pass both tests and are their own quotients.
//
// The lower limit is kept because a black pixel's colour is its history alone:
// a history that fades below 2^-100 otherwise lost its last place to the
// inexact residual.  It costs an integer operation per numerator.
__device__ __forceinline__ uint32_t magnitude_key(float a) { return 2u * __float_as_uint(a) - 1u; }   // 0: the largest
__device__ __forceinline__ bool divides_fast(float d, float most) {
    const float m = fabsf(d);
    return m >= 0x1p-60f && m <= 0x1p60f && most <= 0x1p60f;
}
__device__ __forceinline__ bool divides_fast(float d, float most, uint32_t least) {
    return divides_fast(d, most) && least >= 2u * ((127u - 64u) << 23) - 1u;
}
__device__ __forceinline__ float quotient(float a, float ny, float d) {
    const float nq = a * ny;
    return -__fmaf_rn(__fmaf_rn(nq, d, a), ny, nq);
}
__device__ __forceinline__ float3 divide3(float3 a, float d) {
    const uint32_t least = min(min(magnitude_key(a.x), magnitude_key(a.y)), magnitude_key(a.z));
    if (divides_fast(d, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)), least)) {
        const float ny = -__frcp_rn(d);
        return make_float3(quotient(a.x, ny, d), quotient(a.y, ny, d), quotient(a.z, ny, d));
    }
    return make_float3(a.x / d, a.y / d, a.z / d);
}

// random() (bmfr.cl:162-171): a 32-bit integer hash mapped to [0, 1].
__device__ __forceinline__ float hash_random(uint32_t a) {
    a = (a + 0x7ed55d16u) + (a << 12);
    a = (a ^ 0xc761c23cu) ^ (a >> 19);
    a = (a + 0x165667b1u) + (a << 5);
    a = (a + 0xd3a2646cu) ^ (a << 9);
    a = (a + 0xfd7046c5u) + (a << 3);
    a = (a ^ 0xb55a4f09u) ^ (a >> 16);
    return __uint2float_rn(a) / 4294967296.0f;   // convert_float(UINT_MAX) = 2^32
}

__device__ __forceinline__ uint32_t noise_index(int id, int sub_vector, int feature, int frame) {
    return (uint32_t)id + (uint32_t)sub_vector * (uint32_t)kLocal +
           (uint32_t)feature * (uint32_t)kBlockPixels +
           (uint32_t)frame * (uint32_t)(kBuffers * kBlockPixels);
}

// scale (bmfr.cl:200-205).
__device__ __forceinline__ float scale(float v, float mn, float mx) {
    if (fabsf(mx - mn) > 1.0f) return (v - mn) / (mx - mn);
    return v - mn;
}

__device__ __forceinline__ float round_half(float v) {
    return __half2float(__float2half_rn(v));
}

// Two tmp_data values as binary16 (bmfr.cl:255-265, 468-475): clamped to the
// largest finite value, NaN as 0.
__device__ __forceinline__ __half2 pack_features(float a, float b) {
    uint32_t v;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(b), "f"(a));
    const __half2 h = *reinterpret_cast<__half2*>(&v);
    v &= __heq2_mask(h, h);
    return *reinterpret_cast<__half2*>(&v);
}

__device__ __forceinline__ void hist_store(float* p, int i, float3 v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}
__device__ __forceinline__ void hist_store(__half* p, int i, float3 v) {
    p[3 * i] = __float2half_rn(v.x);
    p[3 * i + 1] = __float2half_rn(v.y);
    p[3 * i + 2] = __float2half_rn(v.z);
}

__device__ __forceinline__ float3 load3(const float* p, int i) {
    return make_float3(p[3 * i], p[3 * i + 1], p[3 * i + 2]);
}
__device__ __forceinline__ void store3(float* p, int i, float3 v) {
    p[3 * i] = v.x;
    p[3 * i + 1] = v.y;
    p[3 * i + 2] = v.z;
}

}  // namespace bmfr
