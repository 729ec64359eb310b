// fit_rows16.cuh — the reference-arithmetic fit of one 32x32 block
// (opencl/bmfr.cl:490-700, binary16 tmp_data) by S teams of 64 threads.
//
// Layout.  Thread i of a team works on rows i + 64*m, m = 0..15, of the
// 1024x13 matrix: the work-items i, i+64, i+128 and i+192 of the reference's
// 256, four rows each.  These are the four operands of the first stage of the
// reference's reduction tree (bmfr.cl:32-33), so that stage runs on the
// thread's own values, and everything a thread does once per column (the
// norm's last stages, the square root, the reciprocal, the loop) is done by
// 2*S warps instead of the eight that one thread per work-item takes.  What
// bounds it, and what that gave, stands at k_fitter_rows16.
//
// The columns lie in shared memory as binary16, rounded at every in-place
// store as the reference's tmp_data is, a thread's 16 rows of a column in two
// 16-byte chunks; S teams take every S-th later column each.  Columns in
// registers (104 of them) unroll every loop over columns: that code spilled
// and waited for instructions more than for anything else.
//
// One pass per column: a later column is read, the previous column's rank-one
// update is applied, the result is stored and its dot product with the
// current column formed while it is in registers.  Every float expression
// rounds as the reference's does (see fit_block.cuh).
#pragma once

#include <type_traits>

#include "fit_block.cuh"
#include "tma.cuh"

namespace bmfr {

constexpr int kTeam = 64;         // threads of a team
constexpr int kRowPairs = 8;      // row pairs per thread: rows i + 128*p and i + 128*p + 64
// 16-byte chunks of the tile: [column][chunk][thread]; raw tmp_data at first.
constexpr int kTileChunks = kBuffers * 2 * kTeam;

struct Rows16Smem {
    alignas(16) float mm[2][12];    // minima and maxima per warp of a team
    float out[12];                  // the column's dot products
    float part1[kTeam];             // first-stage sums of the norm
    float ucl;                      // u[col] from its owner
    int ones[2];                    // column 0 is all ones (per warp of the team that loads it)
    int status;                     // nonzero: a bounded wait ran out
    float Rm[10][10];               // R of the ten feature columns: Rm[x][y], y <= x
    float rhs[10][3];               // rows 0..9 of the three colour columns
    alignas(8) uint64_t bar;        // the raw block's copy
};

// First-stage sums of the dot products, in the tile's columns that are
// finished: value v of thread i.  The XOR keeps the four 8-lane groups of a
// warp that finish values v..v+3 on 32 distinct banks.
__device__ __forceinline__ int part_index(int v, int i) { return v * kTeam + (i ^ ((v & 3) << 3)); }

// Barrier of one group of S teams (named barrier `bar`).
template <int S>
__device__ __forceinline__ void group_sync(int bar) {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(S * kTeam) : "memory");
}

// Feature noise in the order a team reads it: float4 ((f-1)*4 + m/4)*64 + i
// holds rows i + 64*m for four consecutive m.
__device__ __forceinline__ float noise16_value(int entry, int frame) {
    const int c = entry & 3, i = (entry >> 2) & 63, fq = entry >> 8;   // fq = (fb-1)*4 + m/4
    const int row = i + 64 * (4 * (fq & 3) + c);
    return hash_random(noise_index(row, 0, fq / 4 + 1, frame)) - 0.5f;
}

// Stages 2 and 3 of parallel_reduction_sum (bmfr.cl:35-42) on the 64
// first-stage sums at p: lane j of an 8-lane group forms sum_vec[j], then
// every lane adds the eight left to right.
__device__ __forceinline__ float finish_sum(const float* p, int j, int swap = 0) {
    float acc = p[(8 + j) ^ swap];
#pragma unroll
    for (int m = 2; m < 8; ++m) acc = acc + p[(8 * m + j) ^ swap];
    const float s2 = p[j ^ swap] + acc;
    float r = __shfl_sync(kFull, s2, 0, 8);
#pragma unroll
    for (int m = 1; m < 8; ++m) r = r + __shfl_sync(kFull, s2, m, 8);
    return r;
}

// A thread's rows of one column.
struct Rows {
    __half2 h[kRowPairs];
};

__device__ __forceinline__ Rows load_rows(const uint4* tile, int k, int i) {
    Rows x;
    *reinterpret_cast<uint4*>(&x.h[0]) = tile[(2 * k) * kTeam + i];
    *reinterpret_cast<uint4*>(&x.h[4]) = tile[(2 * k + 1) * kTeam + i];
    return x;
}

__device__ __forceinline__ void store_rows(uint4* tile, int k, int i, const Rows& x) {
    tile[(2 * k) * kTeam + i] = *reinterpret_cast<const uint4*>(&x.h[0]);
    tile[(2 * k + 1) * kTeam + i] = *reinterpret_cast<const uint4*>(&x.h[4]);
}

// Half c of column k (rows 512*c .. 512*c + 511) between one warp's registers
// and shared memory, as eight 8x8 matrices of (m, i).  tmp_data arrives in
// rows of 64 halves, 128-byte swizzled (16-byte chunk XOR row & 7); the
// transposed store leaves a thread's eight rows of the half side by side.
// Both use the same 1 KB, read whole before it is written.
__device__ __forceinline__ Rows load_raw_half_column(const uint4* tile, int k, int c) {
    const int lane = threadIdx.x & 31, r = lane & 7, t = lane >> 3;
    const uint32_t row = smem_addr(tile) + (uint32_t)(k * 2048 + (8 * c + r) * 128);
    Rows x;
    uint32_t* v = reinterpret_cast<uint32_t*>(x.h);
#pragma unroll
    for (int n = 0; n < 2; ++n)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[4 * n]), "=r"(v[4 * n + 1]), "=r"(v[4 * n + 2]), "=r"(v[4 * n + 3])
                     : "r"(row + (((4 * n + t) ^ r) << 4))
                     : "memory");
    return x;
}

__device__ __forceinline__ void store_half_column(uint4* tile, int k, int c, const Rows& x) {
    const int lane = threadIdx.x & 31;
    const uint32_t row = smem_addr(tile) + (uint32_t)(k * 2048 + c * 1024 + lane * 16);
    const uint32_t* v = reinterpret_cast<const uint32_t*>(x.h);
#pragma unroll
    for (int n = 0; n < 2; ++n)
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(row + 512 * n),
                     "r"(v[4 * n]), "r"(v[4 * n + 1]), "r"(v[4 * n + 2]), "r"(v[4 * n + 3])
                     : "memory");
}

// One thread's part of the dot product of binary16 columns x and u: the four
// work-items' sums 0 + p0 + p1 + p2 + p3 (bmfr.cl:630-637) and the tree's
// first stage over them.  u0: the float u of the first row, which takes part
// where `row0`.  A binary16 product is exact in float, so every other term
// is one mixed-precision FMA.
__device__ __forceinline__ float dot_rows(const Rows& x, const Rows& u, float u0, bool row0) {
    float s0 = __fmaf_rn(__low2float(x.h[0]), u0, 0.0f);
    if (!row0) s0 = 0.0f;
    float s1 = fma_h(__high2half(x.h[0]), __high2half(u.h[0]), 0.0f);
    float s2 = fma_h(__low2half(x.h[1]), __low2half(u.h[1]), 0.0f);
    float s3 = fma_h(__high2half(x.h[1]), __high2half(u.h[1]), 0.0f);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        s0 = fma_h(__low2half(x.h[2 * q]), __low2half(u.h[2 * q]), s0);
        s1 = fma_h(__high2half(x.h[2 * q]), __high2half(u.h[2 * q]), s1);
        s2 = fma_h(__low2half(x.h[2 * q + 1]), __low2half(u.h[2 * q + 1]), s2);
        s3 = fma_h(__high2half(x.h[2 * q + 1]), __high2half(u.h[2 * q + 1]), s3);
    }
    return s0 + ((s1 + s2) + s3);   // bmfr.cl:33
}

// The column as float pairs with the first column's noise added to features
// 1..9 (bmfr.cl:625-627).
template <bool PLAIN>
__device__ __forceinline__ void noised_rows(const Rows& x, int k, int i, const float4* __restrict__ noise,
                                            NoiseConst nc, float2 (&a)[kRowPairs]) {
#pragma unroll
    for (int p = 0; p < kRowPairs; ++p) a[p] = __half22float2(x.h[p]);
    if (k >= kFeatures) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 r = noise[((k - 1) * 4 + q) * kTeam + i];
        const float2 r01 = make_float2(r.x, r.y), r23 = make_float2(r.z, r.w);
        a[2 * q] = PLAIN ? add_noise_half2(a[2 * q], r01, nc) : add_noise_r2(a[2 * q], r01, nc);
        a[2 * q + 1] = PLAIN ? add_noise_half2(a[2 * q + 1], r23, nc) : add_noise_r2(a[2 * q + 1], r23, nc);
    }
}

// The Householder vector of a finished column and what its update divides by.
struct Reflection {
    float2 u[kRowPairs];
    float ny, b;     // -RN(1/|u|^2), |u|^2
    bool row0;       // the thread's first row takes part
};

// Rank-one update of a column, rounded at the reference's store
// (bmfr.cl:640-652): x - RN(2u*dot / |u|^2).
//
// Every quotient may take Markstein's correction.  |u|^2 of a binary16
// column is 0, at least 2^-48, or not finite.  Where it is 0 or not finite
// the true quotients are NaN (all numerators are then 0, infinite or NaN),
// and so is the sequence's result.  Otherwise a finite dot product (at most
// 2^43) cannot overflow it, and numerators below 2^-100, whose residual would
// round, give quotients below 2^-52, which leave no trace in a binary16
// result.  An infinite or NaN dot product makes infinite or NaN numerators,
// which are their own quotients.
//
// PLAIN: u is 1 but for row 0 (the first column is the constant feature), so
// one quotient serves every other row; and the noise is below 1.
template <bool NOISE, bool PLAIN>
__device__ __forceinline__ Rows update_rows(const Rows& x, int k, int i, const Reflection& f, float dot,
                                            const float4* __restrict__ noise, NoiseConst nc) {
    Rows y;
    const float2 d2 = dup2(2.0f * dot);   // u * 2d rounds as 2u * d
    const float2 ny = dup2(f.ny), b2 = dup2(f.b);
    float2 a[kRowPairs];
    if (NOISE) noised_rows<PLAIN>(x, k, i, noise, nc, a);
    auto subtract = [&](int p, float2 mq) {
        if (NOISE) y.h[p] = __float22half2_rn(add2(a[p], mq));
        else y.h[p] = __floats2half2_rn(add_f32_h(__low2half(x.h[p]), mq.x), add_f32_h(__high2half(x.h[p]), mq.y));
    };
    const bool finite = fabsf(dot) <= 0x1p100f;
    if (PLAIN) {
        const float2 n = make_float2(i == 0 ? f.u[0].x * d2.x : d2.x, d2.x);
        const float2 mq = finite ? neg_quotient(n, ny, b2) : neg2(n);
        subtract(0, mq);
#pragma unroll
        for (int p = 1; p < kRowPairs; ++p) subtract(p, dup2(mq.y));
    } else if (finite) {
#pragma unroll
        for (int p = 0; p < kRowPairs; ++p) subtract(p, neg_quotient(mul2(f.u[p], d2), ny, b2));
    } else {
#pragma unroll
        for (int p = 0; p < kRowPairs; ++p) subtract(p, neg2(mul2(f.u[p], d2)));
    }
    if (!f.row0) y.h[0] = __halves2half2(__low2half(x.h[0]), __high2half(y.h[0]));
    return y;
}

// One Householder column (bmfr.cl:549-655).  MODE 0: the first column, whose
// dot products read features 1..9 with noise added; 1: the second, whose pass
// applies the first column's update to the noised features; 2: the others.
// PLAIN: column 0 is all ones and the noise below 1, as in every frame the
// pipeline makes; the other instance serves callers' own tmp_data and noise
// (a test of the noise inside the loops cost 12 % of the time).  f: the
// previous column's reflection on entry, this one's on return; out holds the
// dot products that go with it.
template <int S, int MODE, bool PLAIN>
__device__ __forceinline__ void qr_column16(int col, int i, int team, Reflection& f, const float4* __restrict__ noise,
                                            NoiseConst nc, Rows16Smem& sm, uint4* tile, int bar) {
    const int lane = threadIdx.x & 31, g = lane >> 3, j = lane & 7, warp = 2 * team + (i >> 5);
    Rows u = load_rows(tile, col, i);
    if (MODE > 0) u = update_rows<MODE == 1, MODE == 1 && PLAIN>(u, col, i, f, sm.out[0], noise, nc);
    const float c0 = __low2float(u.h[0]);
    // Norm of rows >= col+1 (bmfr.cl:553-569); only row i can be above.
    if (team == 0) {
        sm.part1[i] = dot_rows(u, u, c0, i >= col + 1);
        if (i == col) sm.ucl = c0;
        if (i < col) sm.Rm[col][i] = c0;
    }
    group_sync<S>(bar);
    const float norm2 = finish_sum(sm.part1, j);
    const float ucl = sm.ucl;
    // Work-item col's step (bmfr.cl:580-588), evaluated by every thread.
    const float vl = sqrtf(norm2 + ucl * ucl);
    const float ucl_new = ucl - vl;
    const float uls = norm2 + ucl_new * ucl_new;
    if (team == 0 && i == col) sm.Rm[col][col] = vl;
    const float u0 = i == col ? ucl_new : c0;
    const bool row0 = i >= col;

    // The previous update of columns [k, k + N*S) and their dot products with
    // this one (bmfr.cl:606-638); N columns at a time overlap their chains.
    float* part = reinterpret_cast<float*>(tile);
    auto visit = [&](auto columns, int k) {
        constexpr int N = decltype(columns)::value;
        Rows x[N];
        float s[N];
#pragma unroll
        for (int n = 0; n < N; ++n) x[n] = load_rows(tile, k + n * S, i);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            if (MODE == 0) {
                float2 a[kRowPairs];
                noised_rows<PLAIN>(x[n], k + n * S, i, noise, nc, a);
                float2 s01, s23;
                if (PLAIN) {
                    if (i == 0) a[0].x = __fmul_rn(a[0].x, u0);
                    s01 = add2(dup2(0.0f), a[0]);
                    s23 = add2(dup2(0.0f), a[1]);
#pragma unroll
                    for (int q = 1; q < 4; ++q) {
                        s01 = add2(s01, a[2 * q]);
                        s23 = add2(s23, a[2 * q + 1]);
                    }
                } else
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float2 ua = __half22float2(u.h[2 * q]);
                    const float2 ub = __half22float2(u.h[2 * q + 1]);
                    if (q == 0) {
                        ua.x = u0;
                        s01 = fma2(a[0], ua, dup2(-nc.neg_zero));   // 0 + RN(a*u)
                        s23 = fma2(a[1], ub, dup2(-nc.neg_zero));
                    } else {
                        s01 = add2(s01, rmul2(a[2 * q], ua, nc.neg_zero));
                        s23 = add2(s23, rmul2(a[2 * q + 1], ub, nc.neg_zero));
                    }
                }
                s[n] = s01.x + ((s01.y + s23.x) + s23.y);
            } else {
                x[n] = update_rows<MODE == 1, MODE == 1 && PLAIN>(x[n], k + n * S, i, f, sm.out[k + n * S - col], noise, nc);
                s[n] = dot_rows(x[n], u, u0, row0);
            }
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            if (MODE > 0) store_rows(tile, k + n * S, i, x[n]);
            part[part_index((k + n * S - col - 1) & (MODE == 0 ? 7 : 15), i)] = s[n];
        }
    };
    // Stages 2 and 3 of the dot products: four values per warp and turn.
    auto finish = [&](int first, int last) {
#pragma unroll 1
        for (int v0 = first + 4 * warp; v0 < last; v0 += 8 * S) {
            const int slot = (v0 + g) & (MODE == 0 ? 7 : 15);
            const float r = finish_sum(part + slot * kTeam, j, g << 3);
            if (j == 0 && v0 + g < last) sm.out[v0 + g] = r;
        }
    };
    const int end = MODE == 0 ? 9 : kBuffers;   // column 0 alone has room for eight values
    // Later columns in flight per thread.  Teams that share a block overlap
    // each other's chains, and with one column at a time their CTAs fit in 128
    // registers (two at a time there: 294 blocks 21.7 us against 20.9).
    constexpr int kWide = S == 1 ? 2 : 1;
    int k = col + 1 + team;
#pragma unroll 1
    for (; k + (kWide - 1) * S < end; k += kWide * S) visit(std::integral_constant<int, kWide>{}, k);
    if (kWide > 1) {
#pragma unroll 1
        for (; k < end; k += S) visit(std::integral_constant<int, 1>{}, k);
    }
    if (MODE == 0) {
        group_sync<S>(bar);
        finish(0, 8);
        group_sync<S>(bar);
#pragma unroll 1
        for (k = 9 + team; k < kBuffers; k += S) visit(std::integral_constant<int, 1>{}, k);
        group_sync<S>(bar);
        finish(8, 12);
    }
    f.ny = -__frcp_rn(uls);
    f.b = uls;
    f.row0 = row0;
#pragma unroll
    for (int p = 0; p < kRowPairs; ++p) f.u[p] = __half22float2(u.h[p]);
    f.u[0].x = u0;
    if (MODE > 0) {
        group_sync<S>(bar);
        finish(0, kBuffers - 1 - col);
    }
    group_sync<S>(bar);
}

// Back substitution (bmfr.cl:659-699) by one warp, lane c < 3 solving colour
// channel c on its own: the terms of a step are independent until they are
// subtracted, left to right, so nothing waits for another lane.  Quotients
// take Markstein's correction; a value outside the range where that is exact
// sends the block to true divisions.
__device__ __forceinline__ void back_substitute(const Rows16Smem& sm, float* __restrict__ weights_out) {
    const int lane = threadIdx.x & 31, c = lane < 3 ? lane : 2;
    const float own = sm.Rm[lane < kFeatures ? lane : 0][lane < kFeatures ? lane : 0];   // R(lane, lane)
    const float own_y = -__frcp_rn(own);
    bool ok = own >= 0x1p-60f && own <= 0x1p60f;
    float w[kFeatures];
#pragma unroll
    for (int k = kFeatures - 1; k >= 0; --k) {
        const float d = __shfl_sync(kFull, own, k), ny = __shfl_sync(kFull, own_y, k);
        auto quotient = [&](float a) {
            const float m = fabsf(a);
            ok = ok && (m == 0.0f || (m >= 0x1p-60f && m <= 0x1p60f));
            const float nq = a * ny;
            return __fmaf_rn(__fmaf_rn(nq, d, a), ny, nq);   // -RN(a / d)
        };
        float v = -quotient(sm.rhs[k][c]);
#pragma unroll
        for (int x = 1; x < kFeatures; ++x)
            if (x > k) v = v + quotient(sm.Rm[x][k] * w[x]);
        w[k] = v;
    }
    if (!__all_sync(kFull, ok)) {
        // In shared memory's order, solved weights in place of w.
#pragma unroll 1
        for (int k = kFeatures - 1; k >= 0; --k) {
            const float d = sm.Rm[k][k];
            float v = sm.rhs[k][c] / d;
#pragma unroll 1
            for (int x = k + 1; x < kFeatures; ++x) v = v - sm.Rm[x][k] * weights_out[3 * x + c] / d;
            if (lane < 3) weights_out[3 * k + c] = v;
            __syncwarp();
        }
        return;
    }
    if (lane < 3) {
#pragma unroll
        for (int k = 0; k < kFeatures; ++k) weights_out[3 * k + c] = w[k];
    }
}

// The fit of the block whose raw tmp_data lies in `tile`: weights and
// min/max out.
template <int S>
__device__ __forceinline__ void fit_rows16(int i, int team, const float4* __restrict__ noise, NoiseConst nc,
                                           Rows16Smem& sm, uint4* tile, int bar, float* __restrict__ weights_out,
                                           float* __restrict__ mm_out) {
    const int lane = threadIdx.x & 31, warp = i >> 5;
    // The block moves through registers from tmp_data's row order to the
    // threads' chunks, each warp one half of a column in place.  First the
    // columns that keep their values, then features 4..9, which are scaled on
    // the way.
    {
        constexpr int kKept = kBuffers - kScaled, kMine = (kKept + S - 1) / S;
#pragma unroll
        for (int c = 0; c < kMine; ++c) {
            const int n = S * c + team, k = n < kNotScaled ? n : n + kScaled;
            if (n >= kKept) break;
            const Rows x = load_raw_half_column(tile, k, warp);
            store_half_column(tile, k, warp, x);
            if (c == 0 && k == 0) {
                bool ones = true;
#pragma unroll
                for (int p = 0; p < kRowPairs; ++p) ones = ones && __hbeq2(x.h[p], __float2half2_rn(1.0f));
                ones = __all_sync(kFull, ones);
                if (lane == 0) sm.ones[warp] = ones;
            }
        }
    }
    constexpr int kMine = (kScaled + S - 1) / S;
    Rows x[kMine];
    // Min/max of features 4..9 (bmfr.cl:511-535).  Minima and maxima are
    // exact in any order; only the sign of a zero bound can differ from the
    // reference's tree.
#pragma unroll
    for (int c = 0; c < kMine; ++c) {
        const int f = S * c + team;
        if (f >= kScaled) break;
        x[c] = load_raw_half_column(tile, kNotScaled + f, warp);
        __half2 mn = x[c].h[0], mx = x[c].h[0];
#pragma unroll
        for (int p = 1; p < kRowPairs; ++p) {
            mn = __hmin2(mn, x[c].h[p]);
            mx = __hmax2(mx, x[c].h[p]);
        }
        const float lo = warp_min(fminf(INFINITY, fminf(__low2float(mn), __high2float(mn))));
        const float hi = warp_max(fmaxf(-INFINITY, fmaxf(__low2float(mx), __high2float(mx))));
        if (lane == 0) {
            sm.mm[warp][2 * f] = lo;
            sm.mm[warp][2 * f + 1] = hi;
        }
    }
    group_sync<S>(bar);
    if (team == 0 && i < 2 * kScaled)
        mm_out[i] = (i & 1) ? fmaxf(sm.mm[0][i], sm.mm[1][i]) : fminf(sm.mm[0][i], sm.mm[1][i]);
    // scale() (bmfr.cl:200-205), rounded at the store (bmfr.cl:540).  The
    // block's bounds are binary16 values, so the range is at most 131008 and
    // every finite numerator keeps Markstein's correction exact; an infinite
    // range divides finite numerators to zero and the others to NaN.
#pragma unroll
    for (int c = 0; c < kMine; ++c) {
        const int f = S * c + team;
        if (f >= kScaled) break;
        const float mn = fminf(sm.mm[0][2 * f], sm.mm[1][2 * f]);
        const float mx = fmaxf(sm.mm[0][2 * f + 1], sm.mm[1][2 * f + 1]);
        const float d = mx - mn;
        const float2 nm = dup2(-mn), d2 = dup2(d);
        if (!(fabsf(d) > 1.0f)) {
#pragma unroll
            for (int p = 0; p < kRowPairs; ++p) x[c].h[p] = __float22half2_rn(add2(__half22float2(x[c].h[p]), nm));
        } else if (fabsf(d) <= 0x1p60f) {
            const float2 ny = dup2(-__frcp_rn(d));
#pragma unroll
            for (int p = 0; p < kRowPairs; ++p)
                x[c].h[p] = __hneg2(__float22half2_rn(neg_quotient(add2(__half22float2(x[c].h[p]), nm), ny, d2)));
        } else {
#pragma unroll
            for (int p = 0; p < kRowPairs; ++p)
                x[c].h[p] = __float22half2_rn(mul2(add2(__half22float2(x[c].h[p]), nm), dup2(0.0f)));
        }
        store_half_column(tile, kNotScaled + f, warp, x[c]);
    }
    group_sync<S>(bar);

    Reflection f;
    if (sm.ones[0] && sm.ones[1] && fabsf(nc.hi) < 2.0f) {
        qr_column16<S, 0, true>(0, i, team, f, noise, nc, sm, tile, bar);
        qr_column16<S, 1, true>(1, i, team, f, noise, nc, sm, tile, bar);
    } else {
        qr_column16<S, 0, false>(0, i, team, f, noise, nc, sm, tile, bar);
        qr_column16<S, 1, false>(1, i, team, f, noise, nc, sm, tile, bar);
    }
#pragma unroll 1
    for (int col = 2; col < kFeatures; ++col) qr_column16<S, 2, false>(col, i, team, f, noise, nc, sm, tile, bar);

    // Rows 0..9 of the colour columns are the right-hand side
    // (bmfr.cl:596-600 for col >= 10).  The last column's update changes only
    // row 9 of them.
    if (team == 0 && i < kFeatures) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            Rows y = load_rows(tile, kFeatures + c, i);
            if (i == kFeatures - 1) {
                const float n = f.u[0].x * (2.0f * sm.out[c]);
                const float2 mq = fabsf(sm.out[c]) <= 0x1p100f ? neg_quotient(dup2(n), dup2(f.ny), dup2(f.b)) : dup2(-n);
                y.h[0] = __float2half2_rn(add_f32_h(__low2half(y.h[0]), mq.x));
            }
            sm.rhs[i][c] = __low2float(y.h[0]);
        }
    }
    group_sync<S>(bar);
    if (team > 0 || warp > 0) return;
    back_substitute(sm, weights_out);
}

}  // namespace bmfr
