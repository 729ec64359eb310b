// fit_cqr2.cuh — the precision form's fit of one 32x32 block (CholeskyQR2 in
// FP32, binary16 tmp_data; the method is described in fit_block.cuh) by S
// teams of 64 threads, S = 1, 2 or 4.
//
// A thread keeps the scaled and noised feature rows of its 4/S work-items of
// four rows in registers.  With one team it holds 16 rows, so summing the Gram
// entries over the block takes a quarter of the shuffles that 256 threads
// took, and each factorisation, which all wait for, runs in every lane's
// registers instead of on shuffles: 1.5 k cycles instead of 3.3 k, and 1.8 k
// instead of 5.9 k with the solves.
//
// Every sum keeps the order of the 256-thread form (fit_columns_cqr2), whose
// weights these are bit for bit: dark pixels show any other rounding through
// the tone map's root.  That form sums work-item 8*w + j + 64*g over g ^ 2, over
// g ^ 1, over j ^ 4, 2, 1 and over w ^ 1, 2, 4.  One team: thread 8*w + j owns
// all four g; lanes hold j and w & 3, so the steps are lane ^ 4, 2, 1, 8, 16
// and two warps.  Two teams: a thread owns g and g ^ 2; the steps are lane ^ 8,
// 4, 2, 1, 16 and four warps.
#pragma once

#include "fit_block.cuh"
#include "fit_rows16.cuh"

namespace bmfr {

constexpr int kPartials = 96;   // room for a warp's Gram sums: 55 + 30, in chunks of 16

template <int S>
struct Cqr2Smem {
    alignas(16) float part[2 * S][kPartials];   // Gram sums per warp
    float gram[kPartials];
    alignas(16) float2 nR[kGram1 + 1];   // R1: nR[tri(i, j)] = -R1(i, j), twice; its diagonal's reciprocals, not negated
    float mm[2 * S][12];            // minima and maxima per warp
    int status;                     // nonzero: a bounded wait ran out
    alignas(8) uint64_t bar;        // the block's copy
};

// Noise table: float4 (f - 1)*256 + id holds rows id + 256*q of feature f.
__device__ __forceinline__ float noise_quad_value(int entry, int frame) {
    const int q = entry & 3, id = (entry >> 2) & (kLocal - 1), fb = 1 + entry / (4 * kLocal);
    return hash_random(noise_index(id, q, fb, frame)) - 0.5f;
}

// The work-item of thread t, the k-th of its 4/S.
template <int S>
__device__ __forceinline__ int work_item(int t, int k) {
    const int lane = t & 31, warp = t >> 5;
    if (S == 4) return 8 * warp + (lane & 7) + 64 * (lane >> 3);
    if (S == 2) return 8 * (2 * warp + (lane >> 4)) + (lane & 7) + 64 * (((lane >> 3) & 1) + 2 * k);
    return t + 64 * ((k & 1) * 2 + (k >> 1));   // in the order 0, 2, 1, 3
}

// Byte offset within a column of half h of a tile copied with the 128-byte
// swizzle (16-byte chunk XOR row & 7; a column is 16 rows of 64 halves).
__device__ __forceinline__ uint32_t swizzled_in_column(uint32_t h) {
    const uint32_t r = h >> 6, c = h & 63u;
    return (r << 7) | ((((c >> 3) ^ r) & 7u) << 4) | ((c & 7u) << 1);
}

// A work-item's four rows of a column: (rows q0,q1), (rows q2,q3).
struct Quad {
    float2 p[2];
};

__device__ __forceinline__ Quad load_quad(const unsigned char* column, const uint32_t (&off)[4]) {
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __half2float(*reinterpret_cast<const __half*>(column + off[q]));
    Quad x;
    x.p[0] = make_float2(v[0], v[1]);
    x.p[1] = make_float2(v[2], v[3]);
    return x;
}

// The ten features, scaled and noised, of a work-item; `scale`, `nmin`: the
// scaled features' factors and negated minima.
__device__ __forceinline__ void feature_rows(const unsigned char* tile, const float4* __restrict__ noise, int id,
                                             const uint32_t (&off)[4], const float (&nmin)[kScaled],
                                             const float (&scale)[kScaled], float hi, Quad (&a)[kFeatures]) {
#pragma unroll
    for (int k = 0; k < kFeatures; ++k) {
        Quad v = load_quad(tile + k * kBlockPixels * 2, off);
        if (k > 0) {
            const float4 r = noise[(k - 1) * kLocal + id];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (k >= kNotScaled)
                    v.p[h] = mul2(add2(v.p[h], dup2(nmin[k - kNotScaled])), dup2(scale[k - kNotScaled]));
                v.p[h] = fma2(dup2(hi), h ? make_float2(r.z, r.w) : make_float2(r.x, r.y), v.p[h]);
            }
        }
        a[k] = v;
    }
}

// Entry tri(i, j) = R(i, j) or A^T A(i, j), i <= j, and its column j.
__host__ __device__ constexpr int tri(int i, int j) { return j * (j + 1) / 2 + i; }
__host__ __device__ constexpr int tri_column(int e) {
    int j = 0;
    while (tri(0, j + 1) <= e) ++j;
    return j;
}

// Sum of x*y over the work-item's rows.
__device__ __forceinline__ float quad_dot(const Quad& x, const Quad& y) {
    const float2 g = fma2(x.p[1], y.p[1], mul2(x.p[0], y.p[0]));
    return g.x + g.y;
}

// Step e of the forward substitution: a_j -= R(i, j) a_i, or at the diagonal
// a_j /= R(j, j).
__device__ __forceinline__ void substitute(Quad (&a)[kFeatures], int e, float2 r) {
    const int j = tri_column(e), i = e - tri(0, j);
#pragma unroll
    for (int h = 0; h < 2; ++h) a[j].p[h] = i == j ? mul2(a[j].p[h], r) : fma2(r, a[i].p[h], a[j].p[h]);
}

// A 16-byte load that stays where it is written: R1 is the same for every row,
// and kept in registers for all of them it would take 110.
__device__ __forceinline__ float4 load_shared4(const void* p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(smem_addr(p)));
    return v;
}

// A thread's part of Gram entry e: tri(i, j) = column i against column j, then
// (second pass) 55 + 10c + i = column i against colour c, here b.
template <int N>
__device__ __forceinline__ float gram_entry(const Quad (&a)[N][kFeatures], const Quad (&b)[N][3], int e) {
    float g[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        if (e < kGram1) {
            const int j = tri_column(e);
            g[n] = quad_dot(a[n][e - tri(0, j)], a[n][j]);
        } else {
            g[n] = quad_dot(a[n][(e - kGram1) % kFeatures], b[n][(e - kGram1) / kFeatures]);
        }
    }
    if constexpr (N == 1) return g[0];
    else if constexpr (N == 2) return g[0] + g[1];
    else return (g[0] + g[1]) + (g[2] + g[3]);
}

// Entries [16*chunk, 16*chunk + 16) below N summed over the warp into part[]:
// a transposing butterfly, each pair of lanes ending with one entry.
template <int S, int N>
__device__ __forceinline__ void sum_chunk(const Quad (&a)[4 / S][kFeatures], const Quad (&b)[4 / S][3], int chunk,
                                          float* part) {
    const int lane = threadIdx.x & 31;
    float v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = 16 * chunk + k < N ? gram_entry(a, b, 16 * chunk + k) : 0.0f;
    if (S == 4) {
        const float s = warp_transpose_sum<16>(v);
        if ((lane & 1) == 0) part[16 * chunk + (lane >> 1)] = s;
    } else if (S == 1) {
        transpose_step<8, 4>(v, lane);
        transpose_step<4, 2>(v, lane);
        transpose_step<2, 1>(v, lane);
        transpose_step<1, 8>(v, lane);
        v[0] = v[0] + __shfl_xor_sync(kFull, v[0], 16);
        if (lane < 16) part[16 * chunk + ((lane & 7) << 1 | lane >> 3)] = v[0];
    } else {
        transpose_step<8, 8>(v, lane);
        transpose_step<4, 4>(v, lane);
        transpose_step<2, 2>(v, lane);
        transpose_step<1, 1>(v, lane);
        v[0] = v[0] + __shfl_xor_sync(kFull, v[0], 16);
        if (lane < 16) part[16 * chunk + lane] = v[0];
    }
}

// By warp 0, after the barrier behind the passes' sums: Gram entries over the
// group's warps.
template <int S>
__device__ __forceinline__ void sum_partials(Cqr2Smem<S>& sm, int chunks) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int e = 32 * c + lane;
        if (c < chunks && e < kGram2) {
            float s = sm.part[0][e] + sm.part[1][e];
            if constexpr (S >= 2) s = s + (sm.part[2][e] + sm.part[3][e]);
            if constexpr (S == 4) s = s + ((sm.part[4][e] + sm.part[5][e]) + (sm.part[6][e] + sm.part[7][e]));
            sm.gram[e] = s;
        }
    }
    __syncwarp();
}

// Cholesky factorisation of the Gram matrix by every lane on its own, in
// registers: g[tri(i, j)] = R(i, j) and inv[k] = 1 / R(k, k) (0 for a
// dependent column, see fit_block.cuh).  COLOURS: b enters as a right-hand
// column and returns R^-T b.
template <bool COLOURS>
__device__ __forceinline__ void cholesky(const float* gram, float (&g)[kGram1 + 1], float (&inv)[kFeatures],
                                         float (&b)[kFeatures]) {
#pragma unroll
    for (int k = 0; k < kGram1; k += 4) {
        const float4 q = *reinterpret_cast<const float4*>(gram + k);
        g[k] = q.x;
        g[k + 1] = q.y;
        g[k + 2] = q.z;
        g[k + 3] = q.w;
    }
    float least[kFeatures];
#pragma unroll
    for (int k = 0; k < kFeatures; ++k) least[k] = 0x1p-20f * g[tri(k, k)];
#pragma unroll
    for (int k = 0; k < kFeatures; ++k) {
        const float d = g[tri(k, k)];
        const float y = d > least[k] ? rsqrtf(d) : 0.0f;
        inv[k] = y;
        g[tri(k, k)] = d * y;
#pragma unroll
        for (int j = k + 1; j < kFeatures; ++j) g[tri(k, j)] = g[tri(k, j)] * y;
        if (COLOURS) b[k] = b[k] * y;
#pragma unroll
        for (int i = k + 1; i < kFeatures; ++i) {
#pragma unroll
            for (int j = i; j < kFeatures; ++j) g[tri(i, j)] = __fmaf_rn(-g[tri(k, i)], g[tri(k, j)], g[tri(i, j)]);
            if (COLOURS) b[i] = __fmaf_rn(-g[tri(k, i)], b[k], b[i]);
        }
    }
}

// The fit of the block whose tmp_data lies in `tile` (swizzled copy), by
// threads t of S teams.  `release` runs once nobody reads the tile any more.
// REREAD: the warp that factors reads its rows from the tile again afterwards,
// instead of holding them (80 registers with two teams) through the 55 entries
// of the factorisation; in 128 registers that spills (273 blocks 12.3 us
// against 11.9).
template <int S, bool REREAD, typename Release>
__device__ __forceinline__ void fit_cqr2(const unsigned char* tile, const float4* __restrict__ noise, float hi, int t,
                                         Cqr2Smem<S>& sm, int bar, float* __restrict__ weights_out,
                                         float* __restrict__ mm_out, Release&& release) {
    constexpr int kItems = 4 / S;
    const int lane = threadIdx.x & 31, warp = t >> 5;
    // Min/max of features 4..9 (bmfr.cl:511-535), in any order: the column's
    // 16-byte chunks as they lie.
#pragma unroll
    for (int f = 0; f < kScaled; ++f) {
        const uint4* x = reinterpret_cast<const uint4*>(tile + (kNotScaled + f) * kBlockPixels * 2);
        __half2 mn = __float2half2_rn(INFINITY), mx = __float2half2_rn(-INFINITY);
#pragma unroll
        for (int k = 0; k < (S == 1 ? 2 : 1); ++k) {
            if (S == 4 && t >= kBlockPixels / 8) break;
            const uint4 v = x[t + kTeam * k];
            const __half2* h = reinterpret_cast<const __half2*>(&v);
            mn = __hmin2(mn, __hmin2(__hmin2(h[0], h[1]), __hmin2(h[2], h[3])));
            mx = __hmax2(mx, __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
        }
        const float lo = warp_min(fminf(INFINITY, fminf(__low2float(mn), __high2float(mn))));
        const float hi_ = warp_max(fmaxf(-INFINITY, fmaxf(__low2float(mx), __high2float(mx))));
        if (lane == 0) {
            sm.mm[warp][2 * f] = lo;
            sm.mm[warp][2 * f + 1] = hi_;
        }
    }
    group_sync<S>(bar);
    float nmin[kScaled], scale[kScaled];
    {
        // Lane f holds feature f's bounds and its factor (bmfr.cl:200-205).
        const int f = lane < kScaled ? lane : 0;
        float mn = sm.mm[0][2 * f], mx = sm.mm[0][2 * f + 1];
#pragma unroll
        for (int w = 1; w < 2 * S; ++w) {
            mn = fminf(mn, sm.mm[w][2 * f]);
            mx = fmaxf(mx, sm.mm[w][2 * f + 1]);
        }
        const float d = mx - mn;
        const float y = fabsf(d) > 1.0f ? __frcp_rn(d) : 1.0f;
        if (warp == 0 && lane < kScaled) {
            mm_out[2 * lane] = mn;
            mm_out[2 * lane + 1] = mx;
        }
#pragma unroll
        for (int k = 0; k < kScaled; ++k) {
            nmin[k] = -__shfl_sync(kFull, mn, k);
            scale[k] = __shfl_sync(kFull, y, k);
        }
    }
    // Rows of a work-item: the swizzle's XOR does not depend on the column.
    auto offsets = [&](int id, uint32_t (&off)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) off[q] = swizzled_in_column((uint32_t)(q * kLocal + id));
    };
    Quad a[kItems][kFeatures], colours[kItems][3];
#pragma unroll
    for (int n = 0; n < kItems; ++n) {
        uint32_t off[4];
        offsets(work_item<S>(t, n), off);
        feature_rows(tile, noise, work_item<S>(t, n), off, nmin, scale, hi, a[n]);
    }
    // Pass 1: R1 = chol(A^T A).
#pragma unroll
    for (int c = 0; c < 4; ++c) sum_chunk<S, kGram1>(a, colours, c, sm.part[warp]);
    group_sync<S>(bar);
    if (warp == 0) {
        sum_partials<S>(sm, 2);
        float g[kGram1 + 1], inv[kFeatures], none[kFeatures];
        cholesky<false>(sm.gram, g, inv, none);
        if (lane == 0) {
            auto entry = [&](int e) {
                const int j = tri_column(e);
                return e >= kGram1 ? 0.0f : e == tri(j, j) ? inv[j] : -g[e];
            };
#pragma unroll
            for (int e = 0; e < kGram1 + 1; e += 2)
                *reinterpret_cast<float4*>(&sm.nR[e]) = make_float4(entry(e), entry(e), entry(e + 1), entry(e + 1));
        }
        if (REREAD) {
#pragma unroll
            for (int n = 0; n < kItems; ++n) {
                uint32_t off[4];
                offsets(work_item<S>(t, n), off);
                feature_rows(tile, noise, work_item<S>(t, n), off, nmin, scale, hi, a[n]);
            }
        }
    }
    group_sync<S>(bar);
    // Pass 2: Q1 = A R1^-1 row by row, R2 = chol(Q1^T Q1), z = R2^-T Q1^T B.
    // Entries tri(i, j) in order: column j's updates, then its diagonal.
#pragma unroll
    for (int e = 0; e < kGram1 + 1; e += 2) {
        const float4 r = load_shared4(&sm.nR[e]);
#pragma unroll
        for (int n = 0; n < kItems; ++n) {
            substitute(a[n], e, make_float2(r.x, r.y));
            if (e + 1 < kGram1) substitute(a[n], e + 1, make_float2(r.z, r.w));
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sum_chunk<S, kGram2>(a, colours, c, sm.part[warp]);
#pragma unroll
    for (int n = 0; n < kItems; ++n) {
        uint32_t off[4];
        offsets(work_item<S>(t, n), off);
#pragma unroll
        for (int c = 0; c < 3; ++c) colours[n][c] = load_quad(tile + (kFeatures + c) * kBlockPixels * 2, off);
    }
#pragma unroll
    for (int c = 3; c < 6; ++c) sum_chunk<S, kGram2>(a, colours, c, sm.part[warp]);
    group_sync<S>(bar);
    release();
    if (warp > 0) return;
    sum_partials<S>(sm, 3);
    // Lane c < 3 solves colour c: R2 v = z, then R1 w = v.
    const int c = lane < 3 ? lane : 2;
    float g[kGram1 + 1], inv[kFeatures], b[kFeatures];
#pragma unroll
    for (int i = 0; i < kFeatures; ++i) b[i] = sm.gram[kGram1 + kFeatures * c + i];
    cholesky<true>(sm.gram, g, inv, b);
#pragma unroll
    for (int i = kFeatures - 1; i >= 0; --i) {
#pragma unroll
        for (int j = 0; j < kFeatures; ++j)
            if (j > i) b[i] = __fmaf_rn(-g[tri(i, j)], b[j], b[i]);
        b[i] = b[i] * inv[i];
    }
#pragma unroll
    for (int i = kFeatures - 1; i >= 0; --i) {
#pragma unroll
        for (int j = 0; j < kFeatures; ++j)
            if (j > i) b[i] = __fmaf_rn(sm.nR[tri(i, j)].x, b[j], b[i]);
        b[i] = b[i] * sm.nR[tri(i, i)].x;
    }
    if (lane < 3) {
#pragma unroll
        for (int k = 0; k < kFeatures; ++k) weights_out[3 * k + c] = b[k];
    }
}

}  // namespace bmfr
