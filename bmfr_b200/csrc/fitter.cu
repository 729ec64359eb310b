// fitter.cu — standalone fitter kernels (opencl/bmfr.cl:490-700).
//
// k_fitter_rows16: the reference's arithmetic on binary16 tmp_data, groups of
// 64 threads per block of the image (fit_rows16.cuh).  k_fitter_cqr2: the
// precision form's CholeskyQR2, the same way (fit_cqr2.cuh).
//
// k_fitter: everything else.  Persistent CTAs of 256 threads, as many as fit on the SMs.  Each CTA walks
// blocks b = blockIdx.x, + gridDim.x, ...: a block's 13 x 1024 tmp_data
// values arrive in shared memory by one TMA copy and move to registers, and
// the copy of a later block is issued at once so that it overlaps the fit.
//
// Binary16 tmp_data comes in as a 2-D tensor copy (rows of 64 halves, 208
// rows per block) with the 128-byte swizzle: the eight lanes of a warp that
// read one 16-byte chunk of a row meet three other lane groups at rows
// 64 halves apart, which without the swizzle fall in the same four banks
// (four-way conflicts on every load); the swizzle spreads them over 16
// banks.  With the frame's noise table in global memory the CTA keeps two
// tile buffers, so the copy of the block after next is in flight while the
// current one is fitted.  Float tmp_data uses a one-dimensional bulk copy.
//
// There the feature-noise table of the frame is either formed by each CTA in
// its shared memory (the drop-in entry point: no scratch memory, so calls on
// different streams never share state) or read from a table that an earlier
// kernel of the frame pipeline wrote to global memory (smaller CTAs, more of
// them per SM).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "fit_block.cuh"
#include "fit_cqr2.cuh"
#include "fit_rows16.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace bmfr {

constexpr int kTileRows = kBuffers * kBlockPixels / 64;   // 208 rows of 64 halves per block

template <bool HALF_TMP, bool NOISE_GLOBAL>
struct FitterShared {
    using TmpT = typename std::conditional<HALF_TMP, __half, float>::type;
    static constexpr int kStages = (HALF_TMP && NOISE_GLOBAL) ? 2 : 1;
    alignas(1024) TmpT tile[kStages][kBuffers * kBlockPixels];
    FitterSmem sm;
    alignas(8) uint64_t bar[kStages];
    float noise[NOISE_GLOBAL ? 1 : kNoiseTableFloats];
};

// METHOD (FitMethod): the FP32 Householder sequence on binary16 tmp_data, or
// the reference's arithmetic on float tmp_data, which rounds nowhere in
// between; both work on a float tile.
template <bool HALF_TMP, int METHOD, bool NOISE_GLOBAL>
__global__ void __launch_bounds__(256, 2)
    k_fitter(int nblocks, int frame, NoiseConst nc, const void* __restrict__ tmp, const __grid_constant__ CUtensorMap tmap,
             float* __restrict__ weights, float* __restrict__ mins_maxs, const float* __restrict__ noise_g,
             int* __restrict__ status) {
    await_previous_kernel();
    using Shared = FitterShared<HALF_TMP, NOISE_GLOBAL>;
    using TmpT = typename Shared::TmpT;
    constexpr int kStages = Shared::kStages;
    static_assert(METHOD == (HALF_TMP ? kFitHouseholder32 : kFitReference), "");
    extern __shared__ unsigned char smem_raw[];
    // The swizzled copy needs a 1024-byte aligned destination.
    Shared& S = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kTileBytes = kBuffers * kBlockPixels * sizeof(TmpT);
    const char* src = static_cast<const char*>(tmp);
    const int id = work_item_id();
    auto issue = [&](int stage, int blk) {
        mbar_arrive_expect_tx(&S.bar[stage], kTileBytes);
        if constexpr (HALF_TMP) tensor_copy_2d_g2s(S.tile[stage], &tmap, 0, blk * kTileRows, &S.bar[stage]);
        else bulk_copy_g2s(S.tile[stage], src + (size_t)blk * kTileBytes, kTileBytes, &S.bar[stage]);
    };

    if (threadIdx.x == 0) {
        for (int st = 0; st < kStages; ++st) mbar_init(&S.bar[st], 1);
        fence_barrier_init();
        S.sm.status = 0;
        for (int st = 0; st < kStages; ++st)
            if (blockIdx.x + st * (int)gridDim.x < nblocks) issue(st, blockIdx.x + st * gridDim.x);
    }
    if (!NOISE_GLOBAL) fill_noise_table(S.noise, frame);
    const float* noise = NOISE_GLOBAL ? noise_g : S.noise;
    __syncthreads();

    int it = 0;
    for (int b = blockIdx.x; b < nblocks; b += gridDim.x, ++it) {
        const int st = it % kStages;
        const uint32_t phase = (uint32_t)(it / kStages) & 1u;
        if (threadIdx.x == 0 && !mbar_wait_bounded(&S.bar[st], phase)) S.sm.status = kDevTimeout;
        __syncthreads();
        if (S.sm.status) {
            if (threadIdx.x == 0) {
                atomicExch(status, kDevTimeout);
                // let the copies in flight land
                for (int k = 0; k < kStages; ++k)
                    if (b + k * (int)gridDim.x < nblocks) mbar_wait_bounded(&S.bar[(it + k) % kStages], (uint32_t)((it + k) / kStages) & 1u);
            }
            return;
        }
        Tile<false> t;
        const TmpT* tile = S.tile[st];
        // Row k*16 + 4q + id/64 of the tile holds (k, q); its swizzle XOR
        // (low three row bits) does not depend on k.
        uint32_t qoff[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) qoff[q] = swizzled_in_column((uint32_t)(q * kLocal + id));
#pragma unroll
        for (int k = 0; k < kBuffers; ++k) {
            if constexpr (HALF_TMP) {
                const unsigned char* base = reinterpret_cast<const unsigned char*>(tile) + k * kBlockPixels * 2;
                __half v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = *reinterpret_cast<const __half*>(base + qoff[q]);
#pragma unroll
                for (int q = 0; q < 4; ++q) t.set1(k, q, __half2float(v[q]));
            } else {
                const TmpT* col = tile + k * kBlockPixels + id;
#pragma unroll
                for (int q = 0; q < 4; ++q) t.set1(k, q, col[q * kLocal]);
            }
        }
        __syncthreads();   // the buffer is free again
        const int next = b + kStages * (int)gridDim.x;
        if (threadIdx.x == 0 && next < nblocks) issue(st, next);
        fit_block<false, METHOD>(t, noise, nc, S.sm, weights + (size_t)b * kFeatures * 3,
                                 mins_maxs + (size_t)b * kScaled * 2);
    }
}

// The reference-arithmetic fit of binary16 tmp_data (fit_rows16.cuh): G groups
// of S teams per CTA, one CTA per SM or two (kRows16Ctas), each group walking
// blocks of its own.
// The CTA forms the frame's noise table in its shared memory, which its groups
// share; that saves the launch that wrote it to global memory (2.0-2.4 us).
//
// Bound by the dependent steps of each column (norm, square root, dot products,
// update), with FMA and issue slots about half used: 984 blocks issue on 54 %
// of the cycles with the FMA-heavy pipe 45 % active, 8349 blocks on 55 % with
// it 53 % active, and the longest stall is the fixed latency of the operation
// before (1.4 cycles per issue).  More groups on an SM fill the gaps (8349
// blocks: 365 us with four, 318 with five, 295 with six).  One thread per
// work-item, 256 threads per block and the columns in registers, took 47 M warp
// instructions for the 984 blocks of 1280x720, this takes 23 M: 69.5 -> 42.2 us;
// 2135 blocks (1920x1080) 148 -> 87 us; 8349 (3840x2160) 543 -> 294 us.
template <int G>
struct FitterRows16Shared {
    uint4 tile[G][kTileChunks];   // 1024-byte aligned, for the swizzled copy
    Rows16Smem sm[G];
    alignas(16) float noise[kNoiseTableFloats];
};

// CTAs per SM.  A launch does not know what runs beside it: a caller may have
// plans on streams of its own.  With up to two blocks per SM a CTA therefore
// takes at most half of an SM, so that the fits of two streams share it.  Eight
// plans on eight streams, us per round of frames, with CTAs of a whole SM / of
// half / with one thread per work-item: 320x240 127 / 92 / 97, 400x340 201 / 135
// / 163, 640x360 271 / 207 / 263.  Alone, 99 blocks take 16.4 instead of 16.2
// us, 273 blocks 20.8 instead of 20.7.
template <int S, int G>
constexpr int kRows16Ctas = G == 1 || G == 2 ? 2 : 1;
constexpr int kSmemPerSm = 228 * 1024, kSmemPerCta = 2048;   // capacity; a CTA's alignment slack and reserve
static_assert(2 * (sizeof(FitterRows16Shared<2>) + kSmemPerCta) <= kSmemPerSm, "two CTAs of two groups share an SM");

template <int S, int G>
__global__ void __launch_bounds__(kTeam * S * G, kRows16Ctas<S, G>)
    k_fitter_rows16(int nblocks, int frame, NoiseConst nc, const __grid_constant__ CUtensorMap tmap,
                    float* __restrict__ weights, float* __restrict__ mins_maxs, int* __restrict__ status) {
    using Shared = FitterRows16Shared<G>;
    extern __shared__ unsigned char smem_raw[];
    Shared& sh = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kTileBytes = kBuffers * kBlockPixels * sizeof(__half);
    constexpr int kThreads = kTeam * S;
    const int group = threadIdx.x / kThreads, bar = 1 + group;
    const int i = threadIdx.x % kTeam, team = threadIdx.x % kThreads / kTeam;
    // The leader is not in the warp that ends a block with the back
    // substitution, so the next block's copy runs beside it.
    const bool leader = i == 32 && team == S - 1;
    const int first = group * gridDim.x + blockIdx.x, stride = G * gridDim.x;
    Rows16Smem& sm = sh.sm[group];
    uint4* tile = sh.tile[group];
    if (leader) {
        mbar_init(&sm.bar, 1);
        fence_barrier_init();
        sm.status = 0;
    }
    for (int e = threadIdx.x; e < kNoiseTableFloats; e += kThreads * G) sh.noise[e] = noise16_value(e, frame);
    const float4* noise = reinterpret_cast<const float4*>(sh.noise);
    __syncthreads();
    await_previous_kernel();

    uint32_t phase = 0;
    for (int b = first; b < nblocks; b += stride, phase ^= 1u) {
        if (leader) {
            // The tile was last touched by generic loads and stores.
            fence_proxy_async();
            mbar_arrive_expect_tx(&sm.bar, kTileBytes);
            tensor_copy_2d_g2s(tile, &tmap, 0, b * kTileRows, &sm.bar);
            if (!mbar_wait_bounded(&sm.bar, phase)) sm.status = kDevTimeout;
        }
        group_sync<S>(bar);
        if (sm.status) {
            if (leader) {
                atomicExch(status, kDevTimeout);
                mbar_wait_bounded(&sm.bar, phase);   // let the copy in flight land
            }
            return;
        }
        fit_rows16<S>(i, team, noise, nc, sm, tile, bar, weights + (size_t)b * kFeatures * 3,
                      mins_maxs + (size_t)b * kScaled * 2);
    }
}

// The precision form's CholeskyQR2 fit (fit_cqr2.cuh): G groups of S teams per
// CTA, one CTA per SM or two (kCqr2Ctas), as k_fitter_rows16.
//
// Bound by latency at two warps per scheduler, which is what the registers
// allow: 984 blocks issue on 32 % of the cycles with the FMA-heavy pipe 29 %
// active (stalls per issue: instruction fetch 1.5, the operation before 1.1,
// barriers around warp 0's two factorisations 0.7), 8349 blocks on 44 % with it
// 46 % active.  256 threads per block took, against this: 135 blocks 11.7 -> 8.3
// us, 984 (1280x720) 37 -> 23.7, 2135 (1920x1080) 72 -> 44, 8349 (3840x2160)
// 252 -> 152 us.
//
// The fit is straight-line code that each group passes once per block.  Groups
// that have drifted apart fetch it four times over, so from the seventh round
// on it pays to bring them back together (ALIGNED: a barrier of the CTA every
// fourth round): 3680 blocks 79.0 -> 75.2 us, 4736 101 -> 90.5, 8228 179 -> 153
// (156 with a barrier at every round from the fifth on, 152.4 at every second
// round).  In fewer rounds the groups still run side by side and the loop costs
// more than it gives (3000 blocks, six rounds, 63.7 -> 64.1 us; 2400, five, 52.8
// -> 53.5; 2135, four, 44.0 -> 45.2).
constexpr int kAlignRounds = 4;

template <int S, int G>
struct FitterCqr2Shared {
    uint4 tile[G][kTileChunks];   // 1024-byte aligned, for the swizzled copy
    Cqr2Smem<S> sm[G];
    alignas(16) float noise[kNoiseTableFloats];
};

// CTAs per SM, as for k_fitter_rows16; eight plans on eight streams: 320x240 76 /
// 69 / 68, 400x340 138 / 114 / 115, 640x360 189 / 171 / 185.  Alone, 99 blocks
// stay at 8.0 us and 273 blocks take 11.9 instead of 11.0.
template <int S, int G>
constexpr int kCqr2Ctas = G == 1 || G == 2 ? 2 : 1;
static_assert(2 * (sizeof(FitterCqr2Shared<2, 2>) + kSmemPerCta) <= kSmemPerSm, "two CTAs of two groups share an SM");

template <int S, int G, bool ALIGNED>
__global__ void __launch_bounds__(kTeam * S * G, kCqr2Ctas<S, G>)
    k_fitter_cqr2(int nblocks, int frame, NoiseConst nc, const __grid_constant__ CUtensorMap tmap,
                  float* __restrict__ weights, float* __restrict__ mins_maxs, int* __restrict__ status) {
    using Shared = FitterCqr2Shared<S, G>;
    extern __shared__ unsigned char smem_raw[];
    Shared& sh = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kTileBytes = kBuffers * kBlockPixels * sizeof(__half);
    constexpr int kThreads = kTeam * S;
    const int group = threadIdx.x / kThreads, bar = 1 + group, t = threadIdx.x % kThreads;
    const bool leader = t == kThreads - 32;   // not in the warp that solves
    const int first = group * gridDim.x + blockIdx.x, stride = G * gridDim.x;
    Cqr2Smem<S>& sm = sh.sm[group];
    uint4* tile = sh.tile[group];
    auto issue = [&](int blk) {
        fence_proxy_async();   // the tile was last read by generic loads
        mbar_arrive_expect_tx(&sm.bar, kTileBytes);
        tensor_copy_2d_g2s(tile, &tmap, 0, blk * kTileRows, &sm.bar);
    };
    if (leader) {
        mbar_init(&sm.bar, 1);
        fence_barrier_init();
        sm.status = 0;
    }
    for (int e = threadIdx.x; e < kNoiseTableFloats; e += kThreads * G) sh.noise[e] = noise_quad_value(e, frame);
    __syncthreads();
    await_previous_kernel();
    if (leader && first < nblocks) issue(first);

    auto fit = [&](int b, uint32_t phase) {   // false: the block's copy did not arrive
        if (leader && !mbar_wait_bounded(&sm.bar, phase)) sm.status = kDevTimeout;
        group_sync<S>(bar);
        if (sm.status) {
            if (leader) {
                atomicExch(status, kDevTimeout);
                mbar_wait_bounded(&sm.bar, phase);   // let the copy in flight land
            }
            return false;
        }
        fit_cqr2<S, S == 2 && kCqr2Ctas<S, G> == 2>(
            reinterpret_cast<const unsigned char*>(tile), reinterpret_cast<const float4*>(sh.noise), nc.hi, t, sm, bar,
            weights + (size_t)b * kFeatures * 3, mins_maxs + (size_t)b * kScaled * 2, [&] {
                if (leader && b + stride < nblocks) issue(b + stride);
            });
        return true;
    };
    if constexpr (ALIGNED) {
        // The number of rounds is the same in every thread of the CTA; a group
        // without a block left, or whose copy failed, only joins the barriers.
        const int rounds = (nblocks - (int)blockIdx.x + stride - 1) / stride;
        bool live = true;
        for (int r = 0, b = first; r < rounds; ++r, b += stride) {
            if (r % kAlignRounds == kAlignRounds - 1) __syncthreads();
            if (live && b < nblocks) live = fit(b, r & 1);
        }
    } else {
        uint32_t phase = 0;
        for (int b = first; b < nblocks; b += stride, phase ^= 1u)
            if (!fit(b, phase)) return;
    }
}

// The frame's noise table in global memory (kNoiseTableFloats floats).
__global__ void __launch_bounds__(256) k_noise_table(int frame, float* __restrict__ table) {
    await_previous_kernel();
    const int e = blockIdx.x * kLocal + threadIdx.x;
    if (e < kNoiseTableFloats) table[e] = noise_table_value(e, frame);
}

cudaError_t launch_noise_table(int frame, float* table, cudaStream_t s) {
    return launch_chained(k_noise_table, dim3(kNoiseTableFloats / kLocal), dim3(kLocal), 0, s, frame, table);
}

// A barrier that no copy or thread ever completes: thread 0's bounded wait
// runs out after limit_ns and records the timeout as the fitter does.
__global__ void __launch_bounds__(32) k_bounded_wait_probe(int* __restrict__ status, unsigned long long limit_ns) {
    __shared__ alignas(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    __syncwarp();
    if (threadIdx.x == 0 && !mbar_wait_bounded(&bar, 0, limit_ns)) atomicExch(status, kDevTimeout);
}

cudaError_t launch_bounded_wait_probe(int* status, unsigned long long limit_ns, cudaStream_t s) {
    k_bounded_wait_probe<<<1, 32, 0, s>>>(status, limit_ns);
    return cudaGetLastError();
}

// cuTensorMapEncodeTiled from the driver, looked up once.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// binary16 tmp_data of `nblocks` blocks as rows of 64 halves; one box is
// one block (208 rows), swizzled by 128 bytes.
static cudaError_t encode_tmp_map(const void* tmp, int nblocks, CUtensorMap* map) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {64, (cuuint64_t)nblocks * kTileRows};
    const cuuint64_t strides[1] = {128};
    const cuuint32_t box[2] = {64, (cuuint32_t)kTileRows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(tmp), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Allows `smem` bytes per CTA and finds how many CTAs fit on the device.
template <typename Kernel>
static cudaError_t resident_ctas(Kernel kern, int threads, int smem, int dev, int* ctas) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    *ctas = (per_sm > 0 ? per_sm : 1) * sms;
    return cudaSuccess;
}

template <bool HALF_TMP, int METHOD, bool NOISE_GLOBAL>
static cudaError_t launch_fitter_t(int nblocks, int frame, NoiseConst nc, const void* tmp, float* weights,
                                   float* mins_maxs, const float* noise, int* status, cudaStream_t s) {
    auto kern = k_fitter<HALF_TMP, METHOD, NOISE_GLOBAL>;
    const int smem = (int)sizeof(FitterShared<HALF_TMP, NOISE_GLOBAL>) + 1024;   // + alignment slack
    // Resident CTAs per device, found once per device and instantiation.
    // Threads that race on the first call compute the same value, so a
    // relaxed atomic store and load are enough.
    static std::atomic<int> grid_cap[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int cap = grid_cap[dev].load(std::memory_order_relaxed);
    if (cap == 0) {
        e = resident_ctas(kern, kLocal, smem, dev, &cap);
        if (e != cudaSuccess) return e;
        grid_cap[dev].store(cap, std::memory_order_relaxed);
    }
    const int grid = nblocks < cap ? nblocks : cap;
    if (grid <= 0) return cudaSuccess;
    CUtensorMap map;
    std::memset(&map, 0, sizeof map);
    if (HALF_TMP) {
        e = encode_tmp_map(tmp, nblocks, &map);
        if (e != cudaSuccess) return e;
    }
    return launch_chained(kern, dim3(grid), dim3(kLocal), smem, s, nblocks, frame, nc, tmp, map, weights,
                          mins_maxs, noise, status);
}

template <int S, int G>
static cudaError_t launch_rows16_t(int nblocks, int frame, NoiseConst nc, const CUtensorMap& map, float* weights,
                                   float* mins_maxs, int* status, int dev, int ctas, cudaStream_t s) {
    auto kern = k_fitter_rows16<S, G>;
    const int smem = (int)sizeof(FitterRows16Shared<G>) + 1024;   // + alignment slack
    static std::atomic<bool> allowed[64];
    if (!allowed[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        allowed[dev].store(true, std::memory_order_relaxed);
    }
    return launch_chained(kern, dim3(ctas), dim3(kTeam * S * G), smem, s, nblocks, frame, nc, map, weights, mins_maxs,
                          status);
}

template <int S, int G, bool ALIGNED = false>
static cudaError_t launch_cqr2_t(int nblocks, int frame, NoiseConst nc, const CUtensorMap& map, float* weights,
                                 float* mins_maxs, int* status, int dev, int ctas, cudaStream_t s) {
    auto kern = k_fitter_cqr2<S, G, ALIGNED>;
    const int smem = (int)sizeof(FitterCqr2Shared<S, G>) + 1024;   // + alignment slack
    static std::atomic<bool> allowed[64];
    if (!allowed[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        allowed[dev].store(true, std::memory_order_relaxed);
    }
    return launch_chained(kern, dim3(ctas), dim3(kTeam * S * G), smem, s, nblocks, frame, nc, map, weights, mins_maxs,
                          status);
}

// The current device and its SM count, looked up once per device.
static cudaError_t device_sms(int* dev, int* sms) {
    static std::atomic<int> sm_count[64];
    cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    if (*dev < 0 || *dev >= 64) return cudaErrorInvalidDevice;
    *sms = sm_count[*dev].load(std::memory_order_relaxed);
    if (*sms == 0) {
        e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, *dev);
        if (e != cudaSuccess) return e;
        sm_count[*dev].store(*sms, std::memory_order_relaxed);
    }
    return cudaSuccess;
}

// Whether this launch and `beside` blocks of other streams fill the GPU: then
// its blocks are packed onto as few SMs as they fill, with one team each,
// instead of spread for the shortest time, because the SMs it leaves run the
// others.  A step of eight 640x360 streams took 349 us spread and 294 packed
// with CholeskyQR2, 503 and 370 with the reference's arithmetic; five streams
// of 380 blocks together 184 spread and 193 packed.
//
// A packed launch of the reference's arithmetic takes six groups per CTA where
// a launch alone might take seven.  Beside smaller or larger streams that is
// the faster one, beside streams of its own size the slower one (steps of
// 1280x720 with others, us with six / seven: 64x48 128 / 134, 320x240 129 /
// 133, 1920x1080 297 / 311, 3840x2160 808 / 857; one, two or seven of the same
// size 205 / 190, 303 / 283, 796 / 744; 853x481 158 / 149); `beside` does not
// tell them apart.
static bool fills_with_others(int nblocks, int beside, int sms) { return beside > 0 && nblocks + beside > 4 * sms; }

// CTAs of `groups` groups that `nblocks` blocks fill, at most one per SM.
static int packed_ctas(int nblocks, int groups, int sms) {
    const int n = (nblocks + groups - 1) / groups;
    return n < sms ? n : sms;
}

static cudaError_t launch_cqr2(int nblocks, int frame, NoiseConst nc, const void* tmp, float* weights,
                               float* mins_maxs, int* status, cudaStream_t s, int beside) {
    if (nblocks <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = device_sms(&dev, &sms);
    if (e != cudaSuccess) return e;
    CUtensorMap map;
    e = encode_tmp_map(tmp, nblocks, &map);
    if (e != cudaSuccess) return e;
    // Which shape for how many blocks per SM, as for k_fitter_rows16: up to
    // three, several teams shorten a block's chain (144 blocks 8.4 us with four
    // teams, 9.8 with two, 12.0 with one; 400 blocks 13.5 with two, 13.9 with
    // one); beyond, one team per block leaves the fewest sums over threads
    // (1050 blocks 23.8 us against 29.4 with two teams, 3680 blocks 75.2
    // against 87.7).  Four groups of one team fill the registers (255 each).
    const int per_sm = (nblocks + sms - 1) / sms, spread = nblocks < sms ? nblocks : sms;
    auto one_team = [&](int ctas) {
        if (nblocks > (kAlignRounds + 2) * 4 * ctas)   // more than six rounds
            return launch_cqr2_t<1, 4, true>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, ctas, s);
        return launch_cqr2_t<1, 4>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, ctas, s);
    };
    if (fills_with_others(nblocks, beside, sms)) return one_team(packed_ctas(nblocks, 4, sms));
    if (per_sm <= 1) return launch_cqr2_t<4, 1>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    if (per_sm <= 2) return launch_cqr2_t<2, 2>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    if (per_sm <= 3) return launch_cqr2_t<2, 3>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    return one_team(spread);
}

static cudaError_t launch_rows16(int nblocks, int frame, NoiseConst nc, const void* tmp, float* weights,
                                 float* mins_maxs, int* status, cudaStream_t s, int beside) {
    if (nblocks <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = device_sms(&dev, &sms);
    if (e != cudaSuccess) return e;
    CUtensorMap map;
    e = encode_tmp_map(tmp, nblocks, &map);
    if (e != cudaSuccess) return e;
    // Which shape for how many blocks per SM.  Up to three, one block's chain of
    // ten columns is what takes the time, and several teams shorten it: 100
    // blocks 16.6 us with four teams, 17.5 with two, 21.7 with one; 400 blocks
    // 24.7 us with two, 27.5 with one.  Beyond, one team per block costs the
    // fewest operations: 600 blocks 33.9 us against 41.0 with two teams.  A
    // seventh group overloads two of the SM's four schedulers, so a round of
    // seven blocks lasts longer than one of six (3108 blocks: 38.6 against
    // 29.3 us) and pays only where it saves a whole round: 986 blocks 42.3
    // against 52.9 us, 1904 72.0 against 82.2, 2072 79.0 against 82.4, 2812
    // 108.7 against 112.0, 3108 115.9 against 117.2; but 1776 72.0 against
    // 64.1, 2100 96.8 against 86.8, and above 21 blocks per SM the saved round
    // no longer makes up for the longer ones (4144: 153.6 against 147.9).
    const int per_sm = (nblocks + sms - 1) / sms, spread = nblocks < sms ? nblocks : sms;
    if (fills_with_others(nblocks, beside, sms))
        return launch_rows16_t<1, 6>(nblocks, frame, nc, map, weights, mins_maxs, status, dev,
                                     packed_ctas(nblocks, 6, sms), s);
    if (per_sm <= 1) return launch_rows16_t<4, 1>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    if (per_sm <= 2) return launch_rows16_t<2, 2>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    if (per_sm <= 3) return launch_rows16_t<2, 3>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    if (per_sm <= 21 && (per_sm + 6) / 7 < (per_sm + 5) / 6)
        return launch_rows16_t<1, 7>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
    return launch_rows16_t<1, 6>(nblocks, frame, nc, map, weights, mins_maxs, status, dev, spread, s);
}

bool fitter_fills_gpu(bool half_tmp, int qr) { return half_tmp && qr == kFitReference; }

bool fitter_reads_noise_table(bool half_tmp, int qr) { return !half_tmp || qr == kFitHouseholder32; }

cudaError_t launch_fitter(const Geometry& g, int frame, NoiseConst nc, const void* tmp, bool half_tmp,
                          int qr, float* weights, float* mins_maxs, const float* noise_table, int* status,
                          cudaStream_t s, int beside) {
    const int n = g.blocks;
    // The precision-form methods apply to binary16 tmp_data; float tmp_data
    // always takes the reference's arithmetic.
    if (half_tmp && qr == kFitReference) return launch_rows16(n, frame, nc, tmp, weights, mins_maxs, status, s, beside);
    if (half_tmp && qr == kFitCholQR2) return launch_cqr2(n, frame, nc, tmp, weights, mins_maxs, status, s, beside);
    if (noise_table) {
        if (!half_tmp)
            return launch_fitter_t<false, kFitReference, true>(n, frame, nc, tmp, weights, mins_maxs, noise_table,
                                                               status, s);
        return launch_fitter_t<true, kFitHouseholder32, true>(n, frame, nc, tmp, weights, mins_maxs, noise_table,
                                                              status, s);
    }
    if (!half_tmp)
        return launch_fitter_t<false, kFitReference, false>(n, frame, nc, tmp, weights, mins_maxs, nullptr, status,
                                                            s);
    return launch_fitter_t<true, kFitHouseholder32, false>(n, frame, nc, tmp, weights, mins_maxs, nullptr, status,
                                                           s);
}

// ---------------------------------------------------------------------------
// Scratch in a static device array, for callers that cannot allocate.
//
// The fitter's scratch is the frame's noise table (kNoiseTableFloats floats)
// plus the bounded-wait status word.  Both live here in one file-scope device
// array, so launch_fitter_static needs no cudaMalloc.  The table does not
// grow with the image: this fixed size serves every image size a plan
// accepts.  In host code g_fitter_scratch only names the symbol; the device
// address comes from cudaGetSymbolAddress, taken once per device with that
// device current, when the status word is also cleared (on the caller's
// stream, ordered before the call's kernels).  From then on the word is
// sticky: a kernel that gives up a bounded wait sets it, and only
// static_fitter_status_clear (bmfr_fitter_noalloc_check) clears it.
constexpr size_t kStaticStatusOffset = kNoiseTableBytes;             // 36,864
constexpr size_t kStaticScratchBytes = kStaticStatusOffset + 256;    // table + status word
static __device__ __align__(256) unsigned char g_fitter_scratch[kStaticScratchBytes];

static std::mutex g_scratch_mutex;
static void* g_scratch_address[64] = {nullptr};

static cudaError_t static_scratch_address(void** out, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_address[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_fitter_scratch);
        if (e != cudaSuccess) return e;
        e = cudaMemsetAsync(static_cast<unsigned char*>(p) + kStaticStatusOffset, 0, sizeof(int), s);
        if (e != cudaSuccess) return e;
        g_scratch_address[dev] = p;
    }
    *out = g_scratch_address[dev];
    return cudaSuccess;
}

cudaError_t static_fitter_status(int** status, cudaStream_t s) {
    void* base = nullptr;
    const cudaError_t e = static_scratch_address(&base, s);
    if (e != cudaSuccess) return e;
    *status = reinterpret_cast<int*>(static_cast<unsigned char*>(base) + kStaticStatusOffset);
    return cudaSuccess;
}

cudaError_t launch_fitter_static(const Geometry& g, int frame, NoiseConst nc, const void* tmp, bool half_tmp,
                                 int qr, float* weights, float* mins_maxs, cudaStream_t s) {
    void* base = nullptr;
    cudaError_t e = static_scratch_address(&base, s);
    if (e != cudaSuccess) return e;
    float* table = static_cast<float*>(base);
    int* status = reinterpret_cast<int*>(static_cast<unsigned char*>(base) + kStaticStatusOffset);
    if (fitter_reads_noise_table(half_tmp, qr)) {
        e = launch_noise_table(frame, table, s);   // rewrites the table the last call left
        if (e != cudaSuccess) return e;
    }
    return launch_fitter(g, frame, nc, tmp, half_tmp, qr, weights, mins_maxs, table, status, s);
}

}  // namespace bmfr
