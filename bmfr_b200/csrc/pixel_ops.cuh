// pixel_ops.cuh — per-pixel bodies of the BMFR stages (opencl/bmfr.cl),
// shared by the stage kernels and the fused per-block kernel.  Every float
// expression keeps the reference's operation order.
#pragma once

#include "common.cuh"

namespace bmfr {

__device__ __forceinline__ float3 hist_load(const float* p, int i) { return load3(p, i); }
__device__ __forceinline__ float3 hist_load(const __half* p, int i) {
    return make_float3(__half2float(p[3 * i]), __half2float(p[3 * i + 1]), __half2float(p[3 * i + 2]));
}

struct AccumResult {
    float ppx, ppy;      // prev_frame_pixel_f
    float3 color;        // blended colour
    uint8_t accept;
    uint8_t spp;
};

// Reprojection, 4-tap history gather and blend of one pixel
// (bmfr.cl:319-445).  `cur` is the pixel's colour before blending.
// The previous positions and normals of all in-image taps are loaded before
// any tap is tested, so their latencies overlap; the tests and the blend keep
// the reference's order.  Measured (accumulation by events, us, loaded where
// tested / before): 1920x1080 with binary16 histories 72.6 / 63.0, 1280x720
// 39.7 / 34.1; without it the float-history block kernel took 184.7 against
// 170.2.
template <typename HistT>
__device__ __forceinline__ AccumResult accumulate_core(
    const Geometry& g, const AccumArgs& a, int px, int py, float3 wp, float3 nrm, float3 cur,
    const float* __restrict__ prev_n, const float* __restrict__ prev_p,
    const HistT* __restrict__ prev_noisy, const uint8_t* __restrict__ prev_spp) {
    AccumResult r;
    r.ppx = (float)px;
    r.ppy = (float)py;
    r.accept = 0;
    float alpha = 1.0f;
    float3 prev = make_float3(0.f, 0.f, 0.f);
    float sample_spp = 0.0f;
    if (a.frame > 0) {
        const float* m = a.m;
        float uvx = ((m[0] * wp.x + m[4] * wp.y) + m[8] * wp.z) + m[12] * 1.0f;
        float uvy = ((m[1] * wp.x + m[5] * wp.y) + m[9] * wp.z) + m[13] * 1.0f;
        const float w = ((m[3] * wp.x + m[7] * wp.y) + m[11] * wp.z) + m[15] * 1.0f;
        // No lower limit: 1 is added to these quotients.
        if (divides_fast(w, fmaxf(fabsf(uvx), fabsf(uvy)))) {
            const float ny = -__frcp_rn(w);
            uvx = quotient(uvx, ny, w);
            uvy = quotient(uvy, ny, w);
        } else {
            uvx = uvx / w;
            uvy = uvy / w;
        }
        uvx = (uvx + 1.0f) / 2.0f;
        uvy = (uvy + 1.0f) / 2.0f;
        r.ppx = uvx * (float)g.W - a.off_x;
        r.ppy = uvy * (float)g.H - (1.0f - a.off_y);
        const int ix = floor_index(r.ppx), iy = floor_index(r.ppy);
        const float fx = r.ppx - (float)ix, fy = r.ppy - (float)iy;
        const float ofx = 1.0f - fx, ofy = 1.0f - fy;
        const float wts[4] = {ofx * ofy, fx * ofy, ofx * fy, fx * fy};
        const unsigned W = g.W, H = g.H;
        const bool col[2] = {(unsigned)ix < W, (unsigned)ix + 1u < W};
        const bool row[2] = {(unsigned)iy < H, (unsigned)iy + 1u < H};
        // The taps of a row lie side by side: one address per row and buffer.
        const int s0 = (int)((unsigned)iy * W + (unsigned)ix), s1 = (int)((unsigned)s0 + W);
        const float* const p_row[2] = {prev_p + 3 * (ptrdiff_t)s0, prev_p + 3 * (ptrdiff_t)s1};
        const float* const n_row[2] = {prev_n + 3 * (ptrdiff_t)s0, prev_n + 3 * (ptrdiff_t)s1};
        const HistT* const c_row[2] = {prev_noisy + 3 * (ptrdiff_t)s0, prev_noisy + 3 * (ptrdiff_t)s1};
        const uint8_t* const spp_row[2] = {prev_spp + s0, prev_spp + s1};
        float3 tp[4], tn[4];
        bool in[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            in[i] = col[i & 1] && row[i >> 1];
            tp[i] = tn[i] = make_float3(0.f, 0.f, 0.f);
            if (in[i]) {
                tp[i] = load3(p_row[i >> 1], i & 1);
                tn[i] = load3(n_row[i >> 1], i & 1);
            }
        }
        float wt[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float dx = tp[i].x - wp.x, dy = tp[i].y - wp.y, dz = tp[i].z - wp.z;
            const float ex = tn[i].x - nrm.x, ey = tn[i].y - nrm.y, ez = tn[i].z - nrm.z;
            in[i] = in[i] && (dx * dx + dy * dy) + dz * dz < a.pos_lim2 && (ex * ex + ey * ey) + ez * ez < a.nrm_lim2;
            wt[i] = in[i] ? wts[i] : 0.0f;
            if (in[i]) r.accept |= (uint8_t)(1 << i);
        }
        // The accepted taps' histories in one batch; the others add zeros,
        // which change no sum.
        float3 pc[4];
        float ps[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            pc[i] = make_float3(0.f, 0.f, 0.f);
            ps[i] = 0.0f;
            if (in[i]) {
                ps[i] = (float)spp_row[i >> 1][i & 1];
                pc[i] = hist_load(c_row[i >> 1], i & 1);
            }
        }
        float total = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sample_spp = sample_spp + wt[i] * ps[i];
            prev.x = prev.x + wt[i] * pc[i].x;
            prev.y = prev.y + wt[i] * pc[i].y;
            prev.z = prev.z + wt[i] * pc[i].z;
            total = total + wt[i];
        }
        if (total > 0.0f) {
            const uint32_t least = min(min(magnitude_key(prev.x), magnitude_key(prev.y)),
                                       min(magnitude_key(prev.z), magnitude_key(sample_spp)));
            if (divides_fast(total, fmaxf(fmaxf(fabsf(prev.x), fabsf(prev.y)), fmaxf(fabsf(prev.z), sample_spp)),
                             least)) {
                const float ny = -__frcp_rn(total);
                prev.x = quotient(prev.x, ny, total);
                prev.y = quotient(prev.y, ny, total);
                prev.z = quotient(prev.z, ny, total);
                sample_spp = quotient(sample_spp, ny, total);
            } else {
                prev.x = prev.x / total;
                prev.y = prev.y / total;
                prev.z = prev.z / total;
                sample_spp = sample_spp / total;
            }
            alpha = fmaxf(__frcp_rn(sample_spp + 1.0f), a.blend_alpha);
        }
    }
    // convert_uchar_sat_rte(sample_spp) + 1, saturated (bmfr.cl:424-436).
    r.spp = 1;
    if (alpha < 1.0f) r.spp = sample_spp > 254.0f ? 255 : (uint8_t)(__float2int_rn(sample_spp) + 1);
    const float om = 1.0f - alpha;
    r.color = make_float3(alpha * cur.x + om * prev.x, alpha * cur.y + om * prev.y,
                          alpha * cur.z + om * prev.z);
    return r;
}

// Writes the 13 feature/colour values of margin pixel (gx, gy) into the
// block-major tmp_data (bmfr.cl:448-476).
__device__ __forceinline__ void store_tmp_row(const Geometry& g, void* tmp, bool half_tmp, int gx,
                                              int gy, float3 wp, float3 nrm, float3 c) {
    const int xb = gx >> 5, yb = gy >> 5, xin = gx & 31, yin = gy & 31;
    const size_t base = (size_t)(yb * g.MWb + xb) * kBuffers * kBlockPixels + (size_t)(yin * 32 + xin);
    const float f[kBuffers] = {1.0f, nrm.x, nrm.y, nrm.z, wp.x, wp.y, wp.z,
                               wp.x * wp.x, wp.y * wp.y, wp.z * wp.z, c.x, c.y, c.z};
    if (half_tmp) {
        __half* t = static_cast<__half*>(tmp) + base;
        t[0] = __float2half_rn(1.0f);
#pragma unroll
        for (int k = 1; k < kBuffers; k += 2) {
            const __half2 h = pack_features(f[k], f[k + 1]);
            t[k * kBlockPixels] = __low2half(h);
            t[(k + 1) * kBlockPixels] = __high2half(h);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kBuffers; ++k)
            static_cast<float*>(tmp)[base + (size_t)k * kBlockPixels] = f[k] != f[k] ? 0.0f : f[k];
    }
}

// accumulate_noisy_data of margin pixel (gx, gy) (bmfr.cl:310-484), out of
// place: the pixel's colour is read from noisy_in and the blended colour
// goes to the history noisy_out; in-image pixels also write spp,
// prev_frame_pixel and accept.
template <typename HistT>
__device__ __forceinline__ void accumulate_margin_px(
    const Geometry& g, const AccumArgs& a, int gx, int gy, float2* __restrict__ prev_pix,
    uint8_t* __restrict__ accept, const float* __restrict__ cur_n, const float* __restrict__ prev_n,
    const float* __restrict__ cur_p, const float* __restrict__ prev_p, const float* __restrict__ noisy_in,
    HistT* __restrict__ noisy_out, const HistT* __restrict__ prev_noisy, const uint8_t* __restrict__ prev_spp,
    uint8_t* __restrict__ cur_spp, void* __restrict__ tmp) {
    const int2 bo = c_block_offsets[a.frame & 15];
    const int pwx = gx - kBlockEdge / 2 + bo.x;
    const int pwy = gy - kBlockEdge / 2 + bo.y;
    const bool in_image = pwx >= 0 && pwx < g.W && pwy >= 0 && pwy < g.H;
    const int px = mirror(pwx, g.W), py = mirror(pwy, g.H);
    const int lp = py * g.W + px;
    const float3 wp = load3(cur_p, lp);
    const float3 nrm = load3(cur_n, lp);
    const float3 cur = load3(noisy_in, lp);
    const AccumResult r = accumulate_core<HistT>(g, a, px, py, wp, nrm, cur, prev_n, prev_p, prev_noisy, prev_spp);
    store_tmp_row(g, tmp, a.use_half, gx, gy, wp, nrm, r.color);
    if (in_image) {   // bmfr.cl:442, 478-484
        cur_spp[lp] = r.spp;
        hist_store(noisy_out, lp, r.color);
        prev_pix[lp] = make_float2(r.ppx, r.ppy);
        accept[lp] = r.accept;
    }
}

// weighted_sum body (bmfr.cl:712-750).
// Index of the block whose weights pixel (px, py) uses (bmfr.cl:718-722).
__device__ __forceinline__ int pixel_block(const Geometry& g, int frame, int px, int py) {
    const int2 bo = c_block_offsets[frame & 15];
    const int opx = px + kBlockEdge / 2 - bo.x, opy = py + kBlockEdge / 2 - bo.y;
    return (opx / kBlockEdge) + (opy / kBlockEdge) * g.MWb;
}

// w: the block's 30 weights, mm: its 12 min/max values.
__device__ __forceinline__ float3 weighted_sum_px(float3 wp, float3 n, const float* w, const float* mm) {
    const float f[kFeatures] = {1.0f, n.x, n.y, n.z, wp.x, wp.y, wp.z, wp.x * wp.x, wp.y * wp.y, wp.z * wp.z};
    float3 c = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kFeatures; ++k) {
        float v = f[k];
        if (k >= kNotScaled) v = scale(v, mm[(k - kNotScaled) * 2], mm[(k - kNotScaled) * 2 + 1]);
        c.x = c.x + w[3 * k] * v;
        c.y = c.y + w[3 * k + 1] * v;
        c.z = c.z + w[3 * k + 2] * v;
    }
    c.x = c.x < 0.f ? 0.f : c.x;
    c.y = c.y < 0.f ? 0.f : c.y;
    c.z = c.z < 0.f ? 0.f : c.z;
    return c;
}

// A block's weights and feature bounds as a CTA whose pixels all lie in the
// block keeps them in shared memory: the divisions by the bounds' range need
// one reciprocal per block.
struct BlockFit {
    float w[kFeatures * 3 + 2];
    float mn[kScaled], d[kScaled], ny[kScaled];   // minimum, range, -RN(1/range)
};

// Filled by threads t = 0..63 of the CTA; a barrier follows.
__device__ __forceinline__ void prepare_block_fit(BlockFit& f, const float* __restrict__ weights,
                                                  const float* __restrict__ mins_maxs, int block, int t) {
    if (t < kFeatures * 3) f.w[t] = weights[(size_t)block * kFeatures * 3 + t];
    if (t >= 32 && t < 32 + kScaled) {
        const float* mm = mins_maxs + (size_t)block * kScaled * 2 + 2 * (t - 32);
        const float d = mm[1] - mm[0];
        f.mn[t - 32] = mm[0];
        f.d[t - 32] = d;
        f.ny[t - 32] = -__frcp_rn(d);
    }
}

// weighted_sum_px from a prepared block.
__device__ __forceinline__ float3 weighted_sum_block(float3 wp, float3 n, const BlockFit& b) {
    float v[kFeatures] = {1.0f, n.x, n.y, n.z, wp.x, wp.y, wp.z, wp.x * wp.x, wp.y * wp.y, wp.z * wp.z};
#pragma unroll
    for (int k = 0; k < kScaled; ++k) {
        const float a = v[kNotScaled + k] - b.mn[k], d = b.d[k];
        v[kNotScaled + k] = a;
        if (fabsf(d) > 1.0f)   // the same for the whole CTA
            v[kNotScaled + k] = divides_fast(d, fabsf(a), magnitude_key(a)) ? quotient(a, b.ny[k], d) : a / d;
    }
    float3 c = make_float3(0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kFeatures; ++k) {
        c.x = c.x + b.w[3 * k] * v[k];
        c.y = c.y + b.w[3 * k + 1] * v[k];
        c.z = c.z + b.w[3 * k + 2] * v[k];
    }
    c.x = c.x < 0.f ? 0.f : c.x;
    c.y = c.y < 0.f ? 0.f : c.y;
    c.z = c.z < 0.f ? 0.f : c.z;
    return c;
}

// accumulate_filtered_data body (bmfr.cl:778-856); returns the accumulated
// colour and writes the tone-mapped one through `tm`.
// Tone map: clamp(powr(max(0, albedo * acc), 0.454545), 0, 1) (bmfr.cl:853-854).
// powr is evaluated as exp2(0.454545 * log2(x)) on the special function
// unit (__log2f, exp2f): relative error below 1e-6 for x above 1e-3 and a
// negligible absolute error below that (the OpenCL powr it stands for may
// be 16 ulp off); several times cheaper than powf.
__device__ __forceinline__ float tonemap1(float albedo, float acc) {
    const float x = fmaxf(0.0f, albedo * acc);
    const float t = x > 0.0f ? exp2f(0.454545f * __log2f(x)) : 0.0f;
    return fminf(t, 1.0f);
}

template <typename HistT>
__device__ __forceinline__ float3 accumulate_filtered_px(const Geometry& g, int frame, int lp, float3 filt,
                                                         float2 pp, uint8_t acc, uint8_t spp,
                                                         float second_alpha, const HistT* __restrict__ acc_prev,
                                                         float3 albedo, float3* tm) {
    float3 prev = make_float3(0.f, 0.f, 0.f);
    float alpha = 1.0f;
    if (frame > 0 && acc > 0) {
        const int ix = floor_index(pp.x), iy = floor_index(pp.y);
        const float fx = pp.x - (float)ix, fy = pp.y - (float)iy;
        const float ofx = 1.0f - fx, ofy = 1.0f - fy;
        const float wts[4] = {ofx * ofy, fx * ofy, ofx * fy, fx * fy};
        const int s0 = (int)((unsigned)iy * (unsigned)g.W + (unsigned)ix);
        const HistT* const c_row[2] = {acc_prev + 3 * (ptrdiff_t)s0,
                                       acc_prev + 3 * (ptrdiff_t)(int)((unsigned)s0 + (unsigned)g.W)};
        // The accepted taps in one batch of loads; the others add zeros.
        float3 c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            c[i] = make_float3(0.f, 0.f, 0.f);
            if (acc & (1 << i)) c[i] = hist_load(c_row[i >> 1], i & 1);
        }
        float total = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w = acc & (1 << i) ? wts[i] : 0.0f;
            total = total + w;
            prev.x = prev.x + w * c[i].x;
            prev.y = prev.y + w * c[i].y;
            prev.z = prev.z + w * c[i].z;
        }
        if (total > 0.0f) {
            alpha = fmaxf(__frcp_rn((float)spp), second_alpha);
            prev = divide3(prev, total);
        }
    }
    const float om = 1.0f - alpha;
    const float3 a3 = make_float3(alpha * filt.x + om * prev.x, alpha * filt.y + om * prev.y,
                                  alpha * filt.z + om * prev.z);
    *tm = make_float3(tonemap1(albedo.x, a3.x), tonemap1(albedo.y, a3.y), tonemap1(albedo.z, a3.z));
    return a3;
}

// weighted_sum followed by accumulate_filtered_data for image pixel (px, py)
// (bmfr.cl:712-757, 773-856), without stores: returns the accumulated
// colour, and the filtered and tone-mapped colours through `filt`, `tm`.
template <typename HistT>
__device__ __forceinline__ float3 wsacc_core(const Geometry& g, int frame, float second_alpha, int px, int py,
                                             const float* __restrict__ weights,
                                             const float* __restrict__ mins_maxs, const float* __restrict__ cur_n,
                                             const float* __restrict__ cur_p, const float2* __restrict__ prev_pix,
                                             const uint8_t* __restrict__ accept, const float* __restrict__ albedo,
                                             const uint8_t* __restrict__ cur_spp,
                                             const HistT* __restrict__ acc_prev, float3* filt, float3* tm) {
    const int lp = py * g.W + px;
    const int gi = pixel_block(g, frame, px, py);
    const float3 f = weighted_sum_px(load3(cur_p, lp), load3(cur_n, lp), weights + (size_t)gi * kFeatures * 3,
                                     mins_maxs + (size_t)gi * kScaled * 2);
    *filt = f;
    // The accumulation writes the reprojected position and spp of every
    // image pixel, so they are read beside the accept mask instead of after
    // it: the history gather then waits for one round trip, not two.  With
    // no accepted tap they go unused.
    const uint8_t acc = frame > 0 ? accept[lp] : 0;
    const float2 pp = frame > 0 ? prev_pix[lp] : make_float2(0.f, 0.f);
    const uint8_t spp = frame > 0 ? cur_spp[lp] : 1;
    return accumulate_filtered_px(g, frame, lp, f, pp, acc, spp, second_alpha, acc_prev, load3(albedo, lp), tm);
}

// wsacc_core with the stores of the separate stages; `filtered` may be null.
template <typename HistT>
__device__ __forceinline__ void wsacc_px(const Geometry& g, int frame, float second_alpha, int px, int py,
                                         const float* __restrict__ weights, const float* __restrict__ mins_maxs,
                                         const float* __restrict__ cur_n, const float* __restrict__ cur_p,
                                         float* __restrict__ filtered, const float2* __restrict__ prev_pix,
                                         const uint8_t* __restrict__ accept, const float* __restrict__ albedo,
                                         float* __restrict__ tone_mapped, const uint8_t* __restrict__ cur_spp,
                                         const HistT* __restrict__ acc_prev, HistT* __restrict__ acc_cur) {
    const int lp = py * g.W + px;
    float3 f, tm;
    const float3 a3 = wsacc_core<HistT>(g, frame, second_alpha, px, py, weights, mins_maxs, cur_n, cur_p, prev_pix,
                                        accept, albedo, cur_spp, acc_prev, &f, &tm);
    if (filtered) store3(filtered, lp, f);
    hist_store(acc_cur, lp, a3);
    store3(tone_mapped, lp, tm);
}

// taa body (bmfr.cl:873-973).
// YCoCg of one colour, unnormalised (bmfr.cl:184-198).  Products by 2 are
// sums, which overflow where the reference's products do; the product by 0
// (NaN for an infinity) is exact and may be fused.
__device__ __forceinline__ void rgb_to_ycocg(float3 s, float (&ycc)[3]) {
    const float x2 = s.x + s.x, y2 = s.y + s.y, z2 = s.z + s.z;
    ycc[0] = (s.x + y2) + s.z;
    ycc[1] = __fmaf_rn(0.0f, s.y, x2) - z2;
    ycc[2] = (y2 - s.x) - s.z;
}

// The second half of taa (bmfr.cl:904-973) for a pixel whose tonemapped
// colour is `mine` and whose history position pp, with ix, iy its floor, has a
// tap in the image, given the YCoCg bounds of its 3x3 box and its cross:
// history bilinear, clamp, blend.
template <typename HistT>
__device__ __forceinline__ float3 taa_finish(const Geometry& g, float taa_alpha, float2 pp, int ix, int iy,
                                             float3 mine, const float (&mnb)[3], const float (&mxb)[3],
                                             const float (&mnc)[3], const float (&mxc)[3],
                                             const HistT* __restrict__ prev_frame) {
    float3 prev = make_float3(0.f, 0.f, 0.f);
    float total = 0.0f;
    const float fx = pp.x - (float)ix, fy = pp.y - (float)iy;
    const float ofx = 1.0f - fx, ofy = 1.0f - fy;
    const HistT* const row0 = prev_frame + 3 * (ptrdiff_t)(iy * g.W + ix);
    const HistT* const row1 = row0 + 3 * (ptrdiff_t)g.W;
    // The taps in the image in one batch of loads; the others add zeros.
    const float wts[4] = {ofx * ofy, fx * ofy, ofx * fy, fx * fy};
    const bool col[2] = {ix >= 0, ix < g.W - 1}, row[2] = {iy >= 0, iy < g.H - 1};
    float3 s[4];
    bool in[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        in[i] = col[i & 1] && row[i >> 1];
        s[i] = make_float3(0.f, 0.f, 0.f);
        if (in[i]) s[i] = hist_load(i >> 1 ? row1 : row0, i & 1);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float w = in[i] ? wts[i] : 0.0f;
        prev.x = prev.x + w * s[i].x;
        prev.y = prev.y + w * s[i].y;
        prev.z = prev.z + w * s[i].z;
        total = total + w;
    }
    prev = divide3(prev, total);
    float pyc[3];
    rgb_to_ycocg(prev, pyc);
    float cl[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float lo = (mnb[c] + mnc[c]) / 2.0f;
        const float hi = (mxb[c] + mxc[c]) / 2.0f;
        cl[c] = fminf(fmaxf(pyc[c], lo), hi);   // fmin/fmax: the bound where pyc is NaN
    }
    // bmfr.cl:965-967; products by 1/4 round where they are subnormal.
    const float a = cl[0] * 0.25f, b = cl[1] * 0.25f, c = cl[2] * 0.25f;
    const float3 rgb = make_float3((a + b) - c, __fmaf_rn(0.0f, cl[1], a) + c, (a - b) - c);
    const float om = 1.0f - taa_alpha;
    return make_float3(taa_alpha * mine.x + om * rgb.x, taa_alpha * mine.y + om * rgb.y,
                       taa_alpha * mine.z + om * rgb.z);
}

// taa over a strip of R rows per thread.  A warp covers 30 image columns
// x0..x0+29 in lanes 1..30 (lanes 0 and 31 hold the halo columns) and walks
// rows y0..y0+R-1: each thread reads and converts one pixel per row (R+2
// rows with the halo), takes its left and right neighbours by shuffles, and
// keeps a three-row window of horizontal minima and maxima, so a pixel's
// nine neighbours cost about one load and one YCoCg conversion.  Neighbours
// outside the image enter as NaN, which minimum and maximum skip as the
// reference's fmin/fmax do (bmfr.cl:884-902), so the bounds equal the
// reference's up to the sign of a zero bound.
template <int R, typename HistT>
__device__ __forceinline__ void taa_strip(const Geometry& g, int frame, float taa_alpha, int x0, int y0,
                                          const float2* __restrict__ prev_pix, const float* __restrict__ new_frame,
                                          const HistT* __restrict__ prev_frame, HistT* __restrict__ result_hist,
                                          float* __restrict__ result_out) {
    const int lane = threadIdx.x & 31;
    const int x = x0 - 1 + lane;
    const bool col_in = x >= 0 && x < g.W;
    const bool writer = lane >= 1 && lane <= 30 && col_in;
    const float nan = __int_as_float(0x7fffffff);
    float3 rgb[3];
    float own[3][3], hmn[3][3], hmx[3][3];   // [window row][channel]
    // The strip's reprojected positions first: the history gather of each
    // row depends on them, and they depend on nothing here.
    float2 ppre[R];
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
        const int py = y0 + rr;
        ppre[rr] = (writer && py < g.H) ? prev_pix[py * g.W + x] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < R + 2; ++r) {
        const int k = r % 3;
        const int y = y0 - 1 + r;
        const bool in = col_in && y >= 0 && y < g.H;
        const float3 s = in ? load3(new_frame, y * g.W + x) : make_float3(nan, nan, nan);
        rgb[k] = s;
        rgb_to_ycocg(s, own[k]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            // Lanes 0 and 31, the halo columns, take their own as a
            // neighbour and are not written.
            const float v = own[k][c];
            const float vl = __shfl_up_sync(0xffffffffu, v, 1), vr = __shfl_down_sync(0xffffffffu, v, 1);
            hmn[k][c] = min3(vl, v, vr);
            hmx[k][c] = max3(vl, v, vr);
        }
        if (r >= 2) {
            const int up = (r - 2) % 3, mid = (r - 1) % 3, dn = k;
            const int py = y0 + r - 2;
            if (writer && py < g.H) {
                const int lp = py * g.W + x;
                const float2 pp = ppre[r - 2];
                const float3 mine = rgb[mid];
                const int ix = floor_index(pp.x), iy = floor_index(pp.y);
                float3 out = mine;
                if (frame > 0 && (unsigned)ix + 1u <= (unsigned)g.W && (unsigned)iy + 1u <= (unsigned)g.H) {
                    float mnb[3], mxb[3], mnc[3], mxc[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        mnb[c] = min3(hmn[up][c], hmn[mid][c], hmn[dn][c]);
                        mxb[c] = max3(hmx[up][c], hmx[mid][c], hmx[dn][c]);
                        mnc[c] = min3(own[up][c], hmn[mid][c], own[dn][c]);
                        mxc[c] = max3(own[up][c], hmx[mid][c], own[dn][c]);
                    }
                    // A cross, and then perhaps its box, without a number: the
                    // bounds the reference starts from (bmfr.cl:884-888).
                    if (mnc[0] != mnc[0] || mnc[1] != mnc[1] || mnc[2] != mnc[2]) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            mnb[c] = fminf(mnb[c], INFINITY);
                            mxb[c] = fmaxf(mxb[c], -INFINITY);
                            mnc[c] = fminf(mnc[c], INFINITY);
                            mxc[c] = fmaxf(mxc[c], -INFINITY);
                        }
                    }
                    out = taa_finish(g, taa_alpha, pp, ix, iy, mine, mnb, mxb, mnc, mxc, prev_frame);
                }
                hist_store(result_hist, lp, out);
                if (result_out) store3(result_out, lp, out);
            }
        }
    }
}

}  // namespace bmfr
