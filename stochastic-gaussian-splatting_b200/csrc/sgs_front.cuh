// Scatter passes front to back.
//
// Most of what a deep scene's Gaussians draw lies behind other fragments: of 6M Gaussians at 1080p a quarter
// reaches a pixel before the pixel's last winner. Warps take groups of 32 consecutive Gaussians in depth order
// (GroupOrder), blocks among them lower an upper bound of the keys' depths per 8 x 8 pixel tile, and Gaussians
// behind the bounds of all tiles that they touch are dropped, most of them before their projection. Keys only
// decrease during a pass and a bound is never below its tile's keys, so the winners do not depend on any of it. (With
// more than 2^20 Gaussians above 512 pixels under hybrid scheduling, which of them the bin holds, and with that the
// last bit of an alpha, depends on the order of arrival, here as in passes that take them as they lie.)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include "sgs_internal.h"
#include "sgs_rows.cuh"

namespace sgs {

// Quads of tiles whose bounds a refreshing block lowers.
constexpr uint32_t kRefreshQuads = 16u * kOrderedWarps;
// Groups that may still be in flight when the pass has come to a group.
constexpr uint32_t kPassedSlack = 8192;
// Gaussians over more quads of tiles are not tested (a lane goes over all of them).
constexpr uint32_t kMaxTestedQuads = 8;

inline unsigned ordered_blocks(const GroupOrder& o) {
    const unsigned drawing = (o.groups + kOrderedWarps - 1u) / kOrderedWarps;
    return drawing + drawing / (o.refresh_period - 1u) + 1u;
}

// Whether the scene's Gaussians cover the framebuffer so often that depth order pays.
__device__ __forceinline__ bool front_to_back(const AccumulateParams& a) {
    const float4 c = *reinterpret_cast<const float4*>(a.queue->covered_all);
    return c.x + c.y + c.z + c.w > a.groups.min_pixels;
}

__device__ __forceinline__ float3 gaussian_position(const AccumulateParams& a, const uint32_t g) {
    if (a.quant.records != nullptr) return quant_position(a.quant, g, a.quant.records[g].x);
    return make_float3(a.means[3 * g], a.means[3 * g + 1], a.means[3 * g + 2]);
}

__device__ __forceinline__ float dot_plus(const float4 r, const float3 m) {
    return r.x * m.x + r.y * m.y + r.z * m.z + r.w;
}

// Whether Gaussian g lies near one of the other half of its group, on the screen (group_hidden tests rectangles of up to
// 256 pixels) and in depth. In a model that is not in Morton order hardly one does: there the groups' order and tests are
// for nothing, and point splatting, which drops only whole groups, is slower (6M Gaussians at random at 1080p: 457 us
// front to back, 396 as they lie; 8 samples 2289 and 2193 us). Stochastic transparency drops single Gaussians all the
// same (642 and 631 us, 8 samples 2480 and 2690).
__device__ __forceinline__ bool in_compact_group(const AccumulateParams& a, const uint32_t g) {
    const float3 m = gaussian_position(a, g), o = gaussian_position(a, min(g ^ 16u, a.n - 1u));
    const float4 r1 = a.w2c[0], r2 = a.w2c[1], r3 = a.w2c[2];
    const float z = dot_plus(r3, m), zo = dot_plus(r3, o);
    const float dx = (dot_plus(r1, m) / z - dot_plus(r1, o) / zo) * a.cam.focal_x;
    const float dy = (dot_plus(r2, m) / z - dot_plus(r2, o) / zo) * a.cam.focal_y;
    return fabsf(z - zo) <= 0.25f * fabsf(z) && fabsf(dx) <= 128.0f && fabsf(dy) <= 128.0f;
}

// Sorts the groups slice, slice + a.groups.slices, ... by depth (GroupOrder).
template <uint32_t kBlock>
__device__ __forceinline__ void sort_slice(const AccumulateParams& a, const uint32_t slice) {
    constexpr uint32_t kPerThread = kSliceGroups / kBlock;
    static_assert(kGroupBuckets == 4u * kBlock, "a thread sums four buckets");
    __shared__ __align__(16) uint32_t s_count[kGroupBuckets];
    __shared__ uint32_t s_warp[kBlock / 32u];
    for (uint32_t i = threadIdx.x; i < kGroupBuckets; i += kBlock) s_count[i] = 0u;
    const float4 r3 = a.w2c[2];
    float depth[kPerThread];
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) {
        const uint32_t g = slice + (threadIdx.x + k * kBlock) * a.groups.slices;
        if (g >= a.groups.groups) break;
        const uint32_t i = min(g * 32u + 16u, a.n - 1u);
        const float3 m = gaussian_position(a, i);
        depth[k] = r3.x * m.x + r3.y * m.y + r3.z * m.z + r3.w;
    }
    __syncthreads();
    uint32_t bucket[kPerThread], rank[kPerThread];
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) {
        const uint32_t g = slice + (threadIdx.x + k * kBlock) * a.groups.slices;
        if (g >= a.groups.groups) break;
        // what lies before the near plane goes last
        bucket[k] = kGroupBuckets - 1u;
        if (depth[k] > a.cam.near_plane)
            bucket[k] = static_cast<uint32_t>(min(max((__float_as_int(depth[k]) >> kGroupShift) - ((127 - 4) << (23 - kGroupShift)), 0),
                                                  static_cast<int>(kGroupBuckets) - 1));
        rank[k] = atomicAdd(&s_count[bucket[k]], 1u);
    }
    __syncthreads();
    uint4* const own = reinterpret_cast<uint4*>(s_count) + threadIdx.x;  // four buckets per thread
    const uint4 v = *own;
    const uint32_t sum = v.x + v.y + v.z + v.w;
    const uint32_t incl = warp_inclusive_sum(sum, threadIdx.x & 31u);
    if ((threadIdx.x & 31u) == 31u) s_warp[threadIdx.x >> 5] = incl;
    __syncthreads();
    uint32_t first = incl - sum;
#pragma unroll
    for (uint32_t w = 0; w < kBlock / 32u; ++w) first += w < threadIdx.x >> 5 ? s_warp[w] : 0u;
    *own = make_uint4(first, first + v.x, first + v.x + v.y, first + v.x + v.y + v.z);
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) {
        const uint32_t g = slice + (threadIdx.x + k * kBlock) * a.groups.slices;
        if (g >= a.groups.groups) break;
        a.groups.order[(s_count[bucket[k]] + rank[k]) * a.groups.slices + slice] = g;
    }
}

// Whether every pixel of columns [x0, x1] and rows [y0, y1] is nearer than depth `key_hi`, by the bounds of their
// tiles, four per load.
__device__ __forceinline__ bool behind_bounds(const StQueue& q, const uint32_t x0, const uint32_t x1, const uint32_t y0,
                                              const uint32_t y1, const uint32_t key_hi) {
    const uint32_t tx0 = x0 / kBoundTile, tx1 = x1 / kBoundTile, ty0 = y0 / kBoundTile, ty1 = y1 / kBoundTile;
    if ((tx1 / 4u - tx0 / 4u + 1u) * (ty1 - ty0 + 1u) > kMaxTestedQuads) return false;
    for (uint32_t ty = ty0; ty <= ty1; ++ty) {
        for (uint32_t qx = tx0 / 4u; qx <= tx1 / 4u; ++qx) {
            const uint4 b = __ldcg(reinterpret_cast<const uint4*>(
                q.tile_bound + static_cast<size_t>(ty) * q.bound_pitch + 4u * qx));
            uint32_t front = (b.x >= key_hi ? 1u : 0u) | (b.y >= key_hi ? 2u : 0u) | (b.z >= key_hi ? 4u : 0u) |
                             (b.w >= key_hi ? 8u : 0u);
            if (tx0 > 4u * qx) front &= 0xfu << (tx0 - 4u * qx);
            if (tx1 < 4u * qx + 3u) front &= 0xfu >> (4u * qx + 3u - tx1);
            if (front != 0) return false;
        }
    }
    return true;
}

// Extents of a Gaussian without its covariance: the variance along an image axis is at most the largest squared
// scale times the squared length of the axis' row of the Jacobian, the opacity at most 1, and one per cent and a
// pixel cover the rounding. Points of Gaussian point splatting (accumulate_gps.cu) stay within the same extents
// where the ellipse is not too thin, which the dilation grants below 900 times its variance.
// The preactivated layout holds the covariance, whose quadratic form is the variance itself. For Gaussians that are
// stretched along their ray it cancels, down to rounding residue that the projection, which evaluates it in
// another order, does not share. Either evaluation is off by less than 20 roundings (2^-24) of the squared length of
// the axis times the covariance's norm, which the sum of its entries' magnitudes bounds: kFormError of it covers both.
constexpr float kFormError = 4.0e-6f;
// A NaN among the parameters, or a quaternion whose norm overflows, gives a NaN covariance, which the projection
// bounds by the whole framebuffer: no extents are known then (maxima would drop the NaN). The rotation is read for
// this alone.
constexpr float kMaxNormSq = 1.0e37f;
enum Reach { kReachesNothing, kReachesRect, kReachUnknown };
struct ReachRect {
    uint32_t x0, x1, y0, y1, key_hi;
};
__device__ __forceinline__ Reach reach_of(const AccumulateParams& a, const uint32_t g, ReachRect& r) {
    uint4 rec = make_uint4(0u, 0u, 0u, 0u);
    if (a.quant.records != nullptr) rec = a.quant.records[g];
    const float3 m = a.quant.records != nullptr
                         ? quant_position(a.quant, g, rec.x)
                         : make_float3(a.means[3 * g], a.means[3 * g + 1], a.means[3 * g + 2]);
    // Loaded with the mean: after the depth test the rotations cost one sample of 6M Gaussians at 1080p 1.4 %, here
    // nothing.
    const bool plain = a.quant.records == nullptr && a.pre == nullptr;
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
    float4 q = make_float4(1.0f, 0.0f, 0.0f, 0.0f);
    if (plain) s0 = a.scales[3 * g], s1 = a.scales[3 * g + 1], s2 = a.scales[3 * g + 2], q = a.rotations[g];
    const float4 r1 = a.w2c[0], r2 = a.w2c[1], r3 = a.w2c[2];
    const PassCamera& cam = a.cam;
    const float z = dot_plus(r3, m);
    if (z < cam.near_plane - 1.0e-4f * fabsf(cam.near_plane)) return kReachesNothing;
    if (!(z > 0.0f)) return kReachUnknown;
    const float z_rcp = 1.0f / z;
    const float x = dot_plus(r1, m) * z_rcp, y = dot_plus(r2, m) * z_rcp;
    const float xc = fmaxf((-0.15f * cam.width - cam.center_x) / cam.focal_x,
                           fminf(x, (1.15f * cam.width - cam.center_x) / cam.focal_x));
    const float yc = fmaxf((-0.15f * cam.height - cam.center_y) / cam.focal_y,
                           fminf(y, (1.15f * cam.height - cam.center_y) / cam.focal_y));
    const float jx = cam.focal_x * z_rcp, jy = cam.focal_y * z_rcp;
    const float3 ax = make_float3(r1.x - xc * r3.x, r1.y - xc * r3.y, r1.z - xc * r3.z);
    const float3 ay = make_float3(r2.x - yc * r3.x, r2.y - yc * r3.y, r2.z - yc * r3.z);
    float vx, vy;
    if (a.pre != nullptr) {
        const float4 v0 = a.pre[2 * g], v1 = a.pre[2 * g + 1];  // (c11, c12, c13, c22), (c23, c33, ...)
        auto along = [&](const float3 d) {
            return d.x * (v0.x * d.x + 2.0f * (v0.y * d.y + v0.z * d.z)) + d.y * (v0.w * d.y + 2.0f * v1.x * d.z) +
                   v1.y * d.z * d.z;
        };
        const float error = kFormError * (fabsf(v0.x) + fabsf(v0.w) + fabsf(v1.y) +
                                          2.0f * (fabsf(v0.y) + fabsf(v0.z) + fabsf(v1.x)));
        vx = fmaxf(along(ax), 0.0f) + error * (ax.x * ax.x + ax.y * ax.y + ax.z * ax.z);
        vy = fmaxf(along(ay), 0.0f) + error * (ay.x * ay.x + ay.y * ay.y + ay.z * ay.z);
    } else {
        if (a.quant.records != nullptr) s0 = quant_half(rec.z), s1 = quant_half(rec.z >> 16), s2 = quant_half(rec.w);
        const float norm_sq = q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
        const float widest = fmaxf(fmaxf(s0, s1), s2);
        if (!(s0 <= widest && s1 <= widest && s2 <= widest && norm_sq <= kMaxNormSq)) return kReachUnknown;
        const float variance = expf(2.0f * widest);
        vx = variance * (ax.x * ax.x + ax.y * ax.y + ax.z * ax.z);
        vy = variance * (ay.x * ay.x + ay.y * ay.y + ay.z * ay.z);
    }
    const float dilation = (cam.proper_aa ? kDilationProperAA : kDilation) * cam.ss * cam.ss;
    vx = vx * jx * jx + dilation;
    vy = vy * jy * jy + dilation;
    if (!(vx + vy <= 900.0f * dilation)) return kReachUnknown;
    constexpr float kReach = 1.01f * 3.332f;  // sqrt(2 ln 255) = 3.3291
    const float ex = 1.0f + kReach * sqrtf(vx), ey = 1.0f + kReach * sqrtf(vy);
    const float px = x * cam.focal_x + cam.center_x, py = y * cam.focal_y + cam.center_y;
    if (px + ex < 0.0f || px - ex > cam.width || py + ey < 0.0f || py - ey > cam.height) return kReachesNothing;
    const float x_lo = fmaxf(px - ex, 0.0f), x_hi = fminf(px + ex, cam.width - 1.0f);
    const float y_lo = fmaxf(py - ey, 0.0f), y_hi = fminf(py + ey, cam.height - 1.0f);
    if (!(x_lo <= x_hi && y_lo <= y_hi)) return kReachUnknown;
    r.x0 = static_cast<uint32_t>(x_lo);
    r.x1 = static_cast<uint32_t>(x_hi);
    r.y0 = static_cast<uint32_t>(y_lo);
    r.y1 = static_cast<uint32_t>(y_hi);
    r.key_hi = __float_as_uint(0.9999f * z);
    return kReachesRect;
}

// Whether the whole warp's Gaussians lie behind all pixels that they can reach: the tiles of the rectangle around
// all of them, a lane four tiles, against the nearest one's depth. A seventh of the projection's instructions and,
// in the float layout, half of its bytes.
__device__ __forceinline__ bool group_hidden(const AccumulateParams& a, const bool active, const uint32_t g,
                                             const uint32_t lane) {
    constexpr uint32_t kFull = 0xffffffffu;
    ReachRect r;
    const Reach reach = active ? reach_of(a, g, r) : kReachesNothing;
    if (__any_sync(kFull, reach == kReachUnknown)) return false;
    const bool rect = reach == kReachesRect;
    const uint32_t x0 = __reduce_min_sync(kFull, rect ? r.x0 : kFull), x1 = __reduce_max_sync(kFull, rect ? r.x1 : 0u);
    const uint32_t y0 = __reduce_min_sync(kFull, rect ? r.y0 : kFull), y1 = __reduce_max_sync(kFull, rect ? r.y1 : 0u);
    const uint32_t key_hi = __reduce_min_sync(kFull, rect ? r.key_hi : kFull);
    if (x0 > x1) return true;  // nothing to draw
    const uint32_t tx0 = x0 / kBoundTile, tx1 = x1 / kBoundTile, ty0 = y0 / kBoundTile, ty1 = y1 / kBoundTile;
    const uint32_t q0 = tx0 / 4u, columns = tx1 / 4u - q0 + 1u;
    if (columns > 8u) return false;
    const uint32_t log_columns = columns > 4u ? 3u : columns > 2u ? 2u : columns - 1u;  // 1, 2, 4 or 8 lanes a row
    const uint32_t rows_at_once = 32u >> log_columns;
    if (ty1 - ty0 >= 2u * rows_at_once) return false;
    const uint32_t qx = q0 + (lane & ((1u << log_columns) - 1u));
    for (uint32_t ty = ty0 + (lane >> log_columns); ty - (lane >> log_columns) <= ty1; ty += rows_at_once) {
        uint32_t front = 0;
        if (ty <= ty1 && qx <= tx1 / 4u) {
            const uint4 b = __ldcg(reinterpret_cast<const uint4*>(
                a.stq.tile_bound + static_cast<size_t>(ty) * a.stq.bound_pitch + 4u * qx));
            front = (b.x >= key_hi ? 1u : 0u) | (b.y >= key_hi ? 2u : 0u) | (b.z >= key_hi ? 4u : 0u) |
                    (b.w >= key_hi ? 8u : 0u);
            if (tx0 > 4u * qx) front &= 0xfu << (tx0 - 4u * qx);
            if (tx1 < 4u * qx + 3u) front &= 0xfu >> (4u * qx + 3u - tx1);
        }
        if (__any_sync(kFull, front != 0)) return false;
    }
    return true;
}

// Sets the bounds of quad (qx, ty)'s four tiles to the largest depths of their keys in all samples'
// framebuffers: a lane reads a column of eight keys, eight lanes share a tile. `passed`: what is nearer has been
// drawn.
__device__ __forceinline__ void refresh_quad(const AccumulateParams& a, const uint32_t qx, const uint32_t ty,
                                             const uint32_t passed, const uint32_t lane) {
    constexpr uint32_t kFull = 0xffffffffu;
    uint32_t* const bounds = a.stq.tile_bound + (static_cast<size_t>(ty) * a.stq.bound_pitch + 4u * qx);
    const uint4 old = __ldcg(reinterpret_cast<const uint4*>(bounds));
    if (max(max(old.x, old.y), max(old.z, old.w)) < passed) return;  // what is still to come lies behind them all
    const uint32_t x = qx * (4u * kBoundTile) + lane, y0 = ty * kBoundTile;
    const uint32_t rows = x < a.cam.width_int ? min(kBoundTile, a.stq.height - y0) : 0u;
    const unsigned long long* p = a.framebuffer + (static_cast<size_t>(y0) * a.cam.width_int + x);
    auto depth_at = [&](const uint32_t i) {
        return i < rows ? __ldcg(reinterpret_cast<const uint32_t*>(p + static_cast<size_t>(i) * a.cam.width_int) + 1) : 0u;
    };
    // one row first: where each tile has an empty pixel there, the bounds stay as they are
    uint32_t far = depth_at(kBoundTile / 2u);
    uint32_t empty = __ballot_sync(kFull, far == kFull);
    empty |= empty >> 4;
    empty |= empty >> 2;
    empty |= empty >> 1;
    if ((empty & 0x01010101u) == 0x01010101u) return;
    for (uint32_t sm = 0; sm < a.n_samples; ++sm, p += a.fb_stride) {
        uint32_t depth[kBoundTile];  // the keys' high words
#pragma unroll
        for (uint32_t i = 0; i < kBoundTile; ++i) depth[i] = depth_at(i);
#pragma unroll
        for (uint32_t i = 0; i < kBoundTile; ++i) far = max(far, depth[i]);
    }
#pragma unroll
    for (uint32_t o = 1; o < kBoundTile; o <<= 1) far = max(far, __shfl_xor_sync(kFull, far, o));
    // another block's older value may land behind this one: an upper bound all the same
    if ((lane & (kBoundTile - 1u)) == 0) __stcg(bounds + lane / kBoundTile, far);
}

// Every a.groups.refresh_period-th block of the front-to-back pass draws nothing: these go over the framebuffer
// again and again and lower the tiles' bounds, which the blocks after them drop Gaussians by. Blocks start in the
// order of their numbers or nearly so; nothing but the time depends on it. False: the block has done its work;
// true: it draws, as number `block` of the drawing ones.
template <uint32_t kWarps>
__device__ __forceinline__ bool draws(const AccumulateParams& a, uint32_t& block, const bool ordered,
                                      const uint32_t wib, const uint32_t lane) {
    // the quotient, exact below 2^32 (an integer division here took 1 % of the pass)
    const uint32_t round = __double2uint_rz((static_cast<double>(block) + 0.5) * a.groups.refresh_rcp);
    if (block - round * a.groups.refresh_period != a.groups.refresh_period - 1u) {
        block -= round;
        return true;
    }
    if (!ordered) return false;
    const uint32_t quad_columns = a.stq.bound_pitch / 4u;
    const uint32_t quads = quad_columns * a.stq.tiles_y;
    const uint32_t first = (round % ((quads + kRefreshQuads - 1u) / kRefreshQuads)) * kRefreshQuads;
    const uint32_t end = min(first + kRefreshQuads, quads);
    // the depth that the pass has left behind
    const uint32_t at = max((block - round) * kWarps, kPassedSlack) - kPassedSlack;
    const uint32_t middle = min(a.groups.order[min(at, a.groups.groups - 1u)] * 32u + 16u, a.n - 1u);
    const uint32_t passed = __float_as_uint(fmaxf(dot_plus(a.w2c[2], gaussian_position(a, middle)), 0.0f));
    for (uint32_t t = first + wib; t < end; t += kWarps) {
        const uint32_t ty = t / quad_columns;
        refresh_quad(a, t - ty * quad_columns, ty, passed, lane);
    }
    return false;
}

}  // namespace sgs
