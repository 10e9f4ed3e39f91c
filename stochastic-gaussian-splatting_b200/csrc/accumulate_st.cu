// Stochastic-transparency accumulation: the closest accepted fragment per (sub)pixel.
//
// Semantics follow accumulate_scatter.cu:19-77 and scatter_utils.cuh:14-95 of the reference:
// every pixel of a Gaussian's clipped AABB with alpha >= 1/255 accepts the Gaussian when a
// threshold u(frame, Gaussian, pixel) < alpha, and the framebuffer keeps the minimum packed
// (depth_bits << 32 | index) key. The threshold is a stateless function of (frame, Gaussian,
// pixel) and the merge is a minimum, so the result does not depend on which thread evaluates
// which fragment. This file uses that freedom for a B200-oriented schedule:
//
//  * rows, then spans: a warp sorts its 32 Gaussians by their widest span (a bitonic network over
//    the lanes), expands them into AABB rows in that order, 32 rows at a time, and each lane
//    computes the conservative x-span of the alpha >= 1/255 ellipse on its row (the AABB corners,
//    ~45% of its pixels, are never evaluated);
//  * each lane then walks its own row two pixels per step, the alpha exponent of both pixels in
//    packed FP32x2 instructions (fma/mul/sub .f32x2 of sm_100a, each element rounded like the scalar
//    instruction), with no per-pixel owner lookup or shared-memory traffic; the warp steps as often
//    as its longest row needs, and each accepted pixel issues one predicated RED;
//  * a device-side work queue for the Gaussians with larger AABBs, which a persistent kernel takes in
//    parts (no cross-warp tail, no host synchronisation). In sparse scenes a part is a chunk of rows.
//    In dense ones (dense_scene) order_kernel lists the parts in depth order and a part is some
//    tiles of 8 x 8 pixels. Every tile has an upper bound of
//    its keys' depths (tile_bound); one lane per tile drops the tiles that lie behind their bound or
//    off the ellipse, and the warp walks the rest, two pixels per lane, lowering the bounds with the
//    keys it reads. Keys only decrease during a pass, so a dropped fragment could not have won;
//  * deep scenes of millions of Gaussians run front to back (sgs_front.cuh): the pass drops the groups and
//    the Gaussians that lie behind their tiles' bounds (6M at 1080p: 577 us a sample to 395, 283 million
//    warp instructions instead of 469; half of the rows are left, and their walk is what bounds it);
//  * u64 atomicMin (fire-and-forget RED) on the L2-resident framebuffer.
//
// Bit-exactness. The reference's alpha exponent `dx * (cx * dx + cy * dy) + cz * dy * dy` is
// contracted into fused multiply-adds differently by its scatter loops and by its hybrid gather
// kernel (measured on a B200 against the reference's own kernels over ~3.6e10 fragments):
//   scatter (accumulate_st_cu and hybrid::bin_cu):  fma(cz*dy, dy, dx * fma(cx, dx, cy*dy))
//   hybrid gather (hybrid::gather_cu):              fma(dx, fma(cx, dx, cy*dy), (cz*dy)*dy)
// Both forms are written out here with explicitly rounded intrinsics. With hybrid scheduling
// the reference gathers the Gaussians whose AABB exceeds 512 pixels (the first
// min(N, 2^20) of them, accumulate_hybrid.cu:26-27,98-111); those use the gather form.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include "sgs_internal.h"
#include "sgs_front.cuh"
#include "sgs_rows.cuh"

namespace sgs {
namespace {

constexpr uint32_t kBlock = 256;
constexpr uint32_t kWarpsPerBlock = kBlock / 32;
constexpr uint32_t kFullMask = 0xffffffffu;
constexpr uint32_t kQueueBlocksPerSM = 4;
// AABBs with more pixels are queued where the scene is not dense (queued_above).
constexpr uint32_t kMinPixels = kDenseMinPixels << kQueueSteps;
constexpr uint32_t kChunkPixels = 2048;   // pixels per chunk of rows of a queued Gaussian in a sparse scene
constexpr float kSampleMaxCover = 32.0f;  // a sampled Gaussian counts for at most this many framebuffers
constexpr uint32_t kOrderBlock = 512;
constexpr uint32_t kFewEntries = 4096, kManyChunks = 1u << 15;  // GPS: fewer Gaussians and more chunks are not listed
constexpr uint32_t kMaxClaim = 16;     // items a consumer warp takes per atomic on the cursor
constexpr uint32_t kPartQuads = 32;    // quads of four tiles in an item (a part of a queued Gaussian)
// Hybrid scheduling: AABBs above this many pixels are gathered by the reference (accumulate_hybrid.cu:26).
constexpr uint32_t kBinningPixelThreshold = 512;
// Flag in RowGaussian::flags: evaluate with the hybrid gather's contraction.
constexpr uint32_t kGatherFormFlag = 0x80000000u;

// Per-Gaussian constants of the row/span expansion and of a queue entry (64 bytes, four 16-byte words).
struct RowGaussian {
    float mx, my;       // mean2d - 0.5: pixel (x, y) has delta (x - mx, y - my)
    float cx, cy;       // exp2-scaled conic (x, y)
    float cz;           // exp2-scaled conic z
    float opacity;
    SpanConstants span; // conservative row spans (sgs_rows.cuh)
    uint32_t key_lo, key_hi;
    uint32_t x_min;
    uint32_t y_min, w;
    uint32_t row_first; // first row position in the warp's row list (level 1); queue: height
    uint32_t flags;     // kGatherFormFlag
};
static_assert(sizeof(RowGaussian) == kStEntryBytes, "the workspace reserves kStEntryBytes per queue entry");

// Queue entry e: the first q.entries_a entries lie in the queue section, the rest in the borrowed one.
__device__ __forceinline__ RowGaussian* queue_entry(const StQueue& q, const uint32_t e) {
    RowGaussian* const base = static_cast<RowGaussian*>(e < q.entries_a ? q.a : q.b);
    return base + (e < q.entries_a ? e : e - q.entries_a);
}

// Aligned quads of four tiles of the fixed 8 x 8 grid that an AABB touches, and the items its
// Gaussian is cut into.
struct QuadRect {
    uint32_t x0, y0, w, h;
};
__device__ __forceinline__ QuadRect quad_rect(const uint32_t x_min, const uint32_t w, const uint32_t y_min,
                                              const uint32_t h) {
    QuadRect t;
    t.x0 = x_min / (4u * kBoundTile);
    t.y0 = y_min / kBoundTile;
    t.w = (x_min + w - 1u) / (4u * kBoundTile) - t.x0 + 1u;
    t.h = (y_min + h - 1u) / kBoundTile - t.y0 + 1u;
    return t;
}
// scale: log2 of the quads per part over kPartQuads (part_scale).
__device__ __forceinline__ uint32_t part_count(const QuadRect& t, const uint32_t scale) {
    return min((t.w * t.h + (kPartQuads << scale) - 1u) / kPartQuads >> scale, kMaxParts);
}

// Packed FP32x2 arithmetic (sm_100a): two independent round-to-nearest operations per instruction,
// bit-identical to the scalar __fsub_rn / __fmul_rn / __fmaf_rn of each element.
__device__ __forceinline__ unsigned long long f2_pack(const float lo, const float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(const unsigned long long r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ unsigned long long f2_fma(const unsigned long long a, const unsigned long long b,
                                                     const unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long f2_mul(const unsigned long long a, const unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2_add(const unsigned long long a, const unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2_sub(const unsigned long long a, const unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Bits of 1 + u for the white-noise threshold u of pixel x on a row with seed
// gaussian ^ frame * 1973 ^ y * 2699 (pcg_hash of math_utils.h:113-122; ((w >> 22) ^ w) >> 9 is
// written as (w >> 9) ^ (w >> 31)).
__device__ __forceinline__ uint32_t st_threshold_bits(const uint32_t row_seed, const uint32_t x) {
    const uint32_t state = (row_seed ^ (x * 9277u)) * 747796405u + 2891336453u;
    const uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
    return 0x3f800000u | ((word >> 9u) ^ (word >> 31u));
}

// Blue-noise threshold of pixel x on a row whose slice row starts at texel `row_texel`, with the
// Gaussian's x offset bx (math_utils.h:125-136).
__device__ __forceinline__ float st_blue_threshold(const FrameRng& rng, const uint32_t row_texel, const uint32_t x,
                                                   const uint32_t bx) {
    const uint32_t texel = row_texel + ((x + bx) % kBlueNoiseWidth);
    const uint32_t value = (static_cast<uint32_t>(rng.slice[texel]) << 24u) + (1u << 23u) + rng.rotation;
    return static_cast<float>(value >> 8u) * 5.9604644775390625e-8f;
}

// Per-row random-number seed: the white-noise seed of row y, or the blue-noise slice row with the
// Gaussian's x offset in `bx` (math_utils.h:119-136).
template <bool kBlue>
__device__ __forceinline__ uint32_t row_seed(const FrameRng& rng, const uint32_t key_lo, const uint32_t y,
                                             uint32_t& bx) {
    if (kBlue) {
        const uint32_t oy = (key_lo * 0x91E10DA5u) >> 25u;
        bx = (key_lo * 0xC13FA9A9u) >> 25u;
        return ((y + oy) % kBlueNoiseHeight) * kBlueNoiseWidth;
    }
    bx = 0;
    return key_lo ^ (rng.frame * 1973u) ^ (y * 2699u);
}

// Sorting key of Gaussians without rows (they go after every Gaussian with rows).
constexpr uint32_t kNoRowsKey = (1u << 26) - 1u;

// Bitonic sort of one 32-bit value per lane, ascending over the lanes (values distinct).
__device__ __forceinline__ uint32_t warp_sort_ascending(uint32_t v, const uint32_t lane) {
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const uint32_t other = __shfl_xor_sync(kFullMask, v, j);
            const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
            v = keep_min ? min(v, other) : max(v, other);
        }
    }
    return v;
}

// One predicated 64-bit RED.MIN (no branch around it).
__device__ __forceinline__ void red_min_if(unsigned long long* address, const unsigned long long key, const bool pred) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.relaxed.gpu.global.min.u64 [%0], %1;\n\t}" ::"l"(address),
        "l"(key), "r"(static_cast<uint32_t>(pred))
        : "memory");
}

// Each lane walks segment `seg` of `1 << log_segs` equal parts of the span of its row y (when
// valid), two pixels per step; the warp takes as many steps as its longest segment needs
// (scatter_utils.cuh:35-46 per pixel).
template <bool kBlue, bool kHybrid, bool kMulti>
__device__ __forceinline__ void walk_rows(const AccumulateParams& a, const FrameRng& rng, const bool valid,
                                          const RowGaussian& G, const uint32_t y, const uint32_t seg = 0,
                                          const uint32_t log_segs = 0) {
    uint32_t xs = 0, len = 0;
    float dy = 0.0f;
    if (valid) {
        dy = __fsub_rn(static_cast<float>(y), G.my);
        row_span(G.x_min, G.w, G.mx, G.span, dy, xs, len);
        if (log_segs > 0) {
            const uint32_t part = (len + (1u << log_segs) - 1u) >> log_segs;
            const uint32_t skip = min(seg * part, len);
            xs += skip;
            len = min(len - skip, part);
        }
    }
    const uint32_t steps = __reduce_max_sync(kFullMask, len);
    if (steps == 0) return;
    const float cydy = __fmul_rn(G.cy, dy);
    const float czdy = __fmul_rn(G.cz, dy);
    uint32_t bx;
    const uint32_t seed = row_seed<kBlue>(rng, G.key_lo, y, bx);
    const unsigned long long key = (static_cast<unsigned long long>(G.key_hi) << 32) | G.key_lo;
    const bool gather_form = kHybrid && (G.flags & kGatherFormFlag);
    unsigned long long* row = a.framebuffer + (static_cast<size_t>(y) * a.cam.width_int + xs);
    const unsigned long long mx2 = f2_pack(G.mx, G.mx), cx2 = f2_pack(G.cx, G.cx), cydy2 = f2_pack(cydy, cydy);
    const unsigned long long czdy2 = f2_pack(czdy, czdy), dy2 = f2_pack(dy, dy);
    const unsigned long long opacity2 = f2_pack(G.opacity, G.opacity);
    const unsigned long long two = f2_pack(2.0f, 2.0f);
    const float fxs = static_cast<float>(xs);  // pixel coordinates are exact in float
    unsigned long long fx = f2_pack(fxs, fxs + 1.0f);
    for (uint32_t i = 0; i < steps; i += 2) {
        // alpha of pixels xs + i and xs + i + 1 with the reference's contraction of the exponent
        const unsigned long long dx = f2_sub(fx, mx2);
        const unsigned long long inner = f2_fma(cx2, dx, cydy2);
        const unsigned long long e2 =
            gather_form ? f2_fma(dx, inner, f2_mul(czdy2, dy2)) : f2_fma(czdy2, dy2, f2_mul(dx, inner));
        const float2 e = f2_unpack(e2);
        const float2 alpha =
            f2_unpack(f2_mul(opacity2, f2_pack(exp2f(fminf(e.x, 0.0f)), exp2f(fminf(e.y, 0.0f)))));
        const uint32_t x0 = xs + i;
        if (!kMulti) {
            float2 u;
            if (kBlue) {
                u = make_float2(st_blue_threshold(rng, seed, x0, bx), st_blue_threshold(rng, seed, x0 + 1u, bx));
            } else {
                u = f2_unpack(f2_sub(f2_pack(__uint_as_float(st_threshold_bits(seed, x0)),
                                             __uint_as_float(st_threshold_bits(seed, x0 + 1u))),
                                     f2_pack(1.0f, 1.0f)));
            }
            red_min_if(row + i, key, i < len && alpha.x >= kMinAlpha && u.x < alpha.x);
            red_min_if(row + i + 1u, key, i + 1u < len && alpha.y >= kMinAlpha && u.y < alpha.y);
        } else {
            // the same two pixels in every sample of the call: alpha once, one threshold per frame
            const bool in_x = i < len && alpha.x >= kMinAlpha;
            const bool in_y = i + 1u < len && alpha.y >= kMinAlpha;
            unsigned long long* row_s = row;
            for (uint32_t sm = 0; sm < a.n_samples; ++sm, row_s += a.fb_stride) {
                const uint32_t frame = rng.frame + sm;
                float2 u;
                if (kBlue) {
                    const FrameRng rs = frame_rng_at(a, frame);
                    u = make_float2(st_blue_threshold(rs, seed, x0, bx), st_blue_threshold(rs, seed, x0 + 1u, bx));
                } else {
                    // row seeds differ between frames only in the frame term
                    const uint32_t seed_s = seed ^ ((rng.frame * 1973u) ^ (frame * 1973u));
                    u = f2_unpack(f2_sub(f2_pack(__uint_as_float(st_threshold_bits(seed_s, x0)),
                                                 __uint_as_float(st_threshold_bits(seed_s, x0 + 1u))),
                                         f2_pack(1.0f, 1.0f)));
                }
                red_min_if(row_s + i, key, in_x && u.x < alpha.x);
                red_min_if(row_s + i + 1u, key, in_y && u.y < alpha.y);
            }
        }
        fx = f2_add(fx, two);
    }
}

// Whether the tile (tx, ty) may hold a pixel with alpha >= 1/255: the x-extent of the ellipse over the
// tile's rows, a concave function of dy on either side whose maximum lies at +-dy_star or at the end
// of the rows nearest to it, widened like a row's span (sgs_rows.cuh).
__device__ __forceinline__ bool tile_on_ellipse(const RowGaussian& G, const uint32_t tx, const uint32_t ty) {
    if (!(G.span.k2 > 0.0f)) return true;
    const float x0 = static_cast<float>(tx * kBoundTile) - G.mx, y0 = static_cast<float>(ty * kBoundTile) - G.my;
    constexpr float kSide = static_cast<float>(kBoundTile - 1u);
    const float dymax = sqrtf(G.span.dymax2);
    const float eps_y = kSpanPixelMargin + 4.0e-6f * (fabsf(y0) + dymax);
    const float lo = fmaxf(y0 - eps_y, -dymax), hi = fminf(y0 + kSide + eps_y, dymax);
    if (!(lo <= hi)) return lo != lo || hi != hi;
    // right end at dy: slope dy + sqrt(k2 (dymax2 - dy^2)), largest at dy = slope sqrt(dymax2 / (k2 + slope^2))
    const float star = G.span.slope * dymax * rsqrtf(G.span.k2 + G.span.slope * G.span.slope);
    const float dr = fminf(fmaxf(star, lo), hi), dl = fminf(fmaxf(-star, lo), hi);
    const float right = fmaf(G.span.slope, dr, sqrtf(G.span.k2 * fmaxf(fmaf(-dr, dr, G.span.dymax2), 0.0f)));
    const float left = fmaf(G.span.slope, dl, -sqrtf(G.span.k2 * fmaxf(fmaf(-dl, dl, G.span.dymax2), 0.0f)));
    const float eps = 0.1f + 1.0e-4f * (fabsf(right) + fabsf(left) + fabsf(x0));
    // written so that a non-finite bound keeps the tile
    return !(right + eps < x0) && !(left - eps > x0 + kSide);
}

// Sparse scenes: rows per chunk of a queued Gaussian of AABB width w (about kChunkPixels pixels, a power
// of two between 1 and 32; each row is walked in 32 / rows segments, so wide footprints keep every lane
// walking) and chunks per item (1 << scale, but for AABBs of more than kMaxParts times that).
__device__ __forceinline__ uint32_t log_chunk_rows(const uint32_t w) {
    const uint32_t rows = max(1u, min(32u, kChunkPixels / max(w, 1u)));
    return 31u - __clz(rows);
}
struct RowParts {
    uint32_t log_rows, chunks, per_part, parts;
};
__device__ __forceinline__ RowParts row_parts(const uint32_t w, const uint32_t h, const uint32_t scale) {
    RowParts r;
    r.log_rows = log_chunk_rows(w);
    r.chunks = (h + (1u << r.log_rows) - 1u) >> r.log_rows;
    r.per_part = max((r.chunks + kMaxParts - 1u) / kMaxParts, 1u << scale);
    r.parts = (r.chunks + r.per_part - 1u) / r.per_part;
    return r;
}

// A lane's two pixels of tile (tx, ty), (lane & 7, lane / 8) and four rows below, and their keys: 0 (which
// nothing can beat) off the image.
struct TilePixels {
    unsigned long long* p;  // the upper pixel in the first sample's framebuffer
    bool img0, img1;
};
__device__ __forceinline__ TilePixels tile_pixels(const AccumulateParams& a, const uint32_t tx, const uint32_t ty,
                                                  const uint32_t lane) {
    const uint32_t x = tx * kBoundTile + (lane & 7u), y = ty * kBoundTile + (lane >> 3);
    TilePixels t;
    t.p = a.framebuffer + (static_cast<size_t>(y) * a.cam.width_int + x);
    t.img0 = x < a.cam.width_int && y < a.stq.height;
    t.img1 = x < a.cam.width_int && y + 4u < a.stq.height;
    return t;
}
struct TileKeys {
    unsigned long long k0, k1;
};
__device__ __forceinline__ TileKeys tile_keys(const TilePixels& t, const size_t offset, const size_t below) {
    TileKeys k;
    k.k0 = t.img0 ? __ldcg(t.p + offset) : 0ull;
    k.k1 = t.img1 ? __ldcg(t.p + offset + below) : 0ull;
    return k;
}

// The warp walks tile (tx, ty) for Gaussian G, a lane the two pixels `px`: those whose key is
// already nearer are left alone, and the largest depth of the tile's keys lowers its bound. `first`:
// the tile's keys in the first sample's framebuffer (read ahead); with several samples per call the
// other framebuffers' keys are read kKeyBatch samples at a time.
template <bool kBlue, bool kHybrid, bool kMulti>
__device__ __forceinline__ void walk_tile(const AccumulateParams& a, const FrameRng& rng, const RowGaussian& G,
                                          const uint32_t tx, const uint32_t ty, const uint32_t lane,
                                          const TilePixels& px, const TileKeys& first) {
    constexpr uint32_t kKeyBatch = kMulti ? 4u : 1u;
    const uint32_t x = tx * kBoundTile + (lane & 7u);
    const uint32_t y0 = ty * kBoundTile + (lane >> 3), y1 = y0 + 4u;
    const bool col = x - G.x_min < G.w;
    const bool in0 = col && y0 - G.y_min < G.row_first, in1 = col && y1 - G.y_min < G.row_first;
    const size_t below = 4u * static_cast<size_t>(a.cam.width_int);
    const unsigned long long key = (static_cast<unsigned long long>(G.key_hi) << 32) | G.key_lo;
    uint32_t* const bound = a.stq.tile_bound + (static_cast<size_t>(ty) * a.stq.bound_pitch + tx);
    if (!kMulti && !__any_sync(kFullMask, (in0 && key < first.k0) || (in1 && key < first.k1))) {
        // nothing of the tile is left to win
        const uint32_t far = __reduce_max_sync(
            kFullMask, max(static_cast<uint32_t>(first.k0 >> 32), static_cast<uint32_t>(first.k1 >> 32)));
        if (lane == 0) atomicMin(bound, far);
        return;
    }

    // alpha of both pixels with the reference's contraction of the exponent
    const float dx = __fsub_rn(static_cast<float>(x), G.mx);
    const unsigned long long dy =
        f2_sub(f2_pack(static_cast<float>(y0), static_cast<float>(y1)), f2_pack(G.my, G.my));
    const unsigned long long cydy = f2_mul(f2_pack(G.cy, G.cy), dy), czdy = f2_mul(f2_pack(G.cz, G.cz), dy);
    const unsigned long long dx2 = f2_pack(dx, dx);
    const unsigned long long inner = f2_fma(f2_pack(G.cx, G.cx), dx2, cydy);
    const bool gather_form = kHybrid && (G.flags & kGatherFormFlag);
    const float2 e = f2_unpack(gather_form ? f2_fma(dx2, inner, f2_mul(czdy, dy))
                                           : f2_fma(czdy, dy, f2_mul(dx2, inner)));
    const float2 alpha = f2_unpack(
        f2_mul(f2_pack(G.opacity, G.opacity), f2_pack(exp2f(fminf(e.x, 0.0f)), exp2f(fminf(e.y, 0.0f)))));
    const bool hit0 = in0 && alpha.x >= kMinAlpha, hit1 = in1 && alpha.y >= kMinAlpha;
    uint32_t bx;
    const uint32_t seed0 = row_seed<kBlue>(rng, G.key_lo, y0, bx);
    const uint32_t seed1 = row_seed<kBlue>(rng, G.key_lo, y1, bx);

    uint32_t farthest = 0;
    const uint32_t n_samples = kMulti ? a.n_samples : 1u;
    size_t offset = 0;
    for (uint32_t base = 0; base < n_samples; base += kKeyBatch, offset += kKeyBatch * a.fb_stride) {
        TileKeys k[kKeyBatch];
#pragma unroll
        for (uint32_t j = 0; j < kKeyBatch; ++j)
            k[j] = base + j == 0          ? first
                   : base + j < n_samples ? tile_keys(px, offset + j * a.fb_stride, below)
                                          : TileKeys{0ull, 0ull};
#pragma unroll
        for (uint32_t j = 0; j < kKeyBatch; ++j) {
            farthest = max(farthest, max(static_cast<uint32_t>(k[j].k0 >> 32), static_cast<uint32_t>(k[j].k1 >> 32)));
            const bool can0 = hit0 && key < k[j].k0, can1 = hit1 && key < k[j].k1;
            if (!__any_sync(kFullMask, can0 || can1)) continue;
            const uint32_t sm = base + j;
            float2 u;
            if (kBlue) {
                const FrameRng rs = kMulti ? frame_rng_at(a, rng.frame + sm) : rng;
                u = make_float2(st_blue_threshold(rs, seed0, x, bx), st_blue_threshold(rs, seed1, x, bx));
            } else {
                // row seeds differ between frames only in the frame term
                const uint32_t df = kMulti ? (rng.frame * 1973u) ^ ((rng.frame + sm) * 1973u) : 0u;
                u = f2_unpack(f2_sub(f2_pack(__uint_as_float(st_threshold_bits(seed0 ^ df, x)),
                                             __uint_as_float(st_threshold_bits(seed1 ^ df, x))),
                                     f2_pack(1.0f, 1.0f)));
            }
            unsigned long long* const p = px.p + (kMulti ? offset + j * a.fb_stride : 0u);
            red_min_if(p, key, can0 && u.x < alpha.x);
            red_min_if(p + below, key, can1 && u.y < alpha.y);
        }
    }
    farthest = __reduce_max_sync(kFullMask, farthest);
    if (lane == 0 && farthest != 0xffffffffu) atomicMin(bound, farthest);
}

// Whether the Gaussians above kDenseMinPixels cover the framebuffer many times over, by the clear pass's
// sample. Then nearly all of what lies behind the first few surfaces is culled in the queue, so that it
// takes all of them, in depth order; elsewhere the row walker is the faster one for footprints of up to
// some 2000 pixels, and ordering a short queue costs more than it saves.
__device__ __forceinline__ bool dense_scene(const AccumulateParams& a) {
    const float4 c = *reinterpret_cast<const float4*>(a.queue->covered);
    return c.x + c.y + c.z + c.w > a.stq.dense_pixels;
}

// AABBs above this many pixels are queued: in a dense scene all above kDenseMinPixels if the queue holds them, else
// those of the next larger size that it holds. A warp draws what finds the queue full by itself, which takes long where
// that are Gaussians of many thousand pixels (2M Gaussians and 24,000 large ones at 1920x1080, room for 0.53 of 1.30
// million above 256: 2631 us a sample; of the larger ones that it holds 1367; with a queue for 2048 and more 1731). A
// few per cent past the room cost less than the next size (1M Gaussians at 1280x720, room for all: 455 and 539 us), but
// not front to back (kFrontRoom).
constexpr float kRoom = 1.05f;
// Front to back, what finds the queue full comes last and together: single warps with 32 Gaussians of thousands of pixels
// each. Such passes leave some room, and scenes whose large Gaussians may not fit are drawn as they lie (5M Gaussians
// around the camera, 1600x900: 6382 us a sample front to back, 1738; 2.7M: 2090, 608; 5M faint ones 4720, 1561).
constexpr float kFrontRoom = 0.95f;
__device__ __forceinline__ uint32_t queued_above(const AccumulateParams& a, const bool dense, const float share = kRoom) {
    const float room = share * static_cast<float>(a.stq.capacity);
    uint32_t step = kQueueSteps;
#pragma unroll
    for (uint32_t i = kQueueSteps; i-- > 0;) {
        const float4 n = *reinterpret_cast<const float4*>(a.queue->larger[i]);
        if (n.x + n.y + n.z + n.w <= room) step = i;
    }
    return dense ? kDenseMinPixels << step : kMinPixels;
}

// How much larger than usual (log2) the parts of queued Gaussians are, so that the list has room for all that the clear pass
// expects. Gaussians whose parts found the list full were drawn by their own warps (53,000 of up to 3.7 million pixels at
// 2560x1448, 21,700 of them without a place: 134 ms a sample, 1.9 ms with larger parts).
__device__ __forceinline__ uint32_t part_scale(const AccumulateParams& a, const bool dense) {
    auto sum_of = [](const float* const v) {  // (the same in every kernel)
        const float4 n = *reinterpret_cast<const float4*>(v);
        return __fadd_rn(__fadd_rn(n.x, n.y), __fadd_rn(n.z, n.w));
    };
    const float parts = sum_of(a.queue->parts[dense ? 0 : 1]);
    const float list = static_cast<float>(a.stq.list_capacity);
    if (parts <= 0.9f * list) return 0u;
    const float entries = fminf(sum_of(a.queue->larger[dense ? 0u : kQueueSteps - 1u]), static_cast<float>(a.stq.capacity));
    // at most 2^12, where no Gaussian has more than four parts
    const float scale = __fdiv_rn(parts, 0.9f * fmaxf(__fsub_rn(list, entries), 0.25f * list));
    return 32u - __clz(static_cast<uint32_t>(fminf(scale, 4095.0f)));
}

// How a scatter pass takes its Gaussians: a warp 32 of them, several warps the same 32 (small scenes), or a warp
// 32 of them front to back, dropping those behind their tiles' bounds.
enum ScatterMode { kPlain, kSplitRows, kFrontToBack };

// One thread per Gaussian (accumulate_scatter.cu:19-77 for the projection and the AABB).
// Held to as many blocks as leave 64 registers (front to back and one sample: 56), at the price of some spills; with
// the registers that need none fewer warps hide the latencies. Per call with spills and without: split rows and 8
// samples, 30k Gaussians at 640x480, 671 and 693 us, hybrid with blue noise, 100k, 1103 and 1114; front to back, 6M at
// 1920x1080, 398 and 409 us (8 bytes), hybrid 404 and 422 (32), blue noise 433 and 441 (24), both 436 and 449 (68).
template <bool kBlue, bool kHybrid, bool kMulti, ScatterMode kMode>
__global__ void __launch_bounds__(kMode == kFrontToBack ? kOrderedWarps * 32u : kBlock,
                                  kMode == kFrontToBack ? (kMulti ? 32u : 36u) / kOrderedWarps : 4u)
st_scatter_kernel(const AccumulateParams a) {
    constexpr uint32_t kWarps = kMode == kFrontToBack ? kOrderedWarps : kWarpsPerBlock;
    __shared__ RowGaussian s_gauss[kWarps][32];
    __shared__ uint32_t s_rank[kWarps][32];

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t wib = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t upto_mask = kFullMask >> (31u - lane);
    // kSplit (small scenes): 2^log_row_split warps share 32 Gaussians, each walking every 2^log_row_split-th
    // batch of their rows (all project them; the first one queues the large ones)
    wait_for_pass_before();
    constexpr bool kSplit = kMode == kSplitRows;
    uint32_t block = blockIdx.x;
    bool ordered = false, dense = false;
    uint32_t queue_above = kMinPixels, scale = 0;
    if (kMode == kFrontToBack) {
        ordered = front_to_back(a);
        dense = dense_scene(a);
        if (dense) {
            queue_above = queued_above(a, true, ordered ? kFrontRoom : kRoom);
            if (ordered && queue_above == kMinPixels) {  // none of the sizes is sure to fit
                ordered = false;
                queue_above = queued_above(a, true);
            }
        }
        if (!draws<kWarps>(a, block, ordered, wib, lane)) return;
    }
    uint32_t gwarp = block * kWarps + wib;
    const uint32_t log_split = kSplit ? a.stq.log_row_split : 0u;
    const uint32_t sub = gwarp & ((1u << log_split) - 1u);
    if (kMode == kFrontToBack && ordered) {
        if (gwarp >= a.groups.groups) return;
        gwarp = a.groups.order[gwarp];
    }
    const uint32_t idx = (gwarp >> log_split) * 32u + lane;
    bool active = idx < a.n;
    const uint32_t g = active ? idx : a.n - 1;

    if (kMode == kFrontToBack && ordered && group_hidden(a, active, g, lane)) return;

    // Loaded while the projection waits for its own loads: after it, the scatter pass over 400k large Gaussians took 73 us
    // instead of 68. Deep scenes are seldom dense and load the sizes only then.
    if (kMode != kFrontToBack) {
        dense = dense_scene(a);
        queue_above = queued_above(a, dense);
        if (dense) scale = part_scale(a, true);
    }
    Projected p;
    if (!project_gaussian(active, g, a.means, a.scales, a.rotations, a.opacities, a.w2c, a.cam, p, a.pre, a.quant)) return;
    const FrameRng rng = frame_rng(a);

    const PixelRect rect = pixel_rect(p.bounds, a.cam);
    uint32_t count = active ? rect.width * rect.height : 0u;
    RowGaussian G;
    G.mx = p.mean2d.x - 0.5f;
    G.my = p.mean2d.y - 0.5f;
    const float3 ce = conic_for_exp2(p.conic);
    G.cx = ce.x;
    G.cy = ce.y;
    G.cz = ce.z;
    G.opacity = p.opacity;
    const unsigned long long key = pack_fragment(p.depth, g);
    G.key_lo = static_cast<uint32_t>(key);
    G.key_hi = static_cast<uint32_t>(key >> 32);
    G.x_min = rect.x_min;
    G.y_min = rect.y_min;
    G.w = rect.width;
    G.row_first = 0;
    G.flags = 0;
    G.span = span_constants(G.cx, G.cy, G.cz, G.opacity);

    if (kHybrid) {
        // the reference gathers the first min(N, 2^20) Gaussians with more than 512 pixels (warps sharing
        // their Gaussians only run with fewer than that, when all are gathered)
        const bool binned = active && count > kBinningPixelThreshold;
        const uint32_t ballot = __ballot_sync(kFullMask, binned);
        if (ballot != 0) {
            const uint32_t leader = __ffs(ballot) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&a.queue->binned, static_cast<unsigned>(__popc(ballot)));
            base = __shfl_sync(kFullMask, base, leader);
            if (binned && base + __popc(ballot & lt_mask) < a.max_binned) G.flags = kGatherFormFlag;
        }
    }

    if (kMode == kFrontToBack && ordered) {
        if (count != 0 && behind_bounds(a.stq, rect.x_min, rect.x_min + rect.width - 1u, rect.y_min,
                                        rect.y_min + rect.height - 1u, G.key_hi)) {
            active = false;
            count = 0;
        }
        if (!__any_sync(kFullMask, count != 0)) return;
    }

    // larger footprints: an entry in the work queue (or kept here when it is full); one atomic per warp
    bool keep_big = false;
    bool has_rows = count > 0;
    const bool large = count > queue_above;
    const bool want = large && sub == 0;
    if (large) has_rows = false;
    const uint32_t big = __ballot_sync(kFullMask, want);
    if (big != 0) {
        const uint32_t leader = __ffs(big) - 1;
        uint32_t e = 0;
        if (lane == leader) e = atomicAdd(&a.queue->st_entries, static_cast<uint32_t>(__popc(big)));
        e = __shfl_sync(kFullMask, e, leader) + __popc(big & lt_mask);
        const bool fits = want && e < a.stq.capacity;
        if (kMode == kFrontToBack || !dense) scale = part_scale(a, dense);
        const uint32_t parts =
            !fits   ? 0u
            : dense ? part_count(quad_rect(rect.x_min, rect.width, rect.y_min, rect.height), scale)
                    : row_parts(rect.width, rect.height, scale).parts;
        const uint32_t incl = warp_inclusive_sum(parts, lane);
        uint32_t item = 0;
        if (lane == 31 && incl != 0) item = atomicAdd(&a.queue->st_items, incl);
        item = __shfl_sync(kFullMask, item, 31) + (incl - parts);
        const bool listed = fits && item + parts <= a.stq.list_capacity;
        if (fits) {
            RowGaussian st = G;
            st.row_first = listed ? rect.height : 0u;  // no rows: the order pass skips the entry
            *queue_entry(a.stq, e) = st;
        }
        if (!dense) {
            for (uint32_t i = 0; i < parts && item + i < a.stq.list_capacity; ++i)
                a.stq.list[item + i] = listed ? i << kItemEntryBits | e : kNoItem;
        } else {
            count_at_depth(a.stq.histogram, G.key_hi, listed ? parts : 0u, lane);
        }
        keep_big = want && !listed;
        if (keep_big) atomicAdd(&a.queue->overflow, 1u);
    }

    // level 1: the rows of this warp's Gaussians, end to end, the Gaussians ordered by their widest
    // span so that the 32 rows walked together have similar lengths (a warp walks as long as its
    // longest row); Gaussians without rows go last
    uint32_t width_key = kNoRowsKey;
    if (has_rows) {
        uint32_t widest = G.w;
        if (G.span.k2 > 0.0f) {
            const float est = 2.0f * sqrtf(G.span.k2 * G.span.dymax2) + 2.0f;
            if (est < static_cast<float>(widest)) widest = static_cast<uint32_t>(est);
        }
        width_key = min(widest, kNoRowsKey - 1u);
    }
    const uint32_t sorted = warp_sort_ascending((width_key << 5) | lane, lane);  // lane i: i-th smallest
    const uint32_t src_lane = sorted & 31u;
    s_rank[wib][src_lane] = lane;
    const uint32_t h = has_rows ? rect.height : 0u;
    const uint32_t h_sorted = __shfl_sync(kFullMask, h, src_lane);
    const uint32_t incl_sorted = warp_inclusive_sum(h_sorted, lane);
    const uint32_t total_rows = __shfl_sync(kFullMask, incl_sorted, 31);
    __syncwarp();
    const uint32_t rank = s_rank[wib][lane];
    const uint32_t row_first = __shfl_sync(kFullMask, incl_sorted - h_sorted, rank);
    if (has_rows) {
        RowGaussian st = G;
        st.row_first = row_first;
        s_gauss[wib][rank] = st;
    }
    __syncwarp();
    int prev = -1;
    for (uint32_t base = sub * 32u; base < total_rows; base += 32u << log_split) {
        const uint32_t rel = row_first - base;
        const uint32_t bits = __reduce_or_sync(kFullMask, (has_rows && rel < 32u) ? (1u << rel) : 0u);
        if (kSplit) prev = __popc(__ballot_sync(kFullMask, has_rows && row_first < base)) - 1;
        const int owner = prev + __popc(bits & upto_mask);
        prev += __popc(bits);
        const uint32_t r = base + lane;
        const bool valid = r < total_rows;
        const RowGaussian rg = s_gauss[wib][valid ? owner : 0];
        const uint32_t y = rg.y_min + (r - rg.row_first);
        walk_rows<kBlue, kHybrid, kMulti>(a, rng, valid, rg, y);
    }

    // queue overflow: the warp processes its kept large Gaussians, 32 rows at a time
    uint32_t pending = __ballot_sync(kFullMask, keep_big);
    while (pending) {
        const uint32_t src = __ffs(pending) - 1;
        pending &= pending - 1;
        const uint32_t bh = __shfl_sync(kFullMask, rect.height, src);
        __syncwarp();
        if (lane == src) s_gauss[wib][0] = G;
        __syncwarp();
        const RowGaussian bg = s_gauss[wib][0];
        for (uint32_t r0 = 0; r0 < bh; r0 += 32)
            walk_rows<kBlue, kHybrid, kMulti>(a, rng, r0 + lane < bh, bg, bg.y_min + r0 + lane);
    }
}

// Lists the queue's items in depth order (buckets of 1/32 octave). Every block sums the producers'
// histogram itself, counts its own slice of the entries per bucket in shared memory, takes each
// bucket's share with one atomic and places its items there.
// kGps: the entries of GPS hybrid scheduling (accumulate_gps.cu), when the list has room for all of them. Few
// Gaussians of many points are taken as they came: they hide little of one another, and gps_chunks_kernel, with twice
// the warps, draws faster (2033 Gaussians of 70 million points, 2560x1440: calls of 490 us, listed 540; 15,859 of 580
// million: 2140 us, listed 1330). Few points are listed, which spreads them over more warps.
template <bool kGps>
__global__ void __launch_bounds__(kOrderBlock) order_kernel(const AccumulateParams a) {
    constexpr uint32_t kPerThread = kDepthBuckets / kOrderBlock;
    __shared__ uint32_t s_first[kDepthBuckets], s_count[kDepthBuckets];
    __shared__ uint32_t s_warp[kOrderBlock / 32];
    wait_for_pass_before();
    if (!kGps && !dense_scene(a)) return;  // the producers have listed the items as they came
    const uint32_t n = kGps ? static_cast<uint32_t>(min(a.queue->packed >> kQueueEntryShift,
                                                        static_cast<unsigned long long>(min(a.max_binned, a.q.capacity))))
                            : min(a.queue->st_entries, a.stq.capacity);
    if (kGps && n < kFewEntries && (a.queue->packed & kQueueChunkMask) >= kManyChunks) {
        if (blockIdx.x == 0 && threadIdx.x == 0) a.queue->st_listed = kNotListed;
        return;
    }
    const uint32_t per_block = max(kOrderBlock, (n + gridDim.x - 1u) / gridDim.x);
    const uint32_t begin = min(blockIdx.x * per_block, n), end = min(begin + per_block, n);
    if (begin >= end) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t v[kPerThread], sum = 0;
#pragma unroll
    for (uint32_t i = 0; i < kPerThread; ++i) {
        v[i] = a.stq.histogram[threadIdx.x * kPerThread + i];
        sum += v[i];
        s_count[threadIdx.x * kPerThread + i] = 0u;
    }
    const uint32_t incl = warp_inclusive_sum(sum, lane);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t first = incl - sum;
    for (uint32_t w = 0; w < warp; ++w) first += s_warp[w];
#pragma unroll
    for (uint32_t i = 0; i < kPerThread; ++i) {
        s_first[threadIdx.x * kPerThread + i] = first;
        first += v[i];
    }
    __shared__ uint32_t s_total;
    if (threadIdx.x == kOrderBlock - 1u) s_total = first;
    __syncthreads();
    const bool fits = s_total <= a.stq.list_capacity;  // ST: always
    if (blockIdx.x == 0 && threadIdx.x == 0) a.queue->st_listed = fits ? s_total : kNotListed;
    if (!fits) return;
    const uint32_t scale = kGps ? 0u : part_scale(a, true);
    auto parts_of = [&](const uint32_t e, uint32_t& bucket) {
        if (kGps) {
            bucket = depth_bucket(static_cast<uint32_t>(a.q.key[e] >> 32));
            return gps_parts(a.q.count[e]).parts;
        }
        const RowGaussian* const G = queue_entry(a.stq, e);
        const uint32_t h = G->row_first;
        bucket = depth_bucket(G->key_hi);
        return h != 0 ? part_count(quad_rect(G->x_min, G->w, G->y_min, h), scale) : 0u;
    };
    for (uint32_t e = begin + threadIdx.x; e < end; e += kOrderBlock) {
        uint32_t bucket;
        const uint32_t parts = parts_of(e, bucket);
        atomicAdd(&s_count[bucket], parts);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < kPerThread; ++i) {
        const uint32_t bucket = threadIdx.x * kPerThread + i;
        if (s_count[bucket] != 0)
            s_first[bucket] += atomicAdd(a.stq.histogram + kDepthBuckets + bucket, s_count[bucket]);
    }
    __syncthreads();
    for (uint32_t e = begin + threadIdx.x; e < end; e += kOrderBlock) {
        uint32_t bucket;
        const uint32_t parts = parts_of(e, bucket);
        const uint32_t at = atomicAdd(&s_first[bucket], parts);
        for (uint32_t i = 0; i < parts; ++i) a.stq.list[at + i] = i << kItemEntryBits | e;
    }
}

// Persistent consumer of the queue, front to back: a warp takes some items at a time, lays their quads
// end to end and compares 32 quads of tile bounds at a time, one 16-byte load per lane; the tiles in
// front of their bounds are tested against the ellipse, one per lane, and those that remain are
// walked, the next tile's keys read ahead. Short queues are dealt out in pieces of items.
// Four blocks per SM spill up to 32 bytes where three would not: 500k training Gaussians, 800x800, 8 samples, 1142 us
// per call with four, 1161 with three; hybrid 400k heavy-tailed ones at 1279x719, one sample 436 and 466, 4 samples 1015
// and 970.
template <bool kBlue, bool kHybrid, bool kMulti>
__global__ void __launch_bounds__(kBlock, kQueueBlocksPerSM) st_queue_kernel(const AccumulateParams a) {
    __shared__ RowGaussian s_gauss[kWarpsPerBlock][32];
    __shared__ uint2 s_part[kWarpsPerBlock][32];     // first quad of the part, minus its place in the claim; quad columns
    __shared__ uint8_t s_tiles[kWarpsPerBlock][128];  // tiles in front of their bounds: lane << 2 | tile of its quad
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t upto_mask = kFullMask >> (31u - lane);
    wait_for_pass_before();
    const bool dense = dense_scene(a);
    const uint32_t n_items = dense ? a.queue->st_listed : min(a.queue->st_items, a.stq.list_capacity);
    if (n_items == 0) return;
    const FrameRng rng = frame_rng(a);
    const uint32_t n_warps = kWarpsPerBlock * gridDim.x;
    __shared__ uint32_t s_scale;  // not a register for all of the loop
    if (threadIdx.x == 0) s_scale = part_scale(a, dense);
    __syncthreads();
    if (!dense) {
        // row chunks as they came, each lane a segment of a row, without a look at the keys
        uint32_t c = blockIdx.x + wib * gridDim.x;
        while (c < n_items) {
            uint32_t next = 0;
            if (lane == 0) next = atomicAdd(&a.queue->next_chunk, 1u);
            const uint32_t item = a.stq.list[c];
            if (item != kNoItem) {
                const RowGaussian G = *queue_entry(a.stq, item & kItemEntryMask);
                const RowParts r = row_parts(G.w, G.row_first, s_scale);
                const uint32_t chunk = (item >> kItemEntryBits) * r.per_part;
                const uint32_t end = min(chunk + r.per_part, r.chunks);
                for (uint32_t k = chunk; k < end; ++k) {
                    const uint32_t row = (k << r.log_rows) + (lane & ((1u << r.log_rows) - 1u));
                    walk_rows<kBlue, kHybrid, kMulti>(a, rng, row < G.row_first, G, G.y_min + row, lane >> r.log_rows,
                                                      5u - r.log_rows);
                }
            }
            c = n_warps + __shfl_sync(kFullMask, next, 0);
        }
        return;
    }
    uint32_t log_split = 0;
    while (log_split < 4u && (n_items << log_split) < 4u * n_warps) ++log_split;
    const uint32_t n_parts = n_items << log_split;
    // The first claim is the warp's number; each next one is taken while the current is walked. Claims
    // grow with the depth taken: most of what lies there is culled, and long claims in front of the
    // queue would take items out of their order.
    uint32_t c0 = blockIdx.x + wib * gridDim.x, claim = 1;
    while (c0 < n_parts) {
        const uint32_t next_claim = log_split == 0 ? min(1u + c0 / n_warps, kMaxClaim) : 1u;
        uint32_t next = 0;
        if (lane == 0) next = atomicAdd(&a.queue->next_chunk, next_claim);
        const uint32_t item = lane < claim && c0 + lane < n_parts ? a.stq.list[(c0 + lane) >> log_split] : kNoItem;
        RowGaussian G;
        uint32_t quads = 0, first = 0, columns = 1;
        if (item != kNoItem) {
            G = *queue_entry(a.stq, item & kItemEntryMask);
            const QuadRect r = quad_rect(G.x_min, G.w, G.y_min, G.row_first);
            const uint32_t all = r.w * r.h, parts = part_count(r, s_scale);
            const uint32_t size = (all + parts - 1u) / parts;
            first = min((item >> kItemEntryBits) * size, all);
            quads = min(size, all - first);
            columns = r.w;
            // a short queue's items are dealt out in pieces
            const uint32_t piece = (quads + (1u << log_split) - 1u) >> log_split;
            const uint32_t skip = min(piece * ((c0 + lane) & ((1u << log_split) - 1u)), quads);
            first += skip;
            quads = min(piece, quads - skip);
        }
        const uint32_t incl = warp_inclusive_sum(quads, lane);
        const uint32_t start = incl - quads;
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        const uint32_t slot = __popc(__ballot_sync(kFullMask, quads != 0) & lt_mask);
        __syncwarp();
        if (quads != 0) {
            s_gauss[wib][slot] = G;
            s_part[wib][slot] = make_uint2(first - start, columns);
        }
        __syncwarp();
        int prev = -1;
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t rel = start - base;
            const uint32_t bits = __reduce_or_sync(kFullMask, (quads != 0 && rel < 32u) ? (1u << rel) : 0u);
            uint32_t owner = static_cast<uint32_t>(prev + __popc(bits & upto_mask));
            prev += __popc(bits);
            const bool valid = base + lane < total;
            if (!valid) owner = 0;
            const uint2 part = s_part[wib][owner];
            const uint32_t t = base + lane + part.x;
            const uint32_t row = t / part.y;
            const uint32_t x_min = s_gauss[wib][owner].x_min;
            const uint32_t qx = x_min / (4u * kBoundTile) + (t - row * part.y);
            const uint32_t ty = s_gauss[wib][owner].y_min / kBoundTile + row;
            uint32_t front = 0;
            if (valid) {
                const uint4 bound = __ldcg(reinterpret_cast<const uint4*>(
                    a.stq.tile_bound + static_cast<size_t>(ty) * a.stq.bound_pitch + 4u * qx));
                const uint32_t key_hi = s_gauss[wib][owner].key_hi;
                front = (bound.x >= key_hi ? 1u : 0u) | (bound.y >= key_hi ? 2u : 0u) | (bound.z >= key_hi ? 4u : 0u) |
                        (bound.w >= key_hi ? 8u : 0u);
                // the AABB's tiles of the quad
                const uint32_t lo = x_min / kBoundTile, hi = (x_min + s_gauss[wib][owner].w - 1u) / kBoundTile;
                if (lo > 4u * qx) front &= 0xfu << (lo - 4u * qx);
                if (hi < 4u * qx + 3u) front &= 0xfu >> (4u * qx + 3u - hi);
            }
            if (!__any_sync(kFullMask, front != 0)) continue;
            const uint32_t n_front = __popc(front);
            const uint32_t place = warp_inclusive_sum(n_front, lane);
            const uint32_t n_tiles = __shfl_sync(kFullMask, place, 31);
            uint8_t* at = s_tiles[wib] + (place - n_front);
            for (uint32_t i = 0; i < 4u; ++i)
                if (front & (1u << i)) *at++ = static_cast<uint8_t>(lane << 2 | i);
            __syncwarp();
            for (uint32_t j = 0; j < n_tiles; j += 32) {
                const uint32_t tile = s_tiles[wib][min(j + lane, n_tiles - 1u)];
                const uint32_t tx = 4u * __shfl_sync(kFullMask, qx, tile >> 2) + (tile & 3u);
                const uint32_t tyy = __shfl_sync(kFullMask, ty, tile >> 2);
                const uint32_t own = __shfl_sync(kFullMask, owner, tile >> 2);
                uint32_t todo =
                    __ballot_sync(kFullMask, j + lane < n_tiles && tile_on_ellipse(s_gauss[wib][own], tx, tyy));
                if (todo == 0) continue;
                uint32_t src = __ffs(todo) - 1;
                uint32_t wx = __shfl_sync(kFullMask, tx, src), wy = __shfl_sync(kFullMask, tyy, src);
                const size_t below = 4u * static_cast<size_t>(a.cam.width_int);
                TilePixels px = tile_pixels(a, wx, wy, lane);
                TileKeys keys = tile_keys(px, 0, below);
                for (;;) {
                    const uint32_t gauss = __shfl_sync(kFullMask, own, src);
                    todo &= todo - 1;
                    src = todo != 0 ? __ffs(todo) - 1 : src;
                    const uint32_t nx = __shfl_sync(kFullMask, tx, src), ny = __shfl_sync(kFullMask, tyy, src);
                    const TilePixels npx = tile_pixels(a, nx, ny, lane);
                    TileKeys ahead = keys;
                    if (todo != 0) ahead = tile_keys(npx, 0, below);
                    walk_tile<kBlue, kHybrid, kMulti>(a, rng, s_gauss[wib][gauss], wx, wy, lane, px, keys);
                    if (todo == 0) break;
                    px = npx;
                    wx = nx;
                    wy = ny;
                    keys = ahead;
                }
            }
            __syncwarp();
        }
        c0 = n_warps + __shfl_sync(kFullMask, next, 0);
        claim = next_claim;
    }
}

__device__ __forceinline__ void clear_keys(unsigned long long* __restrict__ fb, const size_t n_fb,
                                           WorkQueue* __restrict__ queue, const size_t tid, const size_t stride) {
    ulonglong2* fb2 = reinterpret_cast<ulonglong2*>(fb);
    const size_t n2 = n_fb / 2;
    for (size_t i = tid; i < n2; i += stride) fb2[i] = make_ulonglong2(kEmptyFragment, kEmptyFragment);
    if (tid == 0) {
        if (n_fb & 1) fb[n_fb - 1] = kEmptyFragment;
        if (queue != nullptr) {
            queue->packed = 0;
            queue->next_chunk = 0;
            queue->overflow = 0;
            queue->error = 0;
            queue->binned = 0;
            queue->st_entries = 0;
            queue->st_items = 0;
            queue->st_listed = 0;
        }
    }
}

__device__ __forceinline__ void clear_bounds(const StQueue& q, const size_t tid, const size_t stride) {
    for (size_t i = tid; i < static_cast<size_t>(q.bound_pitch) * q.tiles_y + q.n_blocks; i += stride)
        q.tile_bound[i] = 0xffffffffu;
    for (size_t i = tid; i < 2u * kDepthBuckets; i += stride) q.histogram[i] = 0u;
}

// q.tile_bound null: no tile bounds and no depth histogram.
__global__ void clear_kernel(unsigned long long* __restrict__ fb, const size_t n_fb, WorkQueue* __restrict__ queue,
                             const StQueue q) {
    wait_for_pass_before();
    const size_t tid = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    clear_keys(fb, n_fb, queue, tid, stride);
    if (q.tile_bound != nullptr) clear_bounds(q, tid, stride);
}

// The clear of a stochastic-transparency pass: also the tile bounds and the depth histogram, and, in
// the first kSampleBlocks blocks, the AABB pixels of one Gaussian per thread evenly over the scene, from
// which dense_scene tells how often the larger ones cover the framebuffer.
__global__ void __launch_bounds__(kBlock) st_clear_kernel(const AccumulateParams a, const size_t n_fb) {
    wait_for_pass_before();
    if (blockIdx.x < kSampleBlocks) {
        __shared__ float4 s_sum[kWarpsPerBlock];
        __shared__ uint32_t s_larger[kQueueSteps][kWarpsPerBlock];
        const uint32_t t = blockIdx.x * kBlock + threadIdx.x;
        const uint32_t step = max(a.n / (kSampleBlocks * kBlock), 1u);
        bool active = t < a.n;
        const uint32_t g = active ? t * step : a.n - 1u;
        // the projection loads the mean first and the rest after it; here their latency is all there is
        if (a.quant.records == nullptr && a.pre == nullptr) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.scales + 3 * g));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.rotations + g));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.opacities + g));
        }
        const bool points = a.stq.capacity == 0;  // of point splatting, which has no such queue
        const bool compact = !points || in_compact_group(a, g);
        Projected p;
        float pixels = 0.0f, larger = 0.0f, own = 0.0f, parts = 0.0f, chunks = 0.0f;
        if (project_gaussian(active, g, a.means, a.scales, a.rotations, a.opacities, a.w2c, a.cam, p, a.pre, a.quant) &&
            active) {
            const PixelRect rect = pixel_rect(p.bounds, a.cam);
            own = static_cast<float>(rect.width) * static_cast<float>(rect.height);
            // a faint Gaussian hides little of what lies behind it; the weight is 1 in the mean over scenes whose opacity
            // logits are N(0, 2^2)
            pixels = fminf(2.5f * p.opacity, 1.25f) *
                     fminf(own * static_cast<float>(step), kSampleMaxCover * a.cam.width * a.cam.height);
            larger = own > static_cast<float>(kDenseMinPixels) ? pixels : 0.0f;
            // what passes in depth order drop before it is drawn or queued: groups and Gaussians of few tiles (2.7M Gaussians
            // around the camera, 1600x900, 11,387 times covered, 15 times by these: 77 ms front to back, 16 as they lie)
            if (!compact || own > static_cast<float>(kMinPixels)) pixels = 0.0f;
            // a sampled Gaussian counts for at most 1/32 of the list
            const float most = static_cast<float>(a.stq.list_capacity) * 0.03125f;
            if (own > static_cast<float>(kDenseMinPixels))
                parts = fminf(static_cast<float>(part_count(quad_rect(rect.x_min, rect.width, rect.y_min, rect.height), 0u)) *
                                  static_cast<float>(step), most);
            if (own > static_cast<float>(kMinPixels))
                chunks = fminf(static_cast<float>(row_parts(rect.width, rect.height, 0u).parts) * static_cast<float>(step), most);
        }
        for (uint32_t o = 16; o > 0; o >>= 1) {
            pixels += __shfl_xor_sync(kFullMask, pixels, o);
            larger += __shfl_xor_sync(kFullMask, larger, o);
            parts += __shfl_xor_sync(kFullMask, parts, o);
            chunks += __shfl_xor_sync(kFullMask, chunks, o);
        }
        if ((threadIdx.x & 31u) == 0) s_sum[threadIdx.x >> 5] = make_float4(larger, pixels, parts, chunks);
        for (uint32_t i = 0; i < kQueueSteps; ++i) {
            const uint32_t above = __ballot_sync(kFullMask, own > static_cast<float>(kDenseMinPixels << i));
            if ((threadIdx.x & 31u) == 0) s_larger[i][threadIdx.x >> 5] = __popc(above);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t w = 1; w < kWarpsPerBlock; ++w) {
                larger += s_sum[w].x, pixels += s_sum[w].y;
                parts += s_sum[w].z, chunks += s_sum[w].w;
            }
            a.queue->parts[0][blockIdx.x] = parts;
            a.queue->parts[1][blockIdx.x] = chunks;
            a.queue->covered[blockIdx.x] = larger;
            a.queue->covered_all[blockIdx.x] = pixels;
            for (uint32_t i = 0; i < kQueueSteps; ++i) {
                uint32_t sum = 0;
                for (uint32_t w = 0; w < kWarpsPerBlock; ++w) sum += s_larger[i][w];
                a.queue->larger[i][blockIdx.x] = static_cast<float>(sum) * static_cast<float>(step);
            }
        }
        return;
    }
    uint32_t others = kSampleBlocks;
    if (a.groups.order != nullptr) {
        others += a.groups.slices;
        if (blockIdx.x < others) {
            sort_slice<kBlock>(a, blockIdx.x - kSampleBlocks);
            return;
        }
    }
    const size_t stride = static_cast<size_t>(gridDim.x - others) * kBlock;
    const size_t tid = static_cast<size_t>(blockIdx.x - others) * kBlock + threadIdx.x;
    clear_keys(a.framebuffer, n_fb, a.queue, tid, stride);
    clear_bounds(a.stq, tid, stride);
}

template <bool kBlue, bool kHybrid, bool kMulti>
cudaError_t launch_st(const AccumulateParams& p, const unsigned grid, const int num_sms, cudaStream_t stream) {
    cudaError_t err;
    if (p.groups.order != nullptr)
        err = launch_pass(st_scatter_kernel<kBlue, kHybrid, kMulti, kFrontToBack>, ordered_blocks(p.groups),
                          kOrderedWarps * 32u, p, stream);
    else if (p.stq.log_row_split != 0)
        err = launch_pass(st_scatter_kernel<kBlue, kHybrid, kMulti, kSplitRows>, grid, kBlock, p, stream);
    else
        err = launch_pass(st_scatter_kernel<kBlue, kHybrid, kMulti, kPlain>, grid, kBlock, p, stream);
    if (err == cudaSuccess && !isinf(p.stq.dense_pixels))
        err = launch_pass(order_kernel<false>, static_cast<unsigned>(num_sms), kOrderBlock, p, stream);
    if (err == cudaSuccess)
        err = launch_pass(st_queue_kernel<kBlue, kHybrid, kMulti>, static_cast<unsigned>(num_sms) * kQueueBlocksPerSM,
                          kBlock, p, stream);
    return err;
}

template <bool kMulti>
cudaError_t launch_st_variant(const AccumulateParams& p, const unsigned grid, const int num_sms, cudaStream_t stream) {
    const bool blue = p.blue_noise != nullptr;
    if (blue && p.hybrid) return launch_st<true, true, kMulti>(p, grid, num_sms, stream);
    if (blue) return launch_st<true, false, kMulti>(p, grid, num_sms, stream);
    if (p.hybrid) return launch_st<false, true, kMulti>(p, grid, num_sms, stream);
    return launch_st<false, false, kMulti>(p, grid, num_sms, stream);
}

}  // namespace

namespace {
unsigned clear_blocks(const size_t n_fb, const int num_sms) {
    const size_t need = (n_fb / 2 + kBlock - 1) / kBlock;
    const size_t cap = static_cast<size_t>(num_sms) * 16;
    return static_cast<unsigned>(need > cap ? cap : (need < 1 ? 1 : need));
}
}  // namespace

cudaError_t launch_clear(unsigned long long* framebuffer, const size_t n_fb, WorkQueue* queue, const StQueue& stq,
                         const int num_sms, cudaStream_t stream) {
    const size_t n = n_fb + static_cast<size_t>(stq.bound_pitch) * stq.tiles_y / 2;
    return launch_pass_with(0, clear_kernel, dim3(clear_blocks(n, num_sms)), kBlock, stream, framebuffer, n_fb, queue, stq);
}

cudaError_t launch_order_gps(const AccumulateParams& p, const int num_sms, cudaStream_t stream) {
    return launch_pass(order_kernel<true>, static_cast<unsigned>(num_sms), kOrderBlock, p, stream);
}

cudaError_t launch_clear_st(const AccumulateParams& p, const size_t n_fb, const int num_sms, cudaStream_t stream) {
    const unsigned others = kSampleBlocks + (p.groups.order != nullptr ? p.groups.slices : 0u);
    return launch_pass_with(0, st_clear_kernel, dim3(others + clear_blocks(n_fb, num_sms)), kBlock, stream, p, n_fb);
}

cudaError_t launch_accumulate_st(const AccumulateParams& p, const int num_sms, cudaStream_t stream) {
    if (p.n == 0) return cudaSuccess;
    const unsigned grid = (((p.n + 31u) / 32u << p.stq.log_row_split) + kWarpsPerBlock - 1u) / kWarpsPerBlock;
    return p.n_samples > 1 ? launch_st_variant<true>(p, grid, num_sms, stream)
                           : launch_st_variant<false>(p, grid, num_sms, stream);
}

}  // namespace sgs
