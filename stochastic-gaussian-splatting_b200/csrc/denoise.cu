// Learned resolve: a 6-layer 3x3 convolutional denoiser on BF16 tensor cores (tcgen05, FP32 in TMEM).
//
// The reference has no learned resolve; plain progressive averaging (resolve.cu, Static mode) is the
// fallback and the yardstick of its error. This file holds every kernel of the denoiser:
//   conv3x3_tma_kernel    implicit-GEMM 3x3 convolution, zero padding 1, stride 1, of BF16 inputs loaded
//                         by TMA. Forward layers (bias + ReLU, or bias + residual for the last layer) and
//                         data gradients (flipped, transposed weights; the ReLU mask of the layer below fused).
//   conv3x3_kernel        the first layer on FP16 features (sgs_conv3x3 alone; whole calls convert them first).
//   conv3x3_wgrad_tma_kernel weight and bias gradients of one layer with BF16 input, summed over all pixels.
//   conv3x3_wgrad_kernel  those of the first layer on FP16 features (sgs_conv3x3_wgrad alone).
//   train_*               one training step's weight packing, gradient staging and unpacking.
//   features_*            the 8-channel FP16 input built from the per-sample renders.
//
// Activations are NHWC BF16 [batch][height][width][channels], channels 16 or 32. A CTA
// computes an 8 x 16 pixel tile (M = 128) at a time: it stages the 10 x 18 input halo in
// shared memory as [8-channel chunk][halo pixel][8 channels], so that for every tap (dy, dx) the A
// operand is a K-major no-swizzle view of the halo starting (dy * 10 + dx) * 16 bytes in: the 8
// pixels of a tile row are 16 bytes apart (one core matrix), tile rows 160 bytes apart (SBO), the
// next 8 channels one chunk (2880 bytes) away (LBO). The weights of all 9 taps stay resident in
// shared memory as [tap][chunk][output channel][8] (K-major B). One elected thread issues the
// 9 * CIN / 16 MMAs (M 128, N COUT, K 16) into a 32-column TMEM accumulator and commits them to an
// mbarrier; all four warps then read their 32 TMEM lanes (= 32 pixels) back with tcgen05.ld and
// run the epilogue. Several CTAs share an SM (about 30 KB of shared memory each), so one CTA's
// halo loads overlap another's MMAs and epilogue.
//
// The weight gradient is a GEMM over pixels: dW[tap][co][ci] = sum_p dZ[p][co] * X[p + tap][ci].
// Per tile conv3x3_wgrad_kernel builds an im2col block in shared memory, [group][pixel][8], group =
// (tap, 8-channel chunk) plus one group whose first channel is 1 (its row of the product is the
// bias gradient), and multiplies it as an MN-major A (M = 128 rows of (tap, channel)) with the
// tile's output gradient as an MN-major B (N = COUT). Accumulators stay in TMEM across all the
// tiles a CTA handles and are added to the global gradient once at the end.
//
// Every wait on an mbarrier is bounded: when it runs out the kernel sets an error word (read by
// sgs_denoise_status), stops, waits once more with a bound, releases its TMEM and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "sgs_b200.h"
#include "sgs_internal.h"
#include "sgs_tcgen05.cuh"

namespace sgs {
namespace dn {

constexpr int kTileW = 8;
constexpr int kTileH = 16;
constexpr int kHaloW = kTileW + 2;
constexpr int kHaloH = kTileH + 2;
constexpr int kHaloPx = kHaloW * kHaloH;  // 180
constexpr int kTilePx = kTileW * kTileH;  // 128 = MMA M
constexpr int kThreads = 128;
constexpr uint32_t kWaitLimit = 1u << 20;

enum Epilogue { kEpiRelu = SGS_CONV_RELU, kEpiFinal = SGS_CONV_FINAL, kEpiMask = SGS_CONV_MASK };

__device__ unsigned int g_error;

struct ConvArgs {
    const void* in;
    void* out;
    const uint4* weights;
    const float* bias;
    const uint4* mask;
    const uint4* residual;
    int batch, height, width, tiles_x, tiles_y, n_tiles;
};

struct WgradArgs {
    const void* in;
    const uint4* grad_out;
    float* grad_w;
    float* grad_b;
    int batch, height, width, tiles_x, tiles_y, n_tiles;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t half2_to_bf162(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack_bf16(f.x, f.y);
}

__device__ __forceinline__ uint4 half8_to_bf16x8(uint4 v) {
    return make_uint4(half2_to_bf162(v.x), half2_to_bf162(v.y), half2_to_bf162(v.z), half2_to_bf162(v.w));
}

struct TileXY {
    int b, x0, y0;
};

__device__ __forceinline__ TileXY tile_xy(int t, int tiles_x, int tiles_y) {
    const int tx = t % tiles_x;
    const int rest = t / tiles_x;
    return {rest / tiles_y, tx * kTileW, (rest % tiles_y) * kTileH};
}

// Stages the 10 x 18 halo of the tile at (x0, y0) as [chunk][halo pixel][8] BF16, zero outside the
// image, from 8 FP16 channels per pixel; channels 8..15 are zero.
constexpr int kFeatureChannels = 16;  // as staged
__device__ __forceinline__ void load_halo(const void* in, uint4* halo, const TileXY& t, int height, int width) {
    const uint4* src = static_cast<const uint4*>(in);
    for (int p = threadIdx.x; p < kHaloPx; p += kThreads) {
        const int gx = t.x0 - 1 + p % kHaloW, gy = t.y0 - 1 + p / kHaloW;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (gx >= 0 && gx < width && gy >= 0 && gy < height)
            v = half8_to_bf16x8(__ldg(src + (static_cast<size_t>(t.b) * height + gy) * width + gx));
        halo[p] = v;
        halo[kHaloPx + p] = make_uint4(0u, 0u, 0u, 0u);
    }
}

template <int N>
__device__ __forceinline__ void load_accumulator(uint32_t taddr, float (&acc)[N]) {
    static_assert(N % 16 == 0, "16-column loads");
#pragma unroll
    for (int h = 0; h < N / 16; ++h) {
        float v[16];
        tc::tmem_ld16(taddr + 16 * h, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[16 * h + i] = v[i];
    }
    tc::tmem_wait_ld();
}

// Epilogue of one output pixel (thread m of the tile owns pixel m = 8 * row + column): bias and
// ReLU, bias and residual (final layer), or the ReLU mask of the layer below (data gradient).
// kPlanar: the BF16 output is stored as 8-channel planes [batch][channel / 8][y][x][8] (the layout of
// the denoiser's internal activations: a warp's store covers 128 contiguous bytes per tile row, and a
// halo box of one plane is a 160-byte run per row) instead of NHWC.
template <int COUT, int EPI, bool kPlanar = false>
__device__ __forceinline__ void store_pixel(const ConvArgs& a, const TileXY& tile, int m, const float (&acc)[COUT],
                                            const float (&bias)[COUT]) {
    const int x = tile.x0 + (m & 7), y = tile.y0 + (m >> 3);
    if (x >= a.width || y >= a.height) return;
    const size_t pixel = (static_cast<size_t>(tile.b) * a.height + y) * a.width + x;
    if constexpr (EPI == kEpiFinal) {
        const uint4 r = __ldg(a.residual + pixel);
        const float2 rg = __half22float2(*reinterpret_cast<const __half2*>(&r.x));
        const float2 bx = __half22float2(*reinterpret_cast<const __half2*>(&r.y));
        float* out = static_cast<float*>(a.out) + pixel * 3;
        out[0] = acc[0] + bias[0] + rg.x;
        out[1] = acc[1] + bias[1] + rg.y;
        out[2] = acc[2] + bias[2] + bx.x;
    } else {
        const size_t plane = static_cast<size_t>(a.height) * a.width;
        const size_t first = kPlanar ? (static_cast<size_t>(tile.b) * (COUT / 8) * plane + static_cast<size_t>(y) * a.width + x)
                                     : pixel * (COUT / 8);
        const size_t step = kPlanar ? plane : 1;
        uint4* out = static_cast<uint4*>(a.out) + first;
#pragma unroll
        for (int q = 0; q < COUT / 8; ++q) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = acc[8 * q + i] + bias[8 * q + i];
            if constexpr (EPI == kEpiRelu) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = fmaxf(v[i], 0.0f);
            } else {
                const uint4 mk = __ldg(a.mask + pixel * (COUT / 8) + q);
                const uint32_t mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!(bf16_lo(mw[i]) > 0.0f)) v[2 * i] = 0.0f;
                    if (!(bf16_hi(mw[i]) > 0.0f)) v[2 * i + 1] = 0.0f;
                }
            }
            out[q * step] = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                                       pack_bf16(v[6], v[7]));
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1) conv3x3_kernel(const ConvArgs a) {
    constexpr int COUT = 32;
    constexpr int KC = kFeatureChannels / 8;
    constexpr int kWeightVecs = 9 * KC * COUT;
    constexpr int kHaloVecs = KC * kHaloPx;
    constexpr uint32_t kIdesc = tc::instr_desc_bf16(kTilePx, COUT, false, false);

    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint4* w_s = reinterpret_cast<uint4*>(smem_raw);
    uint4* halo = w_s + kWeightVecs;
    uint64_t* bar_s = reinterpret_cast<uint64_t*>(halo + kHaloVecs);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar_s + 1);
    const int tid = threadIdx.x, warp = tid >> 5;

    for (int i = tid; i < kWeightVecs; i += kThreads) w_s[i] = __ldg(a.weights + i);
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(slot), 32);
    if (tid == 0) tc::mbar_init(tc::smem_u32(bar_s), 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    const uint32_t bar = tc::smem_u32(bar_s);
    const uint32_t halo_a = tc::smem_u32(halo);
    const uint32_t w_a = tc::smem_u32(w_s);

    float bias[COUT];
#pragma unroll
    for (int n = 0; n < COUT; ++n) bias[n] = __ldg(a.bias + n);

    uint32_t phase = 0;
    bool failed = false;
    for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x) {
        const TileXY tile = tile_xy(t, a.tiles_x, a.tiles_y);
        load_halo(a.in, halo, tile, a.height, a.width);
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
                for (int j = 0; j < KC / 2; ++j) {
                    const uint32_t a_addr = halo_a + ((2 * j) * kHaloPx + (tap / 3) * kHaloW + tap % 3) * 16;
                    const uint32_t b_addr = w_a + ((tap * KC + 2 * j) * COUT) * 16;
                    tc::mma_bf16(tmem, tc::smem_desc(a_addr, kHaloPx * 16, kHaloW * 16),
                                 tc::smem_desc(b_addr, COUT * 16, 128), kIdesc, (tap | j) != 0 ? 1u : 0u);
                }
            }
            tc::commit(bar);
        }
        __syncwarp();
        const bool ok = tc::mbar_wait(bar, phase, kWaitLimit);
        phase ^= 1u;
        __syncwarp();
        tc::fence_after_sync();
        float acc[COUT];
        load_accumulator<COUT>(tmem + (static_cast<uint32_t>(warp * 32) << 16), acc);

        if (ok) store_pixel<COUT, kEpiRelu>(a, tile, tid, acc, bias);
        tc::fence_before_sync();
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
    }
    if (failed) {
        if (tid == 0) atomicExch(&g_error, 1u);
        tc::mbar_wait(bar, phase ^ 1u, kWaitLimit);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 32);
    }
}

// Warp-specialised variant for BF16 inputs, persistent over tiles. Warp 4 (one lane) loads each
// tile's halo with TMA, one 8 x 10 x 18 box per 8-channel chunk of a 4-D tensor map over the NHWC
// input (zero fill outside the image), into a ring of kStages halo slots; warp 5 (one lane) issues
// the tile's MMAs into one of two TMEM accumulators and commits them to the slot's "empty" and the
// accumulator's "full" barrier; warps 0-3 drain the accumulator (tcgen05.ld), release it and run
// the epilogue while the next tile's loads and MMAs are in flight.
constexpr int kStages = 3;
constexpr int kTmaThreads = 192;
constexpr int kTmaCols = 64;  // two 32-column accumulators

template <int CIN, int COUT>
struct TmaConv {
    static constexpr int KC = CIN / 8;
    static constexpr int kWeightVecs = 9 * KC * COUT;
    // TMA destinations start on 128-byte boundaries: chunks 184 pixels (2944 bytes) apart
    static constexpr int kChunkPx = 184;
    static constexpr int kHaloVecs = KC * kChunkPx;
    static constexpr uint32_t kHaloBytes = kHaloVecs * 16;
    static constexpr uint32_t kTxBytes = KC * kHaloPx * 16;  // bytes the KC boxes deliver
    static constexpr int kBars = 2 * kStages + 4;
    static constexpr size_t kSmem =
        static_cast<size_t>(kWeightVecs + kStages * kHaloVecs) * 16 + kBars * 8 + 16 + 128;
    static_assert((kChunkPx * 16) % 128 == 0 && (kWeightVecs * 16) % 128 == 0, "128-byte TMA destinations");
};

// kPlanarIn, kPlanar: input, BF16 output in the 8-channel-plane layout of store_pixel (the input's tensor map is then
// over [batch][plane][y][x * 8 + channel] and a chunk's halo is one box of 10 x 18 pixels).
// Held to 4 CTAs per SM (80 registers, no spills): 0.357 against 0.365 ms per 1080p denoiser call at
// the 3 that 90 registers allow.
template <int CIN, int COUT, int EPI, bool kPlanarIn, bool kPlanar>
__global__ void __launch_bounds__(kTmaThreads, 4) conv3x3_tma_kernel(const __grid_constant__ CUtensorMap in_map,
                                                                  const ConvArgs a) {
    using S = TmaConv<CIN, COUT>;
    constexpr uint32_t kIdesc = tc::instr_desc_bf16(kTilePx, COUT, false, false);
    static_assert(COUT <= kTmaCols / 2, "two accumulators");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint4* w_s = reinterpret_cast<uint4*>(smem_raw + ((128u - (tc::smem_u32(smem_raw) & 127u)) & 127u));
    uint4* halo = w_s + S::kWeightVecs;
    uint64_t* bars = reinterpret_cast<uint64_t*>(halo + kStages * S::kHaloVecs);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + S::kBars);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // barriers: full[s], empty[s] (halo slots), acc_full[k], acc_empty[k] (accumulators)
    const uint32_t bar0 = tc::smem_u32(bars);
#define SGS_FULL(st) (bar0 + 8u * (st))
#define SGS_EMPTY(st) (bar0 + 8u * (kStages + (st)))
#define SGS_ACC_FULL(k) (bar0 + 8u * (2 * kStages + (k)))
#define SGS_ACC_EMPTY(k) (bar0 + 8u * (2 * kStages + 2 + (k)))

    for (int i = tid; i < S::kWeightVecs; i += kTmaThreads) w_s[i] = __ldg(a.weights + i);
    tc::fence_async_smem();
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(slot), kTmaCols);
    if (tid == 0) {
        for (int st = 0; st < kStages; ++st) {
            tc::mbar_init(SGS_FULL(st), 1);
            tc::mbar_init(SGS_EMPTY(st), 1);
        }
        for (int k = 0; k < 2; ++k) {
            tc::mbar_init(SGS_ACC_FULL(k), 1);
            tc::mbar_init(SGS_ACC_EMPTY(k), 4);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // everything above reads only the weights, which are older than the kernel before
    wait_for_pass_before();
    tc::launch_dependents();
    const uint32_t tmem = *slot;
    const uint32_t halo_a = tc::smem_u32(halo);
    const uint32_t w_a = tc::smem_u32(w_s);
    bool failed = false;
    int issued = 0;  // producer: tiles whose loads were issued; MMA: tiles whose MMAs were committed

    if (warp == 4) {
        if (lane == 0) {
            for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++issued) {
                const int st = issued % kStages;
                const uint32_t ph = (issued / kStages) & 1u;
                if (issued >= kStages && !tc::mbar_wait(SGS_EMPTY(st), ph ^ 1u, kWaitLimit)) {
                    failed = true;
                    break;
                }
                const TileXY tile = tile_xy(t, a.tiles_x, a.tiles_y);
                tc::mbar_arrive_expect_tx(SGS_FULL(st), S::kTxBytes);
#pragma unroll
                for (int c = 0; c < S::KC; ++c) {
                    const uint32_t dst = halo_a + (st * S::kHaloVecs + c * S::kChunkPx) * 16;
                    if constexpr (kPlanarIn)  // x in elements: 8 per pixel, so always a 16-byte multiple
                        tc::tma_load_4d(dst, &in_map, SGS_FULL(st), (tile.x0 - 1) * 8, tile.y0 - 1, c, tile.b);
                    else
                        tc::tma_load_4d(dst, &in_map, SGS_FULL(st), c * 8, tile.x0 - 1, tile.y0 - 1, tile.b);
                }
            }
        }
    } else if (warp == 5) {
        if (lane == 0) {
            for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++issued) {
                const int st = issued % kStages, k = issued & 1;
                const uint32_t ph = (issued / kStages) & 1u, aph = (issued >> 1) & 1u;
                if (!tc::mbar_wait(SGS_FULL(st), ph, kWaitLimit) ||
                    (issued >= 2 && !tc::mbar_wait(SGS_ACC_EMPTY(k), aph ^ 1u, kWaitLimit))) {
                    failed = true;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t h = halo_a + st * S::kHaloBytes;
#pragma unroll
                for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
                    for (int j = 0; j < S::KC / 2; ++j) {
                        const uint32_t a_addr = h + ((2 * j) * S::kChunkPx + (tap / 3) * kHaloW + tap % 3) * 16;
                        const uint32_t b_addr = w_a + ((tap * S::KC + 2 * j) * COUT) * 16;
                        tc::mma_bf16(tmem + k * (kTmaCols / 2), tc::smem_desc(a_addr, S::kChunkPx * 16, kHaloW * 16),
                                     tc::smem_desc(b_addr, COUT * 16, 128), kIdesc, (tap | j) != 0 ? 1u : 0u);
                    }
                }
                tc::commit(SGS_EMPTY(st));
                tc::commit(SGS_ACC_FULL(k));
            }
        }
    } else {
        float bias[COUT];
#pragma unroll
        for (int n = 0; n < COUT; ++n) bias[n] = (EPI == kEpiMask) ? 0.0f : __ldg(a.bias + n);
        int i = 0;
        for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++i) {
            const int k = i & 1;
            const bool ok = __all_sync(0xFFFFFFFFu, tc::mbar_wait(SGS_ACC_FULL(k), (i >> 1) & 1u, kWaitLimit));
            if (!ok) {
                failed = true;
                break;
            }
            tc::fence_after_sync();
            float acc[COUT];
            load_accumulator<COUT>(tmem + (static_cast<uint32_t>(warp * 32) << 16) + k * (kTmaCols / 2), acc);
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(SGS_ACC_EMPTY(k));
            store_pixel<COUT, EPI, kPlanar>(a, tile_xy(t, a.tiles_x, a.tiles_y), tid, acc, bias);
        }
    }

    if (__syncthreads_or(failed)) {
        if (tid == 0) atomicExch(&g_error, 1u);
        // let this CTA's own copies and MMAs in flight finish (bounded) before its memory goes away
        if (warp == 4 && lane == 0)
            for (int q = issued - 1; q >= 0 && q >= issued - kStages; --q)
                tc::mbar_wait(SGS_FULL(q % kStages), (q / kStages) & 1u, kWaitLimit);
        if (warp == 5 && lane == 0 && issued > 0)
            tc::mbar_wait(SGS_ACC_FULL((issued - 1) & 1), ((issued - 1) >> 1) & 1u, kWaitLimit);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kTmaCols);
    }
#undef SGS_FULL
#undef SGS_EMPTY
#undef SGS_ACC_FULL
#undef SGS_ACC_EMPTY
}

// Weight-gradient geometry of the FP16 features: im2col groups of 8 rows, (tap, chunk) for tap-major order,
// then the bias group, then a zero group. M-tile m reads groups start(m) .. start(m) + 15 and owns (adds to
// the gradient) groups [own(m), own(m + 1)).
struct Wgrad {
    static constexpr int COUT = 32;
    static constexpr int KC = kFeatureChannels / 8;
    static constexpr int KCO = COUT / 8;
    static constexpr int kConvGroups = 9 * KC;
    static constexpr int kBiasGroup = kConvGroups;
    static constexpr int kMTiles = 2;
    static constexpr int kGroups = 20;
    static constexpr int kCols = kMTiles * COUT;
    static constexpr int kHaloVecs = KC * kHaloPx;
    static constexpr int kGradVecs = KCO * kTilePx;
    static constexpr int kColVecs = kGroups * kTilePx;
    static constexpr size_t kSmem = static_cast<size_t>(kHaloVecs + kGradVecs + kColVecs) * 16 + 16;
    static constexpr int kSecond = kGroups - 16;
    __host__ __device__ static constexpr int start(int m) { return m * kSecond; }
    __host__ __device__ static constexpr int own(int m) { return m == 0 ? 0 : m == kMTiles ? kGroups : 16 * m; }
    static_assert(kBiasGroup < kGroups, "bias group allocated");
    static_assert(kCols == 64, "a power of two of TMEM columns");
};

__global__ void __launch_bounds__(kThreads) conv3x3_wgrad_kernel(const WgradArgs a) {
    using G = Wgrad;
    constexpr int CIN = kFeatureChannels, COUT = G::COUT;
    constexpr uint32_t kIdesc = tc::instr_desc_bf16(kTilePx, COUT, true, true);
    constexpr uint32_t kGroupBytes = kTilePx * 16;  // 2048

    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint4* halo = reinterpret_cast<uint4*>(smem_raw);
    uint4* grad_s = halo + G::kHaloVecs;
    uint4* col = grad_s + G::kGradVecs;
    uint64_t* bar_s = reinterpret_cast<uint64_t*>(col + G::kColVecs);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar_s + 1);
    const int tid = threadIdx.x, warp = tid >> 5;

    // constant groups: the bias group (first channel 1.0 for every pixel) and the zero padding
    for (int i = G::kBiasGroup * kTilePx + tid; i < G::kColVecs; i += kThreads)
        col[i] = make_uint4(i < (G::kBiasGroup + 1) * kTilePx ? 0x3F80u : 0u, 0u, 0u, 0u);
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(slot), G::kCols);
    if (tid == 0) tc::mbar_init(tc::smem_u32(bar_s), 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    const uint32_t bar = tc::smem_u32(bar_s);
    const uint32_t col_a = tc::smem_u32(col);
    const uint32_t grad_a = tc::smem_u32(grad_s);

    uint32_t phase = 0;
    bool failed = false;
    bool first = true;
    for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x) {
        const TileXY tile = tile_xy(t, a.tiles_x, a.tiles_y);
        load_halo(a.in, halo, tile, a.height, a.width);
        for (int i = tid; i < G::kGradVecs; i += kThreads) {
            const int k = i / G::KCO, c = i % G::KCO;
            const int x = tile.x0 + (k & 7), y = tile.y0 + (k >> 3);
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (x < a.width && y < a.height)
                v = __ldg(a.grad_out + ((static_cast<size_t>(tile.b) * a.height + y) * a.width + x) * G::KCO + c);
            grad_s[c * kTilePx + k] = v;
        }
        __syncthreads();
        for (int i = tid; i < G::kConvGroups * kTilePx; i += kThreads) {
            const int g = i >> 7, k = i & 127;
            const int tap = g / G::KC, c = g % G::KC;
            col[i] = halo[c * kHaloPx + ((k >> 3) + tap / 3) * kHaloW + (k & 7) + tap % 3];
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int m = 0; m < G::kMTiles; ++m) {
#pragma unroll
                for (int kk = 0; kk < kTilePx / 16; ++kk) {
                    const uint64_t ad = tc::smem_desc(col_a + G::start(m) * kGroupBytes + kk * 256, 128, kGroupBytes);
                    const uint64_t bd = tc::smem_desc(grad_a + kk * 256, 128, kGroupBytes);
                    tc::mma_bf16(tmem + m * COUT, ad, bd, kIdesc, (first && kk == 0) ? 0u : 1u);
                }
            }
            tc::commit(bar);
        }
        first = false;
        __syncwarp();
        const bool ok = tc::mbar_wait(bar, phase, kWaitLimit);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
    }
    if (failed) {
        if (tid == 0) atomicExch(&g_error, 1u);
        tc::mbar_wait(bar, phase ^ 1u, kWaitLimit);
    } else if (!first) {
        __syncwarp();
        tc::fence_after_sync();
#pragma unroll
        for (int m = 0; m < G::kMTiles; ++m) {
            float acc[COUT];
            load_accumulator<COUT>(tmem + (static_cast<uint32_t>(warp * 32) << 16) + m * COUT, acc);
            const int g = G::start(m) + (tid >> 3), ch = tid & 7;
            if (g >= G::own(m) && g < G::own(m + 1)) {
                if (g < G::kConvGroups) {
                    const int tap = g / G::KC, ci = (g % G::KC) * 8 + ch;
#pragma unroll
                    for (int n = 0; n < COUT; ++n) atomicAdd(a.grad_w + (tap * COUT + n) * CIN + ci, acc[n]);
                } else if (g == G::kBiasGroup && ch == 0) {
#pragma unroll
                    for (int n = 0; n < COUT; ++n) atomicAdd(a.grad_b + n, acc[n]);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, G::kCols);
    }
}

// Weight and bias gradients of a layer with BF16 input, persistent and warp-specialised. Warp 4 loads,
// per tile, the input halo with TMA three times, shifted by the taps' dx (one box of 8 channels x 8 x 18
// pixels each, zero fill outside the image), and the tile's output gradient; warp 5 multiplies them,
// pixels as K. A row of 8 pixels is one core matrix, so the taps' dy are row offsets, and one MMA of
// M = 128 holds the rows (dx, input channel) of one dy, then the bias row (a constant group of ones)
// and rows that nothing reads. No im2col copy: with it a tile took 7.9 us, loads, copies and MMAs in
// turn (55 us per 16 x 128 x 128 layer). The accumulators stay in TMEM over all of a CTA's tiles.
template <int CIN, int COUT>
struct WgradTma {
    static constexpr int KC = CIN / 8;
    static constexpr int KCO = COUT / 8;
    static constexpr int kStages = 4;
    static constexpr uint32_t kGroup = kTileW * kHaloH * 16;  // one 8-channel group of a shifted halo
    static constexpr int kOnes = 3 * KC;                      // the group after the three shifts
    static constexpr uint32_t kGradOffset = (kOnes + 1) * kGroup;
    static constexpr uint32_t kGradGroup = kTilePx * 16;
    static constexpr uint32_t kStage = kGradOffset + KCO * kGradGroup;
    static constexpr uint32_t kTxBytes = kOnes * kGroup + KCO * kGradGroup;
    // the rows that nothing reads lie in 16 groups from a stage's start, at most 16 tile rows further
    static constexpr uint32_t kReach = 15 * kGroup + 18 * kTileW * 16;
    static constexpr uint32_t kPad = kReach > kStage ? kReach - kStage : 0;
    static constexpr int kCols = 3 * COUT <= 64 ? 64 : 128;
    static constexpr int kBars = 2 * kStages + 1;
    static constexpr size_t kSmem = static_cast<size_t>(kStages) * kStage + kPad + kBars * 8 + 16 + 128;
    static_assert(kGroup % 128 == 0 && kGradOffset % 128 == 0 && kStage % 128 == 0, "128-byte TMA destinations");
    static_assert(kOnes < 16, "the bias group is a row group of the MMA");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kTmaThreads) conv3x3_wgrad_tma_kernel(const __grid_constant__ CUtensorMap in_map,
                                                                       const __grid_constant__ CUtensorMap grad_map,
                                                                       const WgradArgs a) {
    using G = WgradTma<CIN, COUT>;
    constexpr uint32_t kIdesc = tc::instr_desc_bf16(kTilePx, COUT, true, true);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* const base = smem_raw + ((128u - (tc::smem_u32(smem_raw) & 127u)) & 127u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + G::kStages * G::kStage + G::kPad);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + G::kBars);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar0 = tc::smem_u32(bars);
    const uint32_t done = bar0 + 8u * (2 * G::kStages);
#define SGS_FULL(st) (bar0 + 8u * (st))
#define SGS_EMPTY(st) (bar0 + 8u * (G::kStages + (st)))
    for (int st = 0; st < G::kStages; ++st)
        for (uint32_t i = tid; i < G::kGroup / 16; i += kTmaThreads)
            reinterpret_cast<uint4*>(base + st * G::kStage + G::kOnes * G::kGroup)[i] = make_uint4(0x3F80u, 0u, 0u, 0u);
    tc::fence_async_smem();
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(slot), G::kCols);
    if (tid == 0)
        for (int i = 0; i < G::kBars; ++i) tc::mbar_init(bar0 + 8u * i, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    // everything above touches nothing but shared memory and TMEM; the layer's data gradient, launched behind this
    // kernel, may load its weights and set up from here on
    wait_for_pass_before();
    tc::launch_dependents();
    const uint32_t tmem = *slot;
    const uint32_t smem0 = tc::smem_u32(base);
    bool failed = false;
    int issued = 0;  // producer: tiles whose loads were issued; MMA: tiles whose MMAs were committed

    if (warp == 4) {
        if (lane == 0) {
            for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++issued) {
                const int st = issued % G::kStages;
                if (issued >= G::kStages &&
                    !tc::mbar_wait(SGS_EMPTY(st), ((issued / G::kStages) & 1u) ^ 1u, kWaitLimit)) {
                    failed = true;
                    break;
                }
                const TileXY tile = tile_xy(t, a.tiles_x, a.tiles_y);
                const uint32_t dst = smem0 + st * G::kStage;
                tc::mbar_arrive_expect_tx(SGS_FULL(st), G::kTxBytes);
#pragma unroll
                for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                    for (int c = 0; c < G::KC; ++c)
                        tc::tma_load_4d(dst + (dx * G::KC + c) * G::kGroup, &in_map, SGS_FULL(st), c * 8,
                                        tile.x0 - 1 + dx, tile.y0 - 1, tile.b);
#pragma unroll
                for (int c = 0; c < G::KCO; ++c)
                    tc::tma_load_4d(dst + G::kGradOffset + c * G::kGradGroup, &grad_map, SGS_FULL(st), c * 8, tile.x0,
                                    tile.y0, tile.b);
            }
        }
    } else if (warp == 5) {
        if (lane == 0) {
            for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++issued) {
                const int st = issued % G::kStages;
                if (!tc::mbar_wait(SGS_FULL(st), (issued / G::kStages) & 1u, kWaitLimit)) {
                    failed = true;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t in = smem0 + st * G::kStage, grad = in + G::kGradOffset;
#pragma unroll
                for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                    for (int kk = 0; kk < kTilePx / 16; ++kk)
                        tc::mma_bf16(tmem + dy * COUT, tc::smem_desc(in + (dy + 2 * kk) * (kTileW * 16), 128, G::kGroup),
                                     tc::smem_desc(grad + kk * 256, 128, G::kGradGroup), kIdesc,
                                     (issued | kk) != 0 ? 1u : 0u);
                tc::commit(SGS_EMPTY(st));
            }
            if (!failed) tc::commit(done);
        }
    } else {
        // the CTA's sums, once its last tile's MMAs are through
        const uint32_t tiles = (a.n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;  // one wait's limit for each
        const bool ok = __all_sync(0xFFFFFFFFu, tc::mbar_wait(done, 0, kWaitLimit * min(tiles, 4000u)));
        failed = !ok;
        if (ok) {
            tc::fence_after_sync();
            const int group = tid >> 3, ch = tid & 7;
#pragma unroll
            for (int dy = 0; dy < 3; ++dy) {
                float acc[COUT];
                load_accumulator<COUT>(tmem + (static_cast<uint32_t>(warp * 32) << 16) + dy * COUT, acc);
                if (group < G::kOnes) {
                    const int tap = dy * 3 + group / G::KC, ci = group % G::KC * 8 + ch;
#pragma unroll
                    for (int n = 0; n < COUT; ++n) atomicAdd(a.grad_w + (tap * COUT + n) * CIN + ci, acc[n]);
                } else if (group == G::kOnes && ch == 0 && dy == 0) {
#pragma unroll
                    for (int n = 0; n < COUT; ++n) atomicAdd(a.grad_b + n, acc[n]);
                }
            }
        }
    }
    if (__syncthreads_or(failed)) {
        if (tid == 0) atomicExch(&g_error, 1u);
        // let this CTA's own copies and MMAs in flight finish (bounded) before its memory goes away
        if (warp == 4 && lane == 0)
            for (int q = issued - 1; q >= 0 && q >= issued - G::kStages; --q)
                tc::mbar_wait(SGS_FULL(q % G::kStages), (q / G::kStages) & 1u, kWaitLimit);
        if (warp == 5 && lane == 0 && issued > 0)
            tc::mbar_wait(SGS_EMPTY((issued - 1) % G::kStages), ((issued - 1) / G::kStages) & 1u, kWaitLimit);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, G::kCols);
    }
#undef SGS_FULL
#undef SGS_EMPTY
}

// FP16 features as BF16, so that the first layer's halo comes by TMA like the others' (64 to 41 us for both
// kernels per 1080p frame).
__global__ void __launch_bounds__(256) features_bf16_kernel(const uint4* __restrict__ features,
                                                            uint4* __restrict__ out, const uint32_t n_px) {
    wait_for_pass_before();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i < n_px) out[i] = half8_to_bf16x8(__ldg(features + i));
}

// ---- training step: packing, staging, unpacking ------------------------------------------------

constexpr int kTrainLayers = SGS_DENOISE_LAYERS;
__host__ __device__ constexpr int model_in(int l) { return l == 0 ? 7 : 32; }
__host__ __device__ constexpr int model_out(int l) { return l == kTrainLayers - 1 ? 3 : 32; }
__host__ __device__ constexpr int staged_in(int l) { return l == 0 ? 16 : 32; }
__host__ __device__ constexpr int staged_out(int l) { return l == kTrainLayers - 1 ? 16 : 32; }
// elements of the forward weights, of the weight-gradient sums (8 input channels in the first layer) and
// of the parameters before layer l
__host__ __device__ constexpr int packed_before(int l) {
    int n = 0;
    for (int i = 0; i < l; ++i) n += 9 * staged_in(i) * staged_out(i);
    return n;
}
__host__ __device__ constexpr int sums_before(int l) {
    int n = 0;
    for (int i = 0; i < l; ++i) n += 9 * (i == 0 ? 8 : 32) * staged_out(i);
    return n;
}
__host__ __device__ constexpr int params_before(int l) {
    int n = 0;
    for (int i = 0; i < l; ++i) n += (9 * model_in(i) + 1) * model_out(i);
    return n;
}
__host__ __device__ constexpr int bias_before(int l) { return 32 * l; }
constexpr int kPacked = packed_before(kTrainLayers), kSums = sums_before(kTrainLayers);
constexpr int kParams = params_before(kTrainLayers), kBiases = 32 * (kTrainLayers - 1) + 16;

struct TrainParams {
    const float* weights[kTrainLayers];  // W[co][ci][3][3]
    const float* biases[kTrainLayers];
};

// Forward weights of all layers as BF16 [tap][ci / 8][co][ci % 8] and FP32 biases, zero-padded to the staged
// channels, and (the blocks behind them) the FP16 features as BF16.
constexpr int kPackBlocks = (kPacked + kBiases + 255) / 256;
__global__ void __launch_bounds__(256) train_pack_kernel(const TrainParams p, __nv_bfloat16* __restrict__ weights,
                                                         float* __restrict__ biases, const uint4* __restrict__ features,
                                                         uint4* __restrict__ features_bf16, const uint32_t n_px) {
    wait_for_pass_before();
    if (blockIdx.x >= kPackBlocks) {
        const uint32_t i = (blockIdx.x - kPackBlocks) * 256u + threadIdx.x;
        if (i < n_px) features_bf16[i] = half8_to_bf16x8(__ldg(features + i));
        return;
    }
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < kPacked) {
        int l = 0;
        while (l + 1 < kTrainLayers && i >= packed_before(l + 1)) ++l;
        const int si = staged_in(l), so = staged_out(l), mi = model_in(l), mo = model_out(l);
        const int r = i - packed_before(l);
        const int ci = r / (so * 8) % (si / 8) * 8 + r % 8, co = r / 8 % so, tap = r / (si * so);
        weights[i] = __float2bfloat16_rn(ci < mi && co < mo ? p.weights[l][(co * mi + ci) * 9 + tap] : 0.0f);
    } else if (i < kPacked + kBiases) {
        const int r = i - kPacked, l = r / 32;
        biases[r] = r % 32 < model_out(l) ? p.biases[l][r % 32] : 0.0f;
    }
}

// Data-gradient weights of the layers above the first, BF16 [tap][co / 8][ci][co % 8] = W[co][ci][8 - tap], and
// (the blocks behind them) the output gradient as BF16 with 16 channels.
constexpr int kDgradBlocks = (kPacked - packed_before(1) + 255) / 256;
__global__ void __launch_bounds__(256) train_stage_kernel(const TrainParams p, __nv_bfloat16* __restrict__ weights,
                                                          const float* __restrict__ grad, uint4* __restrict__ staged,
                                                          const uint32_t n_px) {
    wait_for_pass_before();
    if (blockIdx.x >= kDgradBlocks) {
        const uint32_t i = (blockIdx.x - kDgradBlocks) * 256u + threadIdx.x;
        if (i >= n_px) return;
        const float* const g = grad + 3 * static_cast<size_t>(i);
        staged[2 * static_cast<size_t>(i)] = make_uint4(pack_bf16(g[0], g[1]), pack_bf16(g[2], 0.0f), 0u, 0u);
        staged[2 * static_cast<size_t>(i) + 1] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    const int i = packed_before(1) + blockIdx.x * 256 + threadIdx.x;
    if (i >= kPacked) return;
    int l = 1;
    while (l + 1 < kTrainLayers && i >= packed_before(l + 1)) ++l;
    const int si = staged_in(l), so = staged_out(l), mi = model_in(l), mo = model_out(l);
    const int r = i - packed_before(l);
    const int co = r / (si * 8) % (so / 8) * 8 + r % 8, ci = r / 8 % si, tap = r / (si * so);
    weights[i - packed_before(1)] =
        __float2bfloat16_rn(ci < mi && co < mo ? p.weights[l][(co * mi + ci) * 9 + 8 - tap] : 0.0f);
}

// Parameter gradients W1[co][ci][3][3], b1, ..., back to back from the sums [tap][co][ci] and bias sums.
__global__ void __launch_bounds__(256) train_unpack_kernel(const float* __restrict__ sums, float* __restrict__ grads) {
    wait_for_pass_before();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= kParams) return;
    int l = 0;
    while (l + 1 < kTrainLayers && i >= params_before(l + 1)) ++l;
    const int mi = model_in(l), mo = model_out(l), so = staged_out(l), si = l == 0 ? 8 : 32;
    const int r = i - params_before(l);
    if (r < 9 * mi * mo) {
        const int tap = r % 9, ci = r / 9 % mi, co = r / (9 * mi);
        grads[i] = sums[sums_before(l) + (tap * so + co) * si + ci];
    } else {
        grads[i] = sums[kSums + bias_before(l) + (r - 9 * mi * mo)];
    }
}

// ---- input features -----------------------------------------------------------------------

// accum per pixel: float4 (sum r, sum g, sum b, sum alpha), float4 (sum depth, sum lum^2,
// winner changes, last winner index bits).
__global__ void features_accumulate_kernel(const float* __restrict__ image, const float* __restrict__ alpha,
                                           const float* __restrict__ depth,
                                           const unsigned long long* __restrict__ framebuffer,
                                           float4* __restrict__ accum, uint32_t n_px, int first) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_px) return;
    const float r = image[3 * i], g = image[3 * i + 1], b = image[3 * i + 2];
    const float al = alpha[i], d = depth[i];
    const float lum = 0.2126f * r + 0.7152f * g + 0.0722f * b;
    const uint32_t idx = framebuffer != nullptr ? static_cast<uint32_t>(framebuffer[i]) : 0xFFFFFFFFu;
    float4 s0 = make_float4(r, g, b, al);
    float4 s1 = make_float4(d, lum * lum, 0.0f, __uint_as_float(idx));
    if (!first) {
        const float4 p0 = accum[2 * i], p1 = accum[2 * i + 1];
        s0 = make_float4(p0.x + r, p0.y + g, p0.z + b, p0.w + al);
        s1 = make_float4(p1.x + d, p1.y + lum * lum, p1.z + (__float_as_uint(p1.w) != idx ? 1.0f : 0.0f), s1.w);
    }
    accum[2 * i] = s0;
    accum[2 * i + 1] = s1;
}

// features per pixel, FP16: mean r, g, b, mean alpha, mean depth * depth_scale, standard error of
// the mean luminance, fraction of consecutive samples whose winner changed, 0.
__global__ void features_finalize_kernel(const float4* __restrict__ accum, uint4* __restrict__ features,
                                         uint32_t n_px, uint32_t n_samples, float depth_scale) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_px) return;
    const float inv = 1.0f / static_cast<float>(n_samples);
    const float4 s0 = accum[2 * i], s1 = accum[2 * i + 1];
    const float r = s0.x * inv, g = s0.y * inv, b = s0.z * inv;
    const float lum = 0.2126f * r + 0.7152f * g + 0.0722f * b;
    const float var = fmaxf(s1.y * inv - lum * lum, 0.0f);
    const float se = sqrtf(var * inv);
    const float change = s1.z / static_cast<float>(n_samples > 1 ? n_samples - 1 : 1);
    const __half2 h0 = __floats2half2_rn(r, g), h1 = __floats2half2_rn(b, s0.w * inv);
    const __half2 h2 = __floats2half2_rn(s1.x * inv * depth_scale, se), h3 = __floats2half2_rn(change, 0.0f);
    features[i] = make_uint4(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1),
                             *reinterpret_cast<const uint32_t*>(&h2), *reinterpret_cast<const uint32_t*>(&h3));
}

// ---- host side --------------------------------------------------------------------------------

int sm_count() {
    static int count = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        if (count <= 0) count = 148;
    });
    return count;
}

// CTAs of `kernel` that fit on one SM, from its shared memory (with the maximum carveout), registers
// and threads; at most `cap`. (The occupancy query answers for the default carveout, which keeps
// these small-footprint kernels at one CTA per SM.)
template <typename Kernel>
int resident_ctas(Kernel kernel, size_t smem, int cap, int threads = kThreads) {
    int dev = 0, smem_sm = 0, regs_sm = 0;
    cudaFuncAttributes attr{};
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
            cudaSuccess ||
        cudaFuncGetAttributes(&attr, kernel) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev) != cudaSuccess)
        return 0;
    const size_t per_cta = smem + attr.sharedSizeBytes + 1024;  // 1 KB reserved per CTA
    int blocks = static_cast<int>(static_cast<size_t>(smem_sm) / per_cta);
    const int regs = attr.numRegs > 0 ? attr.numRegs * threads : 1;
    if (regs_sm / regs < blocks) blocks = regs_sm / regs;
    if (2048 / threads < blocks) blocks = 2048 / threads;
    return blocks < cap ? blocks : cap;
}

cudaError_t launch_conv(const ConvArgs& a, cudaStream_t stream) {
    constexpr int kChunks = kFeatureChannels / 8;
    constexpr size_t smem = static_cast<size_t>(9 * kChunks * 32 + kChunks * kHaloPx) * 16 + 16;
    static const int per_sm = resident_ctas(conv3x3_kernel, smem, 8);
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    const int grid = a.n_tiles < sm_count() * per_sm ? a.n_tiles : sm_count() * per_sm;
    conv3x3_kernel<<<grid, kThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

// cuTensorMapEncodeTiled from the driver, looked up through the runtime (no libcuda link).
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// 4-D map over a BF16 NHWC tensor [batch][height][width][channels] with a box of 8 channels x
// box_w x box_h pixels x 1 image.
bool nhwc_map(CUtensorMap* map, const void* base, int batch, int height, int width, int channels, int box_w, int box_h) {
    const auto fn = encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(channels), static_cast<cuuint64_t>(width),
                                static_cast<cuuint64_t>(height), static_cast<cuuint64_t>(batch)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(channels) * 2,
                                   static_cast<cuuint64_t>(width) * channels * 2,
                                   static_cast<cuuint64_t>(height) * width * channels * 2};
    const cuuint32_t box[4] = {8, static_cast<cuuint32_t>(box_w), static_cast<cuuint32_t>(box_h), 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same halo boxes over activations in 8-channel planes, [batch][channels / 8][y][x][8]: dimension 0
// runs over x * 8 + channel, so a plane's box is 10 pixels (160 bytes) wide and 18 rows high.
bool planar_halo_map(CUtensorMap* map, const void* base, int batch, int height, int width, int channels) {
    const auto fn = encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(width) * 8, static_cast<cuuint64_t>(height),
                                static_cast<cuuint64_t>(channels / 8), static_cast<cuuint64_t>(batch)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(width) * 16,
                                   static_cast<cuuint64_t>(height) * width * 16,
                                   static_cast<cuuint64_t>(channels / 8) * height * width * 16};
    const cuuint32_t box[4] = {kHaloW * 8, kHaloH, 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// in_channels: the tensor's channels where fewer than CIN (the others read zeros). overlap: the launch
// before in the stream does not write this one's weights and has waited for all before it, so this one's
// start (weights, barriers, tensor memory) may overlap its end (programmatic dependent launch: 359 to
// 345 us per 1080p denoiser call).
template <int CIN, int COUT, int EPI, bool kPlanarIn = false, bool kPlanar = kPlanarIn>
cudaError_t launch_conv_tma(const ConvArgs& a, cudaStream_t stream, int in_channels = CIN, bool overlap = false) {
    using S = TmaConv<CIN, COUT>;
    auto kernel = conv3x3_tma_kernel<CIN, COUT, EPI, kPlanarIn, kPlanar>;
    static const int per_sm = resident_ctas(kernel, S::kSmem, 512 / kTmaCols, kTmaThreads);
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    CUtensorMap map;
    const bool mapped = kPlanarIn ? planar_halo_map(&map, a.in, a.batch, a.height, a.width, CIN)
                                : nhwc_map(&map, a.in, a.batch, a.height, a.width, in_channels, kHaloW, kHaloH);
    if (!mapped) return cudaErrorInvalidValue;
    const int grid = a.n_tiles < sm_count() * per_sm ? a.n_tiles : sm_count() * per_sm;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(kTmaThreads);
    config.dynamicSmemBytes = S::kSmem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, map, a);
}

cudaError_t launch_wgrad(const WgradArgs& a, cudaStream_t stream) {
    using G = Wgrad;
    // TMEM columns bound the CTAs per SM: 512 / kCols
    static const int per_sm = resident_ctas(conv3x3_wgrad_kernel, G::kSmem, 512 / G::kCols);
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    const int grid = a.n_tiles < sm_count() * per_sm ? a.n_tiles : sm_count() * per_sm;
    conv3x3_wgrad_kernel<<<grid, kThreads, G::kSmem, stream>>>(a);
    return cudaGetLastError();
}

template <int CIN, int COUT>
cudaError_t launch_wgrad_tma(const WgradArgs& a, cudaStream_t stream) {
    using G = WgradTma<CIN, COUT>;
    auto kernel = conv3x3_wgrad_tma_kernel<CIN, COUT>;
    static const int per_sm = resident_ctas(kernel, G::kSmem, 512 / G::kCols, kTmaThreads);
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    CUtensorMap in_map, grad_map;
    if (!nhwc_map(&in_map, a.in, a.batch, a.height, a.width, CIN, kTileW, kHaloH) ||
        !nhwc_map(&grad_map, a.grad_out, a.batch, a.height, a.width, COUT, kTileW, kTileH))
        return cudaErrorInvalidValue;
    const int grid = a.n_tiles < sm_count() * per_sm ? a.n_tiles : sm_count() * per_sm;
    // its set-up overlaps the end of the kernel before, which it waits for (and with it for all before that one)
    return launch_pass_with(G::kSmem, kernel, dim3(grid), kTmaThreads, stream, in_map, grad_map, a);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

size_t weights_bytes(int in_channels, int out_channels) {
    const int cin = in_channels == 8 ? 16 : in_channels;
    return static_cast<size_t>(9) * cin * out_channels * 2;
}

int check_shape(int batch, int height, int width) {
    if (batch <= 0 || height <= 0 || width <= 0)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: batch, height and width must be positive");
    const long long tiles =
        static_cast<long long>(batch) * ((height + kTileH - 1) / kTileH) * ((width + kTileW - 1) / kTileW);
    if (tiles > 0x7FFFFFFFll)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: too many pixels for one call");
    return SGS_OK;
}

// Buffers of a training step: `saved` (BF16 features, the five hidden activations, the packed weights and
// biases) from forward to backward, `scratch` (BF16 gradients of the output and of two hidden layers in
// turn, data-gradient weights, weight-gradient sums) in the backward.
struct TrainLayout {
    uint32_t n_px;
    size_t act_bytes;
    size_t features, acts, weights, biases, saved;
    size_t grad16, grad32, dgrad, sums, scratch;
};

TrainLayout train_layout(int batch, int height, int width) {
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    TrainLayout L{};
    const size_t px = static_cast<size_t>(batch) * height * width;
    L.n_px = static_cast<uint32_t>(px);
    L.act_bytes = up(px * SGS_DENOISE_WIDTH * 2);
    L.acts = up(px * 16);
    L.weights = L.acts + (kTrainLayers - 1) * L.act_bytes;
    L.biases = L.weights + up(kPacked * 2);
    L.saved = L.biases + up(kBiases * 4);
    L.grad32 = up(px * 32);
    L.dgrad = L.grad32 + 2 * L.act_bytes;
    L.sums = L.dgrad + up((kPacked - packed_before(1)) * 2);
    L.scratch = L.sums + up((kSums + kBiases) * 4);
    return L;
}

// Layer shapes of the denoiser: (input channels as the ABI counts them, output channels, epilogue).
constexpr int kLayers = SGS_DENOISE_LAYERS;
constexpr int kLayerIn[kLayers] = {8, 32, 32, 32, 32, 32};
constexpr int kLayerOut[kLayers] = {32, 32, 32, 32, 32, 16};

}  // namespace dn
}  // namespace sgs

using namespace sgs;
using namespace sgs::dn;

extern "C" {

size_t sgs_conv3x3_weights_size(int32_t in_channels, int32_t out_channels) {
    return weights_bytes(in_channels, out_channels);
}

int sgs_conv3x3(const sgs_conv3x3_args* p, void* stream_ptr) {
    if (p == nullptr) return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: null descriptor");
    if (int st = check_shape(p->batch, p->height, p->width)) return st;
    if (p->input == nullptr || p->output == nullptr || p->weights == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: input, output and weights are required");
    if (!aligned16(p->input) || !aligned16(p->weights) || !aligned16(p->mask) || !aligned16(p->residual) ||
        (p->epilogue != SGS_CONV_FINAL && !aligned16(p->output)))
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: arrays must be 16-byte aligned");
    if (p->epilogue != SGS_CONV_MASK && p->bias == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: bias is required");
    if (p->epilogue == SGS_CONV_MASK && p->mask == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: the mask epilogue needs a mask");
    if (p->epilogue == SGS_CONV_FINAL && p->residual == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: the final epilogue needs the features");
    ConvArgs a{p->input, p->output, static_cast<const uint4*>(p->weights), p->bias,
               static_cast<const uint4*>(p->mask), static_cast<const uint4*>(p->residual),
               p->batch, p->height, p->width, (p->width + kTileW - 1) / kTileW, (p->height + kTileH - 1) / kTileH, 0};
    a.n_tiles = a.batch * a.tiles_x * a.tiles_y;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    const int ci = p->in_channels, co = p->out_channels, epi = p->epilogue;
    cudaError_t err;
    if (ci == 8 && co == 32 && epi == SGS_CONV_RELU)
        err = launch_conv(a, stream);
    else if (ci == 32 && co == 32 && epi == SGS_CONV_RELU)
        err = launch_conv_tma<32, 32, kEpiRelu>(a, stream);
    else if (ci == 32 && co == 16 && epi == SGS_CONV_FINAL)
        err = launch_conv_tma<32, 16, kEpiFinal>(a, stream);
    else if (ci == 32 && co == 32 && epi == SGS_CONV_MASK)
        err = launch_conv_tma<32, 32, kEpiMask>(a, stream);
    else if (ci == 16 && co == 32 && epi == SGS_CONV_MASK)
        err = launch_conv_tma<16, 32, kEpiMask>(a, stream);
    else
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3: unsupported shape %d -> %d, epilogue %d", ci, co,
                            epi);
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "conv3x3: %s", cudaGetErrorString(err));
    return SGS_OK;
}

int sgs_conv3x3_wgrad(const void* input, int32_t in_channels, const void* grad_output, int32_t out_channels,
                      int32_t batch, int32_t height, int32_t width, float* grad_weights, float* grad_bias,
                      void* stream_ptr) {
    if (int st = check_shape(batch, height, width)) return st;
    if (input == nullptr || grad_output == nullptr || grad_weights == nullptr || grad_bias == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3_wgrad: all arrays are required");
    if (!aligned16(input) || !aligned16(grad_output))
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3_wgrad: arrays must be 16-byte aligned");
    WgradArgs a{input, static_cast<const uint4*>(grad_output), grad_weights, grad_bias, batch, height, width,
                (width + kTileW - 1) / kTileW, (height + kTileH - 1) / kTileH, 0};
    a.n_tiles = a.batch * a.tiles_x * a.tiles_y;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    cudaError_t err;
    if (in_channels == 8 && out_channels == 32)
        err = launch_wgrad(a, stream);
    else if (in_channels == 32 && out_channels == 32)
        err = launch_wgrad_tma<32, 32>(a, stream);
    else if (in_channels == 32 && out_channels == 16)
        err = launch_wgrad_tma<32, 16>(a, stream);
    else
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "conv3x3_wgrad: unsupported shape %d -> %d", in_channels,
                            out_channels);
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "conv3x3_wgrad: %s", cudaGetErrorString(err));
    return SGS_OK;
}

int sgs_denoise_features_accumulate(const float* image, const float* alpha, const float* depth,
                                    const uint64_t* framebuffer, float* accum, uint32_t n_pixels, int32_t first,
                                    void* stream_ptr) {
    if (image == nullptr || alpha == nullptr || depth == nullptr || accum == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise features: image, alpha, depth and accum are required");
    if (!aligned16(accum)) return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise features: accum not aligned");
    if (n_pixels == 0) return SGS_OK;
    features_accumulate_kernel<<<(n_pixels + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
        image, alpha, depth, reinterpret_cast<const unsigned long long*>(framebuffer), reinterpret_cast<float4*>(accum),
        n_pixels, first);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise features: %s", cudaGetErrorString(err));
    return SGS_OK;
}

int sgs_denoise_features_finalize(const float* accum, uint32_t n_pixels, uint32_t n_samples, float depth_scale,
                                  void* features, void* stream_ptr) {
    if (accum == nullptr || features == nullptr || n_samples == 0)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise features: accum, features and n_samples > 0 required");
    if (!aligned16(accum) || !aligned16(features))
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise features: arrays must be 16-byte aligned");
    if (n_pixels == 0) return SGS_OK;
    features_finalize_kernel<<<(n_pixels + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
        reinterpret_cast<const float4*>(accum), static_cast<uint4*>(features), n_pixels, n_samples, depth_scale);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise features: %s", cudaGetErrorString(err));
    return SGS_OK;
}

size_t sgs_denoise_weights_size(void) {
    size_t total = 0;
    for (int l = 0; l < kLayers; ++l) total += weights_bytes(kLayerIn[l], kLayerOut[l]);
    return total;
}

size_t sgs_denoise_scratch_size(int32_t batch, int32_t height, int32_t width) {
    if (batch <= 0 || height <= 0 || width <= 0) return 0;
    return static_cast<size_t>(2) * batch * height * width * SGS_DENOISE_WIDTH * 2;
}

int sgs_denoise(const void* features, int32_t batch, int32_t height, int32_t width, const void* weights,
                const float* biases, void* scratch, size_t scratch_bytes, float* output, void* stream_ptr) {
    if (int st = check_shape(batch, height, width)) return st;
    if (features == nullptr || weights == nullptr || biases == nullptr || scratch == nullptr || output == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise: all arrays are required");
    if (scratch_bytes < sgs_denoise_scratch_size(batch, height, width) || !aligned16(scratch))
        return record_error(SGS_ERROR_WORKSPACE, "denoise: scratch needs %zu bytes, 16-byte aligned",
                            sgs_denoise_scratch_size(batch, height, width));
    if (!aligned16(features) || !aligned16(weights))
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise: features and weights must be 16-byte aligned");
    // the hidden activations live only in the scratch, so they use the 8-channel-plane layout (wider
    // halo boxes, coalesced stores); the same arithmetic as the NHWC layers of sgs_conv3x3
    unsigned char* act[2] = {static_cast<unsigned char*>(scratch),
                             static_cast<unsigned char*>(scratch) + sgs_denoise_scratch_size(batch, height, width) / 2};
    const unsigned char* w = static_cast<const unsigned char*>(weights);
    const float* b = biases;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    const int tiles_x = (width + kTileW - 1) / kTileW, tiles_y = (height + kTileH - 1) / kTileH;
    // the features as BF16 lie in the buffer that the second layer writes
    const uint32_t n_px = static_cast<uint32_t>(static_cast<size_t>(batch) * height * width);
    if (const cudaError_t err = launch_pass_with(0, features_bf16_kernel, dim3((n_px + 255) / 256), 256, stream,
                                                 static_cast<const uint4*>(features), reinterpret_cast<uint4*>(act[1]),
                                                 n_px);
        err != cudaSuccess)
        return record_error(SGS_ERROR_CUDA, "denoise features: %s", cudaGetErrorString(err));
    for (int l = 0; l < kLayers; ++l) {
        const bool last = l == kLayers - 1;
        ConvArgs a{act[(l + 1) & 1], last ? static_cast<void*>(output) : act[l & 1],
                   reinterpret_cast<const uint4*>(w), b, nullptr,
                   last ? static_cast<const uint4*>(features) : nullptr, batch, height, width, tiles_x, tiles_y, 0};
        a.n_tiles = batch * tiles_x * tiles_y;
        cudaError_t err;
        if (l == 0)  // the features' channels 8..15 lie outside the tensor and read zeros
            err = launch_conv_tma<16, 32, kEpiRelu, false, true>(a, stream, 8, true);
        else if (!last)
            err = launch_conv_tma<32, 32, kEpiRelu, true>(a, stream, 32, true);
        else
            err = launch_conv_tma<32, 16, kEpiFinal, true>(a, stream, 32, true);
        if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise layer %d: %s", l + 1, cudaGetErrorString(err));
        w += weights_bytes(kLayerIn[l], kLayerOut[l]);
        b += kLayerOut[l];
    }
    return SGS_OK;
}

size_t sgs_denoise_train_params(void) { return kParams; }

size_t sgs_denoise_train_saved_size(int32_t batch, int32_t height, int32_t width) {
    if (batch <= 0 || height <= 0 || width <= 0) return 0;
    return train_layout(batch, height, width).saved;
}

size_t sgs_denoise_train_scratch_size(int32_t batch, int32_t height, int32_t width) {
    if (batch <= 0 || height <= 0 || width <= 0) return 0;
    return train_layout(batch, height, width).scratch;
}

int sgs_denoise_train_forward(const void* features, int32_t batch, int32_t height, int32_t width,
                              const float* const* params, void* saved, size_t saved_bytes, float* output,
                              void* stream_ptr) {
    if (int st = check_shape(batch, height, width)) return st;
    if (features == nullptr || params == nullptr || saved == nullptr || output == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise train: all arrays are required");
    const TrainLayout L = train_layout(batch, height, width);
    if (saved_bytes < L.saved || !aligned16(saved))
        return record_error(SGS_ERROR_WORKSPACE, "denoise train: the saved buffer needs %zu bytes, 16-byte aligned",
                            L.saved);
    if (!aligned16(features)) return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise train: features not aligned");
    TrainParams p;
    for (int l = 0; l < kTrainLayers; ++l) {
        p.weights[l] = params[2 * l];
        p.biases[l] = params[2 * l + 1];
        if (p.weights[l] == nullptr || p.biases[l] == nullptr)
            return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise train: null parameter");
    }
    unsigned char* const base = static_cast<unsigned char*>(saved);
    auto* weights = reinterpret_cast<__nv_bfloat16*>(base + L.weights);
    float* biases = reinterpret_cast<float*>(base + L.biases);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    cudaError_t err = launch_pass_with(0, train_pack_kernel, dim3(kPackBlocks + (L.n_px + 255) / 256), 256, stream, p,
                                       weights, biases, static_cast<const uint4*>(features),
                                       reinterpret_cast<uint4*>(base + L.features), L.n_px);
    ConvArgs a{};
    a.batch = batch;
    a.height = height;
    a.width = width;
    a.tiles_x = (width + kTileW - 1) / kTileW;
    a.tiles_y = (height + kTileH - 1) / kTileH;
    a.n_tiles = batch * a.tiles_x * a.tiles_y;
    a.residual = static_cast<const uint4*>(features);
    for (int l = 0; l < kTrainLayers && err == cudaSuccess; ++l) {
        a.in = base + (l == 0 ? L.features : L.acts + (l - 1) * L.act_bytes);
        a.out = l == kTrainLayers - 1 ? static_cast<void*>(output) : base + L.acts + l * L.act_bytes;
        a.weights = reinterpret_cast<const uint4*>(weights + packed_before(l));
        a.bias = biases + bias_before(l);
        // the features' channels 8..15 lie outside the tensor and read zeros
        err = l == 0                  ? launch_conv_tma<16, 32, kEpiRelu>(a, stream, 8)
              : l < kTrainLayers - 1 ? launch_conv_tma<32, 32, kEpiRelu>(a, stream, 32, true)
                                      : launch_conv_tma<32, 16, kEpiFinal>(a, stream, 32, true);
    }
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise train forward: %s", cudaGetErrorString(err));
    return SGS_OK;
}

int sgs_denoise_train_backward(const float* grad_output, int32_t batch, int32_t height, int32_t width,
                               const float* const* weights, const void* saved, void* scratch, size_t scratch_bytes,
                               float* grads, void* stream_ptr) {
    if (int st = check_shape(batch, height, width)) return st;
    if (grad_output == nullptr || weights == nullptr || saved == nullptr || scratch == nullptr || grads == nullptr)
        return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise train: all arrays are required");
    const TrainLayout L = train_layout(batch, height, width);
    if (scratch_bytes < L.scratch || !aligned16(scratch) || !aligned16(saved))
        return record_error(SGS_ERROR_WORKSPACE, "denoise train: scratch needs %zu bytes, 16-byte aligned", L.scratch);
    TrainParams p{};
    for (int l = 0; l < kTrainLayers; ++l) {
        p.weights[l] = weights[l];
        if (p.weights[l] == nullptr) return record_error(SGS_ERROR_INVALID_ARGUMENT, "denoise train: null weights");
    }
    const unsigned char* const kept = static_cast<const unsigned char*>(saved);
    unsigned char* const work = static_cast<unsigned char*>(scratch);
    auto* dgrad = reinterpret_cast<__nv_bfloat16*>(work + L.dgrad);
    float* sums = reinterpret_cast<float*>(work + L.sums);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
    cudaError_t err = cudaMemsetAsync(sums, 0, (kSums + kBiases) * sizeof(float), stream);
    if (err == cudaSuccess) {
        err = launch_pass_with(0, train_stage_kernel, dim3(kDgradBlocks + (L.n_px + 255) / 256), 256, stream, p, dgrad,
                               grad_output, reinterpret_cast<uint4*>(work + L.grad16), L.n_px);
    }
    const int tiles_x = (width + kTileW - 1) / kTileW, tiles_y = (height + kTileH - 1) / kTileH;
    const void* gz = work + L.grad16;
    for (int l = kTrainLayers - 1; l >= 0 && err == cudaSuccess; --l) {
        const unsigned char* in = kept + (l == 0 ? L.features : L.acts + (l - 1) * L.act_bytes);
        const WgradArgs w{in, static_cast<const uint4*>(gz), sums + sums_before(l), sums + kSums + bias_before(l),
                          batch, height, width, tiles_x, tiles_y, batch * tiles_x * tiles_y};
        err = l == 0                  ? launch_wgrad_tma<8, 32>(w, stream)
              : l < kTrainLayers - 1 ? launch_wgrad_tma<32, 32>(w, stream)
                                      : launch_wgrad_tma<32, 16>(w, stream);
        if (l == 0 || err != cudaSuccess) break;
        void* const out = work + L.grad32 + (l & 1) * L.act_bytes;
        ConvArgs a{gz, out, reinterpret_cast<const uint4*>(dgrad + packed_before(l) - packed_before(1)), nullptr,
                   reinterpret_cast<const uint4*>(in), nullptr, batch, height, width, tiles_x, tiles_y, w.n_tiles};
        err = l < kTrainLayers - 1 ? launch_conv_tma<32, 32, kEpiMask>(a, stream, 32, true)
                                    : launch_conv_tma<16, 32, kEpiMask>(a, stream, 16, true);
        gz = out;
    }
    if (err == cudaSuccess) {
        err = launch_pass_with(0, train_unpack_kernel, dim3((kParams + 255) / 256), 256, stream,
                               static_cast<const float*>(sums), grads);
    }
    if (err != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise train backward: %s", cudaGetErrorString(err));
    return SGS_OK;
}

int sgs_denoise_status(void* stream_ptr) {
    const cudaError_t sync = cudaStreamSynchronize(static_cast<cudaStream_t>(stream_ptr));
    if (sync != cudaSuccess) return record_error(SGS_ERROR_CUDA, "denoise: %s", cudaGetErrorString(sync));
    unsigned int flag = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&flag, g_error, sizeof(flag)) != cudaSuccess ||
        cudaMemcpyToSymbol(g_error, &zero, sizeof(zero)) != cudaSuccess)
        return record_error(SGS_ERROR_CUDA, "denoise: cannot read the error word");
    if (flag != 0) return record_error(SGS_ERROR_CUDA, "denoise: a tensor-core wait ran out of its bound");
    return SGS_OK;
}

}  // extern "C"
