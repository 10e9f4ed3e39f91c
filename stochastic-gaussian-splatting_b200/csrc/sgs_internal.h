// Internal host-side interface between the C ABI (render_abi.cu) and the kernel files.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>
#include "sgs_gps_parts.h"
#include "sgs_project.cuh"

namespace sgs {

// Stochastic transparency queues AABBs above kDenseMinPixels << step pixels in dense scenes, by the first step whose
// Gaussians the queue holds, and above kDenseMinPixels << kQueueSteps elsewhere.
constexpr uint32_t kDenseMinPixels = 256;
constexpr uint32_t kQueueSteps = 3;

// Large-Gaussian work queue shared by the ST and GPS accumulate passes. Entries are appended
// with one 64-bit atomicAdd on `packed` = (entry count << 40) | chunk count, so every entry's
// first chunk index is known at insertion and increases with the entry index.
struct WorkQueue {
    unsigned long long packed;   // (entries << 40) | chunks, reserved by producers
    unsigned int next_chunk;     // work-stealing cursor of the consumer kernel
    unsigned int overflow;       // producers that found the queue full (processed in place)
    unsigned int error;          // nonzero when a consumer met an inconsistent entry
    unsigned int binned;         // hybrid ST: Gaussians the reference would gather, in arrival order
    unsigned int st_entries;     // ST: entries and list items reserved by producers
    unsigned int st_items;
    unsigned int st_listed;      // items the order pass has listed (GPS: or kNotListed)
    alignas(16) float covered[4];      // AABB pixels of the scene's larger Gaussians, weighted by opacity, estimated by
                                       // kSampleBlocks blocks of the clear pass
    alignas(16) float covered_all[4];  // the same of all its Gaussians of at most kDenseMinPixels << kQueueSteps pixels (GPS:
                                       // of those in compact groups)
    alignas(16) float larger[kQueueSteps][4];  // Gaussians with AABBs above kDenseMinPixels << step, estimated likewise
    alignas(16) float parts[2][4];             // parts of the queued ones in a dense and in a sparse scene, likewise
};
static_assert(offsetof(WorkQueue, covered) % 16 == 0 && offsetof(WorkQueue, covered_all) % 16 == 0 &&
              offsetof(WorkQueue, larger) % 16 == 0 && offsetof(WorkQueue, parts) % 16 == 0, "read as float4");
constexpr unsigned long long kQueueEntryShift = 40;
constexpr unsigned long long kQueueChunkMask = (1ull << kQueueEntryShift) - 1;
// Producers queue chunk indices below this, so the consumers' cursor (which overshoots the last chunk
// by at most one claim per warp) cannot wrap around.
constexpr unsigned long long kMaxQueueChunks = 0xffffffffull - (1ull << 24);
// First-chunk value of a queue entry left unused because its chunks would pass
// kMaxQueueChunks (above every chunk index, so the entry search never returns it).
constexpr uint32_t kUnusedQueueEntry = 0xffffffffu;

// Scratch of the allocation-free render (render_no_alloc.cu). The stochastic-transparency queue takes
// more than 15/16 of 2^18 entries only while a one-sample workspace stays within it.
constexpr size_t kNoAllocScratchBytes = size_t(64) << 20;

// ---- queues in depth order, depth bounds per tile (stochastic transparency; binned GPS Gaussians) ----
constexpr uint32_t kStEntryBytes = 64;
constexpr uint32_t kBoundTile = 8;        // pixels per side of a tile with a depth bound
constexpr uint32_t kBlockTiles = 8;       // tiles per side of a block with a depth bound
constexpr uint32_t kDepthBuckets = 1024;  // 1/32 octave each over view depths of 2^-16 .. 2^16
constexpr uint32_t kSampleBlocks = 4;
// A list item is a part (32 quads of tiles, at most kMaxParts parts) of an entry: part << kItemEntryBits | entry.
constexpr uint32_t kItemEntryBits = 20;
constexpr uint32_t kItemEntryMask = (1u << kItemEntryBits) - 1u;
constexpr uint32_t kMaxParts = 1u << (32u - kItemEntryBits);
constexpr uint32_t kNoItem = 0xffffffffu;  // an unused list place (the last entry has no such part: kMaxStEntries)
constexpr uint32_t kMaxStEntries = kItemEntryMask;
constexpr uint32_t kItemsPerEntry = 4;     // list places per entry, at least
constexpr uint32_t kMaxItems = 1u << 23;

struct StQueue {
    void* a;                        // the first entries_a entries, kStEntryBytes each
    void* b;                        // the others
    uint32_t entries_a;
    uint32_t capacity;              // entries in all, at most kMaxStEntries
    float dense_pixels;             // covered pixels above which the scene counts as dense
    uint32_t log_row_split;         // warps sharing 32 Gaussians in the scatter pass
    uint32_t* list;                 // items in the consumers' order
    uint32_t list_capacity;
    uint32_t* histogram;            // items per depth bucket, then the order pass's cursors
    uint32_t* tile_bound;           // per tile, an upper bound of its keys' depth bits; null: not kept
    uint32_t* block_bound;          // the same per block of 8 x 8 tiles, behind the tiles' bounds (GPS; ST leaves it)
    uint32_t blocks_x, n_blocks;
    uint32_t bound_pitch, tiles_y;  // tiles per row (a multiple of 4) and rows
    uint32_t height;                // framebuffer rows
};

// Scatter passes in depth order: groups of 32 consecutive Gaussians (neighbours in a Morton-ordered model), sorted
// by the depth of their middle one. The clear pass sorts every `slices`-th group in one block; as each of these
// slices is an even sample of the scene, the r-th groups of all of them lie at nearly the same depth, and the
// order takes these together, so that no sum over the blocks is needed.
constexpr uint32_t kSliceGroups = 1024;  // groups per slice, at most
constexpr uint32_t kGroupBuckets = 1024;  // 1/64 octave each over view depths of 2^-4 .. 2^12
constexpr int kGroupShift = 17;           // depth bits below a bucket's
// Warps per block of a front-to-back pass: many of its warps end early, and a block keeps its place until its last
// warp has ended (6M Gaussians at 1080p: 426 us with 8 warps a block, 399 with 4, 399 with 2; point splatting 305, 293
// and 294).
constexpr uint32_t kOrderedWarps = 4;
struct GroupOrder {
    uint32_t* order;          // groups front to back; null: the pass takes them as they come
    uint32_t groups;
    uint32_t slices;
    uint32_t refresh_period;  // every refresh_period-th block of the pass lowers tile bounds
    double refresh_rcp;       // 1 / refresh_period
    float min_pixels;         // covered pixels above which the pass runs in depth order
};

// Depth bucket of a key's high word; depths off the range share the end buckets (the order only
// decides how much is culled, never the winners).
__device__ __forceinline__ uint32_t depth_bucket(const uint32_t depth_bits) {
    const int b = static_cast<int>(depth_bits >> 18) - ((127 - 16) << 5);
    return static_cast<uint32_t>(min(max(b, 0), static_cast<int>(kDepthBuckets) - 1));
}

// Adds `items` (0: none) to the histogram at the depth of `key_hi`, one atomic per bucket of the warp
// (neighbours in Morton order mostly share theirs; a dense scene's Gaussians have some 60 in all).
__device__ __forceinline__ void count_at_depth(uint32_t* __restrict__ histogram, const uint32_t key_hi,
                                               const uint32_t items, const uint32_t lane) {
    const uint32_t bucket = items != 0 ? depth_bucket(key_hi) : 0xffffffffu;
    const uint32_t peers = __match_any_sync(0xffffffffu, bucket);
    const uint32_t sum = __reduce_add_sync(peers, items);
    if (sum != 0 && lane == __ffs(peers) - 1u) atomicAdd(histogram + bucket, sum);
}

// The items of the binned GPS Gaussians: sgs_gps_parts.h.
constexpr uint32_t kNotListed = 0xffffffffu;  // WorkQueue::st_listed: the chunks are taken as they came

// Per-entry arrays of the GPS large-Gaussian queue (structure of arrays, 16-byte aligned).
struct QueueArrays {
    unsigned long long* key;  // packed fragment key
    float4* geom;             // mean2d, L.x, L.y
    float4* geom2;            // L.z, power threshold, opacity_rcp, dilog
    uint4* meta;              // conic x/y/z bits, first chunk
    uint32_t* count;          // number of points
    uint32_t capacity;
};

// Queue entry owning chunk c: the last e in [0, n) with meta[e].w (the entry's first chunk,
// nondecreasing in e, meta[0].w = 0) <= c. A 32-ary search by the whole warp (every lane calls it
// with the same arguments): each step the lanes read 32 evenly spaced first chunks at once and a
// ballot keeps the segment that holds the answer, so 2^20 entries take 4 rounds of loads instead
// of 20 dependent ones.
__device__ __forceinline__ uint32_t queue_entry_of_chunk(const uint4* __restrict__ meta, const uint32_t n,
                                                         const uint32_t c, const uint32_t lane) {
    uint32_t lo = 0, hi = n;  // the answer lies in [lo, hi)
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) >> 5;
        const uint32_t idx = lo + lane * step;
        const bool le = lane == 0u || (idx < hi && meta[idx].w <= c);
        const uint32_t k = 31u - __clz(__ballot_sync(0xffffffffu, le));
        lo += k * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// Scratch carved out of the caller's workspace by layout_workspace().
struct Workspace {
    unsigned long long* framebuffer;  // P_fb packed keys
    float4* samples;                  // P_fb (rgb, depth)
    float4* reuse_weights;            // P_fb when spatial reuse is on
    WorkQueue* queue;
    QueueArrays q;
    size_t bytes;
};

struct AccumulateParams {
    const float* means;
    const float* scales;
    const float4* rotations;
    const float* opacities;
    const float4* w2c;
    unsigned long long* framebuffer;
    uint32_t n;
    uint32_t frame_idx;               // used when frame_ptr is null
    const uint32_t* frame_ptr;        // device-resident frame index, or null
    uint32_t frame_offset;            // added to either: sample s of a call whose passes run per sample
    PassCamera cam;
    const uint8_t* blue_noise;        // (64, 128, 128) volume; null: white noise
    uint32_t max_fragments;           // GPS point cap per Gaussian
    uint32_t max_binned;              // hybrid: binned Gaussian capacity (accumulate_hybrid*.cu max_binned)
    bool hybrid;                      // hybrid scheduling
    WorkQueue* queue;
    QueueArrays q;
    StQueue stq;
    GroupOrder groups;
    uint32_t n_samples;               // samples of one call (frames frame .. frame + n_samples - 1)
    size_t fb_stride;                 // framebuffer elements between consecutive samples' framebuffers
    const float4* pre;                // preactivated layout (2 float4 per Gaussian) or null
    QuantizedModel quant;             // quantised layout (records == null: the float32 arrays)
};

// Frame-dependent random-number state of one call: the frame index (from device memory when the
// caller keeps it there) and the blue-noise slice and rotation it selects (render.cu:77-82).
struct FrameRng {
    uint32_t frame;
    const uint8_t* slice;
    uint32_t rotation;
};

// The random-number state of frame `frame`.
__device__ __forceinline__ FrameRng frame_rng_at(const AccumulateParams& a, const uint32_t frame) {
    FrameRng r;
    r.frame = frame;
    r.slice = a.blue_noise != nullptr
                  ? a.blue_noise + static_cast<size_t>(frame % kBlueNoiseDepth) * kBlueNoiseWidth * kBlueNoiseHeight
                  : nullptr;
    r.rotation = (frame / kBlueNoiseDepth) * 0x9E3779B9u;
    return r;
}

__device__ __forceinline__ FrameRng frame_rng(const AccumulateParams& a) {
    return frame_rng_at(a, (a.frame_ptr != nullptr ? *a.frame_ptr : a.frame_idx) + a.frame_offset);
}

// Launch of a pass whose kernel begins with wait_for_pass_before(): its launch overlaps the end of the pass before
// it, which it then waits for with all that pass wrote.
template <typename... Params, typename... Args>
cudaError_t launch_pass_with(const size_t shared_bytes, void (*kernel)(Params...), const dim3 blocks,
                             const unsigned threads, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = blocks;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, args...);
}
template <typename P>
cudaError_t launch_pass(void (*kernel)(P), const unsigned blocks, const unsigned threads, const P& p,
                        cudaStream_t stream) {
    return launch_pass_with(0, kernel, dim3(blocks), threads, stream, p);
}

cudaError_t launch_clear(unsigned long long* framebuffer, size_t n_fb, WorkQueue* queue, const StQueue& stq,
                         int num_sms, cudaStream_t stream);
cudaError_t launch_order_gps(const AccumulateParams& p, int num_sms, cudaStream_t stream);
cudaError_t launch_clear_st(const AccumulateParams& p, size_t n_fb, int num_sms, cudaStream_t stream);
cudaError_t launch_accumulate_st(const AccumulateParams& p, int num_sms, cudaStream_t stream);
cudaError_t launch_accumulate_gps(const AccumulateParams& p, int num_sms, cudaStream_t stream);
cudaError_t launch_quantize(const float* means, const float* scales, const float4* rotations, const float* opacities,
                            const float* sh, uint32_t sh_floats, uint32_t n, uint4* records, float4* chunks,
                            __half* sh_half, cudaStream_t stream);
cudaError_t launch_composite(const float* image, const float* depth, const float* alpha, const float* background,
                             uint32_t n, float* rgb, float* depth_out, float* alpha_out, cudaStream_t stream);
cudaError_t launch_preactivate(const float* scales, const float4* rotations, const float* opacities, uint32_t n,
                              float4* out, cudaStream_t stream);
cudaError_t launch_atomic_min_probe(unsigned long long* slots, uint64_t n_slots, uint32_t ops, uint32_t blocks,
                                    uint32_t pattern, uint32_t seed, cudaStream_t stream);

struct ResolveParams {
    const float* means;
    const float* scales;
    const float4* rotations;
    const float* opacities;
    const float* sh;
    const float4* w2c;
    const float* cam_position;
    const unsigned long long* framebuffer;
    float4* samples;
    float4* reuse_weights;
    uint2* k_prims;
    float4* k_occl;
    const float* hist_image;
    const float* hist_depth;
    const float* hist_alpha;
    const float* hist_weight_mass;
    const float4* v2pv;
    float* image;
    float* depth;
    float* alpha;
    float* weight_mass;
    uint32_t n_fb;
    uint32_t n_pixels;
    uint32_t sh_bases;
    uint32_t width, height, ss;
    float focal_x, focal_y, center_x, center_y, far_plane;  // image pixels (resolve)
    PassCamera cam;                                          // framebuffer (sample)
    bool spatial_reuse;
    bool sh_vec4;    // degree-3 SH at a 16-byte aligned base: winners load their coefficients as float4
    uint32_t* frame_counter;  // device-resident frame index advanced by the last pass, or null
    int temporal_mode;
    uint32_t n_samples;       // samples merged by one call (the first in temporal_mode, the rest Static)
    size_t fb_stride;         // framebuffer elements between consecutive samples' framebuffers
    QuantizedModel quant;     // quantised layout (records == null: the float32 arrays)
};

cudaError_t launch_sample_resolve(const ResolveParams& p, cudaStream_t stream);

// Backward pass of stochastic transparency (backward_st.cu).
struct BackwardParams {
    const float* means;
    const float* scales;
    const float4* rotations;
    const float* opacities;
    const float* sh;
    const float4* w2c;
    const float* cam_position;
    uint32_t n;
    uint32_t sh_bases;
    bool sh_vec4;                            // degree-3 SH at a 16-byte aligned base
    PassCamera cam;                          // framebuffer camera
    uint32_t width;                          // image width (pixels)
    uint32_t ss;
    const unsigned long long* framebuffer;   // the sample's winners
    const float4* samples;                   // the sample's winner colour and depth
    const float* grad_image;                 // (H, W, 3) upstream gradient of the image
    const float* grad_alpha;                 // (H, W) or null
    const float* grad_depth;                 // (H, W) or null
    float grad_scale;                        // weight of this sample in the output / ss^2
    float* colors;                           // (N, 3) per-Gaussian colour
    double* accum;                           // (N, 10) projected-quantity gradients
    float* d_means;
    float* d_scales;
    float* d_rotations;
    float* d_opacities;
    float* d_sh;
    // fused form over S samples: per framebuffer pixel and sample, the winner key and
    // T = grad_scale (g . c_w + g_d z_w), interleaved [pixel][sample]
    unsigned long long* pix_keys;
    float* pix_terms;
    uint32_t* pix_far;                       // per pixel, the largest depth bits of the samples' winners
    uint32_t* tile_far;                      // per 8 x 8 tile, the largest of those
    uint32_t tiles_x, tiles_y;
    // queues of Gaussians with huge and with large footprints, walked in row chunks by a persistent kernel
    WorkQueue* bw_queue;                     // two
    void* bw_entries;                        // WalkEntry per place (backward_st.cu), bw_slots in all
    uint4* bw_meta;                          // per queue bw_capacity: y_min, height, log2 rows per chunk, first chunk
    uint32_t* bw_index;                      // Gaussian index per place
    uint32_t bw_capacity, bw_slots;
    int num_sms;
    uint32_t n_samples;                      // S
    uint32_t sample;                         // the sample whose terms sample_terms writes
    uint32_t n_fb;                           // framebuffer pixels
};

cudaError_t launch_backward_colors(const BackwardParams& p, cudaStream_t stream);
cudaError_t launch_backward_fragments(const BackwardParams& p, cudaStream_t stream);
cudaError_t launch_backward_projection(const BackwardParams& p, cudaStream_t stream);
cudaError_t launch_backward_sample_terms(const BackwardParams& p, cudaStream_t stream);
cudaError_t launch_backward_framebuffer_terms(const BackwardParams& p, cudaStream_t stream);
cudaError_t launch_backward_fragments_samples(const BackwardParams& p, cudaStream_t stream);

// Sets the calling thread's sgs_last_error() message (printf format) and returns `status`.
int record_error(int status, const char* fmt, ...);

}  // namespace sgs
