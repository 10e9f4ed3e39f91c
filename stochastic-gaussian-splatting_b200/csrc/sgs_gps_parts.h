// How the points of a binned Gaussian (point splatting with hybrid scheduling) are dealt out: plain C++, so
// that its arithmetic can be checked on the host for every count up to the point cap's 2^32 - 1.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SGS_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SGS_HOST_DEVICE inline
#endif

namespace sgs {

constexpr uint32_t kChunkPoints = 256;  // accumulate_hybrid_gps.cu:19

// Chunks of a queue that is taken as it came.
SGS_HOST_DEVICE uint32_t gps_chunks(const uint32_t count) {
    return count / kChunkPoints + (count % kChunkPoints != 0u ? 1u : 0u);
}

// Items of a queue in depth order: kGpsItemPoints points each (more where a Gaussian would have more than
// kMaxGpsParts items, so that the items of 2^20 entries stay below 2^31); an unused entry has none.
constexpr uint32_t kGpsItemPoints = 2048;
constexpr uint32_t kMaxGpsParts = 1024;
struct GpsParts {
    uint32_t parts, points;
};
SGS_HOST_DEVICE GpsParts gps_parts(const uint32_t count) {
    GpsParts p;
    const uint32_t items = count / kGpsItemPoints + (count % kGpsItemPoints != 0u ? 1u : 0u);
    p.points = (items + kMaxGpsParts - 1u) / kMaxGpsParts * kGpsItemPoints;
    p.parts = count != 0u ? count / p.points + (count % p.points != 0u ? 1u : 0u) : 0u;
    return p;
}

// The points [first, first + n) of item `part` of a Gaussian of `count` points.
struct GpsItemPoints {
    uint32_t first, n;
};
SGS_HOST_DEVICE GpsItemPoints gps_item_points(const uint32_t count, const uint32_t part) {
    const uint32_t points = gps_parts(count).points;
    GpsItemPoints i;
    i.first = part * points;
    i.n = points < count - i.first ? points : count - i.first;
    return i;
}

}  // namespace sgs
