// How the persistent edit kernel (hd_edit_persist.cu) splits a level over its
// CTAs, and its grid barrier's word: plain arithmetic, also compiled by a host
// compiler (its test).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HD_SPLIT __host__ __device__ __forceinline__
#else
#define HD_SPLIT inline
#endif

namespace hd {

constexpr uint32_t kPT = 1024; // threads per CTA of the persistent edit kernel (one CTA per SM)

HD_SPLIT uint32_t chunk_len(uint32_t n, uint32_t parts, uint32_t align)
{
    const uint32_t per = (n + parts - 1) / parts;
    return (per + align - 1) / align * align;
}

// Grid phases split a level into one chunk per CTA, a multiple of the warp
// width long (so that a warp's 32 consecutive slots fall in at most two
// chunks): every CTA gets work once a level holds 32 entries per CTA.
constexpr uint32_t kChunkAlign = 32;

// Chunk of level entries a descend flag is counted in (the grid's top-down
// chunking of that level).
HD_SPLIT uint32_t td_chunk(uint32_t i, uint32_t n, uint32_t G) { return i / chunk_len(n, G, kChunkAlign); }

// Chunks of a sorted level (their digit counts' rows) that the scatters sum
// themselves, the least length of a chunk, and the chunks of n elements: at
// most kSumRows of at most kPT elements for as long as they do, else as many
// as hold kChunkAlign elements; never more than the G CTAs, as CTA k works
// chunk k and the digit counts have a row a CTA (a device of fewer than
// kSumRows SMs gets longer chunks).
constexpr uint32_t kSumRows = 32;
constexpr uint32_t kSortChunk = 256;
HD_SPLIT uint32_t sort_chunks(uint32_t n, uint32_t G)
{
    const uint32_t few = (n + kSortChunk - 1) / kSortChunk;
    const uint32_t want = few <= kSumRows      ? few
                          : n <= kSumRows * kPT ? kSumRows
                                                : (n + kChunkAlign - 1) / kChunkAlign;
    return want < 1 ? 1 : want < G ? want : G;
}

// The grid barrier's word: the arrivals of a launch, which only grow, and on top
// the flag of a CTA that gave up (63 bits of arrivals never reach it).
constexpr unsigned long long kBarrierAbort = 1ull << 63;
HD_SPLIT unsigned long long barrier_arrivals(unsigned long long word) { return word & ~kBarrierAbort; }
HD_SPLIT bool barrier_aborted(unsigned long long word) { return (word & kBarrierAbort) != 0; }
// The arrivals at which the k-th barrier of G CTAs is passed
HD_SPLIT unsigned long long barrier_target(uint32_t k, uint32_t G) { return (unsigned long long)k * G; }

} // namespace hd
