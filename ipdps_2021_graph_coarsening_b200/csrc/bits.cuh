// bits.cuh -- one bit per vertex in shared memory, and rows cut by length.
//
// Passes that look up a small fact of every entry's destination (its part, or
// whether it is listed) gather from a bitmap in the block's shared memory: a
// gather that misses L1 is served at about half a sector a clock and SM, a
// shared-memory one at about nine.  200 KB hold 1.6M vertices; larger graphs
// gather the bitmap through L1.
#pragma once
#include <stdint.h>

namespace sgpb {

constexpr uint32_t kBitsMaxWords = 51200;   // 200 KB
// rows of more entries are summed by a whole block
constexpr uint32_t kLongRow = 1024;

__host__ __device__ __forceinline__ uint32_t bit_words(uint32_t n) { return (n + 31) / 32; }

__device__ __forceinline__ uint32_t bit_of(const uint32_t *bits, uint32_t v) {
    return (bits[v >> 5] >> (v & 31u)) & 1u;
}

// the bitmap into shared memory (nothing when it stays in global memory);
// the caller synchronises
__device__ __forceinline__ void bits_load(const uint32_t *__restrict__ g, uint32_t words, uint32_t *s) {
    for (uint32_t k = threadIdx.x; k < words; k += blockDim.x) s[k] = __ldcg(g + k);
}

}  // namespace sgpb
