// Copies of byte spans at any alignment by words, each lane's share a host function too (checked there against
// pages that may not be touched).
#pragma once

#include "common.cuh"

namespace cb {

__host__ __device__ __forceinline__ uint32_t first4(long long n) { return n < 4 ? (uint32_t)n : 4u; }

// The 4-byte words of a destination span of len bytes at d (those that hold one of its bytes), from s, by
// LANES lanes of which this is number l.  Source words are read when they hold a byte of the span; a span of no
// bytes (or fewer) touches nothing: its source may be the end of an allocation.
template <uint32_t LANES>
__host__ __device__ __forceinline__ void copy_words(const uint8_t* s, uint8_t* d, long long len, uint32_t l) {
    if (len <= 0) return;
    constexpr int U = 4;  // words in flight per lane
    const uint32_t k = (uint32_t)(uintptr_t)d & 3u;
    for (long long q0 = 4LL * l - k; q0 < len; q0 += 4 * LANES * U) {  // the word's place in the span
        uint32_t x[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long q = q0 + 4LL * LANES * u;
            x[u] = q >= len ? 0u : q >= 0 ? ld_bytes4(s + q, first4(len - q)) : ld_bytes4(s, first4(len)) << (8 * k);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long q = q0 + 4LL * LANES * u;
            if (q >= len) break;
            if (q >= 0 && q + 4 <= len) {
                *reinterpret_cast<uint32_t*>(d + q) = x[u];
            } else {
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (q + t >= 0 && q + t < len) d[q + t] = (uint8_t)(x[u] >> (8 * t));
            }
        }
    }
}

}  // namespace cb
