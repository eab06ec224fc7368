// Copies of byte spans (at most MAX_SPAN bytes at a time) at any alignment, each lane's share a host function too
// (checked there against pages that may not be touched).
#pragma once

#include "common.cuh"

namespace cb {

constexpr int MAX_SPAN = 1 << 30;

// The word that starts sh bits into lo and goes on in hi.
__host__ __device__ __forceinline__ uint32_t shift_in(uint32_t lo, uint32_t hi, uint32_t sh) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, sh);
#else
    return (uint32_t)((lo | (uint64_t)hi << 32) >> sh);
#endif
}

__host__ __device__ __forceinline__ uint32_t first4(int n) { return n < 4 ? (uint32_t)n : 4u; }

// The 4-byte words of a destination span of len bytes at d (those that hold one of its bytes), from s, by
// LANES lanes of which this is number l.  Source words are read when they hold a byte of the span; a span of no
// bytes (or fewer) touches nothing: its source may be the end of an allocation.
template <uint32_t LANES>
__host__ __device__ __forceinline__ void copy_words(const uint8_t* s, uint8_t* d, int len, uint32_t l) {
    if (len <= 0) return;
    constexpr int U = 4;  // words in flight per lane
    const uint32_t k = (uint32_t)(uintptr_t)d & 3u;
    for (int q0 = 4 * (int)l - (int)k; q0 < len; q0 += 4 * (int)LANES * U) {  // the word's place in the span
        uint32_t x[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + 4 * (int)LANES * u;
            x[u] = q >= len ? 0u : q >= 0 ? ld_bytes4(s + q, first4(len - q)) : ld_bytes4(s, first4(len)) << (8 * k);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + 4 * (int)LANES * u;
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

// The same for a long span, by 16-byte blocks of the destination: each from the aligned source block or two that hold
// its bytes (a block that holds one byte of the span lies in pages of its allocation).  U blocks are in flight per lane,
// 2 U where source and destination share their alignment.
template <uint32_t LANES, int U>
__host__ __device__ __forceinline__ void copy_long(const uint8_t* s, uint8_t* d, int len, uint32_t l) {
    if (len < 64) return copy_words<LANES>(s, d, len, l);
    const int head = (int)(-(uintptr_t)d & 15);
    const uint32_t at = (uint32_t)((uintptr_t)(s + head) & 15), sh = 8 * (at & 3);
    const uint4* sv = reinterpret_cast<const uint4*>(s + head - at);
    uint4* dv = reinterpret_cast<uint4*>(d + head);
    const int nv = (len - head) >> 4;
    if (at == 0) {
        constexpr int V = 2 * U;
        for (int q = (int)l; q < nv; q += (int)LANES * V) {
            uint4 x[V];
#pragma unroll
            for (int u = 0; u < V; u++)
                if (q + u * (int)LANES < nv) x[u] = sv[q + u * (int)LANES];
#pragma unroll
            for (int u = 0; u < V; u++)
                if (q + u * (int)LANES < nv) dv[q + u * (int)LANES] = x[u];
        }
    } else {
        for (int q = (int)l; q < nv; q += (int)LANES * U) {
            uint4 x[U], y[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (q + u * (int)LANES < nv) {
                    x[u] = sv[q + u * (int)LANES];
                    y[u] = sv[q + u * (int)LANES + 1];
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (q + u * (int)LANES < nv) {
                    const uint4 a = x[u], b = y[u];
                    // the five words from byte `at` (rounded down to a word) on
                    const bool two = at & 8, one = at & 4;
                    const uint32_t p0 = two ? a.z : a.x, p1 = two ? a.w : a.y, p2 = two ? b.x : a.z, p3 = two ? b.y : a.w,
                                   p4 = two ? b.z : b.x, p5 = two ? b.w : b.y;
                    const uint32_t w0 = one ? p1 : p0, w1 = one ? p2 : p1, w2 = one ? p3 : p2, w3 = one ? p4 : p3,
                                   w4 = one ? p5 : p4;
                    dv[q + u * (int)LANES] = make_uint4(shift_in(w0, w1, sh), shift_in(w1, w2, sh), shift_in(w2, w3, sh),
                                                        shift_in(w3, w4, sh));
                }
            }
        }
    }
    copy_words<LANES>(s, d, head, l);
    const int i = head + 16 * nv;
    copy_words<LANES>(s + i, d + i, len - i, l);
}

}  // namespace cb
