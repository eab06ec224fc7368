// The slots of the split inflater's arena (inflate_split.cu), and the members it takes.
#pragma once

#include <cstdint>

namespace cb {
namespace split {

// A member's slot holds its symbols: literal bytes from its start up, sequences (a word each) from its end
// down: bits 24-31 literals before the match, 16-23 match length - 3, 15 set when there is a match, 0-14
// distance - 1.  Symbols take at most 4 bytes per 3 output bytes (matches of length 3); the rest is room
// for sequences without a match (one per 255 literals, and at the end of a segment or block).
constexpr uint32_t SEQ_MATCH = 0x8000u;
constexpr uint32_t SEQ_BAD = 1u;  // without SEQ_MATCH: the match has no valid distance
__host__ __device__ constexpr unsigned long long slot_bytes(uint32_t isize) {
    return (2ull * isize + 64ull + 15ull) & ~15ull;
}

// A position in a member's input is a bit of BITS (the ends of its segments have two flags); its output and its slot
// are counted in 32 bits.  Members beyond that, which no BGZF file holds, are inflated by the one-kernel form.
constexpr uint32_t BITS = (1u << 30) - 1;
constexpr uint32_t MAX_ISIZE = 1u << 30;
__host__ __device__ constexpr bool in_reach(uint32_t in_len, uint32_t isize) {
    return in_len <= BITS / 16 && isize <= MAX_ISIZE;
}
static_assert(slot_bytes(MAX_ISIZE) < 1ull << 32, "a slot is counted in 32 bits");

}  // namespace split
}  // namespace cb
