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

// The decode's scratch, apart from the members' output: jobs may share their output or have it read meanwhile, and a
// member's lanes are not bounded by its size (with the output as scratch three took part in one of 1,000 bytes: 8,000 GEX
// members of them 404 us, now 315; 65 KB members as before).  Every member in flight (at most FLIGHT: 18 warps on 148 SMs,
// twice for two ranges) has scratch_bytes, four times the members' mean size (a lane's run holds its symbols with some
// room, and 21 lanes take part from 4,096 bytes on) up to 64 KiB.
constexpr long long FLIGHT = 2 * 18 * 148;
constexpr uint32_t SCRATCH_MIN = 4096, SCRATCH_MAX = 65536;
constexpr long long in_flight(long long n_jobs) { return n_jobs < FLIGHT ? n_jobs : FLIGHT; }
constexpr uint32_t scratch_bytes(long long n_jobs, unsigned long long out_bytes) {
    const unsigned long long s = n_jobs > 0 ? (out_bytes / (unsigned long long)n_jobs * 4 + 4095) & ~4095ull : 0;
    return s < SCRATCH_MIN ? SCRATCH_MIN : s > SCRATCH_MAX ? SCRATCH_MAX : (uint32_t)s;
}
// What the arena (without 80 bytes a job) and the scratch take together for out_bytes of output.
constexpr unsigned long long arena_and_scratch(long long n_jobs, unsigned long long out_bytes) {
    return 2 * out_bytes + (unsigned long long)in_flight(n_jobs) * scratch_bytes(n_jobs, out_bytes);
}
// The scratch per member of a workspace that has `room` for the two: that of the most output it is large enough for
// (so of out_bytes, where it was made for them), or none.
constexpr uint32_t scratch_for(long long n_jobs, unsigned long long room) {
    for (uint32_t s = SCRATCH_MAX; s; s -= 4096) {
        const unsigned long long all = (unsigned long long)in_flight(n_jobs) * s;
        if (all <= room && scratch_bytes(n_jobs, (room - all) / 2) >= s) return s;
    }
    return 0;
}

}  // namespace split
}  // namespace cb
