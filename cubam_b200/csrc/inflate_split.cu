// Raw-DEFLATE inflater for BGZF members, form 3: the Huffman decode, the copy and the CRC32 as kernels of their own.
//
// Replaces cubam's nvcompBatchedDeflateDecompressAsync call and its status/size check
// (src/cubam/bgzf.py:587-611) with the CRC32 check added (cubam's reader does not check it,
// docs/reading.md:48-51).  DEFLATE is RFC 1951.
//
//  1. k_decode: one member per CTA of W warps (W = 8, 4, 2 or 1, fewer the more members there are), its
//     32 W lanes decoding as many segments of the member's bits at once.  A Huffman decoder that starts
//     at a wrong bit falls in step with the true symbols soon (on BAM members after 64 bits in half of
//     the cases, after 512 in 99.5% and after 768 in 99.97%), so every lane starts OVERLAP bits before its
//     segment and notes the first symbol that begins in it; that must be where the lane before stopped, and
//     a lane for which it is not decodes its segment again from there.  (Codes of nearly one length do not
//     fall in step: uniform 7-bit bytes need up to 12 such passes at one warp and 92 at eight, and 20,000
//     members of 65 KB of them take 40 ms, 26 with a member per lane; as many of BAM records 7.4.)  The lanes
//     share one set of code tables in shared memory.  Each lane writes its symbols, literal bytes and 4-byte
//     sequences of a literal count and a match, to a run of its own in the scratch of the members in flight;
//     the warps then put the runs together in the member's slot of an arena in HBM.
//     k_literals copies the members that have no match.
//  2. k_copy: one member per CTA of W warps.  They take 64 W sequences at a time, place them by a prefix
//     sum of their lengths and write the output in rounds of 128 bytes per warp, a 4-byte word per lane,
//     to a ring in shared memory (the sources of matches) and to HBM.
//  3. k_crc: the CRC32 of every member's output, W warps per member, in registers.
//  4. Members whose symbols do not fit their slot are inflated by the one-kernel form
//     (cb_inflate_listed, inflate.cu).
//
// What bounds them: with many members the issue of instructions (decode 0.53 per cycle and scheduler, copy
// 0.68, at the 18 and 22 warps per SM that fit, of which 16.4 and 18.9 were active); with few, the chain of
// steps of one lane and of rounds of one member, which is why a member takes more warps then.  Measured, in
// ms (one serial decoder per member, in one kernel, before; a warp per member in between):
//   39 GEX members (10,000 records)      decode 0.17 (0.46), copy 0.15 (0.43), CRC32 0.01; one kernel 4.2
//   about 70,000 (18 million records)    decode 12.6, copy 13.6, CRC32 1.9; all of it 47 with a member per lane
//
// Every loop is bounded: a decode step consumes input bits, bounded per member, a repair round
// confirms at least one more segment; every shared-memory index is masked or checked; arena and
// scratch writes stay within the member's, output writes within its output range.

#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "crc.cuh"
#include "spans.cuh"
#include "split_slots.cuh"

namespace cb {
namespace split {

// RFC 1951 3.2.5 in closed form: length symbol i = sym - 257 (0-28), distance symbol i (0-29).
__device__ __forceinline__ void len_code(uint32_t i, uint32_t& base, uint32_t& ext) {
    if (i < 4) {
        base = 3 + i;
        ext = 0;
    } else if (i == 28) {
        base = 258;
        ext = 0;
    } else {
        ext = (i >> 2) - 1;
        base = 3 + ((4u | (i & 3u)) << ext);
    }
}
__device__ __forceinline__ void dist_code(uint32_t i, uint32_t& base, uint32_t& ext) {
    if (i < 4) {
        base = 1 + i;
        ext = 0;
    } else {
        ext = (i >> 1) - 1;
        base = 1 + ((2u | (i & 1u)) << ext);
    }
}

// RFC 1951 3.2.7: order of the code length code lengths.
__constant__ uint8_t kClOrder[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// ---------------------------------------------------------------- workspace

// Workspace: [0, 256) queue counters; per job 32 bytes (u32 list of the members for the one-kernel
// form, u32 status, u64 arena slot, u32 literals, u32 sequences); the arena after that, 256-byte
// aligned.  Job j's slot is the prefix sum of slot_bytes over the jobs before it (k_slots), so the arena
// holds 2 sum(ISIZE) + 80 n_jobs bytes at most, whatever the jobs' output offsets are.
constexpr size_t WS_HEAD = 256;
constexpr size_t PER_JOB = 32;
constexpr int JW = PER_JOB / 4;           // words per job
constexpr int PARTS = 2;                  // ranges of jobs of the pipelined form, each with two queue counters
constexpr int Q_LISTED = 2 * PARTS;       // queue counter: members for the one-kernel form (and its queue)
constexpr uint32_t ST_LISTED = 0x100;     // internal status: on that list
constexpr uint32_t ST_LITERALS = 0x200;   // internal status: its output written by k_literals
__host__ __device__ __forceinline__ size_t arena_offset(long long n_jobs) {
    return (WS_HEAD + PER_JOB * (size_t)n_jobs + 255) & ~(size_t)255;
}
// The arena slot of every job: one CTA; thread t sums a contiguous run of jobs, a block scan joins
// the runs, and each thread writes its run's offsets.
constexpr int SLOT_NT = 1024;
__global__ void __launch_bounds__(SLOT_NT) k_slots(const cb_member_job* __restrict__ jobs, int64_t n_jobs,
                                                   const int64_t* __restrict__ d_n_jobs, uint8_t* ws) {
    // Each warp takes a contiguous segment of jobs, read coalesced with eight loads per lane in
    // flight: a first pass sums the segment's slots, the warps' sums are scanned, a second pass
    // writes the slot offsets.
    constexpr int NW = SLOT_NT / 32, U = 8;
    __shared__ unsigned long long wbase[NW + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long n = n_jobs;
    if (d_n_jobs) n = min((long long)n, (long long)*d_n_jobs);
    const long long seg = ((n + NW - 1) / NW + 32 * U - 1) / (32 * U) * (32 * U);
    const long long a = min((long long)warp * seg, n), b = min(a + seg, n);
    unsigned long long sum = 0;
    for (long long j0 = a; j0 < b; j0 += 32 * U) {
        uint32_t isz[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const long long j = j0 + k * 32 + lane;
            isz[k] = j < b ? jobs[j].isize : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; k++) sum += j0 + k * 32 + lane < b ? (unsigned long long)slot_bytes(isz[k]) : 0ull;
    }
    for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
    if (lane == 0) wbase[warp] = sum;
    __syncthreads();
    if (warp == 0) {
        const unsigned long long x = lane < NW ? wbase[lane] : 0ull;
        unsigned long long tot;
        const unsigned long long e = warp_exclusive_scan(x, tot);
        __syncwarp();
        if (lane < NW) wbase[lane] = e;
    }
    __syncthreads();
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(ws + WS_HEAD);
    unsigned long long carry = wbase[warp];
    for (long long j0 = a; j0 < b; j0 += 32 * U) {
        uint32_t isz[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const long long j = j0 + k * 32 + lane;
            isz[k] = j < b ? jobs[j].isize : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
            const long long j = j0 + k * 32 + lane;
            const unsigned long long v = j < b ? (unsigned long long)slot_bytes(isz[k]) : 0ull;
            unsigned long long t;
            const unsigned long long x = warp_exclusive_scan(v, t);
            if (j < b) slot[(JW / 2) * j + 1] = carry + x;
            carry += t;
        }
    }
}

__device__ __forceinline__ void report(cb_inflate_summary* summary, uint32_t* job_status, long long j, uint32_t st) {
    if (job_status) job_status[j] = st;
    if (st != CB_OK) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&summary->n_bad), 1ull);
        atomicMin(reinterpret_cast<long long*>(&summary->first_bad), j);
        atomicMax(&summary->status, (int)st);
    }
}

// ---------------------------------------------------------------- k_decode: one member per CTA of W warps

// Entries of the literal/length table: bits 0-5 the bits of the code and its extra bits (32: a code longer
// than the table resolves), 6-9 the code length, 16-23 the literal or the length base - 3, and
// flags; a literal has none.
constexpr uint32_t F_MATCH = 1u << 31, F_EOB = 1u << 30, F_BAD = 1u << 29;
// Entries of the distance table: bits 0-9 as above, 16-30 the distance base - 1, 31 set for a distance
// (so the upper half is SEQ_MATCH | base - 1); a symbol that is none has bits 16-31 SEQ_BAD.
constexpr uint32_t SLOW = F_BAD | 32;  // (as a second literal: none)
constexpr int ROOT = 9, DROOT = 8;     // bits that index the root tables
constexpr uint32_t LNG = 512;          // entries for the longer literal/length codes, after the root's
constexpr uint32_t DST = (1u << ROOT) + LNG;
// bits a lane decodes before its segment to fall in step (a lane that did not costs its warp a second pass: all
// of form 3 on 2,320 members, in us, with 384 1226, 512 1210, 640 1180, 768 1190, 1024 1188)
constexpr uint32_t OVERLAP = 640;
constexpr uint32_t SEG_MIN = 128;      // bits of a segment, at least
constexpr uint32_t WINDOW = 179200;    // bits of a window of segments: a zlib block of 16,383 BAM symbols
// bytes of scratch per lane, at least (or one lane decodes alone): more lanes for small members, with the more overlap (in
// us, with 128, 192 and 256: 4,000 GEX members of 700 bytes 187 187 192, 400 of text of 3,000 133 121 126)
constexpr uint32_t RUN_MIN = 192;
constexpr int ROWS = 16;               // words of input kept per lane
constexpr int STEPS = 8;               // decode steps between refills
constexpr uint32_t LSTAGE = 32, SSTAGE = 16;  // staged literals (bytes) and sequences per lane
constexpr uint32_t LC_MAX = 235;       // literals before a match, about (one sequence holds up to 255)
static_assert(2 * STEPS + 15 <= (int)LSTAGE && STEPS + 4 <= (int)SSTAGE && LC_MAX + 2 * STEPS <= 255,
              "staging holds a round and what is left of the last");

// Per member (a CTA of W warps): the code tables and what the warps tell each other.
struct DecTables {
    uint32_t tab[(1 << ROOT) + LNG + (1 << DROOT)];  // literal/length codes, then (from DST) distances
    uint32_t lfirst[17], lindex[17], dfirst[17], dindex[17];  // canonical codes by length, left-justified to 15 bits
    uint32_t lcount[16], dcount[16];
    uint16_t lsym[288];             // symbols in canonical order
    uint16_t dsym[32];
    unsigned long long job;
    uint32_t say[9];
};
// Per warp.  The input is columns, word r of lane l at r * 32 + l (rows ROWS, ROWS + 1 repeat rows 0, 1);
// the staging of a lane is contiguous, with odd word strides.
struct DecWarp {
    uint32_t in[(ROWS + 2) * 32];
    uint32_t lst[32 * (LSTAGE / 4 + 1)];  // while a header is read: the code lengths (bytes)
    uint32_t sst[32 * (SSTAGE + 1)];      // while a header is read: the code-length code's table (bytes)
};
template <int W> struct DecMember {
    DecTables t;
    uint32_t ends[32 * W], sums[2][W];
    DecWarp w[W];
};

__device__ __forceinline__ uint32_t lit_entry(uint32_t s, uint32_t L) {
    if (s < 256) return L | (L << 6) | (s << 16);
    if (s == 256) return F_EOB | L | (L << 6);
    if (s >= 286) return F_BAD | L | (L << 6);
    uint32_t base, ext;
    len_code(s - 257, base, ext);
    return F_MATCH | (L + ext) | (L << 6) | ((base - 3) << 16);
}
__device__ __forceinline__ uint32_t dist_entry(uint32_t s, uint32_t L) {
    if (s >= 30) return L | (L << 6) | (SEQ_BAD << 16);
    uint32_t base, ext;
    dist_code(s, base, ext);
    return (L + ext) | (L << 6) | ((SEQ_MATCH | (base - 1)) << 16);
}

// The lowest n bits set (n < 32).
__device__ __forceinline__ uint32_t low_bits(uint32_t n) {
#ifdef __CUDA_ARCH__
    uint32_t m;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(n));
    return m;
#else
    return (1u << n) - 1u;
#endif
}

// Spread entries written at the first slot of each code over the slots up to the next one (rows of 32).
__device__ __forceinline__ void fill_forward(uint32_t* tab, int n) {
    const int lane = threadIdx.x & 31;
    const uint32_t incl = 0xFFFFFFFFu >> (31 - lane);
    uint32_t carry = 0;
    for (int i = 0; i < n; i += 32) {
        const uint32_t v = tab[i + lane];
        const uint32_t below = __ballot_sync(FULL, v != 0) & incl;
        const uint32_t f = __shfl_sync(FULL, v, below ? 31 - __clz(below) : 0);
        const uint32_t x = below ? f : carry;
        tab[i + lane] = x;
        carry = __shfl_sync(FULL, x, 31);
    }
    __syncwarp();
}

// The decode tables of lens[0:nsym) (code lengths, at most 15; nsym <= 288, or 32 for distances), built
// by the whole warp.  Tables are indexed by code bits first bit highest, so a code's slots are adjacent:
// its entry is written at the first one and spread.  `limit` gets the first code longer than the root
// (left-justified to 15 bits; past all codes when there is none); the LNG entries after the root's are
// of 2^lsh codes each from there.  Acceptance as zlib's
// inflate: an over-subscribed code is an error, an incomplete one too unless its longest code has
// length 1.  Returns false on error (the same in every lane).
template <bool LIT>
__device__ __noinline__ bool build_tables(DecTables& W, const uint8_t* lens, int nsym, uint32_t& limit, uint32_t& lsh) {
    constexpr int NB = LIT ? 9 : 1, RB = LIT ? ROOT : DROOT;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* root = W.tab + (LIT ? 0u : DST);
    uint32_t* first = LIT ? W.lfirst : W.dfirst;
    uint32_t* index = LIT ? W.lindex : W.dindex;
    uint32_t* count = LIT ? W.lcount : W.dcount;
    if (lane < 16) count[lane] = 0;
    __syncwarp();
    uint32_t lr[NB];  // each symbol's code length, and its rank within the length
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const int s = b * 32 + lane;
        const uint32_t L = s < nsym ? lens[s] : 0u;
        const uint32_t peers = __match_any_sync(FULL, L);
        const uint32_t at = count[L];
        __syncwarp();
        if ((peers & lt) == 0) count[L] = at + __popc(peers);
        __syncwarp();
        lr[b] = L | ((at + __popc(peers & lt)) << 4);
    }
    const uint32_t cnt = lane >= 1 && lane < 16 ? count[lane] : 0u;
    uint32_t tot;
    // codes up to each length, left-justified (at most 288 << 14 < 2^23), and their number, in one sum
    const uint32_t before = warp_exclusive_scan(((lane < 16 ? cnt << (15 - lane) : 0u) << 9) | cnt, tot);
    const uint32_t total = tot >> 9;
    const int maxlen = 31 - __clz(__ballot_sync(FULL, cnt != 0) | 1u);
    if (total > 32768u || (total < 32768u && maxlen > 1)) return false;
    if (lane < 17) {
        first[lane] = lane < 16 ? before >> 9 : total;
        index[lane] = before & 511u;
    }
    const uint32_t lim = __shfl_sync(FULL, before >> 9, RB + 1);
    const uint32_t span = total - lim;
    limit = span ? lim : 32768u;
    lsh = span <= LNG ? 0u : 32u - (uint32_t)__clz((int)((span - 1) / LNG));
    const int slots = LIT ? (int)((span + (1u << lsh) - 1) >> lsh) : 0;  // at most LNG
    uint32_t* lng = W.tab + (1 << ROOT);
    for (int i = lane; i < (1 << RB); i += 32) root[i] = 0;
    for (int i = lane; i < ((slots + 31) & ~31); i += 32) lng[i] = 0;
    __syncwarp();
    const uint32_t lmax = 15 - lsh;  // longest code with slots of lng
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const uint32_t s = b * 32 + lane, L = lr[b] & 15u, r = lr[b] >> 4;
        if (L) {
            const uint32_t c = first[L] + (r << (15 - L));
            const uint32_t e = LIT ? lit_entry(s, L) : dist_entry(s, L);
            if (L <= (uint32_t)RB) {
                root[c >> (15 - RB)] = e;
            } else {
                (LIT ? W.lsym : W.dsym)[index[L] + r] = (uint16_t)s;
                if (LIT && L <= lmax) lng[(c - lim) >> lsh] = e;
            }
        }
    }
    if (lane == 0) {
        if (span) root[lim >> (15 - RB)] = SLOW;
        if (total < 32768u) root[total >> (15 - RB)] = LIT ? F_BAD | 1u : (SEQ_BAD << 16) | 1u;
        if (LIT && span && first[lmax + 1] < total) lng[(first[lmax + 1] - lim) >> lsh] = SLOW;
    }
    __syncwarp();
    fill_forward(root, 1 << RB);
    fill_forward(lng, (slots + 31) & ~31);
    return true;
}

// The entry of a code whose next 15 bits are c (first bit highest), found by the limits of the code
// lengths from L0 up.
template <bool LIT>
__device__ __noinline__ uint32_t long_entry(const DecTables& W, uint32_t c, uint32_t L0) {
    const uint32_t* first = LIT ? W.lfirst : W.dfirst;
    uint32_t L = L0;
    while (L < 15 && c >= first[L + 1]) L++;
    const uint32_t i = (LIT ? W.lindex : W.dindex)[L] + ((c - first[L]) >> (15 - L));
    if (c >= first[16] || i >= (LIT ? 288u : 32u)) return LIT ? F_BAD | 1u : (SEQ_BAD << 16) | 1u;
    return LIT ? lit_entry(W.lsym[i], L) : dist_entry(W.dsym[i], L);
}

// Word w of the input (words nvalid and up read as zero); block k: words 4k to 4k + 3.
__device__ __forceinline__ uint32_t load_word(const uint32_t* wbase, uint32_t nvalid, uint32_t w) {
    return w < nvalid ? __ldg(wbase + w) : 0u;
}
__device__ __forceinline__ uint4 load_block(const uint32_t* wbase, uint32_t nvalid, uint32_t k) {
    const uint32_t w = 4 * k;
    if (w + 3 < nvalid) return __ldg(reinterpret_cast<const uint4*>(wbase) + k);
    return make_uint4(load_word(wbase, nvalid, w), load_word(wbase, nvalid, w + 1), load_word(wbase, nvalid, w + 2),
                      load_word(wbase, nvalid, w + 3));
}

// The warp's reader of block headers: lane l holds word base + l of the input.
struct HeadBits {
    const uint32_t* wbase;
    uint32_t nvalid, base, word;
    __device__ __forceinline__ void at(uint32_t p) {  // words from bit p on
        base = p >> 5;
        word = load_word(wbase, nvalid, base + (threadIdx.x & 31));
    }
    __device__ __forceinline__ void cover(uint32_t p) {  // at least the 96 bits from p on
        if ((p >> 5) - base > 28u) at(p);
    }
    __device__ __forceinline__ uint32_t get(uint32_t p) const {  // 32 bits from bit p (per lane) on
        const uint32_t w = (p >> 5) - base;
        return __funnelshift_r(__shfl_sync(FULL, word, w), __shfl_sync(FULL, word, w + 1), p);
    }
};

// The code lengths of a dynamic block whose header fields start at bit p (after the three header bits),
// into lens; p is left after them.  The 32 lanes decode the code at 32 bit positions at once; which of
// those are symbols follows from the chain that starts at the first (pointer doubling).  Returns
// literal/length codes | all codes << 16, or 0 on error.
__device__ __noinline__ uint32_t read_lengths(DecTables& W, HeadBits& hb, uint32_t& p, uint8_t* lens, uint32_t* tab4) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    hb.cover(p);
    const uint32_t h = hb.get(p);
    const uint32_t hlit = (h & 31u) + 257, hdist = ((h >> 5) & 31u) + 1, hclen = ((h >> 10) & 15u) + 4;
    p += 14;
    if (hlit > 286 || hdist > 30) return 0;
    // the code-length code: lane s its symbol's length and code (left-justified to 7 bits)
    uint8_t* cl = reinterpret_cast<uint8_t*>(W.lcount);
    if (lane < 16) W.lcount[lane] = 0;
    for (int i = lane; i < 80; i += 32) reinterpret_cast<uint32_t*>(lens)[i] = 0;
    __syncwarp();
    hb.cover(p);
    const uint32_t x3 = hb.get(p + 3 * (lane < 19 ? lane : 0)) & 7u;
    if (lane < (int)hclen) cl[kClOrder[lane]] = (uint8_t)x3;
    p += 3 * hclen;
    __syncwarp();
    const uint32_t L = lane < 19 ? cl[lane] : 0u;
    const uint32_t space = L ? 128u >> L : 0u;
    uint32_t code = 0;
    for (int t = 0; t < 19; t++) {
        const uint32_t Lt = __shfl_sync(FULL, L, t);
        if (Lt && (Lt < L || (Lt == L && t < lane))) code += 128u >> Lt;
    }
    if (__reduce_add_sync(FULL, space) != 128u) return 0;
    // tab: 128 entries of a byte: length << 5 | symbol, never 0
    uint8_t* tab = reinterpret_cast<uint8_t*>(tab4);
    tab4[lane] = 0;
    __syncwarp();
    if (L) tab[code] = (uint8_t)((L << 5) | lane);
    __syncwarp();
    {  // spread each entry up to the next one, four slots per lane
        uint32_t v = tab4[lane];
        const uint32_t last = v >> 24 ? v >> 24 : (v >> 16) & 255u ? (v >> 16) & 255u : (v >> 8) & 255u ? (v >> 8) & 255u : v & 255u;
        const uint32_t below = __ballot_sync(FULL, v != 0) & lt;
        uint32_t c = __shfl_sync(FULL, last, below ? 31 - __clz(below) : 0);
        uint32_t y = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t b = (v >> (8 * k)) & 255u;
            c = b ? b : c;
            y |= c << (8 * k);
        }
        tab4[lane] = y;
    }
    __syncwarp();
    const uint32_t total = hlit + hdist;
    uint32_t ci = 0, last = 0;
    while (ci < total) {
        hb.cover(p);
        const uint32_t x = hb.get(p + lane);
        const uint32_t t = tab[__brev(x) >> 25];
        const uint32_t CL = t >> 5, s = t & 31u;
        const uint32_t eb = s < 16 ? 0u : s == 16 ? 2u : s == 17 ? 3u : 7u;
        const uint32_t n = CL + eb;
        const uint32_t ext = (x >> CL) & ((1u << eb) - 1u);
        // the symbols: positions reached from lane 0
        uint32_t reach = 1u << lane, nx = lane + n;
#pragma unroll
        for (int r = 0; r < 5; r++) {
            const uint32_t orr = __shfl_sync(FULL, reach, nx & 31u), onx = __shfl_sync(FULL, nx, nx & 31u);
            if (nx < 32) {
                reach |= orr;
                nx = onx;
            }
        }
        reach = __shfl_sync(FULL, reach, 0);
        const uint32_t exit = __shfl_sync(FULL, nx, 0);
        const bool on = (reach >> lane) & 1u;
        const uint32_t rep = !on ? 0u : s < 16 ? 1u : (s == 18 ? 11u : 3u) + ext;
        uint32_t tot;
        const uint32_t pos = ci + warp_exclusive_scan(rep, tot);
        const bool act = on && pos < total;
        if (__any_sync(FULL, act && (pos + rep > total || (s == 16 && pos == 0)))) return 0;
        // a repeat copies the length before it: the nearest earlier symbol that is not one
        const uint32_t own = __ballot_sync(FULL, act && s != 16);
        const uint32_t sv = s < 16 ? s : 0u;
        const uint32_t prior = own & lt;
        const uint32_t pv = __shfl_sync(FULL, sv, prior ? 31 - __clz(prior) : 0);
        const uint32_t v = s != 16 ? sv : prior ? pv : last;
        if (act && v)  // lengths start at zero
            for (uint32_t r = 0; r < rep; r++) lens[pos + r] = (uint8_t)v;
        last = own ? __shfl_sync(FULL, sv, 31 - __clz(own)) : last;
        if (ci + tot >= total) {
            const uint32_t end = __ballot_sync(FULL, act && pos + rep == total);
            p = __shfl_sync(FULL, p + lane + n, __ffs(end) - 1);
        } else {
            p += exit;
        }
        ci += tot;
    }
    __syncwarp();
    if (lens[256] == 0) return 0;  // no end-of-block code
    return hlit | (total << 16);
}

// What a lane has decoded of its segment.
struct LaneOut {
    uint32_t nl, ns, lc;   // literals, sequences, literals since the last sequence
    uint32_t fl, fs;       // stored in the slot so far
    uint32_t stop;         // 0, 1 at an end-of-block code, 2 at an invalid code
    bool over;             // more than the run holds (counted on, not stored)
};

// Store 16 staged literals or 4 staged sequences to the lane's run (cap bytes: literals from its start up,
// sequences from its end down), when it holds them.  fl and fs are multiples of 16 and 4.
__device__ __forceinline__ void store_lits(const DecWarp& W, LaneOut& o, uint8_t* run, uint32_t cap) {
    const uint32_t* c = W.lst + (threadIdx.x & 31) * (LSTAGE / 4 + 1) + ((o.fl & (LSTAGE - 1)) >> 2);
    if (16 + o.fl + 4 * o.fs > cap) o.over = true;
    if (!o.over) *reinterpret_cast<uint4*>(run + o.fl) = make_uint4(c[0], c[1], c[2], c[3]);
    o.fl += 16;
}
__device__ __forceinline__ void store_seqs(const DecWarp& W, LaneOut& o, uint8_t* run, uint32_t cap) {
    const uint32_t* c = W.sst + (threadIdx.x & 31) * (SSTAGE + 1) + (o.fs & (SSTAGE - 1));
    o.fs += 4;
    if (o.fl + 4 * o.fs > cap) o.over = true;
    if (!o.over) *reinterpret_cast<uint4*>(run + cap - 4 * o.fs) = make_uint4(c[3], c[2], c[1], c[0]);
}

// A lane's input: 16 words in its column; the block after them is loaded a round ahead.
struct LaneIn {
    const uint32_t* wbase;
    uint32_t nvalid, fill;  // words up to fill are in the column
    bool coming;            // next is being loaded
    uint4 next;
};
__device__ __forceinline__ void put_block(uint32_t* col, uint32_t fill, uint4 v) {
    uint32_t* c = col + (fill & (ROWS - 1)) * 32;
    c[0] = v.x;
    c[32] = v.y;
    c[64] = v.z;
    c[96] = v.w;
    if ((fill & (ROWS - 1)) == 0) {
        col[ROWS * 32] = v.x;
        col[(ROWS + 1) * 32] = v.y;
    }
}
__device__ __forceinline__ void start_input(LaneIn& in, uint32_t* col, uint32_t p) {
    const uint32_t k = p >> 7;
    const uint4 a = load_block(in.wbase, in.nvalid, k), b = load_block(in.wbase, in.nvalid, k + 1),
                c = load_block(in.wbase, in.nvalid, k + 2);
    put_block(col, 4 * k, a);
    put_block(col, 4 * k + 4, b);
    put_block(col, 4 * k + 8, c);
    in.fill = 4 * k + 12;
    in.coming = false;
}
// Take the block that was loaded and load the next one when there is room for it; returns the bit up to
// which steps may start (a step reads three words).
__device__ __forceinline__ uint32_t refill(LaneIn& in, uint32_t* col, uint32_t p) {
    if (in.coming) {
        put_block(col, in.fill, in.next);
        in.fill += 4;
    }
    in.coming = in.fill - (p >> 5) <= ROWS - 4;
    if (in.coming) in.next = load_block(in.wbase, in.nvalid, in.fill >> 2);
    return (in.fill - 2) * 32;
}

// A symbol whose codes the tables do not resolve or that takes more than 32 bits (rare): x its first 32
// bits, hi the next ones.  Returns its bits; e, d: its entries, y: the bits after the literal/length.
__device__ __noinline__ uint32_t slow_symbol(const DecTables& W, uint32_t x, uint32_t hi, uint32_t lsh, uint32_t& e,
                                             uint32_t& d, uint32_t& y) {
    if ((e & 63u) == 32u) e = long_entry<true>(W, __brev(x) >> 17, 15 - lsh);
    const uint32_t n = e & 63u;
    y = __funnelshift_r(x, hi, n);
    d = W.tab[DST + (__brev(y) >> (32 - DROOT))];
    if ((d & 63u) == 32u) d = long_entry<false>(W, __brev(y) >> 17, DROOT + 1);
    return n + (e & F_MATCH ? d & 63u : 0u);
}

// One symbol at bit p of the lane's input, or two literals when the second one's code is in the root table
// and starts below `end` (so that segments end at the same symbols whatever was taken together); p moves
// past them.  With STORE they are staged and the lane stops at an end-of-block or invalid code (end
// becomes 0); without, every code is passed over.  Literals and matches take the same path (a warp has
// both at nearly every step): one access to the tables gives a match's distance code or the second
// literal.  lim: where the codes longer than the root begin; lim2: the table index of the first of them, as
// lim - (index << lsh).
template <bool STORE>
__device__ __forceinline__ void decode_step(const DecTables& T, DecWarp& W, uint32_t* col, uint32_t& p, uint32_t& end, uint32_t lim,
                                            uint32_t lim2, uint32_t lsh, LaneOut& o) {
    const uint32_t* r = col + ((p >> 5) & (ROWS - 1)) * 32;
    const uint32_t w0 = r[0], w1 = r[32];
    const uint32_t x = __funnelshift_r(w0, w1, p);
    const uint32_t c = __brev(x) >> 17;
    uint32_t e = T.tab[c >= lim ? (c - lim2) >> lsh : c >> (15 - ROOT)];
    uint32_t y = __funnelshift_r(x, 0u, e);  // shifts by bits 0-4
    const uint32_t cy = __brev(y), n = e & 63u;
    uint32_t d = T.tab[e & F_MATCH ? DST + (cy >> (32 - DROOT)) : cy >> (32 - ROOT)];
    const bool lit2 = e < F_BAD && d < F_BAD && p + n < end;
    uint32_t t = n + (lit2 || (e & F_MATCH) ? d & 63u : 0u);
    if (t >= 32) t = slow_symbol(T, x, __funnelshift_r(w1, r[64], p), lsh, e, d, y);
    p += t;
    if (STORE) {
        const int lane = threadIdx.x & 31;
        const bool match = (e & F_MATCH) != 0, lit = e < F_BAD;
        const uint32_t len3 = ((e >> 16) & 255u) + __funnelshift_r(x & low_bits(e & 31u), 0u, e >> 6);
        const uint32_t dist = (d >> 16) + __funnelshift_r(y & low_bits(d & 31u), 0u, d >> 6);
        const uint32_t q = (o.lc << 24) | (len3 << 16) | dist;
        if (match) W.sst[lane * (SSTAGE + 1) + (o.ns & (SSTAGE - 1))] = q;
        uint8_t* l = reinterpret_cast<uint8_t*>(W.lst) + lane * (LSTAGE + 4);
        if (lit) l[o.nl & (LSTAGE - 1)] = (uint8_t)(e >> 16);
        if (lit2) l[(o.nl + 1) & (LSTAGE - 1)] = (uint8_t)(d >> 16);
        const uint32_t k = (uint32_t)lit + lit2;
        o.nl += k;
        o.ns += match;
        o.lc = match ? 0u : o.lc + k;
        if (e & (F_EOB | F_BAD)) {
            o.stop = e & F_BAD ? 2u : 1u;
            end = 0;
        }
    }
}

// Barrier and vote over a member's W warps (W == 1: a CTA may hold several members).
template <int W> __device__ __forceinline__ void sync_member() {
    if (W == 1) __syncwarp();
    else __syncthreads();
}
template <int W> __device__ __forceinline__ bool any_of_member(bool x) {
    return W == 1 ? __any_sync(FULL, x) != 0 : __syncthreads_or(x) != 0;
}

// Exclusive sums over the member's threads of two values; their totals in ta and tb.
template <int W>
__device__ __forceinline__ void cta_scan2(DecMember<W>& M, uint32_t& a, uint32_t& b, uint32_t& ta, uint32_t& tb) {
    const int warp = threadIdx.x >> 5;
    a = warp_exclusive_scan(a, ta);
    b = warp_exclusive_scan(b, tb);
    if (W == 1) return;
    if ((threadIdx.x & 31) == 0) {
        M.sums[0][warp] = ta;
        M.sums[1][warp] = tb;
    }
    __syncthreads();
    ta = tb = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
        if (w == warp) {
            a += ta;
            b += tb;
        }
        ta += M.sums[0][w];
        tb += M.sums[1][w];
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t run_byte(const uint8_t* p) { return __ldcg(p); }

// Move a run of n literals and k sequences (cap bytes) to dl and down from ds, by one warp: its loads are
// issued ahead of its stores, eight words of each per lane.
__device__ __forceinline__ void move_run(const uint8_t* run, uint32_t cap, uint32_t n, uint32_t k, uint8_t* dl,
                                         uint32_t* ds) {
    constexpr uint32_t U = 8;
    const uint32_t lane = threadIdx.x & 31, h = min(n, (uint32_t)(-(intptr_t)dl & 3));
    const uint32_t nw = (n - h) >> 2, tail = (n - h) & 3u;
    const uint32_t* lw = reinterpret_cast<const uint32_t*>(run);
    const uint32_t* sq = reinterpret_cast<const uint32_t*>(run + cap) - 1;
    uint32_t* d = reinterpret_cast<uint32_t*>(dl + h);
    // byte h + 4 i on of the literals in word i, and the head's and tail's bytes
    const uint32_t hb = lane < h ? run_byte(run + lane) : 0u;
    const uint32_t tb = lane < tail ? run_byte(run + n - tail + lane) : 0u;
    for (uint32_t i0 = 0; i0 < k || i0 < nw; i0 += 32 * U) {
        uint32_t q[U], a[U], b[U];
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            const uint32_t i = i0 + 32 * u + lane;
            q[u] = i < k ? __ldcg(sq - i) : 0u;
            a[u] = i < nw ? __ldcg(lw + i) : 0u;
            b[u] = i < nw && h ? __ldcg(lw + i + 1) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            const uint32_t i = i0 + 32 * u + lane;
            if (i < k) ds[-(int)i] = q[u];
            if (i < nw) d[i] = __funnelshift_r(a[u], b[u], 8 * h);
        }
    }
    if (lane < h) dl[lane] = (uint8_t)hb;
    if (lane < tail) dl[n - tail + lane] = (uint8_t)tb;
}

// Write n bytes to any dst, by one warp: word(i, h) gives the source's bytes h + 4 i to h + 4 i + 3, of which
// h = 0 to 3 are before dst's first whole word.
template <class F> __device__ __forceinline__ void put_bytes(uint8_t* dst, uint32_t n, F word) {
    const uint32_t lane = threadIdx.x & 31, h = min(n, (uint32_t)(-(intptr_t)dst & 3));
    if (lane < h) dst[lane] = (uint8_t)(word(0, 0) >> (8 * lane));
    const uint32_t nw = (n - h) >> 2, tail = (n - h) & 3u;
    uint32_t* d = reinterpret_cast<uint32_t*>(dst + h);
    for (uint32_t i = lane; i < nw; i += 32) d[i] = word(i, h);
    if (lane < tail) dst[n - tail + lane] = (uint8_t)(word(nw, h) >> (8 * lane));
}

// The Huffman-coded symbols of one block from bit p0 on, added to the nl literals and ns sequences in the
// member's slot, by the whole CTA; p0, nl and ns are left after them.  scratch: scratch_n bytes, 16-byte
// aligned, for the lanes' runs before they are put together.  CB_OK, CB_ERR_INFLATE or ST_LISTED (they do
// not fit the slot), the same in every thread.
template <int W>
__device__ uint32_t decode_block(DecMember<W>& M, LaneIn& in, uint32_t& p0, uint32_t E, uint8_t* slot, uint32_t slot_n,
                                 uint32_t& nl, uint32_t& ns, uint8_t* scratch, uint32_t scratch_n, uint32_t limit,
                                 uint32_t lsh) {
    constexpr uint32_t T = 32 * W;
    const uint32_t tid = threadIdx.x % T, lane = tid & 31;
    DecWarp& D = M.w[tid >> 5];
    uint32_t* col = D.in + lane;
    const uint32_t lim2 = limit - ((1u << ROOT) << lsh);
    const uint32_t most = max(1u, min(T, scratch_n / RUN_MIN));  // lanes with room for a run
    for (;;) {  // windows of up to T segments
        if (p0 >= E) return CB_ERR_INFLATE;
        const uint32_t R = E - p0;
        const uint32_t seg = max(SEG_MIN, (min(R, WINDOW) + most - 1) / most);
        const uint32_t A = min(most, (R + seg - 1) / seg);
        const uint32_t b0 = p0 + tid * seg, b1 = min(b0 + seg, E);
        const bool act = tid < A;
        LaneOut o;
        uint32_t p = tid * seg <= OVERLAP ? p0 : b0 - OVERLAP;
        if (act) start_input(in, col, p);
        __syncwarp();
        {
            const uint32_t end = act ? b0 : 0u;
            while (__any_sync(FULL, p < end)) {
                uint32_t to = 0;
                if (p < end) to = min(end, refill(in, col, p));
#pragma unroll 1
                for (int k = 0; k < STEPS; k++)
                    if (p < to) decode_step<false>(M.t, D, col, p, to, limit, lim2, lsh, o);
            }
        }
        uint32_t s = p;  // the first symbol of the lane's segment
        if (act) start_input(in, col, p);  // (decoded again from there, a segment gives the same sequences)
        const uint32_t cap = (scratch_n / A) & ~15u;
        uint8_t* run = scratch + tid * cap;
        bool need = act, direct = false;
        uint32_t F, al, as, tl, ts, my_l, my_s;
        o.stop = 0;
        for (;;) {
            uint32_t end = 0;
            if (need) {
                o.nl = o.ns = o.lc = o.fl = o.fs = o.stop = 0;
                o.over = false;
                end = b1;
            }
            while (__any_sync(FULL, p < end)) {
                uint32_t to = 0;
                if (p < end) to = min(end, refill(in, col, p));
#pragma unroll 1
                for (int k = 0; k < STEPS; k++)
                    if (p < to) decode_step<true>(M.t, D, col, p, to, limit, lim2, lsh, o);
                if (need) {
                    if (o.stop) end = 0;
                    if (!direct) {
                        while (o.nl - o.fl >= 16) store_lits(D, o, run, cap);
                        while (o.ns - o.fs >= 4) store_seqs(D, o, run, cap);
                    }
                    // a sequence's literal count has 8 bits; the literals after the last match have one of their own
                    if (o.lc > LC_MAX || (p >= end && o.lc)) {
                        D.sst[lane * (SSTAGE + 1) + (o.ns & (SSTAGE - 1))] = o.lc << 24;
                        o.ns++;
                        o.lc = 0;
                    }
                    if (direct) {  // to their places, one by one (rare)
                        for (; o.fl < o.nl && o.fl < my_l; o.fl++)
                            slot[nl + al + o.fl] =
                                reinterpret_cast<const uint8_t*>(D.lst)[lane * (LSTAGE + 4) + (o.fl & (LSTAGE - 1))];
                        for (; o.fs < o.ns && o.fs < my_s; o.fs++)
                            reinterpret_cast<uint32_t*>(slot + slot_n)[-1 - (int)(ns + as + o.fs)] =
                                D.sst[lane * (SSTAGE + 1) + (o.fs & (SSTAGE - 1))];
                    } else if (o.ns - o.fs >= 4 || (p >= end && o.ns > o.fs)) {
                        store_seqs(D, o, run, cap);
                    }
                    if (p >= end) {
                        need = false;
                        if (!direct && o.nl > o.fl) store_lits(D, o, run, cap);
                    }
                }
            }
            // every segment up to the block's end must begin where the one before it ended
            M.ends[tid] = p | (act ? o.stop << 30 : 0u);
            sync_member<W>();
            F = A - 1;
            for (uint32_t w = 0; w < T && w < A; w += 32) {
                const uint32_t stopped = __ballot_sync(FULL, M.ends[w + lane] >> 30);
                if (stopped) {
                    F = w + __ffs((int)stopped) - 1;
                    break;
                }
            }
            const uint32_t pe = tid ? M.ends[tid - 1] & BITS : p0;
            need = tid > 0 && tid <= F && s != pe;
            if (any_of_member<W>(need)) {
                if (need) s = p = pe;
            } else {
                if (direct) break;
                my_l = al = tid <= F ? o.nl : 0u;
                my_s = as = tid <= F ? o.ns : 0u;
                cta_scan2<W>(M, al, as, tl, ts);
                direct = any_of_member<W>(tid <= F && o.over);  // some run was too short: decode them again
                if (!direct || nl + tl + 4ull * ((unsigned long long)ns + ts) > slot_n) break;
                need = tid <= F;
                p = s;
            }
            if (need) start_input(in, col, p);
            __syncwarp();
        }
        const uint32_t stop = M.ends[F] >> 30;
        p0 = M.ends[F] & BITS;
        if (stop == 2 || p0 > E) return CB_ERR_INFLATE;
        if (nl + tl + 4ull * ((unsigned long long)ns + ts) > slot_n) return ST_LISTED;
        if (!direct) {
            // the runs, one after another, to the slot: each warp its lanes'
            const uint32_t w0 = tid & ~31u;
            for (uint32_t r = 0; r < 32 && w0 + r <= F; r++) {
                const uint32_t n = __shfl_sync(FULL, my_l, r), k = __shfl_sync(FULL, my_s, r);
                const uint32_t dl = nl + __shfl_sync(FULL, al, r), ds = ns + __shfl_sync(FULL, as, r);
                move_run(scratch + (w0 + r) * cap, cap, n, k, slot + dl, reinterpret_cast<uint32_t*>(slot + slot_n) - 1 - ds);
            }
        }
        nl += tl;
        ns += ts;
        sync_member<W>();  // the next window writes scratch and ends
        if (stop) return CB_OK;
    }
}

// One member's symbols into its slot, by the whole CTA, with scratch_n bytes of scratch.  CB_OK, CB_ERR_INFLATE or
// ST_LISTED, the same in every thread.
template <int W>
__device__ uint32_t decode_member(DecMember<W>& M, const cb_member_job& job, uint8_t* slot, uint8_t* scratch,
                                  uint32_t scratch_n, uint32_t& nl, uint32_t& ns) {
    const uint32_t tid = threadIdx.x % (32 * W), lane = tid & 31, warp = tid >> 5;
    LaneIn in;
    const uintptr_t src = (uintptr_t)job.in;
    in.wbase = reinterpret_cast<const uint32_t*>(src & ~(uintptr_t)15);
    in.nvalid = (uint32_t)((src + job.in_len + 8 - (uintptr_t)in.wbase) >> 2);
    uint32_t p = (uint32_t)(src & 15) * 8;
    const uint32_t s0 = p, E = p + job.in_len * 8u;
    const uint32_t slot_n = (uint32_t)slot_bytes(job.isize);
    uint8_t* lens = reinterpret_cast<uint8_t*>(M.w[0].lst);
    nl = ns = 0;
    if (!in_reach(job.in_len, job.isize)) return ST_LISTED;
    for (;;) {
        if (p > E) return CB_ERR_INFLATE;
        if (warp == 0) {  // the block's header, and its code lengths
            HeadBits hb;
            hb.wbase = in.wbase;
            hb.nvalid = in.nvalid;
            hb.at(p);
            const uint32_t h = hb.get(p), btype = (h >> 1) & 3u;
            uint32_t q = p + 3, a = 288, b = 32, bad = btype == 3;
            if (btype == 0) {
                q = s0 + ((q - s0 + 7) & ~7u);
                const uint32_t y = hb.get(q);
                q += 32;
                a = y & 0xFFFFu;
                bad = a != (~y >> 16) || q > E || 8ull * a > E - q;
            } else if (btype == 1) {
                for (int i = lane; i < 320; i += 32) lens[i] = i < 144 ? 8 : i < 256 ? 9 : i < 280 ? 7 : i < 288 ? 8 : 5;
            } else if (btype == 2) {
                const uint32_t r = read_lengths(M.t, hb, q, lens, M.w[0].sst);
                bad = r == 0;
                a = r & 0xFFFFu;
                b = (r >> 16) - a;
            }
            if (lane == 0) {
                M.t.say[0] = h & 7u;
                M.t.say[1] = q;
                M.t.say[2] = a;
                M.t.say[3] = b;
                M.t.say[4] = bad;
            }
        }
        sync_member<W>();
        const uint32_t h = M.t.say[0], na = M.t.say[2], nb = M.t.say[3];
        p = M.t.say[1];
        const bool final_block = h & 1u;
        if (M.t.say[4]) return CB_ERR_INFLATE;
        if ((h >> 1) == 0) {
            const uint32_t k = (na + 254) / 255;
            if (nl + na + 4ull * ((unsigned long long)ns + k) > slot_n) return ST_LISTED;
            // stored bytes, a part per warp
            const uint32_t part = ((na + W - 1) / W + 3) & ~3u, from = min(na, warp * part), n = min(na, from + part) - from;
            const uint32_t pb = p + 8 * from;
            put_bytes(slot + nl + from, n, [&](uint32_t i, uint32_t h2) {
                const uint32_t bit = pb + 8 * (4 * i + h2), w = bit >> 5;
                return __funnelshift_r(load_word(in.wbase, in.nvalid, w), load_word(in.wbase, in.nvalid, w + 1), bit);
            });
            for (uint32_t i = tid; i < k; i += 32 * W)
                reinterpret_cast<uint32_t*>(slot + slot_n)[-1 - (int)(ns + i)] = min(255u, na - 255 * i) << 24;
            p += 8 * na;
            nl += na;
            ns += k;
            sync_member<W>();  // say is written again
        } else {
            uint32_t limit, lsh;
            if (warp == 0) {
                const bool ok = build_tables<true>(M.t, lens, (int)na, limit, lsh);
                if (lane == 0) {
                    M.t.say[5] = ok;
                    M.t.say[6] = limit;
                    M.t.say[7] = lsh;
                }
            }
            if (warp == (W > 1 ? 1u : 0u)) {
                uint32_t dl, dsh;
                const bool ok = build_tables<false>(M.t, lens + na, (int)nb, dl, dsh);
                if (lane == 0) M.t.say[8] = ok;
            }
            sync_member<W>();
            limit = M.t.say[6];
            lsh = M.t.say[7];
            if (!M.t.say[5] || !M.t.say[8]) return CB_ERR_INFLATE;
            const uint32_t st = decode_block<W>(M, in, p, E, slot, slot_n, nl, ns, scratch, scratch_n, limit, lsh);
            if (st != CB_OK) return st;
        }
        if (final_block) return p > E ? (uint32_t)CB_ERR_INFLATE : (uint32_t)CB_OK;
    }
}

template <int W>
__global__ void __launch_bounds__(W == 1 ? 64 : W * 32, W == 1 ? 9 : 16 / W)
    k_decode(const cb_member_job* __restrict__ jobs, int64_t n_jobs, const int64_t* __restrict__ d_n_jobs,
             uint32_t* job_status, cb_inflate_summary* summary, uint8_t* ws, uint8_t* arena,
             unsigned long long arena_bytes, uint8_t* scratch, uint32_t scratch_n, bool list_unfit, long long j0, long long j1,
             int qi) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    constexpr int MEMBERS = W == 1 ? 2 : 1;  // per CTA
    scratch += (unsigned long long)(blockIdx.x * MEMBERS + threadIdx.x / (32 * W)) * scratch_n;
    DecMember<W>& M = reinterpret_cast<DecMember<W>*>(smem_raw)[threadIdx.x / (32 * W)];
    const bool first = threadIdx.x % (32 * W) == 0;
    unsigned long long* queue = reinterpret_cast<unsigned long long*>(ws);
    uint32_t* per_job = reinterpret_cast<uint32_t*>(ws + WS_HEAD);
    long long n = n_jobs;
    if (d_n_jobs) n = min((long long)n, (long long)*d_n_jobs);
    n = min(n, j1);  // this launch's jobs: [j0, j1)
    for (;;) {
        if (first) M.t.job = atomicAdd(queue + qi, 1ull);
        sync_member<W>();
        const long long j = j0 + (long long)M.t.job;
        if (j >= n) break;
        const cb_member_job job = jobs[j];
        const unsigned long long so = reinterpret_cast<const unsigned long long*>(per_job)[(JW / 2) * j + 1];
        uint32_t nl = 0, ns = 0;
        const uint32_t st = so + slot_bytes(job.isize) <= arena_bytes
                                ? decode_member<W>(M, job, arena + so, scratch, scratch_n, nl, ns)
                            : list_unfit ? ST_LISTED
                                         : (uint32_t)CB_ERR_CAPACITY;
        sync_member<W>();
        if (first) {
            per_job[JW * j + 1] = st;
            per_job[JW * j + 4] = nl;
            per_job[JW * j + 5] = ns;
            if (st == ST_LISTED) per_job[JW * atomicAdd(queue + Q_LISTED, 1ull)] = (uint32_t)j;
            else report(summary, job_status, j, st);
        }
    }
}

// ---------------------------------------------------------------- k_literals: members without a match
// Members of literals alone (stored blocks, or codes without matches) from their slots to their places, before k_copy,
// which takes literals in groups of a few sequences of at most 255 and most of them byte by byte: in us, all of form 3
// without this kernel and with it, of members of 65 KB of stored blocks: 3,000 1448 769, 20,000 7808 2724.  (In k_copy or
// k_decode itself the code for it cost all other members 1 to 16%, in k_crc 3%.)  A CTA looks at LOOK members at a time, 64
// bytes each, and its two warps take those it finds; it is small, to find room beside the other range's kernels.
constexpr int LOOK = 8;
__global__ void __launch_bounds__(64) k_literals(const cb_member_job* __restrict__ jobs, int64_t n_jobs,
                                                  const int64_t* __restrict__ d_n_jobs, uint8_t* out_base, uint8_t* ws,
                                                  const uint8_t* arena, long long j0, long long j1) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* per_job = reinterpret_cast<uint32_t*>(ws + WS_HEAD);
    long long n = n_jobs;
    if (d_n_jobs) n = min((long long)n, (long long)*d_n_jobs);
    n = min(n, j1);
    for (long long jb = j0 + (long long)LOOK * blockIdx.x; jb < n; jb += (long long)LOOK * gridDim.x) {
        bool found = false;
        if (lane < LOOK && jb + lane < n) {
            const uint32_t st = *reinterpret_cast<volatile uint32_t*>(per_job + JW * (jb + lane) + 1);
            // (another warp may have copied it)
            found = (st == CB_OK || st == ST_LITERALS) && per_job[JW * (jb + lane) + 4] == jobs[jb + lane].isize;
        }
        const uint32_t all = __ballot_sync(FULL, found);
        for (uint32_t left = all, k = 0; left; left &= left - 1, k++) {
            if (k % 2 != warp) continue;
            const long long j = jb + __ffs((int)left) - 1;
            const uint32_t isize = jobs[j].isize, ns = per_job[JW * j + 5];
            const uint8_t* lits = arena + reinterpret_cast<const unsigned long long*>(per_job)[(JW / 2) * j + 1];
            const uint32_t* sq = reinterpret_cast<const uint32_t*>(lits + slot_bytes(isize)) - 1;
            uint32_t more = 0;
            for (uint32_t i = lane; i < ns; i += 32) more |= __ldcg(sq - i) & 0xFFFFFFu;
            if (__any_sync(FULL, more != 0)) continue;  // a match, of no valid distance
            copy_long<32, 2>(lits, out_base + jobs[j].out_off, (int)isize, lane);
            if (lane == 0) per_job[JW * j + 1] = ST_LITERALS;
        }
    }
}

// ---------------------------------------------------------------- k_copy: one member per CTA of W warps

constexpr uint32_t LINE = 128;            // output bytes of a warp's round: a word per lane
constexpr uint32_t FAR_WORDS = 8, FAR_LEN = 4 * FAR_WORDS - 3;  // of a fetched source, at most

// A group's tokens are the literal runs and matches of its sequences, numbered 4 t + 1 to 4 t + 4 for thread
// t's two (so numbers rise along the output).  tok: above bit 16 what to add to a byte's place (from the
// group's first line) to get its source's offset from the ring's start in shared memory; T_NEAR: a match
// closer than a round, some of whose bytes may have their source in the same round, with its distance in
// bits 0-11 (all ones in other tokens: far from any round).  The few tokens with T_WRAP (a source across the
// ring's end) or T_DIRECT (one read from HBM: a literal with T_PLAIN) find it through aux: the distance above
// bit 16 and the start, or for T_PLAIN what to add to get a literal's place in the slot.
constexpr uint32_t T_WRAP = 1u << 12, T_DIRECT = 1u << 13, T_PLAIN = 1u << 14, T_NEAR = 1u << 15, T_FAR = 0xFFFu;
constexpr uint32_t T_FLAGS = T_NEAR | T_WRAP | T_DIRECT;

// RING_: bytes of output kept in shared memory: sources up to RING_ - GMAX - SPAN bytes back read it, older
// ones the output already stored.
template <uint32_t RING_, int W_>
struct CopyCfg {
    static constexpr int W = W_;
    static constexpr uint32_t T = 32 * W_, RING = RING_, RMASK = RING_ - 1;
    static constexpr uint32_t SPAN = LINE * W_;   // output bytes of a round of all warps
    static constexpr uint32_t GMAX = 1152 * W_;   // output bytes of a group of 64 sequences per warp, at most
    static constexpr uint32_t FAR_N = W_ == 8 ? 32 : 40;  // sources fetched from HBM per warp and group
    static constexpr uint32_t LITS = 256 * W_;    // literals of a group held in shared memory
    static_assert((RING_ & (RING_ - 1)) == 0 && RING_ >= GMAX + 2 * SPAN + 512 && RING_ <= 16384, "ring size");
    static_assert(GMAX >= 2 * (255 + 258), "two sequences fit a group");
    static_assert(2 * SPAN < T_FAR && 4 * T < 65536, "a token's number and a near distance have their bits");
    using Id = typename std::conditional<W_ == 1, uint8_t, uint16_t>::type;
    struct alignas(16) Smem {
        uint8_t ring[RING_];
        uint32_t lit[LITS / 4];           // the group's first literals
        uint32_t far[W_][2][FAR_N * FAR_WORDS];  // fetched sources of this group and the next
        uint32_t tok[4 * T + 4], aux[4 * T + 4];
        alignas(8) Id map[GMAX + SPAN];   // per byte of the group's lines: the number of the token that starts there
        uint16_t head[(GMAX + SPAN) / LINE + 1];  // W > 1: per line, the token of its first byte
        uint8_t missing[T];               // W > 1: per word of a round, the bytes that wait for others
        unsigned long long sums[W_], job;
        uint32_t count[W_];
    };
};

// Copy the 4 bytes at src to dst in shared memory without waiting, and wait for this thread's copies.
__device__ __forceinline__ void copy_async4(uint32_t* dst, const uint8_t* src) {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
#else
    *dst = *reinterpret_cast<const uint32_t*>(src);
#endif
}
__device__ __forceinline__ void wait_async() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.wait_all;\n" ::: "memory");
#endif
}

// All ones, shifted left by n (0 from 32 on).
__device__ __forceinline__ uint32_t shl_clamp(uint32_t n) { return __funnelshift_lc(0u, 0xFFFFFFFFu, n); }

// Positions below are slots: bytes from the 128-byte line of the member's first output byte (a bytes
// before it).  A group is 64 sequences per warp, two per thread.  Its output is written in rounds of one
// line per warp, a word per lane: each byte of the word belongs to the last token that starts at or before
// it.
template <class C>
__global__ void __launch_bounds__(C::T, C::W == 1 ? 28 : 1)
    k_copy(const cb_member_job* __restrict__ jobs, int64_t n_jobs, const int64_t* __restrict__ d_n_jobs,
           uint8_t* out_base, uint32_t* job_status, cb_inflate_summary* summary, uint8_t* ws,
           const uint8_t* arena, long long j0, long long j1, int qi) {
    constexpr int W = C::W;
    constexpr uint32_t T = C::T;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    typename C::Smem& M = *reinterpret_cast<typename C::Smem*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint8_t* smem = M.ring;
    uint32_t* ring4 = reinterpret_cast<uint32_t*>(M.ring);
    const uint32_t LIT_AT = (uint32_t)(reinterpret_cast<const uint8_t*>(M.lit) - smem);
    const uint32_t FAR_AT = (uint32_t)(reinterpret_cast<const uint8_t*>(M.far[warp]) - smem);
    constexpr uint32_t NOT_OLD = 255, FAR_N = C::FAR_N;
    unsigned long long* queue = reinterpret_cast<unsigned long long*>(ws) + qi;  // this launch's counter
    uint32_t* per_job = reinterpret_cast<uint32_t*>(ws + WS_HEAD);
    long long n = n_jobs;
    if (d_n_jobs) n = min((long long)n, (long long)*d_n_jobs);
    n = min(n, j1);  // this launch's jobs: [j0, j1)
    auto sync = [&]() {
        if (W == 1) __syncwarp();
        else __syncthreads();
    };
    auto any = [&](bool x) { return W == 1 ? __any_sync(FULL, x) != 0 : __syncthreads_or(x) != 0; };
    for (uint32_t i = tid; i < C::GMAX + C::SPAN; i += T) M.map[i] = 0;
    if (tid == 0) M.tok[0] = T_FAR;  // bytes before the group's first

    for (;;) {
        if (tid == 0) M.job = atomicAdd(queue, 1ull);
        sync();
        const long long j = j0 + (long long)M.job;
        sync();
        if (j >= n) break;
        if (per_job[JW * j + 1] != CB_OK) continue;  // k_decode reported or listed it, or k_literals copied it
        const cb_member_job job = jobs[j];
        const uint8_t* lits = arena + reinterpret_cast<const unsigned long long*>(per_job)[(JW / 2) * j + 1];
        const uint2* sq = reinterpret_cast<const uint2*>(lits + slot_bytes(job.isize)) - 1;  // sequences 1, 0
        const uint32_t nl = per_job[JW * j + 4], ns = per_job[JW * j + 5];
        const uint32_t a = (uint32_t)((uintptr_t)(out_base + job.out_off) & (LINE - 1));
        uint8_t* base = out_base + job.out_off - a;  // slot 0
        const uint32_t Eend = a + job.isize;
        uint32_t P = a, st = CB_OK;
        uint32_t g = 0, lbase = 0;  // sequences (an even number) and literals done
        uint32_t lw0, lw1;
        auto load_lits = [&]() {  // the group's first literals
            const uint32_t l = (lbase & ~3u) + 4 * tid;
            lw0 = l < nl ? __ldcg(reinterpret_cast<const uint32_t*>(lits + l)) : 0u;
            lw1 = l + 4 * T < nl ? __ldcg(reinterpret_cast<const uint32_t*>(lits + l + 4 * T)) : 0u;
        };
        uint2 seq;
        auto load_seqs = [&](uint32_t from) {  // this thread's two sequences of a group
            const uint32_t i = from + 2 * tid;
            seq = i < ns ? __ldcg(sq - (i >> 1)) : make_uint2(0, 0);
            if (i + 1 >= ns) seq.x = 0;
        };
        // The plan of the group of seq that starts at P: this thread's literals and match lengths, output bytes and
        // literals before them and of the group, its sequences, whether it is invalid, and where sources older
        // than the ring come to `far` (f0, f1), of which those before `done` are on their way from here on.
        uint32_t s0, s1, c0, m0, c1, m1, eb, el, glen, glit, cnt, f0, f1, half = 0;
        bool bad;
        auto plan = [&](uint32_t done) {
            s0 = seq.y;
            s1 = seq.x;
            c0 = s0 >> 24;
            m0 = s0 & SEQ_MATCH ? ((s0 >> 16) & 255u) + 3 : 0u;
            c1 = s1 >> 24;
            m1 = s1 & SEQ_MATCH ? ((s1 >> 16) & 255u) + 3 : 0u;
            const bool none0 = (s0 & 0xFFFFu) && !m0, none1 = (s1 & 0xFFFFu) && !m1;
            const uint32_t vb = c0 + m0 + c1 + m1, vl = c0 + c1;
            if (W == 1) {
                uint32_t gv;
                const uint32_t ex = warp_exclusive_scan(vb | (vl << 16), gv);
                eb = ex & 0xFFFFu;
                el = ex >> 16;
                glen = gv & 0xFFFFu;
                glit = gv >> 16;
            } else {
                unsigned long long wt;
                unsigned long long ex = warp_exclusive_scan((unsigned long long)vb | ((unsigned long long)vl << 32), wt);
                if (lane == 0) M.sums[warp] = wt;
                __syncthreads();
                unsigned long long tot = 0;
#pragma unroll
                for (int w = 0; w < W; w++) {
                    if (w == (int)warp) ex += tot;
                    tot += M.sums[w];
                }
                eb = (uint32_t)ex;
                el = (uint32_t)(ex >> 32);
                glen = (uint32_t)tot;
                glit = (uint32_t)(tot >> 32);
            }
            cnt = min(2 * T, ns - g);
            if (glen > C::GMAX) {  // the threads whose sequences end within GMAX bytes (at least one)
                const uint32_t mine = __popc(__ballot_sync(FULL, eb + vb <= C::GMAX));
                uint32_t keep = mine;
                if (W > 1) {
                    if (lane == 0) M.count[warp] = mine;
                    __syncthreads();  // and every thread has read sums
                    keep = 0;
#pragma unroll
                    for (int w = 0; w < W; w++) keep += M.count[w];
                }
                if (W == 1) {
                    glen = __shfl_sync(FULL, eb + vb, keep - 1);
                    glit = __shfl_sync(FULL, el + vl, keep - 1);
                } else {
                    if (tid == keep - 1) M.sums[0] = (unsigned long long)(eb + vb) | ((unsigned long long)(el + vl) << 32);
                    __syncthreads();
                    glen = (uint32_t)M.sums[0];
                    glit = (uint32_t)(M.sums[0] >> 32);
                }
                cnt = min(cnt, 2 * keep);
                if (tid >= keep) {
                    c0 = m0 = c1 = m1 = 0;
                    eb = glen;
                    el = glit;
                }
            }
            const uint32_t R0 = P & ~(LINE - 1), p0 = P - R0, pe = p0 + glen;
            const uint32_t y0 = P + eb + c0, y1 = y0 + m0 + c1;  // the matches' slots
            const uint32_t d0 = (s0 & 0x7FFFu) + 1, d1 = (s1 & 0x7FFFu) + 1, x0 = y0 - d0, x1 = y1 - d1;
            bad = any(none0 || none1 || (m0 && d0 > y0 - a) || (m1 && d1 > y1 - a)) || glen > Eend - P;
            const uint32_t old = R0 + (pe + C::SPAN - 1) / C::SPAN * C::SPAN;  // the ring will hold old - RING on
            const bool old0 = m0 && x0 + C::RING < old, old1 = m1 && x1 + C::RING < old;
            f0 = old0 ? FAR_N : NOT_OLD;
            f1 = old1 ? FAR_N : NOT_OLD;
            const bool get0 = !bad && old0 && m0 <= FAR_LEN && x0 + m0 <= done;
            const bool get1 = !bad && old1 && m1 <= FAR_LEN && x1 + m1 <= done;
            const uint32_t any0 = __ballot_sync(FULL, get0), any1 = __ballot_sync(FULL, get1);
            if (any0 | any1) {
                auto fetch = [&](uint32_t f, uint32_t x, uint32_t m) {
                    const uint32_t nw = ((x & 3u) + m + 3) >> 2;
                    const uint8_t* q = base + (x & ~3u);
                    uint32_t* to = M.far[warp][half] + FAR_WORDS * f;
#pragma unroll
                    for (uint32_t k = 0; k < FAR_WORDS; k++)
                        if (k < nw) copy_async4(to + k, q + 4 * k);
                };
                if (get0) f0 = min(FAR_N, (uint32_t)__popc(any0 & lt));
                if (get1) f1 = min(FAR_N, (uint32_t)(__popc(any0) + __popc(any1 & lt)));
                if (f0 < FAR_N) fetch(f0, x0, m0);
                if (f1 < FAR_N) fetch(f1, x1, m1);
            }
        };
        load_seqs(0);
        load_lits();
        if (ns) {
            plan(a);
            load_seqs(cnt);
        }
        while (g < ns) {
            if (bad) {
                st = CB_ERR_INFLATE;
                break;
            }
            M.lit[tid] = lw0;
            M.lit[tid + T] = lw1;
            // places from the group's first line: its start, this thread's, and after each of its parts
            const uint32_t R0 = P & ~(LINE - 1), P0 = P, p0 = P - R0, pe = p0 + glen;
            const uint32_t b0 = p0 + eb, b1 = b0 + c0, b2 = b1 + m0, b3 = b2 + c1;
            const uint32_t d0 = (s0 & 0x7FFFu) + 1, d1 = (s1 & 0x7FFFu) + 1;
            const uint32_t l0 = (lbase & 3u) + el, l1 = l0 + c0, lit0 = lbase & ~3u;
            const uint32_t x0 = R0 + b1 - d0, x1 = R0 + b3 - d1;
            const uint32_t far_at = FAR_AT + half * (4 * FAR_WORDS * FAR_N);
            {
                auto place = [&](uint32_t id, uint32_t start, uint32_t len) {
                    M.map[start] = (typename C::Id)id;
                    if (W > 1)  // and the lines whose first byte is the token's
                        for (uint32_t L = (start + LINE - 1) / LINE; L * LINE < start + len; L++) M.head[L] = (uint16_t)id;
                };
                auto literals = [&](uint32_t id, uint32_t start, uint32_t c, uint32_t l) {
                    place(id, start, c);
                    const bool held = l + c <= C::LITS;
                    M.tok[id] = (((held ? LIT_AT + l : 0u) - start) << 16) | (held ? T_FAR : T_FAR | T_DIRECT | T_PLAIN);
                    M.aux[id] = lit0 + l - start;
                };
                auto match = [&](uint32_t id, uint32_t start, uint32_t len, uint32_t d, uint32_t x, uint32_t f) {
                    place(id, start, len);
                    const uint32_t at = x & C::RMASK;
                    const bool is_old = f != NOT_OLD, held = is_old ? f < FAR_N : at + len <= C::RING;
                    M.tok[id] = (((!held ? 0u : is_old ? far_at + 4 * FAR_WORDS * f + (x & 3u) : at) - start) << 16) |
                                (!held ? (is_old ? T_FAR | T_DIRECT : T_FAR | T_WRAP) : d < C::SPAN ? T_NEAR | d : T_FAR);
                    M.aux[id] = start | (d << 16);
                };
                if (c0) literals(4 * tid + 1, b0, c0, l0);
                if (m0) match(4 * tid + 2, b1, m0, d0, x0, f0);
                if (c1) literals(4 * tid + 3, b2, c1, l1);
                if (m1) match(4 * tid + 4, b3, m1, d1, x1, f1);
                if (W > 1 && tid == 0 && p0) M.head[0] = 0;
            }
            // the next group is planned, and its old sources and the sequences after it loaded, while this one is
            // written (with 32 old sources, fetched when their own group was planned, 61,825 members took 25.3 ms
            // of decode, copy and CRC32, now 22.7: with 24 of them 26.9, 32 23.9, 48 23.1)
            wait_async();
            g += cnt;
            lbase += glit;
            P += glen;
            half ^= 1;
            load_lits();
            if (g < ns) {
                plan(P0 & ~3u);  // (the word that P0 lies in is stored by this group)
                load_seqs(g + cnt);
            }
            sync();
            uint32_t carry = 0;
            const uint32_t full0 = a > R0 ? a - R0 : 0u, full1 = Eend - R0;  // whole words of the member
            for (uint32_t sr = 0; sr < pe; sr += C::SPAN) {
                const uint32_t rr = sr + LINE * warp, rel = rr + 4 * lane, w = R0 + rel;
                // the numbers of the tokens that start in the word
                uint32_t m[4];
                if (W == 1) {
                    const uint32_t x = *reinterpret_cast<const uint32_t*>(M.map + rel);
                    *reinterpret_cast<uint32_t*>(M.map + rel) = 0;
#pragma unroll
                    for (int k = 0; k < 4; k++) m[k] = (x >> (8 * k)) & 255u;
                } else {
                    const uint2 x = *reinterpret_cast<const uint2*>(M.map + rel);
                    *reinterpret_cast<uint2*>(M.map + rel) = make_uint2(0, 0);
                    m[0] = x.x & 0xFFFFu;
                    m[1] = x.x >> 16;
                    m[2] = x.y & 0xFFFFu;
                    m[3] = x.y >> 16;
                    carry = rr < pe ? M.head[rr / LINE] : 0u;
                }
                // the token of the byte before the word: the last one that starts in a lane below, else the
                // line's first (W > 1) or the last of the line before
                const uint32_t mlast = max(max(m[0], m[1]), max(m[2], m[3]));
                const uint32_t below = __ballot_sync(FULL, mlast != 0) & lt;
                uint32_t id = __shfl_sync(FULL, mlast, below ? 31 - __clz((int)below) : 0);
                if (!below) id = carry;
                uint32_t ids[4], tk[4], v[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    id = max(id, m[k]);
                    ids[k] = id;
                    tk[k] = M.tok[id];
                    v[k] = W == 1 ? smem[(int)(rel + k) + ((int)tk[k] >> 16)] : smem[(rel + k + (tk[k] >> 16)) & 0xFFFFu];
                }
                if (W == 1) carry = __shfl_sync(FULL, id, 31);
                uint32_t word = __byte_perm(__byte_perm(v[0], v[1], 0x40), __byte_perm(v[2], v[3], 0x40), 0x5410);
                if (rr == 0 && rel < p0) {  // bytes before the group's first are there already
                    const uint32_t mine = shl_clamp(8 * (p0 - rel));
                    word = (word & mine) | (ring4[(w & C::RMASK) >> 2] & ~mine);
                }
                const uint32_t fl = tk[0] | tk[1] | tk[2] | tk[3];
                uint32_t pend = 0;  // bytes whose source is written in this round
                const int left = (int)(pe - rel), fresh = (int)max(sr, p0);  // from fresh on
                if (__any_sync(FULL, left > 0 && (fl & T_FLAGS))) {
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((int)(rel + k - (tk[k] & T_FAR)) >= fresh) pend |= 1u << k;
                    pend &= ~shl_clamp((uint32_t)max(left, 0));
                    if (__any_sync(FULL, left > 0 && (fl & (T_WRAP | T_DIRECT)))) {
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            if ((tk[k] & (T_WRAP | T_DIRECT)) && k < left) {
                                const uint32_t ax = M.aux[ids[k]], x = w + k - (ax >> 16);
                                uint32_t b = 0;
                                if (tk[k] & T_DIRECT) b = __ldcg(tk[k] & T_PLAIN ? lits + (uint32_t)(rel + k + ax) : base + x);
                                else if ((int)(x - R0) >= fresh) pend |= 1u << k;
                                else b = M.ring[x & C::RMASK];
                                word = (word & ~(0xFFu << (8 * k))) | (b << (8 * k));
                            }
                        }
                    }
                }
                if (any(pend != 0)) {
                    // their sources; a match that overlaps itself repeats the bytes before its start
                    int px[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        px[k] = 0x7FFFFFFF;
                        if (pend >> k & 1) {
                            const uint32_t ax = M.aux[ids[k]], d = ax >> 16;
                            const int start = (int)(ax & 0xFFFFu);
                            px[k] = (int)(rel + k - d);
                            if (px[k] >= start) {  // (the quotient of small numbers; half keeps it off the integers)
                                const int n = px[k] - start;
                                px[k] = start - (int)d + n - (int)d * (int)__fdividef((float)n + 0.5f, (float)d);
                            }
                        }
                    }
                    if (W > 1) {
                        M.missing[tid] = (uint8_t)pend;
                        ring4[(w & C::RMASK) >> 2] = word;
                        __syncthreads();
                    }
                    do {
                        // at each pass the bytes whose sources are there (W == 1: lie below the first missing)
                        int Q = 0;
                        if (W == 1) {
                            Q = (int)__reduce_min_sync(FULL, pend ? rel + __ffs((int)pend) - 1 : 0x7FFFFFFFu);
                            ring4[(w & C::RMASK) >> 2] = word;
                            __syncwarp();
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            bool ready = px[k] < Q;
                            if (W > 1 && (pend >> k & 1))
                                ready = px[k] < fresh || !(M.missing[(px[k] - sr) >> 2] >> (px[k] & 3) & 1);
                            if (ready) {
                                word = (word & ~(0xFFu << (8 * k))) | ((uint32_t)M.ring[(R0 + px[k]) & C::RMASK] << (8 * k));
                                pend &= ~(1u << k);
                                px[k] = 0x7FFFFFFF;
                            }
                        }
                        sync();
                        if (W > 1) {
                            M.missing[tid] = (uint8_t)pend;
                            ring4[(w & C::RMASK) >> 2] = word;
                        }
                    } while (any(pend != 0));
                }
                ring4[(w & C::RMASK) >> 2] = word;
                if (rel < pe && rel + 4 > p0) {
                    if (rel >= full0 && rel + 4 <= full1) {
                        // (a word that the group ends in is left to the next one: only final bytes are ever stored)
                        if (rel + 4 <= pe) *reinterpret_cast<uint32_t*>(base + w) = word;
                    } else {  // the member's first or last word: its own bytes only
                        for (uint32_t s = max(w, P0); s < min(w + 4, R0 + pe); s++) base[s] = (uint8_t)(word >> (8 * (s - w)));
                    }
                }
                sync();
            }
        }
        wait_async();
        if (st == CB_OK && P != Eend) st = CB_ERR_INFLATE;
        if (tid == 0 && st != CB_OK) {
            per_job[JW * j + 1] = st;
            report(summary, job_status, j, st);
        }
    }
}

// ---------------------------------------------------------------- k_crc: one member per W warps
// The rows of crc.cuh, in registers, eight at a time with the next eight being loaded.  What bounds it is the
// latency of memory: 4.5 GB of output 2.06 ms (2.42 without the load ahead; 39 members 12.5 us, 20.8).  (Tables for
// every byte took a shared-memory access with conflicts per byte.)

constexpr int CRC_NT = 256;

// Eight rows (128 bytes each) of a message of len bytes, whose lane's first word is at byte q (negative
// positions are zero bytes): as words of the message where the rows reach its first four bytes, which are
// inverted (the CRC's initial value), else as the aligned words with x the one after the last row's (lane 0's).
__device__ __forceinline__ void crc_load(const uint8_t* m, uint32_t len, long long q, bool head, uint32_t (&w)[8], uint32_t& x) {
    if (head) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int p = (int)(q + 128 * i), at = max(p, 0);
            uint32_t y = p > -4 ? ld_bytes4(m + at, len - (uint32_t)at) : 0u;
            if (p < 0) y = p > -4 ? y << (-8 * p) : 0u;
            if (len >= 4 && p < 4 && p > -4) y ^= p < 0 ? FULL << (-8 * p) : FULL >> (8 * p);
            w[i] = y;
        }
    } else {
        const uintptr_t ad = (uintptr_t)(m + q);
        const uint32_t* wp = reinterpret_cast<const uint32_t*>(ad & ~(uintptr_t)3);
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = __ldg(wp + 32 * i);
        x = (ad & 3) && (threadIdx.x & 31) == 0 ? __ldg(wp + 256) : 0u;
    }
}

// W warps per member, each a part of its 4,096-byte steps; parts are joined by x^(8 bytes after).
template <int W>
__global__ void __launch_bounds__(CRC_NT)
    k_crc(const cb_member_job* __restrict__ jobs, int64_t n_jobs, const int64_t* __restrict__ d_n_jobs,
          const uint8_t* __restrict__ out_base, uint32_t* job_status, cb_inflate_summary* summary, uint8_t* ws,
          long long j0, long long j1) {
    __shared__ uint32_t fold[4][256];
    __shared__ uint32_t parts[CRC_NT / 32];
    init_crc_fold(fold);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* per_job = reinterpret_cast<uint32_t*>(ws + WS_HEAD);
    long long n = n_jobs;
    if (d_n_jobs) n = min((long long)n, (long long)*d_n_jobs);
    n = min(n, j1);
    constexpr int PER = CRC_NT / 32 / W;  // members per CTA at a time
    for (long long jb = j0 + (long long)blockIdx.x * PER; jb < n; jb += (long long)gridDim.x * PER) {
        const long long j = jb + warp / W;
        uint32_t c = 0, want = 0;
        const uint32_t st = j < n ? per_job[JW * j + 1] : (uint32_t)CB_ERR_INFLATE;
        const bool on = st == CB_OK || st == ST_LITERALS;
        uint32_t len = 0;
        if (on) {
            const cb_member_job job = jobs[j];
            const uint8_t* m = out_base + job.out_off;
            len = job.isize;
            want = job.crc;
            const long long pad = (long long)((4096u - (len & 4095u)) & 4095u);
            const long long iters = ((long long)len + pad) >> 12;
            const long long i0 = iters * (warp % W) / W, i1 = iters * (warp % W + 1) / W;
            uint32_t v[32];
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = 0;
            const uint32_t sh = (uint32_t)((uintptr_t)(m - pad) & 3) * 8;
            auto head = [&](long long row) { return row * 128 - pad < 4; };
            uint32_t w[8], x = 0;
            if (i0 < i1) crc_load(m, len, i0 * 4096 + 4 * lane - pad, head(i0 * 32), w, x);
            for (long long it = i0; it < i1; it++) {
                const bool last = it + 1 == i1;
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 8) {
                    const long long row = it * 32 + r0, nr = row + 8;
                    uint32_t nw[8], nx = 0;  // the next rows are loaded while these are folded
                    if (r0 < 24 || !last) crc_load(m, len, nr * 128 + 4 * lane - pad, head(nr), nw, nx);
                    if (sh && !head(row)) {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const uint32_t hi = __shfl_sync(FULL, lane == 0 ? (i < 7 ? w[(i + 1) & 7] : x) : w[i], (lane + 1) & 31);
                            w[i] = __funnelshift_r(w[i], hi, sh);
                        }
                    }
                    if (last) crc_rows<true>(v, w, r0);
                    else crc_rows<false>(v, w, r0);
#pragma unroll
                    for (int i = 0; i < 8; i++) w[i] = nw[i];
                    x = nx;
                }
            }
            c = crc_fold_rows(fold, v);
            if (W > 1 && i1 < iters) c = gf_mul(c, xpow_from(kCrc.x2n, 32768ull * (unsigned long long)(iters - i1)));
        }
        if (W > 1) {
            if (lane == 0) parts[warp] = c;
            __syncthreads();
            if (warp % W == 0)
                for (int w = 1; w < W; w++) c ^= parts[warp + w];
            __syncthreads();
        }
        if (on && warp % W == 0) {
            const uint32_t crc = len >= 4 ? ~c : crc_finish(c, len);
            if (lane == 0 && crc != want) {
                per_job[JW * j + 1] = CB_ERR_CRC;
                report(summary, job_status, j, CB_ERR_CRC);
            }
        }
    }
}

__global__ void k_split_init(cb_inflate_summary* summary, unsigned long long* queue) {
    summary->status = CB_OK;
    summary->reserved = 0;
    summary->n_bad = 0;
    summary->first_bad = INT64_MAX;
    for (int q = 0; q < Q_LISTED + 2; q++) queue[q] = 0;  // decode and copy counters of up to two job ranges, the list's
}

__global__ void k_split_finish(cb_inflate_summary* summary) {
    if (summary->first_bad == INT64_MAX) summary->first_bad = -1;
}

}  // namespace split
}  // namespace cb

using namespace cb;

int cb_set_error(cudaError_t e);  // abi.cu
int cb_inflate_split_any(const cb_member_job* jobs, int64_t n_jobs, const int64_t* d_n_jobs, uint8_t* out_base,
                         int check_crc, uint32_t* job_status, cb_inflate_summary* summary, void* workspace,
                         size_t workspace_bytes, bool list_unfit, void* stream);
// inflate.cu: the one-kernel form for the jobs list[step * k], k < *count (on the device)
int cb_inflate_listed(const cb_member_job* jobs, const uint32_t* list, int step, const unsigned long long* count,
                      uint8_t* out_base, int check_crc, uint32_t* job_status, cb_inflate_summary* summary,
                      unsigned long long* queue, cudaStream_t s);

namespace {

constexpr int MAX_DEVICES = 64;

// CTAs per SM of a kernel on the current device, setting its shared memory size once per device.
template <class K>
int occupancy(int (&cache)[MAX_DEVICES], K kernel, int threads, size_t smem) {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEVICES) return -1;
    int& b = cache[d];
    if (b > 0) return b;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int occ = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem);
    if (e != cudaSuccess) return -(int)e;
    b = occ > 0 ? occ : 1;
    return b;
}

int fail_occ(int o) { return cb_set_error(o == -1 ? cudaErrorInvalidDevice : (cudaError_t)(-o)); }

// One inflate call's arguments.
struct Call {
    const cb_member_job* jobs;
    int64_t n_jobs;
    const int64_t* d_n_jobs;
    uint8_t* out_base;
    int check_crc;
    uint32_t* job_status;
    cb_inflate_summary* summary;
    uint8_t *ws, *arena;
    unsigned long long arena_bytes;
    uint8_t* scratch;  // decode's, scratch_n bytes per member in flight
    uint32_t scratch_n;
    bool list_unfit;
};

// One launch's jobs: [j0, j1) of the table, and its queue counters (decode at qd, copy at qd + 1).
struct Range {
    long long j0, j1;
    int qd;
    long long s0, s1;  // its members in flight: [s0, s1) of the scratch
};

// CTAs for a persistent grid of `occ` per SM, `members` each at a time, no more than the range has work for.
unsigned grid_for(const Call& c, Range r, int occ, int members) {
    long long grid = (long long)cb_device_sm_count() * occ;
    const long long by_work = (r.j1 - r.j0 + members - 1) / members;
    if (!c.d_n_jobs && by_work < grid) grid = by_work;
    return (unsigned)(grid < 1 ? 1 : grid);
}

// Each kernel takes as many warps per member as keep all members resident at once: one member's serial work
// bounds a call of few, and a second round of members doubles it.  Decode and copy, in us, of 39 / 386 / 773 /
// 1545 / 3090 GEX members: 8 warps 171 333 518 987 1835 and 161 339 531 1022 1893; 4 warps 193 218 393 607 1135
// and 226 249 477 743 1266; 2 warps 255 283 306 536 837 and 343 367 394 760 1170; 1 warp 402 423 455 491 880
// and 535 559 591 630 861.  (Before the copy's bytes were put together in fewer instructions: 4% less now.)
template <int W>
int decode_occupancy() {
    static int cache[MAX_DEVICES];
    constexpr int MEMBERS = W == 1 ? 2 : 1;
    return occupancy(cache, split::k_decode<W>, 32 * W * MEMBERS, MEMBERS * sizeof(split::DecMember<W>));
}
template <class C>
int copy_occupancy() {
    static int cache[MAX_DEVICES];
    static_assert(sizeof(typename C::Smem) < (C::W == 1 ? 32768 : 65536), "a source's offset has 16 bits");
    return occupancy(cache, split::k_copy<C>, C::T, sizeof(typename C::Smem));
}
bool resident(const Call& c, int occ) { return c.n_jobs <= (long long)cb_device_sm_count() * occ; }

template <int W>
int launch_decode(const Call& c, Range r, cudaStream_t s) {
    constexpr int MEMBERS = W == 1 ? 2 : 1, NT = 32 * W * MEMBERS;
    const int o = decode_occupancy<W>();
    if (o <= 0) return fail_occ(o);
    const long long room = (r.s1 - r.s0) / MEMBERS;
    if (room < 1) return CB_ERR_ARG;
    const unsigned grid = grid_for(c, r, o, MEMBERS);
    split::k_decode<W><<<grid < room ? grid : (unsigned)room, NT, MEMBERS * sizeof(split::DecMember<W>), s>>>(
        c.jobs, c.n_jobs, c.d_n_jobs, c.job_status, c.summary, c.ws, c.arena, c.arena_bytes, c.scratch + r.s0 * c.scratch_n,
        c.scratch_n, c.list_unfit, r.j0, r.j1, r.qd);
    return CB_OK;
}

int decode_range(const Call& c, Range r, cudaStream_t s) {
    return resident(c, decode_occupancy<8>())   ? launch_decode<8>(c, r, s)
           : resident(c, decode_occupancy<4>()) ? launch_decode<4>(c, r, s)
           : resident(c, decode_occupancy<2>()) ? launch_decode<2>(c, r, s)
                                                : launch_decode<1>(c, r, s);
}

template <class C>
int launch_copy(const Call& c, Range r, cudaStream_t s) {
    const int o = copy_occupancy<C>();
    if (o <= 0) return fail_occ(o);
    split::k_copy<C><<<grid_for(c, r, o, 1), C::T, sizeof(typename C::Smem), s>>>(
        c.jobs, c.n_jobs, c.d_n_jobs, c.out_base, c.job_status, c.summary, c.ws, c.arena, r.j0, r.j1, r.qd + 1);
    return CB_OK;
}

template <int W>
int launch_crc(const Call& c, Range r, cudaStream_t s) {
    static int cache[MAX_DEVICES];
    const int o = occupancy(cache, split::k_crc<W>, split::CRC_NT, 0);
    if (o <= 0) return fail_occ(o);
    split::k_crc<W><<<grid_for(c, r, o, split::CRC_NT / 32 / W), split::CRC_NT, 0, s>>>(
        c.jobs, c.n_jobs, c.d_n_jobs, c.out_base, c.job_status, c.summary, c.ws, r.j0, r.j1);
    return CB_OK;
}

// Whether members without matches go through k_literals: not where a member has two warps or more, whose copy takes them
// well enough (1,000 of 65 KB 583 us) and the launch and look cost the others 6 us.
bool takes_literals(const Call& c) { return !resident(c, copy_occupancy<split::CopyCfg<8192, 2>>()); }

int copy_range(const Call& c, Range r, cudaStream_t s) {
    using C8 = split::CopyCfg<16384, 8>;
    using C4 = split::CopyCfg<16384, 4>;
    using C2 = split::CopyCfg<8192, 2>;
    const int cw = (int)cb_param(CB_PARAM_COPY_WARPS);
    if (takes_literals(c))
        split::k_literals<<<(unsigned)min((r.j1 - r.j0 + split::LOOK - 1) / split::LOOK, 32768LL), 64, 0, s>>>(
            c.jobs, c.n_jobs, c.d_n_jobs, c.out_base, c.ws, c.arena, r.j0, r.j1);
    int rc;
    if (resident(c, copy_occupancy<C8>())) rc = launch_copy<C8>(c, r, s);
    else if (resident(c, copy_occupancy<C4>())) rc = launch_copy<C4>(c, r, s);
    else if (resident(c, copy_occupancy<C2>())) rc = launch_copy<C2>(c, r, s);
    // 4 KB: 22 warps per SM; with 8 KB 16 (15,456 GEX members when it had 28: 4.04 ms, 8 KB 4.39)
    else if (cw == 12) rc = launch_copy<split::CopyCfg<4096, 1>>(c, r, s);
    else if (cw == 24) rc = launch_copy<split::CopyCfg<8192, 1>>(c, r, s);
    else rc = launch_copy<split::CopyCfg<16384, 1>>(c, r, s);
    if (rc != CB_OK || !c.check_crc) return rc;
    const long long room = (long long)cb_device_sm_count() * 28;  // warps
    return c.n_jobs * 8 <= room   ? launch_crc<8>(c, r, s)
           : c.n_jobs * 4 <= room ? launch_crc<4>(c, r, s)
           : c.n_jobs * 2 <= room ? launch_crc<2>(c, r, s)
                                  : launch_crc<1>(c, r, s);
}

// A pair of side streams for the pipelined form, and the events that join them to the caller's stream.  A caller's
// stream keeps its pair, so that calls on several streams do not wait for one another; a stream beyond SIDES takes the
// pair that was used longest ago (calls then queue behind one another).  Side streams that joined a capture belong to
// it until it ends: no other call may use them meanwhile, or the capture is lost.  The mutex keeps each call's records
// and waits together (a wait takes the event's state when it is called).
struct Side {
    cudaStream_t x = nullptr, y = nullptr, owner = nullptr;
    cudaEvent_t start = nullptr, done_x = nullptr, done_y = nullptr;
    unsigned long long used = 0;  // when, counted in calls; 0: the pair is not made yet
};
constexpr int SIDES = 8;
Side g_side[MAX_DEVICES][SIDES];
unsigned long long g_side_calls = 0;
std::mutex g_side_mu;

// The capture that stream s is part of, 0 for none; -1 (as an unsigned number) for one that was lost or cannot be told.
unsigned long long capture_of(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(s, &st, &id) != cudaSuccess) {
        cudaGetLastError();
        return ~0ull;
    }
    return st == cudaStreamCaptureStatusNone ? 0 : st == cudaStreamCaptureStatusActive ? id : ~0ull;
}

int make_side(Side& sd) {
    // (another thread's capture does not forbid this thread to make streams in this mode)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return cb_set_error(e);
    if (!sd.x) e = cudaStreamCreateWithFlags(&sd.x, cudaStreamNonBlocking);
    if (e == cudaSuccess && !sd.y) e = cudaStreamCreateWithFlags(&sd.y, cudaStreamNonBlocking);
    if (e == cudaSuccess && !sd.start) e = cudaEventCreateWithFlags(&sd.start, cudaEventDisableTiming);
    if (e == cudaSuccess && !sd.done_x) e = cudaEventCreateWithFlags(&sd.done_x, cudaEventDisableTiming);
    if (e == cudaSuccess && !sd.done_y) e = cudaEventCreateWithFlags(&sd.done_y, cudaEventDisableTiming);
    const cudaError_t back = cudaThreadExchangeStreamCaptureMode(&mode);
    return cb_set_error(e != cudaSuccess ? e : back);
}

// The pair for a call on s, under g_side_mu; none (out is null) when other captures hold them all.
int side_for(int dev, cudaStream_t s, Side*& out) {
    out = nullptr;
    const unsigned long long capture = capture_of(s);
    Side *oldest = nullptr, *fresh = nullptr;
    for (Side& sd : g_side[dev]) {
        if (!sd.used) {
            if (!fresh) fresh = &sd;
            continue;
        }
        const unsigned long long of = capture_of(sd.x);
        if (of != 0 && of != capture) continue;
        if (sd.owner == s) {
            out = &sd;
            break;
        }
        if (!oldest || sd.used < oldest->used) oldest = &sd;
    }
    if (!out && fresh) {
        const int rc = make_side(*fresh);
        if (rc != CB_OK) return rc;
        out = fresh;
    }
    if (!out) out = oldest;
    if (out) {
        out->owner = s;
        out->used = ++g_side_calls;
    }
    return CB_OK;
}

// Pipelined: the jobs in two ranges, each decoded and then copied on its own stream, so that the second range's decode and
// the first range's copy fill the warps that the other's end leaves idle: from 20 members per SM, where they take more than
// one round of resident warps (3,865 GEX members 2.45 ms -> 2.12, 15,457 6.95 -> 6.72; 2,320 1.358 -> 1.366; cut at three
// quarters 2.35 and 6.78; in four ranges 2.59 and 7.09).  Only with the job count known on the host, and under capture only
// from 65,536 jobs (or when it is always on).
template <class Captured> bool two_ranges(int64_t n_jobs, Captured captured) {
    const long long pipe = cb_param(CB_PARAM_DECODE_PIPELINE);
    if (n_jobs < 2 || pipe == 0) return false;
    if (pipe == 2 || n_jobs >= 65536) return true;
    return n_jobs >= 20LL * cb_device_sm_count() && !captured();
}

}  // namespace

// Kernels of one call of form 3.
int cb_split_launches(int64_t n_jobs, int check_crc, bool captured) {
    if (n_jobs <= 0) return 2;  // init and finish
    Call c{};
    c.n_jobs = n_jobs;
    const int ranges = two_ranges(n_jobs, [&] { return captured; }) ? 2 : 1;
    return 4 + ranges * (2 + (check_crc ? 1 : 0) + (takes_literals(c) ? 1 : 0));
}

extern "C" size_t cb_inflate_split_workspace_bytes(int64_t n_jobs, int64_t out_bytes) {
    if (n_jobs < 0 || out_bytes < 0) return 0;
    return split::arena_offset(n_jobs) + 80 * (size_t)n_jobs + 32 + split::arena_and_scratch(n_jobs, out_bytes);
}

extern "C" int cb_inflate_split(const cb_member_job* jobs, int64_t n_jobs, const int64_t* d_n_jobs, uint8_t* out_base,
                                int check_crc, uint32_t* job_status, cb_inflate_summary* summary, void* workspace,
                                size_t workspace_bytes, void* stream) {
    return cb_inflate_split_any(jobs, n_jobs, d_n_jobs, out_base, check_crc, job_status, summary, workspace,
                                workspace_bytes, false, stream);
}

int cb_inflate_split_any(const cb_member_job* jobs, int64_t n_jobs, const int64_t* d_n_jobs, uint8_t* out_base,
                         int check_crc, uint32_t* job_status, cb_inflate_summary* summary, void* workspace,
                         size_t workspace_bytes, bool list_unfit, void* stream) {
    if (!summary || !workspace || n_jobs < 0 || workspace_bytes < split::arena_offset(n_jobs) + 16) return CB_ERR_ARG;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    uint8_t* arena = reinterpret_cast<uint8_t*>(((uintptr_t)(ws + split::arena_offset(n_jobs)) + 15) & ~(uintptr_t)15);
    // the scratch of the members in flight at the workspace's end, the arena before it
    const unsigned long long rest = (unsigned long long)(ws + workspace_bytes - arena), fixed = 80ull * n_jobs + 16;
    const long long flight = split::in_flight(n_jobs);
    const uint32_t scratch_n = split::scratch_for(n_jobs, rest > fixed ? rest - fixed : 0);
    const unsigned long long arena_bytes = (rest - (unsigned long long)flight * scratch_n) & ~15ull;
    const Call c{jobs, n_jobs, d_n_jobs, out_base, check_crc, job_status, summary, ws, arena, arena_bytes,
                 arena + arena_bytes, scratch_n, list_unfit};
    auto* queue = reinterpret_cast<unsigned long long*>(ws);
    split::k_split_init<<<1, 1, 0, s>>>(summary, queue);
    if (n_jobs > 0) {
        split::k_slots<<<1, split::SLOT_NT, 0, s>>>(jobs, n_jobs, d_n_jobs, ws);
        const bool two = !d_n_jobs && two_ranges(n_jobs, [&] { return capture_of(s) != 0; });
        int rc = CB_OK;
        std::unique_lock<std::mutex> lock(g_side_mu, std::defer_lock);
        Side* sd = nullptr;
        if (two) {
            int dev = 0;
            const cudaError_t e = cudaGetDevice(&dev);
            if (e != cudaSuccess) return cb_set_error(e);
            if (dev < 0 || dev >= MAX_DEVICES) return CB_ERR_ARG;
            lock.lock();
            if ((rc = side_for(dev, s, sd)) != CB_OK) return rc;
        }
        if (!sd) {
            const Range all{0, n_jobs, 0, 0, flight};
            rc = decode_range(c, all, s);
            if (rc == CB_OK) rc = copy_range(c, all, s);
            if (rc != CB_OK) return rc;
        } else {
            cudaError_t e = cudaEventRecord(sd->start, s);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(sd->x, sd->start, 0);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(sd->y, sd->start, 0);
            if (e != cudaSuccess) return cb_set_error(e);
            const Range ra{0, n_jobs / 2, 0, 0, flight / 2}, rb{n_jobs / 2, n_jobs, 2, flight / 2, flight};
            rc = decode_range(c, ra, sd->x);
            if (rc == CB_OK) rc = decode_range(c, rb, sd->y);
            if (rc == CB_OK) rc = copy_range(c, ra, sd->x);
            if (rc == CB_OK) rc = copy_range(c, rb, sd->y);
            // join both side streams back to the caller's stream whatever happened above
            e = cudaEventRecord(sd->done_x, sd->x);
            if (e == cudaSuccess) e = cudaEventRecord(sd->done_y, sd->y);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(s, sd->done_x, 0);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(s, sd->done_y, 0);
            if (rc != CB_OK) return rc;
            if (e != cudaSuccess) return cb_set_error(e);
        }
        if (lock.owns_lock()) lock.unlock();
        rc = cb_inflate_listed(jobs, reinterpret_cast<const uint32_t*>(ws + split::WS_HEAD), split::JW,
                               queue + split::Q_LISTED,
                               out_base, check_crc, job_status, summary, queue + split::Q_LISTED + 1, s);
        if (rc != CB_OK) return rc;
    }
    split::k_split_finish<<<1, 1, 0, s>>>(summary);
    return cb_set_error(cudaGetLastError());
}
