// CRC32 (zlib's polynomial, reflected) arithmetic shared by the inflater and the compressor.
//
// Spans are checksummed in parallel: each part gets a raw column (the CRC register run over its
// bytes from zero, no pre- or post-inversion), and columns are joined with
// raw(A || B) = raw(A) * x^(8 |B|) + raw(B) in GF(2)[x] modulo the polynomial, the combination
// zlib's crc32_combine is built on.  The zlib CRC of n bytes is then
// raw ^ (0xFFFFFFFF * x^(8 n)) ^ 0xFFFFFFFF.
#pragma once

#include <cstdint>

namespace cb {

// Reflected representation of GF(2)[x] modulo the CRC-32 polynomial: bit 31 is x^0.
constexpr uint32_t POLY = 0xEDB88320u;

__host__ __device__ constexpr uint32_t gf_mul(uint32_t a, uint32_t b) {
    uint32_t p = 0;
    for (int i = 0; i < 32; i++) {
        if (a & 0x80000000u) p ^= b;
        a <<= 1;
        b = (b & 1u) ? (b >> 1) ^ POLY : (b >> 1);
    }
    return p;
}

struct CrcConst {
    uint32_t x2n[32];   // x^(2^k)
    uint32_t seg[5];    // x^(8 * 32 * 2^k): shifts that combine the lane columns
    uint32_t k992;      // x^(8 * 992): one window minus one column
};

__host__ __device__ constexpr uint32_t xpow_from(const uint32_t* x2n, unsigned long long n) {
    uint32_t r = 0x80000000u;  // x^0
    for (int k = 0; n; n >>= 1, k++)
        if (n & 1) r = gf_mul(r, x2n[k]);
    return r;
}

constexpr CrcConst make_crc_const() {
    CrcConst c{};
    uint32_t p = 0x40000000u;  // x^1
    for (int k = 0; k < 32; k++) {
        c.x2n[k] = p;
        p = gf_mul(p, p);
    }
    for (int k = 0; k < 5; k++) c.seg[k] = xpow_from(c.x2n, 8ull * 32ull * (1ull << k));
    c.k992 = xpow_from(c.x2n, 8ull * 992ull);
    return c;
}

// One copy per translation unit (static: the host-side shadows of two units do not collide).
static __constant__ CrcConst kCrc = make_crc_const();

// zlib's CRC of n bytes from their raw column.
__device__ __forceinline__ uint32_t crc_finish(uint32_t raw, unsigned long long n) {
    return raw ^ gf_mul(0xFFFFFFFFu, xpow_from(kCrc.x2n, 8ull * n)) ^ 0xFFFFFFFFu;
}

// Slice-by-8 CRC tables (table t: the CRC of a byte followed by t zero bytes).
__device__ inline void init_crc8(uint32_t (*crc8)[256]) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        uint32_t c = (uint32_t)i;
        for (int k = 0; k < 8; k++) c = (c & 1u) ? (c >> 1) ^ POLY : c >> 1;
        crc8[0][i] = c;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        uint32_t c = crc8[0][i];
        for (int t = 1; t < 8; t++) {
            c = (c >> 8) ^ crc8[0][c & 255];
            crc8[t][i] = c;
        }
    }
}

// The raw column after 8 more bytes (w0 = bytes 0-3, w1 = bytes 4-7, little-endian).
__device__ __forceinline__ uint32_t crc_step8(const uint32_t (*T)[256], uint32_t c, uint32_t w0, uint32_t w1) {
    c ^= w0;
    return T[7][c & 255] ^ T[6][(c >> 8) & 255] ^ T[5][(c >> 16) & 255] ^ T[4][c >> 24] ^ T[3][w1 & 255] ^
           T[2][(w1 >> 8) & 255] ^ T[1][(w1 >> 16) & 255] ^ T[0][w1 >> 24];
}

// ---- CRC by rows: the polynomial P divides P(x^1024) (= P^1024 in characteristic 2), so a message may
// be reduced by P(x^1024) first: rows of 1024 bits (a 4-byte word per lane) take the place of the
// polynomial's single bits, and eliminating a row is an XOR of it into the 14 rows that P's other terms
// name -- seven three-input XORs per row of 128 bytes, in registers.  What is left are 32 rows; each lane
// folds its words of them with a table of x^1024 and the lanes join with one multiplication each.

struct CrcLane {
    uint32_t x1024, k[32];  // x^1024; x^(32 (32 - l)): the bits after lane l's word of a row, and 32 more
};
constexpr CrcLane make_crc_lane() {
    CrcLane c{};
    const CrcConst q = make_crc_const();
    c.x1024 = xpow_from(q.x2n, 1024);
    uint32_t v = xpow_from(q.x2n, 32);
    const uint32_t x32 = v;
    for (int l = 31; l >= 0; l--) {
        c.k[l] = v;
        v = gf_mul(v, x32);
    }
    return c;
}
static __constant__ CrcLane kCrcLane = make_crc_lane();

// v[i] ^= the rows d before it, d over the terms of the polynomial (x^(32 - d)).
template <bool LAST>
__device__ __forceinline__ void crc_rows(uint32_t (&v)[32], const uint32_t (&w)[8], int i0) {
    constexpr int D[13] = {6, 9, 10, 16, 20, 21, 22, 24, 25, 27, 28, 30, 31};
#pragma unroll
    for (int i = 0; i < 32; i++) {
        if (i < i0 || i >= i0 + 8) continue;
        uint32_t x = v[i] ^ w[i & 7];  // v[i] so far: the row 32 before
#pragma unroll
        for (int t = 0; t < 13; t++)
            if (!LAST || D[t] > i) x ^= v[(i - D[t]) & 31];
        v[i] = x;
    }
}

// The table that folds rows together (T[b][v] = v x^(8 (3 - b)) x^1024 in the reflected form), by the CTA.
__device__ __forceinline__ void init_crc_fold(uint32_t (*T)[256]) {
    for (int i = threadIdx.x; i < 1024; i += blockDim.x)
        T[i >> 8][i & 255] = gf_mul((uint32_t)(i & 255) << (8 * (i >> 8)), kCrcLane.x1024);
}

// The raw column of the 4,096 bytes that crc_rows<true> left in v, the same in every lane.
__device__ __forceinline__ uint32_t crc_fold_rows(const uint32_t (*T)[256], const uint32_t (&v)[32]) {
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < 32; i++) c = T[0][c & 255] ^ T[1][(c >> 8) & 255] ^ T[2][(c >> 16) & 255] ^ T[3][c >> 24] ^ v[i];
    return __reduce_xor_sync(FULL, gf_mul(c, kCrcLane.k[threadIdx.x & 31]));
}

}  // namespace cb
