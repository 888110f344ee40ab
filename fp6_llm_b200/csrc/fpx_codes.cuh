// Warp-level re-arrangement of codes between rows and the prepacked layout (device only).
//
// The unit of every weight-format kernel is 64 rows x 32 columns per warp.  Lane 4g+t of the packed layout owns, of such a
// unit, rows {g, g+8, .. g+56} x column pairs (2t, 2t+1) of each of the four 8-column chunks; a thread that reads or writes
// memory wants whole chunks of a row instead (8 codes: 16 bytes of fp16, bw bytes of a code stream).  So lane 4g+s handles
// chunk s of the rows g, g+8, .. on the memory side, and the four lanes of a quad exchange words by a 4 x 4 transpose.
// What is exchanged is already in the byte order of the packed words:
//   b word = [code(r1, 2t+1) | code(r0, 2t+1) | ...] as below: four codes of the row pair r0 = g + 16k, r1 = r0 + 8.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "fpx_layout.h"

namespace fpx {

// Four codes, one per byte: bytes from the top = (r0, odd column), (r1, odd), (r0, even), (r1, even): the order in which the
// packed words hold the codes of one lane (see field_source in fpx_layout.h).
// `lo`/`hi` of a row: its eight codes of a chunk, one per byte, column 0 in the lowest byte of lo.
__device__ __forceinline__ void rows_to_quad_words(uint32_t r0_lo, uint32_t r0_hi, uint32_t r1_lo, uint32_t r1_hi, uint32_t b[4]) {
    b[0] = __byte_perm(r0_lo, r1_lo, 0x1504);
    b[1] = __byte_perm(r0_lo, r1_lo, 0x3726);
    b[2] = __byte_perm(r0_hi, r1_hi, 0x1504);
    b[3] = __byte_perm(r0_hi, r1_hi, 0x3726);
}
// The same for rows whose column 0 is in the HIGHEST byte of `lo` (codes cut from a big-endian stream).
__device__ __forceinline__ void stream_rows_to_quad_words(uint32_t r0_lo, uint32_t r0_hi, uint32_t r1_lo, uint32_t r1_hi, uint32_t b[4]) {
    b[0] = __byte_perm(r0_lo, r1_lo, 0x2637);
    b[1] = __byte_perm(r0_lo, r1_lo, 0x0415);
    b[2] = __byte_perm(r0_hi, r1_hi, 0x2637);
    b[3] = __byte_perm(r0_hi, r1_hi, 0x0415);
}
__device__ __forceinline__ void quad_words_to_rows(const uint32_t b[4], uint32_t& r0_lo, uint32_t& r0_hi, uint32_t& r1_lo, uint32_t& r1_hi) {
    r0_lo = __byte_perm(b[0], b[1], 0x7531);
    r0_hi = __byte_perm(b[2], b[3], 0x7531);
    r1_lo = __byte_perm(b[0], b[1], 0x6420);
    r1_hi = __byte_perm(b[2], b[3], 0x6420);
}

// v[i] of lane j of a quad becomes v[j] of lane i.
__device__ __forceinline__ void quad_transpose(uint32_t v[4], int lane) {
#pragma unroll
    for (int bit = 1; bit <= 2; bit <<= 1) {
        const bool up = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (i & bit) continue;
            const uint32_t send = up ? v[i] : v[i | bit];
            const uint32_t got = __shfl_xor_sync(0xffffffffu, send, bit);
            if (up) v[i] = got; else v[i | bit] = got;
        }
    }
}

// The eight codes of a chunk of the unpacked, MSB-first stream, one per byte, column 0 in the highest byte of lo.  v0: the
// aligned 32-bit word that holds the chunk's first byte, `at`: which of its bytes that is, v1: the next word.  Chunks of 5
// or 6 bytes that start on a multiple of their length always reach into v1 and never past it, those of 4 bytes never do.
template <int BW>
__device__ __forceinline__ void cut_stream_chunk(uint32_t v0, uint32_t v1, uint32_t at, uint32_t& lo, uint32_t& hi) {
    uint32_t a, b;   // codes 0..3 and 4..7 in the lowest 4 * BW bits; what lies above is masked off below
    if constexpr (BW == 6) {
        a = __byte_perm(v0, v1, 0x0012 + 0x0111 * at);
        b = __byte_perm(v0, v1, 0x0345 + 0x0111 * at);
    } else if constexpr (BW == 5) {
        const uint32_t top = __byte_perm(v0, v1, 0x0123 + 0x1111 * at), last = __byte_perm(v0, v1, 0x0004 + at);
        a = top >> 12;
        b = (top << 8) | (last & 0xffu);
    } else {
        a = __byte_perm(v0, v1, 0x0001);
        b = __byte_perm(v0, v1, 0x0023);
    }
    constexpr uint32_t code = (1u << BW) - 1u, even = code | (code << 16), odd = even << 8;
    a = ((a << (16 - 2 * BW)) & 0xffff0000u) | (a & 0xffffu);
    b = ((b << (16 - 2 * BW)) & 0xffff0000u) | (b & 0xffffu);
    lo = ((a << (8 - BW)) & odd) | (a & even);
    hi = ((b << (8 - BW)) & odd) | (b & even);
}

// Four six-bit codes, one per byte, column 0 in the lowest -> 24 bits, code i at bits 6i .. 6i + 5.
__device__ __forceinline__ uint32_t join_codes6(uint32_t c) {
    const uint32_t two = (c & 0x003f003fu) | ((c >> 2) & 0x0fc00fc0u);
    return (two & 0xfffu) | ((two >> 4) & 0xfff000u);
}

template <int BW>
__device__ __forceinline__ void read_stream_chunk(const uint32_t* first, uint32_t at, uint32_t& lo, uint32_t& hi) {
    cut_stream_chunk<BW>(__ldg(first), BW == 4 ? 0u : __ldg(first + 1), at, lo, hi);
}

// Two fp16 patterns sign | (exponent, mantissa) >> (5 - E) from codes in the upper bytes of both halves, left-aligned there.
template <int E_BITS>
__device__ __forceinline__ uint32_t pattern_pair(uint32_t x) {
    constexpr uint32_t below = (0x7fffu >> (5 - E_BITS)) * 0x00010001u;
    return (x & 0x80008000u) | ((x >> (5 - E_BITS)) & below);
}
// value = code value * scale in fp16: the first product (by 2^bias) is exact, the second rounds once, as in the reference.
__device__ __forceinline__ uint32_t scaled_pair(uint32_t pattern, __half2 bias, __half2 scale) {
    const __half2 v = __hmul2(__hmul2(*reinterpret_cast<const __half2*>(&pattern), bias), scale);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// The packed words of one unit, built from its b words: add(k, b) takes, for the row pair k (rows g + 16k, g + 16k + 8),
// b[s] = chunk s; columns 0..15 of the unit are the chunks 0 (first half) and 1 (second half), columns 16..31 the chunks 2, 3.
// word4[j][k], word2[j][k / 2], word1[j]: the lane's words of 16-column block j.
template <int BW>
struct PackedUnit {
    uint32_t w4[2][4], w2[2][2], w1[2];
    __device__ __forceinline__ void add(int k, const uint32_t b[4]) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t h0 = b[2 * j], h1 = b[2 * j + 1];
            w4[j][k] = ((h0 & 0x0f0f0f0fu) << 4) | (h1 & 0x0f0f0f0fu);
            if (BW == 6) {   // bits 7-6 of every byte: chunk half 0 of the even k, then half 1, then the odd k's
                const uint32_t t0 = h0 & 0x30303030u, t1 = h1 & 0x30303030u;
                if (k & 1) w2[j][k >> 1] |= (t0 >> 2) | (t1 >> 4);
                else w2[j][k >> 1] = (t0 << 2) | t1;
            }
            if (BW == 5) {   // bit 7 - (2k + half) of every byte
                const uint32_t t = (((h0 & 0x10101010u) << 3) | ((h1 & 0x10101010u) << 2)) >> (2 * k);
                w1[j] = k ? (w1[j] | t) : t;
            }
        }
    }
    __device__ __forceinline__ void take(int k, uint32_t b[4]) const {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            uint32_t h0 = (w4[j][k] >> 4) & 0x0f0f0f0fu, h1 = w4[j][k] & 0x0f0f0f0fu;
            if (BW == 6) {
                const uint32_t v = w2[j][k >> 1];
                h0 |= (k & 1 ? v << 2 : v >> 2) & 0x30303030u;
                h1 |= (k & 1 ? v << 4 : v) & 0x30303030u;
            }
            if (BW == 5) {
                h0 |= ((w1[j] << (2 * k)) >> 3) & 0x10101010u;
                h1 |= ((w1[j] << (2 * k)) >> 2) & 0x10101010u;
            }
            b[2 * j] = h0;
            b[2 * j + 1] = h1;
        }
    }
    // j0: index of the unit's first 16-column block counted over the matrix, (64-row block) * (cols / 16) + column / 16
    __device__ __forceinline__ void store(uint8_t* packed, uint64_t off2, uint64_t off4, uint64_t j0, int lane) const {
        uint32_t* r4 = reinterpret_cast<uint32_t*>(packed + off4) + j0 * 128 + lane;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) r4[(j * 4 + k) * 32] = w4[j][k];
        if (BW == 6) {
            uint32_t* r2 = reinterpret_cast<uint32_t*>(packed + off2) + j0 * 64 + lane;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int k = 0; k < 2; k++) r2[(j * 2 + k) * 32] = w2[j][k];
        }
        if (BW == 5) {
            uint32_t* r1 = reinterpret_cast<uint32_t*>(packed) + j0 * 32 + lane;
#pragma unroll
            for (int j = 0; j < 2; j++) r1[j * 32] = w1[j];
        }
    }
    __device__ __forceinline__ void load(const uint8_t* packed, uint64_t off2, uint64_t off4, uint64_t j0, int lane) {
        const uint32_t* r4 = reinterpret_cast<const uint32_t*>(packed + off4) + j0 * 128 + lane;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) w4[j][k] = __ldg(r4 + (j * 4 + k) * 32);
        if (BW == 6) {
            const uint32_t* r2 = reinterpret_cast<const uint32_t*>(packed + off2) + j0 * 64 + lane;
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int k = 0; k < 2; k++) w2[j][k] = __ldg(r2 + (j * 2 + k) * 32);
        }
        if (BW == 5) {
            const uint32_t* r1 = reinterpret_cast<const uint32_t*>(packed) + j0 * 32 + lane;
#pragma unroll
            for (int j = 0; j < 2; j++) w1[j] = __ldg(r1 + j * 32);
        }
    }
};

}  // namespace fpx
