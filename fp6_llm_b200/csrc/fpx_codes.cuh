// Warp-level re-arrangement of codes between rows and the prepacked layout (device only).
//
// The unit of every weight-format kernel is 64 rows x 32 columns per warp.  Lane 4g+t of the packed layout owns, of such a
// unit, rows {g, g+8, .. g+56} x column pairs (2t, 2t+1) of each of the four 8-column chunks; a thread that reads or writes
// memory wants whole chunks of a row instead (8 codes: 16 bytes of fp16, bw bytes of a code stream).  So lane 4g+s handles
// chunk s of the rows g, g+8, .. on the memory side, and the four lanes of a quad exchange words by a 4 x 4 transpose.
// What is exchanged is already in the byte order of the packed words:
//   b word = [code(r1, 2t+1) | code(r0, 2t+1) | ...] as below: four codes of the row pair r0 = g + 16k, r1 = r0 + 8.
#pragma once
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
