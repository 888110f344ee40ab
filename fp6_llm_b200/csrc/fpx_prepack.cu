// Weight-format kernels for sm_100a:
//   * prepack:            unpacked MSB-first code streams -> the reference's bit-interleaved
//                         [1-bit | 2-bit | 4-bit] region layout, bit-exact with the CPU packer
//                         (fp6_llm/csrc/utils/weight_prepacking.h:118-196);
//   * dequant (unpacked): the reference's CPU dequantiser on the GPU
//                         (fp6_llm/csrc/utils/weight_dequant.h:10-48);
//   * dequant (packed):   prepacked weights -> fp16 [M, K], for fp16 GEMM comparisons and for checking the packed
//                         format end to end (by the packers' way backwards, fpx_codes.cuh, not by the GEMM's unpack code);
//   * repack:             prepacked weights -> the 128 x 128 tiles of fpx_native.cu;
//   * quantise:           fp16 weights -> row scales, and fp16 weights + row scales -> prepacked weights.
// All are byte shuffles bounded by HBM traffic (bytes in + bytes out).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fpx_codes.cuh"
#include "fpx_internal.h"
#include "fpx_layout.h"

namespace fpx {

namespace {

// A CTA of the kernels below = 64 rows x kWarps * kSlots units of 32 columns (fpx_codes.cuh), warps on neighbouring units.
constexpr int kWarps = 8;
constexpr int kSlots = 2;

// Packs the unpacked stream.  A lane cuts its chunks (8 codes, bw bytes) out of two aligned words, neighbouring lanes and
// warps read neighbouring bytes, and the packed words are put together in registers.  HBM-bound: 30 us = 4.1 TB/s
// on 10240 x 8192 e3m2 codes.  (Gathering every field of every word from shared memory with the closed form of
// field_source took 154 us.)
template <int BW>
__global__ void __launch_bounds__(kWarps * 32)
prepack_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t K, uint32_t ctas_per_row, uint64_t off2,
               uint64_t off4) {
    const uint32_t i = blockIdx.x / ctas_per_row;              // 64-row block
    const uint32_t first_unit = (blockIdx.x - i * ctas_per_row) * kSlots * kWarps;
    const int lane = threadIdx.x & 31, g = lane >> 2, s = lane & 3;
    const uint32_t units = K / 32;
    const size_t row_bytes = (size_t)K * BW / 8;               // a multiple of 8 * BW
    const uint32_t at = ((uint32_t)s * BW) & 3u;               // a unit starts on a word: 4 * BW bytes per row
#pragma unroll 1
    for (int slot = 0; slot < kSlots; slot++) {
        const uint32_t unit = first_unit + slot * kWarps + (threadIdx.x >> 5);
        if (unit >= units) return;
        const uint8_t* src = in + ((size_t)i * kRowsPerBlock + g) * row_bytes + (size_t)unit * (4 * BW) + (s * BW - at);
        PackedUnit<BW> words;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t lo[2], hi[2], b[4];
#pragma unroll
            for (int r = 0; r < 2; r++)
                read_stream_chunk<BW>(reinterpret_cast<const uint32_t*>(src + (size_t)(16 * k + 8 * r) * row_bytes), at, lo[r], hi[r]);
            stream_rows_to_quad_words(lo[0], hi[0], lo[1], hi[1], b);
            quad_transpose(b, lane);
            words.add(k, b);
        }
        words.store(out, off2, off4, (uint64_t)i * (K / 16) + (uint64_t)unit * 2, lane);
    }
}

// Round-to-nearest quantiser fused with the packer: fp16 weights [M, K] and fp16 row scales in, prepacked FPx out,
// without the unpacked tensor in between.  (The reference ships no working quantiser: fp6_llm/csrc/utils/
// weight_quant.h:9-104 truncates and is not bound; the layout it would feed is the packer's above.)
// Code of a weight = nearest representable magnitude of |w / scale|; ties go to the even code; beyond the largest
// magnitude it saturates; the sign bit is the sign of the quotient.
//
// HBM-bound (2 + bw / 8 bytes per weight), so the instructions per weight have to stay near ten.  The exact definition
// (quantize_rtn_code: a division and a compare with every midpoint) took 8660 us on 8192 x 28672 e3m2 weights; this form
// takes 113 us = 5.7 TB/s:
//   * w * (1 / scale), with the reciprocal taken once per row, instead of w / scale.  Only the side of the quotient on which
//     a midpoint lies matters, and for fp16 w and scale the two are equal or at least 2^-16 (relative) apart: w and midpoint *
//     scale are integers below 2^11 and 2^16 in units of a power of two.  The product is within 2^-22 of the quotient, so
//     rounding it to a multiple of 32 units in the last place (2^-18) puts exact ties back on the midpoint, which has at most
//     five significant bits, and moves nothing else across one.
//   * rounding to the format by cvt for e3m2 and e2m3, by one addition of a power of two otherwise (round_code).
//   * a lane reads 16 bytes of a row; the packed words are put together in registers (fpx_codes.cuh).
// Rows whose scale is zero, negative or not finite, and chunks that hold an infinite or NaN weight, take the exact definition.
// Code of the magnitude and sign in the bits of a finite float: 2^(23 - M) times the binade's unit (at least the subnormals'
// binade) is added, so that the addition itself rounds to the format's last bit, ties to even.
template <int E_BITS, int M_BITS>
__device__ __forceinline__ uint32_t round_code(uint32_t u) {
    constexpr int kBias = (1 << (E_BITS - 1)) - 1;
    constexpr uint32_t kMinBinade = (uint32_t)(127 + 1 - kBias) << 23;
    // the largest magnitude: (2 - 2^-M) * 2^(2^E - 1 - bias)
    constexpr uint32_t kTop = ((uint32_t)(127 + (1 << E_BITS) - 1 - kBias) << 23) | (((1u << M_BITS) - 1u) << (23 - M_BITS));
    const uint32_t a = min(u & 0x7fffffffu, kTop);
    const uint32_t binade = max(a & 0x7f800000u, kMinBinade);
    const uint32_t c = binade + ((uint32_t)(23 - M_BITS) << 23);
    const uint32_t t = __float_as_uint(__uint_as_float(a) + __uint_as_float(c));
    return (t - c) + ((binade - kMinBinade) >> (23 - M_BITS)) + ((u >> 31) << (E_BITS + M_BITS));
}

// Eight codes, one per byte, of q[0..7].
template <int E_BITS, int M_BITS>
__device__ __forceinline__ void round_codes8(const float (&q)[8], uint32_t& lo, uint32_t& hi) {
    uint32_t u[8];
#pragma unroll
    for (int i = 0; i < 8; i++) u[i] = (__float_as_uint(q[i]) + 16u) & 0xffffffe0u;
    if constexpr ((E_BITS == 3 && M_BITS == 2) || (E_BITS == 2 && M_BITS == 3)) {
        uint32_t pair[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float even = __uint_as_float(u[2 * i]), odd = __uint_as_float(u[2 * i + 1]);
            uint16_t h;
            if constexpr (E_BITS == 3) asm("cvt.rn.satfinite.e3m2x2.f32 %0, %1, %2;" : "=h"(h) : "f"(odd), "f"(even));
            else asm("cvt.rn.satfinite.e2m3x2.f32 %0, %1, %2;" : "=h"(h) : "f"(odd), "f"(even));
            pair[i] = h;
        }
        lo = pair[0] | (pair[1] << 16);
        hi = pair[2] | (pair[3] << 16);
    } else {
        uint32_t c[8];
#pragma unroll
        for (int i = 0; i < 8; i++) c[i] = round_code<E_BITS, M_BITS>(u[i]);
        lo = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
        hi = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
    }
}

template <int E_BITS, int M_BITS>
__device__ __noinline__ uint2 exact_codes8(uint4 raw, float scale) {
    const uint32_t h[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t out[2] = {0u, 0u};
    for (int i = 0; i < 8; i++) {
        const float w = __half2float(__ushort_as_half((unsigned short)(h[i >> 1] >> (16 * (i & 1)))));
        out[i >> 2] |= quantize_rtn_code(E_BITS, M_BITS, __fdiv_rn(w, scale)) << (8 * (i & 3));
    }
    return make_uint2(out[0], out[1]);
}

template <int E_BITS, int M_BITS>
__global__ void __launch_bounds__(kWarps * 32)
quantize_prepack_kernel(const __half* __restrict__ w, const __half* __restrict__ scales, uint8_t* __restrict__ out,
                        uint32_t K, uint32_t ctas_per_row, uint64_t off2, uint64_t off4, int aligned16) {
    constexpr int BW = 1 + E_BITS + M_BITS;
    __shared__ float row_scale[kRowsPerBlock], row_inv[kRowsPerBlock];   // row_inv 0: the row takes the exact definition
    const uint32_t i = blockIdx.x / ctas_per_row;              // 64-row block
    const uint32_t first_unit = (blockIdx.x - i * ctas_per_row) * kSlots * kWarps;
    const int lane = threadIdx.x & 31, g = lane >> 2, s = lane & 3;
    if (threadIdx.x < kRowsPerBlock) {
        const float sc = __half2float(scales[(size_t)i * kRowsPerBlock + threadIdx.x]);
        row_scale[threadIdx.x] = sc;
        row_inv[threadIdx.x] = (sc > 0.0f && sc < 65536.0f) ? 1.0f / sc : 0.0f;
    }
    __syncthreads();
    const uint32_t units = K / 32;
#pragma unroll 1
    for (int slot = 0; slot < kSlots; slot++) {
        const uint32_t unit = first_unit + slot * kWarps + (threadIdx.x >> 5);
        if (unit >= units) return;
        const __half* src = w + ((size_t)i * kRowsPerBlock + g) * K + (size_t)unit * 32 + s * 8;
        uint4 raw[8];
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const __half* p = src + (size_t)(8 * r) * K;
            if (aligned16) {
                raw[r] = __ldg(reinterpret_cast<const uint4*>(p));
            } else {
                const uint32_t* p4 = reinterpret_cast<const uint32_t*>(p);
                raw[r] = make_uint4(__ldg(p4), __ldg(p4 + 1), __ldg(p4 + 2), __ldg(p4 + 3));
            }
        }
        PackedUnit<BW> words;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t lo[2], hi[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint4 v = raw[2 * k + r];
                const int row = 16 * k + 8 * r + g;
                const float inv = row_inv[row];
                const __half2* h = reinterpret_cast<const __half2*>(&v);
                // 0 * x summed over the chunk: anything but a zero means an infinite or NaN weight
                const __half2 zero = __half2half2(__ushort_as_half((unsigned short)0));
                const __half2 probe = __hfma2(h[0], zero, __hfma2(h[1], zero, __hfma2(h[2], zero, __hmul2(h[3], zero))));
                if (inv == 0.0f || (*reinterpret_cast<const uint32_t*>(&probe) & 0x7fff7fffu) != 0u) {
                    const uint2 c = exact_codes8<E_BITS, M_BITS>(v, row_scale[row]);
                    lo[r] = c.x; hi[r] = c.y;
                } else {
                    float q[8];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float2 f = __half22float2(h[e]);
                        q[2 * e] = f.x * inv;
                        q[2 * e + 1] = f.y * inv;
                    }
                    round_codes8<E_BITS, M_BITS>(q, lo[r], hi[r]);
                }
            }
            __syncwarp();
            uint32_t b[4];
            rows_to_quad_words(lo[0], hi[0], lo[1], hi[1], b);
            quad_transpose(b, lane);
            words.add(k, b);
        }
        words.store(out, off2, off4, (uint64_t)i * (K / 16) + (uint64_t)unit * 2, lane);
    }
}

// Row scales of a quantiser: max|w| of a row divided by the format's largest magnitude, not below 2^-24, as fp16.  One CTA per
// row, 16 bytes per lane and round.  Absolute values of fp16 compare like their bit patterns, with NaN above infinity, so
// the maximum is taken on integers and a NaN in the row comes out as NaN.  HBM-bound: 69 us = 6.8 TB/s on
// 8192 x 28672 (five elementwise and reduction launches in fp32 took 1045 us).
__global__ void __launch_bounds__(256) row_scales_kernel(const __half* __restrict__ w, __half* __restrict__ scales, uint32_t K,
                                                          float inv_top) {
    const uint4* row = reinterpret_cast<const uint4*>(w + (size_t)blockIdx.x * K);
    const uint32_t chunks = K / 8;
    uint32_t m = 0;   // two 16-bit maxima
    auto take = [&](const uint4& v) {
        m = __vmaxu2(m, __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu)));
    };
    uint32_t c = threadIdx.x;
    for (; c + 3 * 256 < chunks; c += 4 * 256) {   // four loads in flight per lane
        const uint4 v0 = __ldg(row + c), v1 = __ldg(row + c + 256), v2 = __ldg(row + c + 512), v3 = __ldg(row + c + 768);
        take(v0); take(v1); take(v2); take(v3);
    }
    for (; c < chunks; c += 256) take(__ldg(row + c));
    m = max(m & 0xffffu, m >> 16);
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ uint32_t part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < 8; i++) m = max(m, part[i]);
        const float s = __half2float(__ushort_as_half((unsigned short)m)) * inv_top;
        scales[blockIdx.x] = __float2half_rn(s < 5.9604644775390625e-8f ? 5.9604644775390625e-8f : s);   // 2^-24; NaN stays
    }
}

// Unpacked codes -> fp16.  A warp takes 1024 columns of a row, a lane four chunks of 8 codes, 32 chunks apart: neighbouring lanes
// read neighbouring bytes (two aligned words per chunk) and write neighbouring 16 bytes.  HBM-bound: 42 us = 5.5 TB/s on
// 10240 x 8192 e3m2 codes (byte loads and a division of the index per chunk took 54 us).
constexpr uint32_t kDequantChunks = 128;   // chunks per warp
template <int E_BITS, int M_BITS>
__global__ void __launch_bounds__(256)
dequant_unpacked_kernel(const uint8_t* __restrict__ in, const __half* __restrict__ scales, __half* __restrict__ out,
                        uint32_t M, uint32_t K, uint32_t warps_per_row, int aligned4) {
    constexpr int BW = 1 + E_BITS + M_BITS;
    const uint32_t id = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t row = id / warps_per_row;
    if (row >= M) return;
    const uint32_t chunks = K / 8, c0 = (id - row * warps_per_row) * kDequantChunks + lane;
    const __half2 bias = __half2half2(__ushort_as_half(bias_half_bits(E_BITS)));
    const __half2 scale = __half2half2(scales[row]);
    const uint8_t* src = in + (size_t)row * chunks * BW;       // a row starts on a word: chunks is a multiple of 8
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * K);
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const uint32_t c = c0 + 32 * u;
        lo[u] = hi[u] = 0u;
        if (c >= chunks) continue;
        const uint32_t byte = c * BW;
        if (aligned4) {
            read_stream_chunk<BW>(reinterpret_cast<const uint32_t*>(src + (byte & ~3u)), byte & 3u, lo[u], hi[u]);
        } else {   // a stream that starts between two words
            uint32_t v[2] = {0u, 0u};
#pragma unroll
            for (int b = 0; b < BW; b++) v[b >> 2] |= (uint32_t)src[byte + b] << (8 * (b & 3));
            cut_stream_chunk<BW>(v[0], v[1], 0u, lo[u], hi[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const uint32_t c = c0 + 32 * u;
        if (c >= chunks) break;
        const uint32_t l = lo[u] << (8 - BW), h = hi[u] << (8 - BW);   // left-aligned in every byte; columns from the top byte down
        uint4 v;
        v.x = scaled_pair(pattern_pair<E_BITS>(__byte_perm(l, 0u, 0x2434)), bias, scale);
        v.y = scaled_pair(pattern_pair<E_BITS>(__byte_perm(l, 0u, 0x0414)), bias, scale);
        v.z = scaled_pair(pattern_pair<E_BITS>(__byte_perm(h, 0u, 0x2434)), bias, scale);
        v.w = scaled_pair(pattern_pair<E_BITS>(__byte_perm(h, 0u, 0x0414)), bias, scale);
        dst[c] = v;
    }
}

// Prepacked codes -> fp16: the way of the packers backwards, so that a lane stores 16 bytes of a row.  HBM-bound: 36 us =
// 6.4 TB/s on 10240 x 8192 e3m2 codes (storing the register pairs of the GEMM's unpack, 4 bytes each, took 70 us).
template <int E_BITS, int M_BITS>
__global__ void __launch_bounds__(kWarps * 32)
dequant_packed_kernel(const uint8_t* __restrict__ packed, const __half* __restrict__ scales, __half* __restrict__ out,
                      uint32_t K, uint32_t ctas_per_row, uint64_t off2, uint64_t off4, int aligned16) {
    constexpr int BW = 1 + E_BITS + M_BITS;
    __shared__ __half row_scale[kRowsPerBlock];
    const uint32_t i = blockIdx.x / ctas_per_row;              // 64-row block
    const uint32_t first_unit = (blockIdx.x - i * ctas_per_row) * kSlots * kWarps;
    const int lane = threadIdx.x & 31, g = lane >> 2, s = lane & 3;
    if (threadIdx.x < kRowsPerBlock) row_scale[threadIdx.x] = scales[(size_t)i * kRowsPerBlock + threadIdx.x];
    __syncthreads();
    const __half2 bias = __half2half2(__ushort_as_half(bias_half_bits(E_BITS)));
    const uint32_t units = K / 32;
#pragma unroll 1
    for (int slot = 0; slot < kSlots; slot++) {
        const uint32_t unit = first_unit + slot * kWarps + (threadIdx.x >> 5);
        if (unit >= units) return;
        PackedUnit<BW> words;
        words.load(packed, off2, off4, (uint64_t)i * (K / 16) + (uint64_t)unit * 2, lane);
        __half* dst = out + ((size_t)i * kRowsPerBlock + g) * K + (size_t)unit * 32 + s * 8;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t b[4], lo[2], hi[2];
            words.take(k, b);
            quad_transpose(b, lane);
            quad_words_to_rows(b, lo[0], hi[0], lo[1], hi[1]);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const __half2 scale = __half2half2(row_scale[16 * k + 8 * r + g]);
                const uint32_t l = lo[r] << (8 - BW), h = hi[r] << (8 - BW);
                uint4 v;
                v.x = scaled_pair(pattern_pair<E_BITS>(__byte_perm(l, 0u, 0x1404)), bias, scale);
                v.y = scaled_pair(pattern_pair<E_BITS>(__byte_perm(l, 0u, 0x3424)), bias, scale);
                v.z = scaled_pair(pattern_pair<E_BITS>(__byte_perm(h, 0u, 0x1404)), bias, scale);
                v.w = scaled_pair(pattern_pair<E_BITS>(__byte_perm(h, 0u, 0x3424)), bias, scale);
                __half* p = dst + (size_t)(16 * k + 8 * r) * K;
                if (aligned16) {
                    *reinterpret_cast<uint4*>(p) = v;
                } else {
                    uint32_t* p4 = reinterpret_cast<uint32_t*>(p);
                    p4[0] = v.x; p4[1] = v.y; p4[2] = v.z; p4[3] = v.w;
                }
            }
        }
    }
}

// Prepacked weights -> tiles of 128 rows x 128 K, six bits per code whatever the format, code i of a row at bits 6i .. 6i + 5.
// The six-bit code of the same value in the tensor-core format with E exponent bits (e3m2 or e2m3) has the same fields with the
// mantissa extended by zeros.  CTA = 64 rows x 256 columns, a warp per unit: the lanes bring the codes into row order as the
// dequantiser does, join eight of them to six bytes and put these into shared memory, where the 64 rows of a tile are one run
// of 6 KB; the CTA then stores that run 16 bytes per thread.  K tiles that reach past K are filled with code 0 (+0).
// HBM-bound: 70 us = 5.0 TB/s on 8192 x 28672 e3m2 weights (writing each row's 12-byte pieces as they came took 105 us).
constexpr int kHalfTileBytes = kRowsPerBlock * kNatRowBytes;
template <int BW>
__global__ void __launch_bounds__(kWarps * 32) native_repack_kernel(const uint8_t* __restrict__ packed, uint8_t* __restrict__ native,
                                                                    uint32_t K, uint32_t ktiles, uint32_t ctas_per_row, uint64_t off2,
                                                                    uint64_t off4) {
    __shared__ __align__(16) uint8_t rows[2][kHalfTileBytes];
    const uint32_t i = blockIdx.x / ctas_per_row;              // 64-row block
    const uint32_t tile0 = (blockIdx.x - i * ctas_per_row) * 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, s = lane & 3;
    const uint32_t unit = tile0 * 4 + warp;
    if (unit < ktiles * 4) {
        PackedUnit<BW> words = {};
        if (unit < K / 32) words.load(packed, off2, off4, (uint64_t)i * (K / 16) + (uint64_t)unit * 2, lane);
        uint8_t* dst = &rows[warp >> 2][g * kNatRowBytes + (warp & 3) * 24 + s * 6];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t b[4], lo[2], hi[2];
            words.take(k, b);
            quad_transpose(b, lane);
            quad_words_to_rows(b, lo[0], hi[0], lo[1], hi[1]);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t first = join_codes6(lo[r] << (6 - BW)), second = join_codes6(hi[r] << (6 - BW));
                uint16_t* p = reinterpret_cast<uint16_t*>(dst + (16 * k + 8 * r) * kNatRowBytes);
                p[0] = (uint16_t)first;
                p[1] = (uint16_t)((first >> 16) | (second << 8));
                p[2] = (uint16_t)(second >> 8);
            }
        }
    }
    __syncthreads();
    constexpr uint32_t kChunks = kHalfTileBytes / 16;
    for (uint32_t c = threadIdx.x; c < 2 * kChunks; c += kWarps * 32) {
        const uint32_t t = c / kChunks, at = c - t * kChunks;
        if (tile0 + t >= ktiles) break;
        uint8_t* dst = native + ((size_t)(i >> 1) * ktiles + tile0 + t) * kNatTileBytes + (i & 1) * kHalfTileBytes;
        reinterpret_cast<uint4*>(dst)[at] = reinterpret_cast<const uint4*>(rows[t])[at];
    }
}

bool shape_ok(int e_bits, int m_bits, size_t M, size_t K) {
    // the packer itself needs 64-row / 64-column granularity (weight_prepacking.h:121-122)
    return format_supported(e_bits, m_bits) && M > 0 && K > 0 && M % 64 == 0 && K % 64 == 0 && M <= 0xffffffffull &&
           K <= 0x7fffffffull;
}

}  // namespace

namespace {
// CTAs of a kernel that takes 64 rows x kWarps * kSlots units per CTA: per row of blocks, and in all (0: too many)
size_t unit_ctas(size_t M, size_t K, uint32_t* per_row) {
    const uint32_t per_cta = kWarps * kSlots;
    *per_row = ((uint32_t)(K / 32) + per_cta - 1) / per_cta;
    const size_t ctas = (M / kRowsPerBlock) * *per_row;
    return ctas <= 0x7fffffffull ? ctas : 0;
}
}  // namespace

cudaError_t launch_prepack(int e_bits, int m_bits, cudaStream_t stream, const void* unpacked, void* packed, size_t M,
                           size_t K) {
    if (!shape_ok(e_bits, m_bits, M, K) || !unpacked || !packed || unpacked == packed) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(unpacked) & 3) || (reinterpret_cast<uintptr_t>(packed) & 3))
        return cudaErrorMisalignedAddress;
    uint32_t per_row = 0;
    const size_t ctas = unit_ctas(M, K, &per_row);
    if (ctas == 0) return cudaErrorInvalidValue;
    const uint8_t* in = static_cast<const uint8_t*>(unpacked);
    uint8_t* out = static_cast<uint8_t*>(packed);
    const int bw = bit_width(e_bits, m_bits);
    const uint64_t off2 = region_offset(bw, 2, M, K), off4 = region_offset(bw, 4, M, K);
    switch (bw) {
        case 4:  prepack_kernel<4><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, per_row, off2, off4); break;
        case 5:  prepack_kernel<5><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, per_row, off2, off4); break;
        default: prepack_kernel<6><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, per_row, off2, off4); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_quantize_prepack(int e_bits, int m_bits, cudaStream_t stream, const __half* weights,
                                    const __half* scales, void* packed, size_t M, size_t K) {
    if (!shape_ok(e_bits, m_bits, M, K) || !weights || !scales || !packed) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(weights) & 3) || (reinterpret_cast<uintptr_t>(packed) & 3))
        return cudaErrorMisalignedAddress;
    uint8_t* out = static_cast<uint8_t*>(packed);
    const int bw = bit_width(e_bits, m_bits);
    const uint64_t off2 = region_offset(bw, 2, M, K), off4 = region_offset(bw, 4, M, K);
    const int aligned16 = (reinterpret_cast<uintptr_t>(weights) & 15) == 0;
    uint32_t per_row = 0;
    const size_t ctas = unit_ctas(M, K, &per_row);
    if (ctas == 0) return cudaErrorInvalidValue;
    FPX_DISPATCH_FORMAT(e_bits, m_bits, (quantize_prepack_kernel<kE, kM><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(weights, scales, out, (uint32_t)K, per_row, off2, off4, aligned16)));
    return cudaGetLastError();
}

cudaError_t launch_row_scales(cudaStream_t stream, const __half* weights, __half* scales, size_t M, size_t K, float top) {
    if (!weights || !scales || M == 0 || M > 0x7fffffffull || K == 0 || K % 8 != 0 || K > 0x7fffffffull || !(top > 0.0f))
        return cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(weights) & 15) return cudaErrorMisalignedAddress;
    row_scales_kernel<<<(unsigned)M, 256, 0, stream>>>(weights, scales, (uint32_t)K, 1.0f / top);
    return cudaGetLastError();
}

cudaError_t launch_dequant_unpacked(int e_bits, int m_bits, cudaStream_t stream, const void* unpacked,
                                    const __half* scales, __half* out, size_t M, size_t K) {
    if (!shape_ok(e_bits, m_bits, M, K) || !unpacked || !scales || !out) return cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(out) & 15) return cudaErrorMisalignedAddress;
    const uint32_t warps_per_row = ((uint32_t)(K / 8) + kDequantChunks - 1) / kDequantChunks;
    const size_t warps = M * warps_per_row;
    if (warps > 0xffffffffull - 8) return cudaErrorInvalidValue;
    const unsigned ctas = (unsigned)((warps + 7) / 8);
    const uint8_t* in = static_cast<const uint8_t*>(unpacked);
    FPX_DISPATCH_FORMAT(e_bits, m_bits, (dequant_unpacked_kernel<kE, kM><<<ctas, 256, 0, stream>>>(in, scales, out, (uint32_t)M, (uint32_t)K, warps_per_row, (reinterpret_cast<uintptr_t>(unpacked) & 3) == 0)));
    return cudaGetLastError();
}

cudaError_t launch_dequant_packed(int e_bits, int m_bits, cudaStream_t stream, const void* packed,
                                  const __half* scales, __half* out, size_t M, size_t K) {
    if (!shape_ok(e_bits, m_bits, M, K) || !packed || !scales || !out) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(packed) & 15) || (reinterpret_cast<uintptr_t>(out) & 3))
        return cudaErrorMisalignedAddress;
    uint32_t per_row = 0;
    const size_t ctas = unit_ctas(M, K, &per_row);
    if (ctas == 0) return cudaErrorInvalidValue;
    const uint8_t* in = static_cast<const uint8_t*>(packed);
    const int bw = bit_width(e_bits, m_bits);
    const uint64_t off2 = region_offset(bw, 2, M, K), off4 = region_offset(bw, 4, M, K);
    const int aligned16 = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    FPX_DISPATCH_FORMAT(e_bits, m_bits, (dequant_packed_kernel<kE, kM><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, scales, out, (uint32_t)K, per_row, off2, off4, aligned16)));
    return cudaGetLastError();
}

cudaError_t launch_native_repack(int e_bits, int m_bits, cudaStream_t stream, const void* packed, void* native, size_t M, size_t K) {
    if (!native_format(e_bits, m_bits) || !packed || !native || packed == native) return cudaErrorInvalidValue;
    if (M == 0 || M % 256 != 0 || K == 0 || K % 64 != 0 || M > 0x7fffffffull || K > 0x7fffffffull) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(packed) & 3) || (reinterpret_cast<uintptr_t>(native) & 15)) return cudaErrorMisalignedAddress;
    const uint32_t ktiles = (uint32_t)((K + kNatTileK - 1) / kNatTileK), per_row = (ktiles + 1) / 2;
    const size_t ctas = (M / kRowsPerBlock) * per_row;
    if (ctas > 0x7fffffffull) return cudaErrorInvalidValue;
    const uint8_t* in = static_cast<const uint8_t*>(packed);
    uint8_t* out = static_cast<uint8_t*>(native);
    const int bw = bit_width(e_bits, m_bits);
    const uint64_t off2 = region_offset(bw, 2, M, K), off4 = region_offset(bw, 4, M, K);
    switch (bw) {
        case 4:  native_repack_kernel<4><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, ktiles, per_row, off2, off4); break;
        case 5:  native_repack_kernel<5><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, ktiles, per_row, off2, off4); break;
        default: native_repack_kernel<6><<<(unsigned)ctas, kWarps * 32, 0, stream>>>(in, out, (uint32_t)K, ktiles, per_row, off2, off4); break;
    }
    return cudaGetLastError();
}

}  // namespace fpx
