// Last step of an output tile, shared by the GEMM kernels: 16 finished fp32 columns of a warp's 32 rows (lane = row) ->
// activation -> fp16 -> memory.
//
// A lane that stored its own row wrote 2 bytes per column, and with the gate/up product every lane computed it for every
// column although only the even ones stored it: 16 shuffles, 16 products with an IEEE division each, 16 two-byte stores per
// 16 columns.  Instead neighbouring lanes exchange what the other needs and take every second column each (one shuffle per
// two columns), lanes two and four apart do the same with the packed halves, and a lane stores 8 bytes (four rows of one
// column): plain 12 shuffles + 4 stores, gate/up 14 shuffles + 8 products + 2 stores.  The tensor cores wait meanwhile (the
// next tile needs the accumulator), so this is main-loop time: a tile of 256 columns with the gate/up product gave up ~17 us
// beside ~50 us of MMAs.  57344 x 8192 gate/up layers in a chain, together with the tile ends on the unpack warps
// (fpx_gemm.cu): 1763 -> 1540 us at 2048 tokens, 397 -> 335 us at 512, where the same layers without the product take 1440 and 346.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "fpx_internal.h"
#include "ptx_sm100.cuh"

namespace fpx {

// silu(gate) * up in fp32, every operation rounded once: 3.29 units of 2^-24 off on average over gates of -30 .. 30, 30.5 at most
// (the exponential's part).  With the hardware's approximate reciprocal instead of the division it was 3.32 and 31.1, and
// whole passes ran 1 - 2 % faster (70B block at 64 tokens 189.7 against 193.4 us, at 512 708 against 715): precision counts.
__device__ __forceinline__ float silu_mul(float gate, float up) { return gate / (1.0f + __expf(-gate)) * up; }

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// f[u] = column n0 + u (u < 16, or < CH when the tile is narrower) of row `row` (row of lane 0 a multiple of 32), biased and
// scaled; columns past N are not stored.  Rows of the targets are 8-byte aligned at every fourth row.
template <int CH>
__device__ __forceinline__ void store_columns(const OutTargets& out, int activation, float (&f)[CH], uint32_t n0, uint32_t N,
                                              uint32_t row, int lane) {
    static_assert(CH == 4 || CH == 8 || CH == 16, "columns per round");
    const bool odd = lane & 1, second = lane & 2, fourth = lane & 4;
    if (activation == kActSiluMul) {   // rows 2c (gate) and 2c + 1 (up) of output channel c sit in neighbouring lanes
        float y[CH / 2];               // channel row / 2 of column 2j + odd
#pragma unroll
        for (int j = 0; j < CH / 2; j++) {
            const float got = __shfl_xor_sync(0xffffffffu, odd ? f[2 * j] : f[2 * j + 1], 1);
            y[j] = silu_mul(odd ? got : f[2 * j], odd ? f[2 * j + 1] : got);
        }
        uint32_t w[CH / 4];            // two channels of column 4j + 2 * second + odd
#pragma unroll
        for (int j = 0; j < CH / 4; j++) {
            const float got = __shfl_xor_sync(0xffffffffu, second ? y[2 * j] : y[2 * j + 1], 2);
            w[j] = second ? pack_half2(got, y[2 * j + 1]) : pack_half2(y[2 * j], got);
        }
        const uint32_t n1 = n0 + 2u * second + odd;
        if constexpr (CH >= 8) {       // four channels of column 8j + 4 * fourth + 2 * second + odd
            __half* dst = out.ptr[0] + out.row0 + ((row & ~7u) >> 1);
#pragma unroll
            for (int j = 0; j < CH / 8; j++) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, fourth ? w[2 * j] : w[2 * j + 1], 4);
                const uint2 v = fourth ? make_uint2(got, w[2 * j + 1]) : make_uint2(w[2 * j], got);
                const uint32_t n = n1 + 8u * j + 4u * fourth;
                if (n < N) *reinterpret_cast<uint2*>(dst + (size_t)n * out.ld) = v;
            }
        } else {                       // four columns: two channels each
            if (n1 < N) *reinterpret_cast<uint32_t*>(out.ptr[0] + (size_t)n1 * out.ld + out.row0 + ((row & ~3u) >> 1)) = w[0];
        }
        return;
    }
    uint32_t w[CH / 2];                // two rows of column 2j + odd
#pragma unroll
    for (int j = 0; j < CH / 2; j++) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? f[2 * j] : f[2 * j + 1], 1);
        w[j] = odd ? pack_half2(got, f[2 * j + 1]) : pack_half2(f[2 * j], got);
    }
    uint2 v[CH / 4];                   // four rows of column 4j + 2 * second + odd
#pragma unroll
    for (int j = 0; j < CH / 4; j++) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, second ? w[2 * j] : w[2 * j + 1], 2);
        v[j] = second ? make_uint2(got, w[2 * j + 1]) : make_uint2(w[2 * j], got);
    }
    const uint32_t n1 = n0 + 2u * second + odd;
    const size_t first = out.row0 + (row & ~3u);
#pragma unroll 1
    for (uint32_t r = 0; r < out.count; r++) {   // one target, or the buffer of every rank
        __half* dst = out.ptr[r] + first;
#pragma unroll
        for (int j = 0; j < CH / 4; j++) {
            const uint32_t n = n1 + 4u * j;
            if (n < N) *reinterpret_cast<uint2*>(dst + (size_t)n * out.ld) = v[j];
        }
    }
}

// Four finished rows m0 .. m0 + 3 (m0 a multiple of 4) of token n: bias, activation, fp16, memory.
__device__ __forceinline__ void store_four_rows(const OutTargets& out, int activation, const __half* bias, float4 acc, uint32_t m0,
                                                uint32_t n) {
    if (bias) {
        acc.x += __half2float(bias[m0]); acc.y += __half2float(bias[m0 + 1]);
        acc.z += __half2float(bias[m0 + 2]); acc.w += __half2float(bias[m0 + 3]);
    }
    if (activation == kActSiluMul) {   // two gate/up pairs -> two output channels
        *reinterpret_cast<uint32_t*>(out.ptr[0] + (size_t)n * out.ld + out.row0 + (m0 >> 1)) =
            pack_half2(silu_mul(acc.x, acc.y), silu_mul(acc.z, acc.w));
        return;
    }
    const uint2 packed = make_uint2(pack_half2(acc.x, acc.y), pack_half2(acc.z, acc.w));
    const size_t at = (size_t)n * out.ld + out.row0 + m0;
    for (uint32_t t = 0; t < out.count; t++) *reinterpret_cast<uint2*>(out.ptr[t] + at) = packed;
}

// End of a tile whose K range a cluster shared: every CTA holds its part as [token][128 rows] fp32 at `part` of its shared
// memory (the pipeline ring, idle by then); the warps of all CTAs take a token each in turn and add the parts in rank order.
// Called by whole warps between the two cluster barriers.
__device__ __forceinline__ void reduce_cluster(const OutTargets& out, int activation, const __half* bias, uint32_t part, uint32_t ctas,
                                               uint32_t rank, uint32_t warps, uint32_t row0, uint32_t n0, uint32_t tokens, int warp,
                                               int lane) {
    for (uint32_t t = (uint32_t)warp * ctas + rank; t < tokens; t += warps * ctas) {
        const uint32_t addr = part + (t * 128u + 4u * (uint32_t)lane) * 4u;
        float4 v[kMaxCluster];
#pragma unroll
        for (uint32_t s = 0; s < (uint32_t)kMaxCluster; s++)
            if (s < ctas) v[s] = ptx::ld_cluster_f4(ptx::mapa(addr, s));
        float4 acc = v[0];
#pragma unroll
        for (uint32_t s = 1; s < (uint32_t)kMaxCluster; s++)
            if (s < ctas) { acc.x += v[s].x; acc.y += v[s].y; acc.z += v[s].z; acc.w += v[s].w; }
        store_four_rows(out, activation, bias, acc, row0 + 4u * (uint32_t)lane, n0 + t);
    }
}

}  // namespace fpx
