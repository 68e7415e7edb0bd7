// Activation quantisation by lanes, for the quantisation kernels and for the one that prepares a dense linear.
#pragma once

#include <cuda_fp8.h>

#include "common.cuh"

namespace nvmoe {
namespace {

__device__ __forceinline__ uint32_t to_e4m3x4(float a, float b, float c, float d) {
    // cvt.rn.satfinite.e4m3x2.f32: round-to-nearest-even, saturating (|x/scale| <= 448 by construction)
    uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
    return lo | (hi << 16);
}

// Sixteen neighbouring bf16 columns a lane, 16-byte aligned at `src`: LANES lanes (a scale block of 16 * LANES columns)
// share a scale. `out` receives the lane's E4M3 bytes, `word` (the same in the eight lanes of 128 columns) the E8M0 bytes
// of their columns; an inactive lane, past the end of the row, adds zeros. Called by a whole warp.
template <uint32_t LANES>
__device__ __forceinline__ void quantize_sixteen(const uint16_t* src, bool active, uint32_t lane, uint32_t (&out)[4], uint32_t& word) {
    uint4 v[2] = {};
    if (active) {
        v[0] = __ldg(reinterpret_cast<const uint4*>(src));
        v[1] = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    }
    const uint32_t w[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) m = fmaxf(m, fmaxf(fabsf(nvmoe_bf16_to_f32(w[i])), fabsf(nvmoe_bf16_to_f32(w[i] >> 16))));
#pragma unroll
    for (uint32_t o = 1u; o < LANES; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float scale = nvmoe_rounded_fp8_scale(m);
    const float inv = __uint_as_float(0x7f000000u - __float_as_uint(scale));  // 1 / scale, exact (a power of two)
#pragma unroll
    for (int i = 0; i < 4; i++)
        out[i] = to_e4m3x4(nvmoe_bf16_to_f32(w[2 * i]) * inv, nvmoe_bf16_to_f32(w[2 * i] >> 16) * inv,
                           nvmoe_bf16_to_f32(w[2 * i + 1]) * inv, nvmoe_bf16_to_f32(w[2 * i + 1] >> 16) * inv);
    // two lanes hold 32 columns: byte (lane % 8) / 2 of the word of their 128
    word = active ? (nvmoe_f32_bits(scale) >> 23) << (8u * ((lane & 7u) >> 1)) : 0u;
    word |= __shfl_xor_sync(0xffffffffu, word, 2);
    word |= __shfl_xor_sync(0xffffffffu, word, 4);
}

// By a warp: the down operands of a route that only the down stage keeps, as if its gate/up frame had never been written.
__device__ __forceinline__ void zero_down_row(const DownRows& down, uint32_t row, uint32_t lane) {
    for (uint32_t c = lane * 16u; c < down.cols; c += 512u)
        *reinterpret_cast<uint4*>(down.q + (size_t)row * down.cols + c) = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t words = (down.cols + 127u) / 128u;
    for (uint32_t c = lane; c < words; c += 32u) *down.scales.at(row, c) = 0x7f7f7f7fu;
}

}  // namespace
}  // namespace nvmoe
