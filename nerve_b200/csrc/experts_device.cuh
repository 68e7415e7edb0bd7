// What the tcgen05 expert kernels of one CTA (experts_tc.cu) and of a CTA pair (experts_pair.cu) share.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace nvmoe {
namespace {

constexpr uint32_t kBlockM = 128u;   // weight rows per operand tile
constexpr uint32_t kBlockK = 128u;   // K elements per operand tile = 4 MMAs of K = 32
constexpr uint32_t kTmaBoxBytes = kBlockM * 64u;   // global bytes of one 128 x 128 box of 4-bit codes
constexpr uint32_t kATileBytes = kBlockM * 128u;   // one byte slot per element
constexpr uint32_t kScaleBlockBytes = 512u;        // 128 rows x 4 scale bytes

struct TileList {
    const uint32_t* tiles;   // (expert << 16) | token tile within the expert
    const uint32_t* count;   // number of entries
};

// SwiGLU of the tensor path: the same expression and roundings as nvmoe_swiglu (accumulators rounded
// to bf16, clamp, g / (1 + exp(-alpha g)) * (u + offset), result rounded to bf16) with the hardware's
// approximate exponential and reciprocal (a few units in the last place of f32, far below the bf16
// rounding that follows) instead of the pinned software forms: a wide token tile spends more issue
// slots on its epilogue than on its MMAs, and the pinned forms cost several times as many.
// The CUDA-core path keeps the pinned forms. swiglu_approx: of values rounded to bf16, not rounded itself; swiglu_bf16_bits:
// of accumulators, the bf16 bits.
__device__ __forceinline__ float swiglu_approx(float g, float u, float limit, float alpha, float up_offset) {
    if (limit > 0.0f) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
    }
    return __fdividef(g, 1.0f + __expf(-alpha * g)) * (u + up_offset);
}
__device__ __forceinline__ uint32_t swiglu_bf16_bits(float gate_acc, float up_acc, float limit, float alpha, float up_offset) {
    const float g = __bfloat162float(__float2bfloat16_rn(gate_acc));
    const float u = __bfloat162float(__float2bfloat16_rn(up_acc));
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(swiglu_approx(g, u, limit, alpha, up_offset)));
}

}  // namespace
}  // namespace nvmoe
