// One token's routing by a warp, for the router kernel and for the kernel that routes and schedules a small call.
#pragma once

#include "common.cuh"

namespace nvmoe {
namespace {

constexpr float kNegInf = -__builtin_huge_valf();

__device__ __forceinline__ float unpack_logit(const uint32_t* row, uint32_t e) {
    uint32_t packed = row[e >> 1];
    return nvmoe_bf16_to_f32((e & 1u) ? (packed >> 16) : packed);
}

__device__ __forceinline__ bool better(float s, uint32_t e, float best, uint32_t best_e) {
    return s > best || (s == best && e < best_e);
}

// warp-wide arg-max of (score, expert) pairs under `better`; all lanes return the winner
__device__ __forceinline__ void warp_argmax(float& s, uint32_t& e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float os = __shfl_xor_sync(0xffffffffu, s, o);
        uint32_t oe = __shfl_xor_sync(0xffffffffu, e, o);
        // an empty candidate carries e == kUnboundSlot and can only win over another empty one
        bool take = (oe != kUnboundSlot) && (e == kUnboundSlot || better(os, oe, s, e));
        if (take) {
            s = os;
            e = oe;
        }
    }
}

// A score as a number whose order is the score's: equal for equal scores (-0 and 0 are), above 0 for every score but a NaN, which is 0.
__device__ __forceinline__ uint32_t score_key(float s) {
    const uint32_t bits = __float_as_uint(__fadd_rn(s, 0.0f));
    return s != s ? 0u : bits ^ ((uint32_t)((int32_t)bits >> 31) | 0x80000000u);
}
// warp_argmax by the warp's integer maximum: of the lanes' (score, expert) pairs the one with the higher score, of equal ones with
// the lower expert; kUnboundSlot stands for no pair. All lanes return the winner. Ten shuffles and five compares in a chain a
// round otherwise: layers, us, one token of 32 experts 38.4 / 37.3 with four rounds of this, tiny layer of 64 25.8 / 25.4.
__device__ __forceinline__ uint32_t warp_best(float s, uint32_t e) {
    const uint32_t key = e == kUnboundSlot ? 0u : score_key(s);
    const uint32_t top = __reduce_max_sync(0xffffffffu, key);
    return __reduce_min_sync(0xffffffffu, top != 0u && key == top ? e : kUnboundSlot);
}

// One step of a lane's sum: bf16 x bf16 (exact in f32) added with one rounding, the products' operands converted by the
// instruction itself.
__device__ __forceinline__ float fma_bf16(uint16_t a, uint16_t b, float c) {
    float d;
    asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(d) : "h"(a), "h"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float read_bias(const void* bias, uint32_t dtype, uint32_t e) {
    if (dtype == NVMOE_BIAS_F32) return reinterpret_cast<const float*>(bias)[e];
    if (dtype == NVMOE_BIAS_BF16) return nvmoe_bf16_to_f32(reinterpret_cast<const uint16_t*>(bias)[e]);
    return 0.0f;
}

// SHORT, for the blocks of a small call that route beside its operands and schedule, which run their code once and wait for every line of it: the functions
// of the scores are calls, one copy for all places. Kernels that only route have them inlined. Layers, us, calls everywhere and no loop unrolled / calls in those
// blocks only: 256 experts of 2048 x 512 in groups, 16 tokens 72.8 / 71.6, 250 151.2 / 149.1; 250 of 64 of 1024 x 512 63.7 / 63.3; 4 of 64 of 256 x 128, 32 routes a
// token, 42.2 / 36.7; 64 of 8 of 256 x 512 23.2 / 23.1; 33 to 200 of 32 of 2880 x 2880 level. router_reg_kernel by itself, 256 experts in groups: 64 tokens
// 8.1 / 6.7, 2048 11.5 / 9.9, 4096 23.2 / 18.9, 16384 50.3 / 48.0; without groups 5.9 / 5.9, 7.9 / 7.9, 17.0 / 17.7, 36.0 / 37.6; 32 experts, 16384 7.3 / 7.0. (Loops over selections unrolled by four
// as well: layers of 256 experts 1 to 3 us more.)
__device__ __noinline__ float call_exp(float v) { return nvmoe_expf(v); }
__device__ __noinline__ float call_divide(float a, float b) { return __fdiv_rn(a, b); }
__device__ __noinline__ float call_sigmoid(float v) { return nvmoe_sigmoidf(v); }
__device__ __noinline__ float call_softplus_root(float v) { return __fsqrt_rn(nvmoe_softplusf(v)); }
__device__ __noinline__ float call_softcap(float v, float cap) { return __fmul_rn(nvmoe_tanhf(__fdiv_rn(v, cap)), cap); }
template <bool SHORT> __device__ __forceinline__ float route_exp(float v) { return SHORT ? call_exp(v) : nvmoe_expf(v); }
template <bool SHORT> __device__ __forceinline__ float route_divide(float a, float b) { return SHORT ? call_divide(a, b) : __fdiv_rn(a, b); }
template <bool SHORT> __device__ __forceinline__ float route_sigmoid(float v) { return SHORT ? call_sigmoid(v) : nvmoe_sigmoidf(v); }
template <bool SHORT> __device__ __forceinline__ float route_softplus_root(float v) { return SHORT ? call_softplus_root(v) : __fsqrt_rn(nvmoe_softplusf(v)); }
template <bool SHORT> __device__ __forceinline__ float route_softcap(float v, float cap) {
    return SHORT ? call_softcap(v, cap) : __fmul_rn(nvmoe_tanhf(__fdiv_rn(v, cap)), cap);
}

// ---- the same router with a token's experts in registers ------------------------------------------
// For up to 32 * EPL experts and at most 32 selections a token; GROUPS: with group-limited masking, for groups of a
// power of two of experts up to 32, which are then a run of lanes: lane l keeps the
// experts l, l + 32, .. in registers, lane r keeps selection r once it is made, and everything the kernel above
// does through shared memory by one lane (the weights, the ascending order, packing, telemetry) is done by the
// lanes side by side. Every sum that has an order keeps it (values travel by shuffle and are added in the same
// sequence); the results are bit for bit those of router_kernel, which remains for the other cases. Called by a whole warp.

// k rounds of arg-max over the experts that `taken` does not name: lane r keeps selection r (expert and value). False if there are fewer than k
// selectable scores.
template <int EPL>
__device__ __forceinline__ bool pick_experts(uint32_t E, uint32_t k, const float (&val)[EPL], const float (&score)[EPL], uint32_t taken, uint32_t& my_e, float& my_v) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    my_e = kUnboundSlot;
    my_v = 0.0f;
    for (uint32_t r = 0; r < k; r++) {
        float best = kNegInf, best_v = 0.0f;
        uint32_t best_e = kUnboundSlot;
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const uint32_t e = lane + 32u * j;
            if (e < E && ((taken >> j) & 1u) == 0u && better(score[j], e, best, best_e)) {
                best = score[j];
                best_e = e;
                best_v = val[j];
            }
        }
        const uint32_t winner = warp_best(best, best_e);
        if (winner == kUnboundSlot) return false;
        // the winner is the best candidate of the lane that owns it
        const float winner_v = __shfl_sync(kFull, best_v, winner & 31u);
        if (lane == (winner & 31u)) taken |= 1u << (winner >> 5);
        if (lane == r) {
            my_e = winner;
            my_v = winner_v;
        }
    }
    return true;
}

// The selection: lane r receives selection r (expert and activated value). False if there are fewer than k selectable scores.
template <bool SHORT, int EPL, bool GROUPS>
__device__ __forceinline__ bool select_experts(const RouterLaunch& p, uint32_t token, uint32_t& my_e, float& my_v) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t E = p.g.routed_experts;
    const uint32_t k = p.g.routed_k;
    const uint32_t kind = p.g.router_kind;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* row = p.logits + (size_t)token * ((E + 1u) / 2u);

    float val[EPL], score[EPL];
#pragma unroll
    for (int j = 0; j < EPL; j++) {
        const uint32_t e = lane + 32u * j;
        val[j] = e < E ? unpack_logit(row, e) : 0.0f;
        score[j] = 0.0f;
    }
    // ---- activation and selection score ---------------------------------------------------
    if (kind == NVMOE_ROUTER_SCORE_TOPK) {
        if (p.g.activation == NVMOE_ACT_SOFTMAX) {
            float smax = kNegInf;
#pragma unroll
            for (int j = 0; j < EPL; j++)
                if (lane + 32u * j < E) smax = fmaxf(smax, val[j]);
            smax = warp_max(smax);
            float lo = 0.0f, hi = 0.0f;  // virtual lanes `lane` and `lane + 32` of a 64-wide group
#pragma unroll
            for (int j = 0; j < EPL; j++) {
                if (lane + 32u * j < E) {
                    val[j] = route_exp<SHORT>(__fsub_rn(val[j], smax));
                    if (j & 1) hi = __fadd_rn(hi, val[j]); else lo = __fadd_rn(lo, val[j]);
                }
            }
            const float sden = warp_butterfly_sum(__fadd_rn(lo, hi));
#pragma unroll
            for (int j = 0; j < EPL; j++) val[j] = route_divide<SHORT>(val[j], sden);
        } else {
#pragma unroll
            for (int j = 0; j < EPL; j++)
                val[j] = p.g.activation == NVMOE_ACT_SIGMOID ? route_sigmoid<SHORT>(val[j]) : route_softplus_root<SHORT>(val[j]);
        }
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const uint32_t e = lane + 32u * j;
            score[j] = e < E ? __fadd_rn(val[j], read_bias(p.bias, p.g.bias_dtype, e)) : 0.0f;
        }
    } else if (kind == NVMOE_ROUTER_TOPK_SOFTMAX) {
#pragma unroll
        for (int j = 0; j < EPL; j++) score[j] = val[j];
    } else {
        const bool sigmoid = p.g.activation == NVMOE_ACT_SIGMOID;
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const uint32_t e = lane + 32u * j;
            float v = val[j];
            if (p.g.logit_softcap > 0.0f) v = route_softcap<SHORT>(v, p.g.logit_softcap);
            val[j] = v;
            score[j] = e < E ? __fadd_rn(sigmoid ? route_sigmoid<SHORT>(v) : v, read_bias(p.bias, p.g.bias_dtype, e)) : 0.0f;
        }
    }

    uint32_t taken = 0u;
    if (GROUPS) {
        // a group's score is the sum of its two best; the experts of the groups outside the topk_group best count as taken
        const uint32_t per = E / p.g.n_group, side = 32u / per;  // groups in a register slot of the warp
        float my_group = kNegInf;
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            float first = lane + 32u * j < E && score[j] > kNegInf ? score[j] : kNegInf, second = kNegInf;
            for (uint32_t o = 1u; o < per; o <<= 1) {
                const float other_first = __shfl_xor_sync(kFull, first, o), other_second = __shfl_xor_sync(kFull, second, o);
                second = fmaxf(fminf(first, other_first), fmaxf(second, other_second));
                first = fmaxf(first, other_first);
            }
            const float group = __shfl_sync(kFull, per >= 2u ? __fadd_rn(first, second) : first, (lane % side) * per);
            if (lane / side == (uint32_t)j) my_group = group;  // lane g keeps group g
        }
        uint32_t kept = 0u;
        for (uint32_t round = 0; round < p.g.topk_group; round++) {
            const bool open = lane < p.g.n_group && ((kept >> lane) & 1u) == 0u && my_group >= kNegInf;  // (not a NaN)
            const uint32_t winner = warp_best(my_group, open ? lane : kUnboundSlot);
            if (winner != kUnboundSlot) kept |= 1u << winner;
        }
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const uint32_t group = (uint32_t)j * side + lane / per;
            if (group >= 32u || ((kept >> group) & 1u) == 0u) taken |= 1u << j;
        }
    }
    return pick_experts<EPL>(E, k, val, score, taken, my_e, my_v);
}

// How many experts every token selects besides.
__device__ __forceinline__ uint32_t always_selected(const RouterLaunch& p) { return p.g.router_kind == NVMOE_ROUTER_SCORE_TOPK ? p.g.always_count : 0u; }

// What a token's selections are counted by.
struct RouteCounts {
    uint32_t experts, k, kind, total_k, total_resources;
};
__device__ __forceinline__ RouteCounts counts_of(const RouterLaunch& p) {
    const uint32_t always = always_selected(p);
    return RouteCounts{p.g.routed_experts, p.g.routed_k, p.g.router_kind, p.g.routed_k + always, p.g.routed_experts + always};
}

// The places of a token's selections in ascending order of the experts: lane r < total_k holds selection r.
__device__ __forceinline__ uint32_t ascending_rank(uint32_t my_e, uint32_t total_k) {
    uint32_t rank = 0u;
    for (uint32_t q = 0; q < total_k; q++) {
        const uint32_t other = __shfl_sync(0xffffffffu, my_e, q);
        if (other < my_e) rank++;
    }
    return rank;
}

// Of a token whose selections the lanes hold (`found`: there are k): lane r < total_k receives the expert and the place of one of its route words, as
// finish_token writes them.
__device__ __forceinline__ void order_token(const RouterLaunch& p, bool found, uint32_t& my_e, uint32_t& rank) {
    const uint32_t lane = threadIdx.x & 31u, k = p.g.routed_k, always = always_selected(p);
    if (!found) my_e = 0u;  // words of zeros
    if (found && lane >= k) my_e = p.g.routed_experts + (lane - k);
    rank = found ? ascending_rank(my_e, k + always) : lane;
}

// Weights, route words and telemetry of such a token (n: counts_of); my_e and rank as above.
template <bool SHORT>
__device__ __forceinline__ void finish_token(const RouterLaunch& p, const RouteCounts& n, uint32_t token, bool found, uint32_t& my_e, float my_v, uint32_t& rank) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t E = n.experts, k = n.k, kind = n.kind, total_k = n.total_k, total_resources = n.total_resources;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* out = p.routes + (size_t)token * total_k;
    if (!found) {
        // no selectable score (NaN logits): fail closed instead of indexing out of bounds
        if (lane == 0u) {
            for (uint32_t r = 0; r < total_k; r++) out[r] = 0u;
            raise_status(p.status, NVMOE_STATUS_ROUTE_NONFINITE);
        }
        my_e = 0u;
        rank = lane;
        return;
    }

    // ---- weights, in the summation orders the shaders fix ----------------------------------
    float w = 0.0f;
    if (kind == NVMOE_ROUTER_SCORE_TOPK) {
        float den = 0.0f;
        if (p.g.normalize_selected)
            for (uint32_t r = 0; r < k; r++) den = __fadd_rn(den, __shfl_sync(kFull, my_v, r));
        w = p.g.normalize_selected ? __fmul_rn(route_divide<SHORT>(my_v, den), p.g.routed_scale) : __fmul_rn(my_v, p.g.routed_scale);
        if (lane >= k && lane < total_k) {
            my_e = E + (lane - k);
            w = p.g.always_weight;
        }
    } else {
        const bool sigmoid = kind == NVMOE_ROUTER_TOPK_ROUTED && p.g.activation == NVMOE_ACT_SIGMOID;
        const bool divide = kind == NVMOE_ROUTER_TOPK_SOFTMAX || p.g.normalize_selected || !sigmoid;
        const float maximum = __shfl_sync(kFull, my_v, 0);
        const float t = sigmoid ? route_sigmoid<SHORT>(my_v) : route_exp<SHORT>(__fsub_rn(my_v, maximum));
        float den = 0.0f;
        for (uint32_t r = 0; r < k; r++) den = __fadd_rn(den, __shfl_sync(kFull, t, r));
        w = divide ? route_divide<SHORT>(t, den) : t;
    }

    // ---- ascending expert id, pack, telemetry ----------------------------------------------------
    rank = ascending_rank(my_e, total_k);
    if (lane < total_k) {
        out[rank] = (nvmoe_f32_to_bf16(w) << 16) | my_e;
        if (p.telemetry) atomicAdd(p.telemetry + my_e, 1u);
    }
    if (p.telemetry) {
        for (uint32_t q = 0; q < total_k; q++) {
            const uint32_t right = __shfl_sync(kFull, my_e, q);
            if (lane < total_k && my_e < right) {
                const uint32_t preceding = my_e * (2u * total_resources - my_e - 1u) / 2u;
                atomicAdd(p.telemetry + total_resources + preceding + right - my_e - 1u, 1u);
            }
        }
    }
}

template <bool SHORT, int EPL, bool GROUPS>
__device__ __forceinline__ void route_token(const RouterLaunch& p, uint32_t token) {
    // (looked up ahead of the selection: behind it, router_reg_kernel with 256 experts in groups takes 10.4 us for 2048 tokens instead of 9.9, 23.7 for 4096 instead of
    // 18.9, 51.9 for 16384 instead of 48.0)
    const RouteCounts n = counts_of(p);
    uint32_t my_e, rank;
    float my_v;
    const bool found = select_experts<SHORT, EPL, GROUPS>(p, token, my_e, my_v);
    finish_token<SHORT>(p, n, token, found, my_e, my_v, rank);
}

}  // namespace
}  // namespace nvmoe
