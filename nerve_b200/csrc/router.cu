// Router projection and the three route-native router forms.
//
//   router_linear_kernel   runtime-rs/shaders/linear_bf16.comp.template:39-95 and
//                          linear_bias_bf16.comp.template:31-84
//   router_kernel          runtime-rs/shaders/moe_router_score_topk_batch1_bf16.comp.template:109-220
//                          runtime-rs/shaders/moe_topk_bf16.comp.template:44-145
//                          runtime-rs/shaders/moe_topk_routed_batch1_bf16.comp.template:71-182
//
// One warp routes one token.  Selection is k rounds of a (score, index) arg-max whose comparator
// is the shaders' own: higher score wins, equal scores go to the lower expert index, a NaN score
// is never chosen.  Route weights use the pinned transcendentals of nvmoe_math.h and the summation
// orders the shaders fix (selection order for the selected-only denominators, index order for
// the softmax-over-all of the routed form); the one order the shaders leave to the hardware, the
// subgroup sum of the score_topk softmax, is pinned to 64 lane-strided partials folded by an xor
// butterfly (32,16,8,4,2,1) — the same definition the CPU checker uses.
#include "router_reg.cuh"

namespace nvmoe {
namespace {

struct WarpSmem {
    float* values;      // activated value (score_topk) or soft-capped logit (routed) or raw logit
    float* score;       // selection score
    uint32_t* flags;    // bit0 selected, bit1 allowed
    uint32_t* top;      // [kMaxTopK]
    float* top_w;       // [kMaxTopK]
    float* group_score; // [32]
};

__global__ void __launch_bounds__(128) router_kernel(RouterLaunch p, uint32_t warps_per_block) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    grid_dependency_sync();
    const uint32_t E = p.g.routed_experts;
    const uint32_t k = p.g.routed_k;
    const uint32_t kind = p.g.router_kind;
    const uint32_t always = kind == NVMOE_ROUTER_SCORE_TOPK ? p.g.always_count : 0u;
    const uint32_t total_k = k + always;
    const uint32_t total_resources = E + always;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t token = blockIdx.x * warps_per_block + warp;
    if (warp >= warps_per_block || token >= p.tokens) return;

    const size_t per_warp = (size_t)E * 12u + kMaxTopK * 8u + 32u * 4u;
    unsigned char* base = smem_raw + per_warp * warp;
    WarpSmem s;
    s.values = reinterpret_cast<float*>(base);
    s.score = s.values + E;
    s.flags = reinterpret_cast<uint32_t*>(s.score + E);
    s.top = s.flags + E;
    s.top_w = reinterpret_cast<float*>(s.top + kMaxTopK);
    s.group_score = s.top_w + kMaxTopK;

    const uint32_t* row = p.logits + (size_t)token * ((E + 1u) / 2u);

    // ---- activation and selection score ---------------------------------------------------
    if (kind == NVMOE_ROUTER_SCORE_TOPK) {
        float smax = kNegInf, sden = 0.0f;
        if (p.g.activation == NVMOE_ACT_SOFTMAX) {
            for (uint32_t e = lane; e < E; e += 32u) smax = fmaxf(smax, unpack_logit(row, e));
            smax = warp_max(smax);
            float lo = 0.0f, hi = 0.0f;  // virtual lanes `lane` and `lane + 32` of a 64-wide group
            for (uint32_t e = lane; e < E; e += 64u) lo = __fadd_rn(lo, nvmoe_expf(__fsub_rn(unpack_logit(row, e), smax)));
            for (uint32_t e = lane + 32u; e < E; e += 64u) hi = __fadd_rn(hi, nvmoe_expf(__fsub_rn(unpack_logit(row, e), smax)));
            sden = warp_butterfly_sum(__fadd_rn(lo, hi));
        }
        for (uint32_t e = lane; e < E; e += 32u) {
            float v = unpack_logit(row, e);
            float a;
            if (p.g.activation == NVMOE_ACT_SIGMOID) {
                a = nvmoe_sigmoidf(v);
            } else if (p.g.activation == NVMOE_ACT_SOFTMAX) {
                a = __fdiv_rn(nvmoe_expf(__fsub_rn(v, smax)), sden);
            } else {
                a = __fsqrt_rn(nvmoe_softplusf(v));
            }
            s.values[e] = a;
            s.score[e] = __fadd_rn(a, read_bias(p.bias, p.g.bias_dtype, e));
        }
    } else if (kind == NVMOE_ROUTER_TOPK_SOFTMAX) {
        for (uint32_t e = lane; e < E; e += 32u) {
            float v = unpack_logit(row, e);
            s.values[e] = v;
            s.score[e] = v;
        }
    } else {
        const bool sigmoid = p.g.activation == NVMOE_ACT_SIGMOID;
        for (uint32_t e = lane; e < E; e += 32u) {
            float v = unpack_logit(row, e);
            if (p.g.logit_softcap > 0.0f)
                v = __fmul_rn(nvmoe_tanhf(__fdiv_rn(v, p.g.logit_softcap)), p.g.logit_softcap);
            s.values[e] = v;
            s.score[e] = __fadd_rn(sigmoid ? nvmoe_sigmoidf(v) : v, read_bias(p.bias, p.g.bias_dtype, e));
        }
    }
    __syncwarp();

    // ---- group-limited mask (extension; n_group == 0 keeps every expert) -------------------
    if (p.g.n_group == 0u) {
        for (uint32_t e = lane; e < E; e += 32u) s.flags[e] = 2u;
    } else {
        const uint32_t per = E / p.g.n_group;
        if (lane < p.g.n_group) {
            float first = kNegInf, second = kNegInf;
            for (uint32_t j = 0; j < per; j++) {
                float v = s.score[lane * per + j];
                if (v > first) {
                    second = first;
                    first = v;
                } else if (v > second) {
                    second = v;
                }
            }
            s.group_score[lane] = per >= 2u ? __fadd_rn(first, second) : first;
        }
        __syncwarp();
        uint32_t kept = 0u;  // computed redundantly by every lane: n_group <= 32
        for (uint32_t round = 0; round < p.g.topk_group; round++) {
            float best = kNegInf;
            uint32_t best_g = kUnboundSlot;
            for (uint32_t g = 0; g < p.g.n_group; g++) {
                if (kept & (1u << g)) continue;
                float v = s.group_score[g];
                if (better(v, g, best, best_g)) {
                    best = v;
                    best_g = g;
                }
            }
            if (best_g != kUnboundSlot) kept |= 1u << best_g;
        }
        for (uint32_t e = lane; e < E; e += 32u) s.flags[e] = (kept >> (e / per)) & 1u ? 2u : 0u;
    }
    __syncwarp();

    // ---- k rounds of arg-max -------------------------------------------------------------
    bool missing = false;
    for (uint32_t r = 0; r < k; r++) {
        float best = kNegInf;
        uint32_t best_e = kUnboundSlot;
        for (uint32_t e = lane; e < E; e += 32u) {
            if (s.flags[e] != 2u) continue;  // not allowed, or already selected (bit0)
            float v = s.score[e];
            if (better(v, e, best, best_e)) {
                best = v;
                best_e = e;
            }
        }
        warp_argmax(best, best_e);
        if (best_e == kUnboundSlot) {
            missing = true;
            break;
        }
        if (lane == 0) {
            s.top[r] = best_e;
            s.flags[best_e] = 3u;
        }
        __syncwarp();
    }

    if (lane != 0) return;
    uint32_t* out = p.routes + (size_t)token * total_k;
    if (missing) {
        // no selectable score (NaN logits): fail closed instead of indexing out of bounds
        for (uint32_t r = 0; r < total_k; r++) out[r] = 0u;
        raise_status(p.status, NVMOE_STATUS_ROUTE_NONFINITE);
        return;
    }

    // ---- weights, in the summation orders the shaders fix ----------------------------------
    if (kind == NVMOE_ROUTER_SCORE_TOPK) {
        float den = 0.0f;
        if (p.g.normalize_selected)
            for (uint32_t r = 0; r < k; r++) den = __fadd_rn(den, s.values[s.top[r]]);
        for (uint32_t r = 0; r < k; r++) {
            float w = s.values[s.top[r]];
            w = p.g.normalize_selected ? __fmul_rn(__fdiv_rn(w, den), p.g.routed_scale) : __fmul_rn(w, p.g.routed_scale);
            s.top_w[r] = w;
        }
        for (uint32_t o = 0; o < always; o++) {
            s.top[k + o] = E + o;
            s.top_w[k + o] = p.g.always_weight;
        }
    } else if (kind == NVMOE_ROUTER_TOPK_SOFTMAX) {
        float maximum = s.values[s.top[0]];
        float den = 0.0f;
        for (uint32_t r = 0; r < k; r++) den = __fadd_rn(den, nvmoe_expf(__fsub_rn(s.values[s.top[r]], maximum)));
        for (uint32_t r = 0; r < k; r++)
            s.top_w[r] = __fdiv_rn(nvmoe_expf(__fsub_rn(s.values[s.top[r]], maximum)), den);
    } else {
        const bool sigmoid = p.g.activation == NVMOE_ACT_SIGMOID;
        float maximum = s.values[s.top[0]];
        float den = 0.0f;
        if (p.g.normalize_selected) {
            for (uint32_t r = 0; r < k; r++) {
                float v = s.values[s.top[r]];
                den = __fadd_rn(den, sigmoid ? nvmoe_sigmoidf(v) : nvmoe_expf(__fsub_rn(v, maximum)));
            }
        } else if (!sigmoid) {
            maximum = kNegInf;
            for (uint32_t e = 0; e < E; e++) maximum = fmaxf(maximum, s.values[e]);
            for (uint32_t e = 0; e < E; e++) den = __fadd_rn(den, nvmoe_expf(__fsub_rn(s.values[e], maximum)));
        }
        for (uint32_t r = 0; r < k; r++) {
            float v = s.values[s.top[r]];
            float w = sigmoid ? nvmoe_sigmoidf(v) : nvmoe_expf(__fsub_rn(v, maximum));
            if (p.g.normalize_selected || !sigmoid) w = __fdiv_rn(w, den);
            s.top_w[r] = w;
        }
    }

    // ---- ascending expert id (insertion sort of the shaders), pack, telemetry ---------------
    for (uint32_t r = 1; r < total_k; r++) {
        uint32_t e = s.top[r];
        float w = s.top_w[r];
        uint32_t ins = r;
        while (ins > 0u && s.top[ins - 1u] > e) {
            s.top[ins] = s.top[ins - 1u];
            s.top_w[ins] = s.top_w[ins - 1u];
            ins--;
        }
        s.top[ins] = e;
        s.top_w[ins] = w;
    }
    for (uint32_t r = 0; r < total_k; r++) {
        out[r] = (nvmoe_f32_to_bf16(s.top_w[r]) << 16) | s.top[r];
        if (p.telemetry) atomicAdd(p.telemetry + s.top[r], 1u);
    }
    if (p.telemetry) {
        for (uint32_t l = 0; l < total_k; l++) {
            uint32_t left = s.top[l];
            for (uint32_t rr = l + 1u; rr < total_k; rr++) {
                uint32_t right = s.top[rr];
                if (left < right) {
                    uint32_t preceding = left * (2u * total_resources - left - 1u) / 2u;
                    atomicAdd(p.telemetry + total_resources + preceding + right - left - 1u, 1u);
                }
            }
        }
    }
}

template <int EPL, bool GROUPS>
__global__ void __launch_bounds__(128) router_reg_kernel(RouterLaunch p) {
    grid_dependency_sync();
    const uint32_t token = blockIdx.x * 4u + (threadIdx.x >> 5);
    if (token < p.tokens) route_token<false, EPL, GROUPS>(p, token);
}

// ---- router projection ----------------------------------------------------------------------
// The shader gives every output row 64 lanes that stride over the packed input words with two
// f32 fma per word and then sums the lanes.  Here a block of 64 threads owns a TT x ET tile of
// (token, output) pairs: thread v plays lane v of every pair in the tile, so each x and w word is
// loaded once per thread and reused across the tile, and the 64 lane sums of a pair are folded
// with the pinned butterfly (step 32 through shared memory, 16..1 by shuffles).

// The 64 lanes' sums of a block's tile, folded in the pinned order (lane v by thread v), rounded and stored.
template <int TT, int ET>
__device__ __forceinline__ void fold_and_store(const float (&acc)[TT][ET], float (&fold)[TT * ET][32], float (&result)[TT * ET], const uint16_t* __restrict__ bias,
                                               uint32_t* __restrict__ logits, uint32_t t0, uint32_t e0, uint32_t tokens, uint32_t outputs) {
    const uint32_t v = threadIdx.x;
    // butterfly step 32: lanes v and v^32 live in different warps
    if (v >= 32u) {
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int b = 0; b < ET; b++) fold[a * ET + b][v - 32u] = acc[a][b];
    }
    __syncthreads();
    if (v < 32u) {
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int b = 0; b < ET; b++) {
                float sum = warp_butterfly_sum(__fadd_rn(acc[a][b], fold[a * ET + b][v]));
                if (v == 0u) result[a * ET + b] = sum;
            }
    }
    __syncthreads();
    // pack pairs of outputs into words; ET is even so a word never straddles two blocks
    const uint32_t out_words = (outputs + 1u) / 2u;
    for (uint32_t i = v; i < TT * (ET / 2); i += 64u) {
        uint32_t a = i / (ET / 2), bw = i % (ET / 2);
        uint32_t t = t0 + a, e = e0 + 2u * bw;
        if (t >= tokens || e >= outputs) continue;
        float lo = result[a * ET + 2u * bw];
        float hi = result[a * ET + 2u * bw + 1u];
        if (bias) {
            lo = __fadd_rn(lo, nvmoe_bf16_to_f32(bias[e]));
            if (e + 1u < outputs) hi = __fadd_rn(hi, nvmoe_bf16_to_f32(bias[e + 1u]));
        }
        uint32_t word = nvmoe_f32_to_bf16(lo);
        if (e + 1u < outputs) word |= nvmoe_f32_to_bf16(hi) << 16;
        logits[(size_t)t * out_words + e / 2u] = word;
    }
}

template <int TT, int ET, int DEPTH>
__global__ void __launch_bounds__(64) router_linear_kernel(const uint16_t* __restrict__ x,
                                                           const uint16_t* __restrict__ w,
                                                           const uint16_t* __restrict__ bias,
                                                           uint32_t* __restrict__ logits, uint32_t tokens,
                                                           uint32_t hidden, uint32_t outputs, CallStart start) {
    __shared__ float fold[TT * ET][32];
    __shared__ float result[TT * ET];
    grid_dependency_sync();
    begin_call(start);
    const uint32_t v = threadIdx.x;
    const uint32_t t0 = blockIdx.y * TT, e0 = blockIdx.x * ET;
    const uint32_t words = hidden / 2u;
    const uint32_t* xw = reinterpret_cast<const uint32_t*>(x);
    const uint32_t* ww = reinterpret_cast<const uint32_t*>(w);
    float acc[TT][ET];
#pragma unroll
    for (int a = 0; a < TT; a++)
#pragma unroll
        for (int b = 0; b < ET; b++) acc[a][b] = 0.0f;

    // The sum order of a lane is fixed (its words in ascending order), the load order is not: the
    // loads of DEPTH steps are issued together so that their latencies overlap.
    for (uint32_t cw0 = v; cw0 < words; cw0 += 64u * DEPTH) {
        uint32_t xr[DEPTH][TT], wr[DEPTH][ET];
#pragma unroll
        for (int u = 0; u < DEPTH; u++) {
            const uint32_t cw = cw0 + 64u * u;
            const bool in = cw < words;
#pragma unroll
            for (int a = 0; a < TT; a++) xr[u][a] = (in && t0 + a < tokens) ? __ldg(xw + (size_t)(t0 + a) * words + cw) : 0u;
#pragma unroll
            for (int b = 0; b < ET; b++) wr[u][b] = (in && e0 + b < outputs) ? __ldg(ww + (size_t)(e0 + b) * words + cw) : 0u;
        }
#pragma unroll
        for (int u = 0; u < DEPTH; u++) {
            if (cw0 + 64u * u >= words) break;  // a step past the end must not even add zeros (-0 + 0 = +0)
#pragma unroll
            for (int a = 0; a < TT; a++) {
                float xl = nvmoe_bf16_to_f32(xr[u][a]), xh = nvmoe_bf16_to_f32(xr[u][a] >> 16);
#pragma unroll
                for (int b = 0; b < ET; b++) {
                    acc[a][b] = __fmaf_rn(xl, nvmoe_bf16_to_f32(wr[u][b]), acc[a][b]);
                    acc[a][b] = __fmaf_rn(xh, nvmoe_bf16_to_f32(wr[u][b] >> 16), acc[a][b]);
                }
            }
        }
    }
    fold_and_store<TT, ET>(acc, fold, result, bias, logits, t0, e0, tokens, outputs);
}

// The same sums for small calls of aligned rows, which wait for the latency of the rows' loads and for the lines of code: the rows are staged whole in shared
// memory by 16-byte asynchronous copies, all under way at once without a register, and a short loop adds them up (4 to 12 KB of code where the loads through
// registers take 16 to 27).
constexpr uint32_t kStagedHidden = 8192u;  // (two blocks of six rows an SM)

template <int TT, int ET>
__global__ void __launch_bounds__(64) router_linear_staged_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, const uint16_t* __restrict__ bias,
                                                                  uint32_t* __restrict__ logits, uint32_t tokens, uint32_t hidden, uint32_t outputs, CallStart start) {
    extern __shared__ __align__(16) uint32_t stage[];  // [token rows, then output rows][words]
    __shared__ float fold[TT * ET][32];
    __shared__ float result[TT * ET];
    const uint32_t v = threadIdx.x, t0 = blockIdx.y * TT, e0 = blockIdx.x * ET, words = hidden / 2u;
    grid_dependency_sync();
    begin_call(start);
#pragma unroll 1
    for (uint32_t r = 0; r < TT + ET; r++) {  // (rows past the last ones repeat them: their sums are not stored)
        const uint32_t* row = reinterpret_cast<const uint32_t*>(r < TT ? x : w) + (size_t)(r < TT ? min(t0 + r, tokens - 1u) : min(e0 + r - TT, outputs - 1u)) * words;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + r * words);
#pragma unroll 4
        for (uint32_t c = 4u * v; c < words; c += 256u)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4u * c), "l"(row + c) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float acc[TT][ET];
#pragma unroll
    for (int a = 0; a < TT; a++)
#pragma unroll
        for (int b = 0; b < ET; b++) acc[a][b] = 0.0f;
#pragma unroll 4
    for (uint32_t c = v; c < words; c += 64u) {  // (the order of the loads through registers: the same sums bit for bit)
        uint32_t xv[TT], wv[ET];
#pragma unroll
        for (int a = 0; a < TT; a++) xv[a] = stage[a * words + c];
#pragma unroll
        for (int b = 0; b < ET; b++) wv[b] = stage[(TT + b) * words + c];
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int b = 0; b < ET; b++) acc[a][b] = fma_bf16((uint16_t)xv[a], (uint16_t)wv[b], acc[a][b]);
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int b = 0; b < ET; b++) acc[a][b] = fma_bf16((uint16_t)(xv[a] >> 16), (uint16_t)(wv[b] >> 16), acc[a][b]);
    }
    fold_and_store<TT, ET>(acc, fold, result, bias, logits, t0, e0, tokens, outputs);
}

// The same projection for large batches, bound by the multiply-adds: an SM does 128 a clock, and every other instruction of
// the loop takes its turn among theirs. A block of 256 threads owns 32 tokens x 16 outputs: the rows of a 512-column chunk are
// staged in shared memory by 16-byte asynchronous copies, three chunks ahead, one barrier a chunk. A warp owns 16 tokens x 8
// outputs and half of the shader's 64 lanes, so that 24 words from shared memory serve 256 multiply-adds, which take their
// operands as bf16: 16384 x 7168 x 256 in 1.46 ms, 70 a clock (with chunks of 256 columns 1.52). With both conversions as
// instructions of their own, tiles of 8 x 8 for both halves of the lanes, two chunks and two barriers a chunk it was 2.04 ms, 50
// a clock; with twelve warps 1.40, but 36 us instead of 27 for 4096 x 2880 x 32. (Packed pairs, fma.rn.f32x2, run at 68
// to 75 whatever surrounds them.) Sums, their order and the roundings are those of router_linear_kernel, bit for bit.
constexpr int kTileTokens = 32, kTileOutputs = 16, kSubTokens = 16, kSubOutputs = 8;
constexpr uint32_t kTileRows = kTileTokens + kTileOutputs, kChunkWords = 256, kChunks = 4;
constexpr uint32_t kRouterTileBytes = kChunks * kTileRows * kChunkWords * 4;
__global__ void __launch_bounds__(256, 1) router_linear_tiled_kernel(const uint16_t* __restrict__ x,
                                                                    const uint16_t* __restrict__ w,
                                                                    const uint16_t* __restrict__ bias,
                                                                    uint32_t* __restrict__ logits, uint32_t tokens,
                                                                    uint32_t hidden, uint32_t outputs, CallStart start) {
    extern __shared__ __align__(16) uint32_t stage[];  // [buffer][token rows, then output rows][word of the chunk]
    __shared__ float result[kTileTokens][kTileOutputs];
    grid_dependency_sync();
    begin_call(start);
    const uint32_t warp = threadIdx.x >> 5, l = threadIdx.x & 31u;
    const uint32_t t0 = blockIdx.y * kTileTokens, e0 = blockIdx.x * kTileOutputs;
    const uint32_t h = warp & 1u;  // lanes l + 32 h of the shader
    const uint32_t ta = ((warp >> 1) & 1u) * kSubTokens, eb = (warp >> 2) * kSubOutputs;  // this warp's corner of the block's tile
    const uint32_t words = hidden / 2u;
    const uint32_t chunks = (words + kChunkWords - 1u) / kChunkWords;
    const uint32_t* xw = reinterpret_cast<const uint32_t*>(x);
    const uint32_t* ww = reinterpret_cast<const uint32_t*>(w);
    // the 16-byte pieces of a chunk this thread copies: rows threadIdx / 32 + 8 i, four words from word 4 l of each 128
    const uint32_t* src[kTileRows / 8];
#pragma unroll
    for (uint32_t i = 0; i < kTileRows / 8; i++) {
        const uint32_t row = warp + 8u * i;
        const bool token_row = row < (uint32_t)kTileTokens;
        const uint32_t index = token_row ? t0 + row : e0 + row - kTileTokens;
        src[i] = index < (token_row ? tokens : outputs) ? (token_row ? xw : ww) + (size_t)index * words + 4u * l : nullptr;
    }
    auto fetch = [&](uint32_t chunk) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + (chunk % kChunks) * (kTileRows * kChunkWords) + warp * kChunkWords + 4u * l);
#pragma unroll
        for (uint32_t i = 0; i < kTileRows / 8; i++) {
#pragma unroll
            for (uint32_t q = 0; q < kChunkWords; q += 128u) {
                const bool ok = chunk * kChunkWords + q + 4u * l < words && src[i] != nullptr;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (i * 8u * kChunkWords + q) * 4u),
                             "l"(ok ? src[i] + chunk * kChunkWords + q : xw), "r"(ok ? 16u : 0u)
                             : "memory");
            }
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    float acc[kSubTokens][kSubOutputs];
#pragma unroll
    for (int a = 0; a < kSubTokens; a++)
#pragma unroll
        for (int b = 0; b < kSubOutputs; b++) acc[a][b] = 0.0f;
    for (uint32_t c = 0; c + 1u < kChunks; c++) {
        if (c < chunks) fetch(c);
        commit();
    }
    for (uint32_t chunk = 0; chunk < chunks; chunk++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kChunks - 2) : "memory");
        __syncthreads();  // this chunk has landed; everyone is through with the one before, whose buffer is filled next
        if (chunk + kChunks - 1u < chunks) fetch(chunk + kChunks - 1u);
        commit();
        const uint32_t* tile = stage + (chunk % kChunks) * (kTileRows * kChunkWords) + 32u * h + l;
        auto step = [&](uint32_t s) {
            uint32_t xr[kSubTokens], wr[kSubOutputs];
#pragma unroll
            for (int b = 0; b < kSubOutputs; b++) wr[b] = tile[(kTileTokens + eb + b) * kChunkWords + 64u * s];
#pragma unroll
            for (int a = 0; a < kSubTokens; a++) xr[a] = tile[(ta + a) * kChunkWords + 64u * s];
#pragma unroll
            for (int a = 0; a < kSubTokens; a++) {
#pragma unroll
                for (int b = 0; b < kSubOutputs; b++) acc[a][b] = fma_bf16((uint16_t)xr[a], (uint16_t)wr[b], acc[a][b]);
#pragma unroll
                for (int b = 0; b < kSubOutputs; b++) acc[a][b] = fma_bf16((uint16_t)(xr[a] >> 16), (uint16_t)(wr[b] >> 16), acc[a][b]);
            }
        };
        if ((chunk + 1u) * kChunkWords <= words) {  // (without a branch between them the second step's words are read under the first's sums)
#pragma unroll
            for (uint32_t s = 0; s < kChunkWords / 64; s++) step(s);
        } else {
            // a lane whose word lies past the row adds nothing (not even zeros: -0 + 0 = +0)
#pragma unroll 1
            for (uint32_t s = 0; s < kChunkWords / 64; s++)
                if (chunk * kChunkWords + 64u * s + 32u * h + l < words) step(s);
        }
    }
    // Butterfly step 32, lane l with lane l + 32: the two warps of a corner hand each other half of their sums (of 8 of the 16
    // tokens) through the chunk buffers and add. Steps 16 .. 1 fold the remaining 64 sums over the lanes by halves: a sum goes on
    // in the half of the lanes that its step chooses, with the operands and the order of the full butterfly.
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    constexpr int kHalf = kSubTokens * kSubOutputs / 2;
    float* exchange = reinterpret_cast<float*>(stage);
    float v[kHalf];
#pragma unroll
    for (int i = 0; i < kHalf; i++) {
        const float low = acc[i / kSubOutputs][i % kSubOutputs], high = acc[kSubTokens / 2 + i / kSubOutputs][i % kSubOutputs];
        exchange[(warp * kHalf + i) * 32u + l] = h == 0u ? high : low;
        v[i] = h == 0u ? low : high;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kHalf; i++) v[i] = __fadd_rn(v[i], exchange[((warp ^ 1u) * kHalf + i) * 32u + l]);
#pragma unroll
    for (int o = 16, n = kHalf / 2; o > 0; o >>= 1, n >>= 1) {
        const bool upper = (l & o) != 0u;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float kept = upper ? v[i + n] : v[i], given = upper ? v[i] : v[i + n];
            v[i] = __fadd_rn(kept, __shfl_xor_sync(0xffffffffu, given, o));
        }
    }
    // (lane bits 16 .. 1 chose bits 32 .. 2 of the sum's number; two sums are left to a lane)
#pragma unroll
    for (uint32_t i = 0; i < 2u; i++) {
        const uint32_t n = 2u * l + i;
        result[ta + h * (kSubTokens / 2) + n / kSubOutputs][eb + n % kSubOutputs] = v[i];
    }
    __syncthreads();
    const uint32_t out_words = (outputs + 1u) / 2u;
    for (uint32_t i = threadIdx.x; i < kTileTokens * (kTileOutputs / 2); i += 256u) {
        const uint32_t a = i / (kTileOutputs / 2), bw = i % (kTileOutputs / 2);
        const uint32_t t = t0 + a, e = e0 + 2u * bw;
        if (t >= tokens || e >= outputs) continue;
        float lo = result[a][2u * bw], hi = result[a][2u * bw + 1u];
        if (bias) {
            lo = __fadd_rn(lo, nvmoe_bf16_to_f32(bias[e]));
            if (e + 1u < outputs) hi = __fadd_rn(hi, nvmoe_bf16_to_f32(bias[e + 1u]));
        }
        uint32_t word = nvmoe_f32_to_bf16(lo);
        if (e + 1u < outputs) word |= nvmoe_f32_to_bf16(hi) << 16;
        logits[(size_t)t * out_words + e / 2u] = word;
    }
}

}  // namespace

static uint32_t router_total_k(const RouterLaunch& p) {
    return p.g.routed_k + (p.g.router_kind == NVMOE_ROUTER_SCORE_TOPK ? p.g.always_count : 0u);
}

bool router_is_small(const RouterLaunch& p) {
    return p.g.routed_experts <= 128u && router_total_k(p) <= 32u && p.g.n_group == 0u && p.g.router_kind <= NVMOE_ROUTER_TOPK_ROUTED &&
           !(p.g.router_kind == NVMOE_ROUTER_TOPK_ROUTED && !p.g.normalize_selected && p.g.activation != NVMOE_ACT_SIGMOID);
}

void configure_router_kernels() {
    cudaFuncSetAttribute(router_linear_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRouterTileBytes);
    cudaFuncSetAttribute(router_linear_staged_kernel<2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * kStagedHidden * 2);
    cudaFuncSetAttribute(router_linear_staged_kernel<1, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * kStagedHidden * 2);
}

void launch_router(const RouterLaunch& p, cudaStream_t stream) {
    const uint32_t E = p.g.routed_experts;
    const uint32_t total_k = router_total_k(p);
    // the routed form's softmax over all experts (neither normalised over the selection nor sigmoid) sums in expert order
    const bool sums_all = p.g.router_kind == NVMOE_ROUTER_TOPK_ROUTED && !p.g.normalize_selected && p.g.activation != NVMOE_ACT_SIGMOID;
    const uint32_t per = p.g.n_group ? E / p.g.n_group : 0u;
    const bool lane_groups = p.g.n_group != 0u && per <= 32u && (per & (per - 1u)) == 0u;
    if (E <= 256u && total_k <= 32u && (p.g.n_group == 0u || lane_groups) && !sums_all && p.g.router_kind <= NVMOE_ROUTER_TOPK_ROUTED) {
        const dim3 grid((p.tokens + 3u) / 4u), block(128);
        if (lane_groups) {
            launch_chained(E <= 32u ? router_reg_kernel<1, true> : E <= 128u ? router_reg_kernel<4, true> : router_reg_kernel<8, true>, grid,
                           block, 0, stream, p);
        } else {
            launch_chained(E <= 32u ? router_reg_kernel<1, false> : E <= 128u ? router_reg_kernel<4, false> : router_reg_kernel<8, false>, grid,
                           block, 0, stream, p);
        }
        return;
    }
    const size_t per_warp = (size_t)E * 12u + kMaxTopK * 8u + 32u * 4u;
    uint32_t warps = E <= 1024u ? 4u : 1u;
    size_t smem = per_warp * warps;
    if (smem > 48u * 1024u)
        cudaFuncSetAttribute(router_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    uint32_t blocks = (p.tokens + warps - 1u) / warps;
    launch_chained(router_kernel, dim3(blocks), dim3(warps * 32u), smem, stream, p, warps);
}

void launch_router_linear(const uint16_t* x, const uint16_t* w, const uint16_t* bias, uint32_t* logits,
                          uint32_t tokens, uint32_t hidden, uint32_t outputs, bool beside, const CallStart& start, cudaStream_t stream) {
    const bool aligned = hidden % 8u == 0u && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0u;
    const dim3 narrow((outputs + 1u) / 2u, tokens), grid((outputs + 3u) / 4u, (tokens + 1u) / 2u);
    if (tokens <= 256u && aligned && hidden <= kStagedHidden && narrow.x * narrow.y <= 256u) {
        // Staged rows, one token by two outputs a block, while that makes few blocks: each has half a row less to wait for and a quarter of the sums. Layers,
        // us, rows through registers / staged 2 x 4 / 1 x 2: 1 token of 32 experts of 2880 columns 26.8 / 26.5 / 25.3, 7 tokens 32.9 / 32.6 / 31.2, 16 (256
        // blocks) 35.9 / 35.4 / 34.5; 128 experts, 1 token 30.7 / 28.8 / 27.5, 4 28.2 / 27.8 / 27.5, but 5 (320 blocks) 29.0 / 28.8 / 29.8; 64 experts, 9
        // tokens (288) 29.3 / 28.9 / 29.3; 256 experts of 7168 columns, 1 token 59.3 / 57.6 / 56.4; of 1024 columns 30.2 / 30.3 / 29.6; 8 experts of 256
        // columns, 64 tokens 23.1 / 23.5 / 22.7.
        launch_chained(router_linear_staged_kernel<1, 2>, narrow, dim3(64), 3u * hidden * 2u, stream, x, w, bias, logits, tokens, hidden, outputs, start);
    } else if (tokens <= 256u && aligned && hidden >= 1536u && hidden <= kStagedHidden && grid.x * grid.y <= 2u * 148u) {
        // Staged rows, 2 x 4, of long rows while every block finds room at once (at 7168 columns an SM holds two). Layers, us, through registers / staged: 64
        // tokens of 32 experts of 2880 columns 39.5 / 39.1, 8 of 256 experts of 7168 77.8 / 75.2, 10 of 64 of 4096 45.9 / 44.1, 40 of 64 of 1536 (160
        // blocks) 38.2 / 37.6; on the other side of the line 16 tokens of 32 of 1024 columns 23.9 / 24.2, 128 of 32 of 2880 (512 blocks) 45.4 / 45.4,
        // 18 of 256 of 7168 (576) 87.9 / 90.0, 64 of 128 of 2880 (1024) 75.7 / 78.0.
        launch_chained(router_linear_staged_kernel<2, 4>, grid, dim3(64), 6u * hidden * 2u, stream, x, w, bias, logits, tokens, hidden, outputs, start);
    } else if (tokens <= 256u) {
        const dim3 wide((outputs + 7u) / 8u, (tokens + 3u) / 4u);
        // Small tiles for small calls, which need the blocks. A tile of 4 x 8 reads half the bytes from L2 per pair, and an SM takes as long for one of its
        // blocks as for all that it holds, where the time of 2 x 4 tiles grows with their number. With eight steps under way an SM holds six wide blocks,
        // with four eight: the most steps that let one wave take the call, and four steps again once a second wave is full. From three blocks an SM on where
        // the operands are made beside the schedule (`beside`), else from five: by itself, with the rows in L2, the wide kernel takes longer below that (7168
        // columns 2.6 17.1 / 20.3 small / wide, 2880 3.5 9.0 / 11.1). Layers, us, small tiles / wide of eight steps, by wide blocks an SM: operands
        // beside, 7168 columns 3.2 209.1 / 206.2, 3.9 218.0 / 215.5, 4.3 226.0 / 225.2, 5.2 252.7 / 247.6; 2880 columns 3.2 64.3 / 63.1, 4.1 66.2 / 65.5, 4.9 68.6 / 67.5;
        // 4096 columns 3.1 64.5 / 65.3, 4.1 78.5 / 78.1, 5.1 83.8 / 80.9; else, 2048 columns 3.2 85.4 / 84.5, 4.1 91.9 / 94.1, 4.5 94.2 / 97.8; 4096 columns 3.1
        // 89.6 / 91.6, 3.5 90.9 / 91.7, 4.1 112.9 / 110.8; 5120 columns 3.7 115.6 / 113.8, 4.1 123.6 / 124.1, 4.3 129.3 / 130.7.
        // Wide of four / eight steps: 5.2 170.5 / 167.2 and 69.9 / 67.9; 5.8 175.8 / 173.9 and 73.6 / 72.4; 6.1 74.1 / 76.7; 6.9 194.1 / 201.1.
        // Four steps against small tiles further on: 8.2 225.6 / 226.0 (small / wide), 9.1 231.5 / 228.4.
        const uint32_t blocks = wide.x * wide.y;
        if (blocks >= (beside ? 3u : 5u) * 148u && blocks <= 6u * 148u) {
            launch_chained(router_linear_kernel<4, 8, 8>, wide, dim3(64), 0, stream, x, w, bias, logits, tokens, hidden, outputs, start);
        } else if ((blocks > 6u * 148u && blocks <= 8u * 148u) || blocks >= 9u * 148u) {
            launch_chained(router_linear_kernel<4, 8, 4>, wide, dim3(64), 0, stream, x, w, bias, logits, tokens, hidden, outputs, start);
        } else if (grid.x * grid.y <= 4u * 148u && (hidden > 2048u || (hidden > 1024u && grid.x * grid.y <= 148u))) {
            // Few blocks of long rows, but too many to be staged, or unaligned: a call waits for the latency of their loads, so that 24 steps (of 128
            // columns) are under way instead of 8. Layers, us, 8 / 24: 100 tokens of 32 experts of 2880 columns 45.6 / 44.9, of 2304 40.9 / 40.3, of 2048
            // 37.6 / 37.6, of 1536 33.2 / 33.8. Beyond four blocks an SM 24 steps lose: 64 tokens of 128 experts of 2880 columns 64.1 / 65.9.
            launch_chained(router_linear_kernel<2, 4, 24>, grid, dim3(64), 0, stream, x, w, bias, logits, tokens, hidden, outputs, start);
        } else {
            launch_chained(router_linear_kernel<2, 4, 8>, grid, dim3(64), 0, stream, x, w, bias, logits, tokens, hidden, outputs, start);
        }
    } else if (aligned) {
        dim3 grid((outputs + kTileOutputs - 1u) / kTileOutputs, (tokens + kTileTokens - 1u) / kTileTokens);
        launch_chained(router_linear_tiled_kernel, grid, dim3(256), kRouterTileBytes, stream, x, w, bias, logits, tokens, hidden, outputs, start);
    } else {
        dim3 grid((outputs + 15u) / 16u, (tokens + 3u) / 4u);
        launch_chained(router_linear_kernel<4, 16, 2>, grid, dim3(64), 0, stream, x, w, bias, logits, tokens, hidden, outputs, start);
    }
}

}  // namespace nvmoe
