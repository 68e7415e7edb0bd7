// The router projection of large calls on the tensor cores, with the results of the pinned one.
//
// A logit is defined as 64 lane-strided f32 chains folded by a butterfly (router.cu), which tensor cores cannot add in that order. But a
// call only gives away which experts a token selects and their weights, for which few of its logits have to be known exactly. So:
//
//   router_filter_kernel   all logits as a bf16 matrix product with f32 sums, and the norms of the token rows and of the router's rows
//   router_refine_kernel   a warp a token: from |product - logit| <= c |x| |w| an interval of every expert's score; experts that cannot be among
//                          the selected ones (nor decide which groups are kept) drop out; the chains of the others in their own order;
//                          selection, weights and telemetry from these as in router_reg.cuh
//
// What is selected, and every bit of the weights, is what all exact logits would give: an expert drops out only if k scores are above the upper end of its own.
// A score is a monotone function of the logit's bf16 value here (the logit itself, or its sigmoid plus the expert's bias: nvmoe_sigmoidf is monotone over
// all bf16 values), so that an interval's ends are the scores of the ends. Rows without a usable bound (NaN, infinities, norms
// that overflow) keep every expert.
//
// The bound, in units u = 2^-24 of |x| |w|, which is at least sum |x_i w_i| over the products, exact in f32, that both sides add up. A chain of
// n = hidden / 64 terms and six folds errs by n + 6. The tensor core adds 16 columns a step: it aligns its 17 addends at the largest and cuts them off
// 2^-25 below that, and cuts the sum to 24 bits (measured, not documented: of addends to 1, 2^-25 still counts and 2^-26 does not; all-positive rows that begin
// with the largest product err by 4.7 u a step), so at most 17 / 2 + 2 u of the largest partial sum or product; kStepUnits are taken, and
// tests/test_gpu_router_product.py holds both on rows made for it, which reach 0.12 of the bound. Partial sums are kept small: after
// every 128 columns they are added to registers, one u each, so that the steps of a row err by no more than those of 128 columns. At hidden 7168 that
// makes 305 u, and two to three of 256 logits a token have to be made exactly; with sums over whole rows in the tensor core 7300 u, and eleven.
#include <cuda.h>
#include <cuda_bf16.h>

#include "experts_tc.cuh"
#include "router_reg.cuh"
#include "tcgen05.cuh"

namespace nvmoe {
namespace {

using namespace tc;

constexpr uint32_t kFlushBlocks = 2u;  // of 64 columns, after which the sums are taken out of the tensor core
constexpr uint32_t kFilterTokens = 128u, kFilterColumns = 64u;  // of a tile: rows of a 128-byte swizzled box
constexpr uint32_t kSumWarps = 16u, kFilterThreads = 32u * (4u + kSumWarps), kFilterMaxSlots = 8u, kFilterSmem = 200u * 1024u;

struct FilterBarriers {
    uint64_t full[kFilterMaxSlots], empty[kFilterMaxSlots], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base, abort;
};

struct FilterKernel {
    const uint16_t* w;
    float* product;   // [splits][tokens][outputs up to a multiple of 16]
    float* x_norm2;   // [splits][tokens] sums of squares; -1 for zeros only
    float* w_norm;    // [outputs]
    uint32_t* status;
    uint32_t tokens, hidden, outputs, n, slots, tmem_columns;
    long long wait_cycles;
    bool withhold;  // (debug) the first CTA leaves out its first stage, whose waits must then give up
    CallStart start;
};

__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ float square_sum(const uint4& v, float sum) {
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        sum = fma_bf16((uint16_t)words[i], (uint16_t)words[i], sum);
        sum = fma_bf16((uint16_t)(words[i] >> 16), (uint16_t)(words[i] >> 16), sum);
    }
    return sum;
}

// 128 tokens by all outputs a CTA, of a part of the columns where that leaves SMs idle (the refinement adds the parts up). Bound by the token rows (16384 x 7168
// are 235 MB). Warp 0 issues the copies, 1 the MMAs, 2 and 3 make the norms of the router's rows (shared out over the CTAs). Sixteen warps, four to a
// quarter of the tokens, make the norms of the token rows from the staged tiles, a quarter of the columns each, and add up a quarter of the outputs.
__global__ void __launch_bounds__(kFilterThreads, 1) router_filter_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map,
                                                                         const FilterKernel p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ FilterBarriers bars;
    __shared__ float row_squares[4][kFilterTokens];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    volatile uint32_t* abort_flag = &bars.abort;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t x_bytes = kFilterTokens * 128u, stage_bytes = x_bytes + p.n * 128u;
    const uint32_t all_blocks = (p.hidden + kFilterColumns - 1u) / kFilterColumns;
    const uint32_t block0 = all_blocks * blockIdx.y / gridDim.y, block1 = all_blocks * (blockIdx.y + 1u) / gridDim.y;
    if (threadIdx.x == 0u) {
        for (uint32_t s = 0; s < p.slots; s++) {
            mbar_init(&bars.full[s], 1u);
            mbar_init(&bars.empty[s], 1u + kSumWarps);  // the MMAs that read it, the warps
        }
        for (uint32_t i = 0; i < 2u; i++) {
            mbar_init(&bars.acc_full[i], 1u);
            mbar_init(&bars.acc_empty[i], kSumWarps);
        }
        mbar_init(&bars.drain, 1u);
        bars.abort = 0u;
        fence_mbar_init();
    }
    __syncthreads();
    if (warp == 1u) {
        tmem_alloc(&bars.tmem_base, p.tmem_columns);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars.tmem_base, token0 = blockIdx.x * kFilterTokens;
    grid_dependency_sync();
    begin_call(p.start);
    if (warp == 0u) {
        if (lane == 0u) {
            uint32_t slot = 0u, parity = 1u;
            for (uint32_t b = block0; b < block1; b++) {
                if (!mbar_wait(&bars.empty[slot], parity, abort_flag, p.wait_cycles)) break;
                const uint32_t at = smem_u32(smem) + slot * stage_bytes;
                if (!p.withhold || b != 0u || blockIdx.x != 0u) {
                    mbar_arrive_expect_tx(&bars.full[slot], stage_bytes);
                    tma_load_2d(at, &x_map, (int)(b * kFilterColumns), (int)token0, &bars.full[slot]);
                    tma_load_2d(at + x_bytes, &w_map, (int)(b * kFilterColumns), 0, &bars.full[slot]);
                }
                if (++slot == p.slots) {
                    slot = 0u;
                    parity ^= 1u;
                }
            }
        }
    } else if (warp == 1u) {
        if (lane == 0u) {
            // f32 sums, bf16 operands, both K-major
            const uint32_t idesc = 1u << 4 | 1u << 7 | 1u << 10 | (p.n >> 3) << 17 | (kFilterTokens >> 4) << 24;
            uint32_t slot = 0u, parity = 0u;
            for (uint32_t b = block0; b < block1; b++) {
                const uint32_t chunk = (b - block0) / kFlushBlocks, at_chunk = (b - block0) % kFlushBlocks, acc = chunk & 1u;
                if (at_chunk == 0u && !mbar_wait(&bars.acc_empty[acc], ((chunk >> 1) & 1u) ^ 1u, abort_flag, p.wait_cycles)) break;
                if (!mbar_wait(&bars.full[slot], parity, abort_flag, p.wait_cycles)) break;
                tc_fence_after();
                const uint32_t at = smem_u32(smem) + slot * stage_bytes;
                const uint64_t a = desc_k_major_sw128(at), w = desc_k_major_sw128(at + x_bytes);
#pragma unroll
                for (uint32_t k = 0; k < kFilterColumns / 16u; k++)  // (32 bytes of a row each)
                    tc_mma_bf16(tmem + acc * p.n, a + 2u * k, w + 2u * k, idesc, at_chunk != 0u || k != 0u ? 1u : 0u);
                tc_commit(&bars.empty[slot]);
                if (at_chunk + 1u == kFlushBlocks || b + 1u == block1) tc_commit(&bars.acc_full[acc]);
                if (++slot == p.slots) {
                    slot = 0u;
                    parity ^= 1u;
                }
            }
            // (nothing of this CTA may still be reading shared memory or using tensor memory when they are released, and another role may give
            // up when this one is through with its loop)
            tc_commit(&bars.drain);
            mbar_wait_winddown(&bars.drain, 0u, kWinddownCycles);
        }
    } else if (warp < 4u) {
        const uint32_t ctas = gridDim.x * gridDim.y;
        for (uint32_t e = (blockIdx.y * gridDim.x + blockIdx.x) * 2u + warp - 2u; e < p.outputs; e += ctas * 2u) {
            float sum = 0.0f;
            for (uint32_t c = lane * 8u; c < p.hidden; c += 256u) sum = square_sum(__ldg(reinterpret_cast<const uint4*>(p.w + (size_t)e * p.hidden + c)), sum);
            sum = warp_butterfly_sum(sum);
            if (lane == 0u) p.w_norm[e] = sqrtf(sum);
        }
    } else {
        const uint32_t quadrant = warp & 3u, part = (warp - 4u) >> 2, row = quadrant * 32u + lane, token = token0 + row;
        uint32_t slot = 0u, parity = 0u, any = 0u, chunk = 0u;
        float squares[2] = {0.0f, 0.0f}, sums[4][16];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int q = 0; q < 16; q++) sums[i][q] = 0.0f;
        // the sums of a chunk, 16 outputs at a time: part, part + 4, ..
        auto flush = [&] {
            const uint32_t acc = chunk & 1u;
            if (!mbar_wait_warp(&bars.acc_full[acc], (chunk >> 1) & 1u, abort_flag, p.wait_cycles)) return false;
            tc_fence_after();
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++) {
                const uint32_t c = 16u * (part + 4u * i);
                if (c >= p.n) continue;
                uint32_t r[16];
                tmem_ld16(tmem + acc * p.n + ((quadrant * 32u) << 16) + c, r);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 16; q++) sums[i][q] = __fadd_rn(sums[i][q], __uint_as_float(r[q]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0u) mbar_arrive(&bars.acc_empty[acc]);
            chunk++;
            return true;
        };
        bool alive = true;
#pragma unroll 1
        for (uint32_t b = block0; alive; b++) {
            const bool last = b == block1;
            if (!last) {
                alive = mbar_wait_warp(&bars.full[slot], parity, abort_flag, p.wait_cycles);
                if (!alive) break;
                const unsigned char* tile = smem + slot * stage_bytes;
#pragma unroll
                for (uint32_t c = 0; c < 2u; c++) {
                    const uint4 v = *reinterpret_cast<const uint4*>(tile + swizzle128_offset(row, 2u * part + c));
                    squares[c] = square_sum(v, squares[c]);
                    any |= v.x | v.y | v.z | v.w;
                }
                __syncwarp();
                if (lane == 0u) mbar_arrive(&bars.empty[slot]);
                if (++slot == p.slots) {
                    slot = 0u;
                    parity ^= 1u;
                }
            }
            // (a block late: the next one's slot is given back before the wait for the sums)
            if (b != block0 && (last || (b - block0) % kFlushBlocks == 0u)) alive = flush();
            if (last) break;
        }
        row_squares[part][row] = (any & 0x7fff7fffu) == 0u ? -1.0f : squares[0] + squares[1];
        named_barrier(1u, 32u * kSumWarps);  // (every one of the warps comes here, through with its loop or given up)
        if (alive && token < p.tokens) {
            const size_t at = (size_t)blockIdx.y * p.tokens + token;
            if (part == 0u) {
                float all = -1.0f;
#pragma unroll
                for (int i = 0; i < 4; i++) all = all < 0.0f ? row_squares[i][row] : row_squares[i][row] < 0.0f ? all : all + row_squares[i][row];
                p.x_norm2[at] = all;
            }
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++) {
                const uint32_t c = 16u * (part + 4u * i);
                if (c >= p.n) continue;
                float4* out = reinterpret_cast<float4*>(p.product + at * p.n + c);
#pragma unroll
                for (int q = 0; q < 4; q++) out[q] = make_float4(sums[i][4 * q], sums[i][4 * q + 1], sums[i][4 * q + 2], sums[i][4 * q + 3]);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1u) {
        tc_fence_after();
        tmem_dealloc(tmem, p.tmem_columns);
    }
    if (*abort_flag && threadIdx.x == 0u) {
        raise_status(p.status, NVMOE_STATUS_WAIT_EXPIRED);
        winddown_pause();
    }
}

__device__ __forceinline__ void add_words(const uint4& x, const uint4& w, float* acc) {
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; q++) acc[q] = fma_bf16((uint16_t)xs[q], (uint16_t)ws[q], acc[q]);
#pragma unroll
    for (int q = 0; q < 4; q++) acc[q] = fma_bf16((uint16_t)(xs[q] >> 16), (uint16_t)(ws[q] >> 16), acc[q]);
}

// The exact sum of router_linear_kernel for a token and an expert by eight lanes: lane l of them plays lanes 4 l .. 4 l + 3 and 32 + 4 l .. of the
// shader's 64 (whose words lie 64 apart), 16 bytes of either a step; the loads of DEPTH steps are issued together. All eight end with the sum.
// Called by a whole warp.
template <int D>
struct Depth {
    static constexpr int value = D;
};
// (volatile: the loads of a group stay together, ahead of the sums)
__device__ __forceinline__ uint4 load_row(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
template <int DEPTH>
__device__ __forceinline__ float exact_sum(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, uint32_t hidden) {
    const uint32_t l = threadIdx.x & 7u, steps = hidden / 128u;
    const uint4* xr = reinterpret_cast<const uint4*>(x) + l;
    const uint4* wr = reinterpret_cast<const uint4*>(w) + l;
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    auto run = [&](auto depth, uint32_t s) {
        constexpr int D = decltype(depth)::value;
        uint4 xv[D][2], wv[D][2];
#pragma unroll
        for (int u = 0; u < D; u++) {
            wv[u][0] = load_row(wr + 16u * (s + u));
            wv[u][1] = load_row(wr + 16u * (s + u) + 8u);
            xv[u][0] = load_row(xr + 16u * (s + u));
            xv[u][1] = load_row(xr + 16u * (s + u) + 8u);
        }
#pragma unroll
        for (int u = 0; u < D; u++) {
            add_words(xv[u][0], wv[u][0], acc);
            add_words(xv[u][1], wv[u][1], acc + 4);
        }
    };
    uint32_t s = 0u;
#pragma unroll 1
    for (; s + DEPTH <= steps; s += DEPTH) run(Depth<DEPTH>{}, s);
#pragma unroll 1
    for (; s < steps; s++) run(Depth<1>{}, s);
    if (hidden % 128u != 0u) add_words(__ldg(xr + 16u * steps), __ldg(wr + 16u * steps), acc);  // (the upper lanes of the shader add nothing)
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        v[q] = __fadd_rn(acc[q], acc[q + 4]);                           // lanes 32 apart
        v[q] = __fadd_rn(v[q], __shfl_xor_sync(0xffffffffu, v[q], 4));  // 16
        v[q] = __fadd_rn(v[q], __shfl_xor_sync(0xffffffffu, v[q], 2));  // 8
        v[q] = __fadd_rn(v[q], __shfl_xor_sync(0xffffffffu, v[q], 1));  // 4
    }
    return __fadd_rn(__fadd_rn(v[0], v[2]), __fadd_rn(v[1], v[3]));     // 2, 1
}

struct RefineKernel {
    RouterLaunch router;
    const uint16_t* x;
    const uint16_t* w;
    const uint16_t* logit_bias;  // or null
    const float* product;
    const float* x_norm2;
    const float* w_norm;
    uint32_t hidden, n, splits;
    float relative;  // of |x| |w|
};

// The largest `count`-th of the lanes' keys (EPL each, 0: none), as warp_best orders them; 0 if there are fewer.
template <int EPL>
__device__ __forceinline__ uint32_t nth_key(uint32_t (&keys)[EPL], uint32_t count) {
    uint32_t top = 0u;
#pragma unroll 1
    for (uint32_t r = 0; r < count; r++) {
        uint32_t best = 0u;
#pragma unroll
        for (int j = 0; j < EPL; j++) best = max(best, keys[j]);
        top = __reduce_max_sync(0xffffffffu, best);
        const uint32_t holders = __ballot_sync(0xffffffffu, best == top);
        if ((threadIdx.x & 31u) == (uint32_t)__ffs(holders) - 1u) {
            bool gone = false;
#pragma unroll
            for (int j = 0; j < EPL; j++) {
                const bool here = !gone && keys[j] == top;
                gone |= here;
                keys[j] = here ? 0u : keys[j];
            }
        }
    }
    return top;
}

// A warp a token; the exact sums of a block's tokens are shared out over all of its lanes, eight a sum.
constexpr uint32_t kRefineWarps = 4u;
constexpr int kRefineDepth = 4;
template <int EPL, bool GROUPS>
__global__ void __launch_bounds__(32 * kRefineWarps, EPL > 4 ? 3 : 4) router_refine_kernel(const RefineKernel p) {
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr float kInf = __builtin_huge_valf();
    __shared__ uint32_t pairs[kRefineWarps * 32 * EPL];  // (token of the block << 16 | expert) whose sums are asked for
    __shared__ float sums[kRefineWarps * 32 * EPL];
    __shared__ uint32_t counts[kRefineWarps];
    grid_dependency_sync();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, token0 = blockIdx.x * kRefineWarps;
    const bool valid = token0 + warp < p.router.tokens;
    const uint32_t token = valid ? token0 + warp : p.router.tokens - 1u;  // (a warp past the last token asks for nothing)
    const nvmoe_geometry& g = p.router.g;
    const uint32_t E = g.routed_experts, k = g.routed_k;
    const bool sigmoid = g.router_kind == NVMOE_ROUTER_SCORE_TOPK;

    // ---- an interval of every expert's logit, then of its score; as ordered keys ----------------------------------------
    // (whatever is loaded is asked for first: the block waits once)
    float product[EPL], w_norm[EPL], logit_bias[EPL], select_bias[EPL];
#pragma unroll
    for (int j = 0; j < EPL; j++) {
        const uint32_t e = min(lane + 32u * j, E - 1u);
        product[j] = __ldg(p.product + (size_t)token * p.n + e);
        w_norm[j] = __ldg(p.w_norm + e);
        logit_bias[j] = p.logit_bias ? nvmoe_bf16_to_f32(__ldg(p.logit_bias + e)) : 0.0f;
        select_bias[j] = sigmoid ? read_bias(p.router.bias, g.bias_dtype, e) : 0.0f;
    }
    float x_norm = __ldg(p.x_norm2 + token);
#pragma unroll 2
    for (uint32_t s = 1; s < p.splits; s++) {
        const size_t at = (size_t)s * p.router.tokens + token;
        const float part = __ldg(p.x_norm2 + at);
#pragma unroll
        for (int j = 0; j < EPL; j++) product[j] += __ldg(p.product + at * p.n + min(lane + 32u * j, E - 1u));
        x_norm = x_norm < 0.0f ? part : part < 0.0f ? x_norm : x_norm + part;
    }
    x_norm = x_norm < 0.0f ? 0.0f : sqrtf(x_norm) + 1e-16f;  // (squares of less than 1e-19 may have been lost)
    auto score_of = [&](float logit, int j) { return sigmoid ? __fadd_rn(nvmoe_sigmoidf(logit), select_bias[j]) : logit; };
    auto logit_of = [&](float sum, int j) { return nvmoe_round_bf16(p.logit_bias ? __fadd_rn(sum, logit_bias[j]) : sum); };
    float val[EPL];                            // the logit of the experts that `known` names
    uint32_t low[EPL], high[EPL], known = 0u;  // keys of the score's ends (0: no expert)
    float low_score[EPL], high_score[EPL];
#pragma unroll
    for (int j = 0; j < EPL; j++) {
        const float a = product[j], norm = w_norm[j] + 1e-16f;
        // (operands below the smallest normal number may count as zeros in the product)
        const float error = fmaf(x_norm * norm, p.relative, x_norm == 0.0f ? 0.0f : fmaf(x_norm + norm, 1e-33f, 1e-30f));
        const bool bounded = x_norm < 1e30f && norm < 1e30f && error < 1e30f && fabsf(a) < 1e30f && fabsf(logit_bias[j]) < 1e30f;
        const float lo = logit_of(a - error, j), hi = logit_of(a + error, j);
        val[j] = hi;
        if (bounded && lo == hi) known |= 1u << j;
        low_score[j] = score_of(lo, j);
        high_score[j] = score_of(hi, j);
        if (!bounded || !(low_score[j] <= high_score[j])) {
            low_score[j] = kNegInf;
            high_score[j] = kInf;
        }
        const bool there = lane + 32u * j < E;
        if (!there) low_score[j] = high_score[j] = kNegInf;
        low[j] = there ? score_key(low_score[j]) : 0u;
        high[j] = there ? score_key(high_score[j]) : 0u;
    }

    // ---- groups that may be kept, and those that are ------------------------------------------------------------------------
    const uint32_t per = GROUPS ? E / g.n_group : 1u, side = GROUPS ? 32u / per : 1u;  // (a group is a run of `per` lanes)
    uint32_t open = 0u, sure = kFull, second_key[EPL];  // groups; and per slot the key of the second best low end of the lane's group
    auto group_of = [&](int j) { return (uint32_t)j * side + lane / per; };
    // the two best of `score` of each lane's groups, all slots side by side
    auto best_two = [&](const float (&score)[EPL], float (&first)[EPL], float (&second)[EPL]) {
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            first[j] = score[j] > kNegInf ? score[j] : kNegInf;
            second[j] = kNegInf;
        }
#pragma unroll 1
        for (uint32_t o = 1u; o < per; o <<= 1) {
#pragma unroll
            for (int j = 0; j < EPL; j++) {
                const float other_first = __shfl_xor_sync(kFull, first[j], o), other_second = __shfl_xor_sync(kFull, second[j], o);
                second[j] = fmaxf(fminf(first[j], other_first), fmaxf(second[j], other_second));
                first[j] = fmaxf(first[j], other_first);
            }
        }
    };
    if (GROUPS) {
        uint32_t group_low = 0u, group_high = 0u;  // lane g keeps group g
        float first[EPL], second[EPL], top[EPL], next[EPL];
        best_two(low_score, first, second);
        best_two(high_score, top, next);
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            second_key[j] = score_key(per >= 2u ? second[j] : first[j]);
            float lo = per >= 2u ? __fadd_rn(first[j], second[j]) : first[j], hi = per >= 2u ? __fadd_rn(top[j], next[j]) : top[j];
            if (!(lo <= hi)) {
                lo = kNegInf;
                hi = kInf;
            }
            lo = __shfl_sync(kFull, lo, (lane % side) * per);
            hi = __shfl_sync(kFull, hi, (lane % side) * per);
            if (lane / side == (uint32_t)j && lane < g.n_group) {
                group_low = score_key(lo);
                group_high = score_key(hi);
            }
        }
        uint32_t keys[1] = {group_low};
        const uint32_t line = nth_key<1>(keys, g.topk_group);
        open = __ballot_sync(kFull, group_high != 0u && group_high >= line);
        uint32_t rivals = 0u;
#pragma unroll 1
        for (uint32_t q = 0; q < g.n_group; q++) {
            const uint32_t other = __shfl_sync(kFull, group_high, q);
            if (q != lane && other >= group_low) rivals++;
        }
        sure = __ballot_sync(kFull, group_low > score_key(kNegInf) && rivals < g.topk_group) & open;
    }
    auto in_groups = [&](uint32_t groups, int j) { return !GROUPS || (group_of(j) < 32u && ((groups >> group_of(j)) & 1u) != 0u); };

    // ---- the logits that matter: first of the two best experts, by any chance, of groups that may be kept or not; then, with the kept groups known, of
    // the experts that may be among the k best
    uint32_t wanted = 0u;
#pragma unroll 1
    for (uint32_t pass = GROUPS && __syncthreads_or(open != sure) ? 0u : 1u; pass < 2u; pass++) {
        uint32_t keys[EPL];
#pragma unroll
        for (int j = 0; j < EPL; j++) keys[j] = in_groups(sure, j) ? low[j] : 0u;
        const uint32_t line = pass == 0u ? 0u : nth_key<EPL>(keys, k);
        wanted = 0u;
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const bool may = pass == 0u ? in_groups(open & ~sure, j) && high[j] >= second_key[j] : in_groups(sure, j) && high[j] >= line;
            if (valid && high[j] != 0u && may) wanted |= 1u << j;
        }
        uint32_t n = 0u, place[EPL];
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const bool mine = ((wanted & ~known) >> j) & 1u;
            const uint32_t all = __ballot_sync(kFull, mine);
            place[j] = n + __popc(all & ((1u << lane) - 1u));
            n += __popc(all);
        }
        if (lane == 0u) counts[warp] = n;
        __syncthreads();
        uint32_t base = 0u, total = 0u;
#pragma unroll
        for (uint32_t v = 0; v < kRefineWarps; v++) {
            if (v == warp) base = total;
            total += counts[v];
        }
#pragma unroll
        for (int j = 0; j < EPL; j++)
            if (((wanted & ~known) >> j) & 1u) pairs[base + place[j]] = warp << 16 | (lane + 32u * j);
        __syncthreads();
#pragma unroll 1
        for (uint32_t at = 4u * warp; at < total; at += 4u * kRefineWarps) {
            const uint32_t mine = min(at + (lane >> 3), total - 1u), pair = pairs[mine];  // (a place past the list repeats its last sum)
            const float sum = exact_sum<kRefineDepth>(p.x + (size_t)(token0 + (pair >> 16)) * p.hidden, p.w + (size_t)(pair & 0xffffu) * p.hidden, p.hidden);
            if ((lane & 7u) == 0u) sums[mine] = sum;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            if (((wanted & ~known) >> j & 1u) == 0u) continue;
            val[j] = logit_of(sums[base + place[j]], j);
            low[j] = high[j] = score_key(score_of(val[j], j));
        }
        known |= wanted;
        if (!GROUPS || pass != 0u) continue;
        float my_group = kNegInf, score[EPL], first[EPL], second[EPL];
#pragma unroll
        for (int j = 0; j < EPL; j++) score[j] = (wanted >> j) & 1u ? score_of(val[j], j) : kNegInf;
        best_two(score, first, second);
#pragma unroll
        for (int j = 0; j < EPL; j++) {
            const float group = __shfl_sync(kFull, per >= 2u ? __fadd_rn(first[j], second[j]) : first[j], (lane % side) * per);
            if (lane / side == (uint32_t)j) my_group = group;
        }
        const uint32_t candidates = open & ~sure;
#pragma unroll 1
        for (uint32_t round = __popc(sure); round < g.topk_group; round++) {
            const bool free = lane < g.n_group && ((candidates & ~sure) >> lane & 1u) != 0u && my_group >= kNegInf;  // (not a NaN)
            const uint32_t winner = warp_best(my_group, free ? lane : kUnboundSlot);
            if (winner != kUnboundSlot) sure |= 1u << winner;
        }
    }
    float score[EPL];
#pragma unroll
    for (int j = 0; j < EPL; j++) {
        score[j] = kNegInf;
        if (((wanted >> j) & 1u) == 0u) continue;
        if (sigmoid) val[j] = nvmoe_sigmoidf(val[j]);
        score[j] = sigmoid ? __fadd_rn(val[j], select_bias[j]) : val[j];
    }
    const uint32_t taken = ~wanted;
    uint32_t my_e, rank;
    float my_v;
    if (!valid) return;
    const bool found = pick_experts<EPL>(E, k, val, score, taken, my_e, my_v);
    finish_token<true>(p.router, counts_of(p.router), token, found, my_e, my_v, rank);
}

constexpr double kStepUnits = 16.0;     // (10.5 by the above)
constexpr uint32_t kFilterSplits = 8u;  // at most

}  // namespace

// Which calls. Product and refinement take 13 us of latency, more with more experts a lane; the tiled projection (router.cu), in blocks of 32
// tokens x 16 outputs, 15 us a round of the SMs at 2880 columns. Layers, us, pinned / filtered (tokens x hidden x experts): 512 x 2880 x 32 69.1 / 67.4,
// 2048 135.9 / 134.2; 2048 x 1024 x 32 81.4 / 80.8, 768 59.9 / 60.8; 512 x 2880 x 128 (one round) 110.7 / 113.5, 768 (two) 128.5 / 119.9, 2048 185.1 / 152.9;
// 257 x 4096 x 64 90.6 / 89.6, 2048 191.0 / 173.3; grouped, 768 x 2048 x 64 111.3 / 115.1, 1536 157.2 / 154.0; 2048 x 7168 x 256 788 / 673;
// 2048 x 512 x 16 64.8 / 66.8. In one round of the tiled blocks that of many experts, or of groups, costs more than it gives, unless the round is nearly full, whose blocks
// share the rows' bandwidth: 300 x 6016 x 192 141.3 / 146.0, 417 x 6976 x 160 (140 blocks) 142.5 / 134.7; grouped, 264 x 7552 x 256 120.7 / 129.4, 363 x 4480 x 128 114.2 / 121.0, 551 x
// 5120 x 128 (144 blocks) 149.8 / 141.0, 630 x 6208 x 64 146.2 / 150.5, 1049 x 7040 x 64 (132) 162.2 / 157.7, 576 x 1792 x 32 57.6 / 58.8, 495 x 2816 x 32 59.4 / 59.8, 602 x 3840 x 16 70.0 /
// 67.8. Of 430 layers drawn around the line the rule takes the slower way by 0.14 % in the mean (0.8 % without these), by 4 % at most.
// (A size that is taken stays so with more tokens: a plan's scratch is sized for its largest call.)
bool router_filter_form(const nvmoe_geometry& g) {
    const bool form = g.router_kind == NVMOE_ROUTER_TOPK_SOFTMAX || (g.router_kind == NVMOE_ROUTER_SCORE_TOPK && g.activation == NVMOE_ACT_SIGMOID);
    const uint32_t total_k = g.routed_k + (g.router_kind == NVMOE_ROUTER_SCORE_TOPK ? g.always_count : 0u), per = g.n_group ? g.routed_experts / g.n_group : 1u;
    return form && g.routed_experts <= 256u && total_k <= 32u && g.hidden_size % 64u == 0u && per <= 32u && (per & (per - 1u)) == 0u;
}
bool router_filter_takes(const nvmoe_geometry& g, uint32_t tokens) {
    if (!router_filter_form(g) || tokens <= 256u) return false;
    const uint64_t blocks = (uint64_t)((tokens + 31u) / 32u) * ((g.routed_experts + 15u) / 16u);
    const uint32_t sms = device_sm_count();
    const uint64_t rounds = (blocks + sms - 1u) / sms;
    uint64_t columns = 1024u + 24u * (uint64_t)g.routed_experts;
    if (rounds == 1u) {
        const bool nearly_full = 10u * blocks >= 9u * (uint64_t)sms;
        if (g.routed_experts > (g.n_group ? 32u : 128u) && !(nearly_full && (!g.n_group || g.routed_experts <= 128u))) return false;
        if (g.n_group && g.routed_experts <= 32u) columns += 1200u;
    }
    return rounds * g.hidden_size >= columns;
}

static uint32_t filter_tiles(uint32_t tokens) { return (tokens + kFilterTokens - 1u) / kFilterTokens; }
static uint32_t filter_splits(uint32_t tokens, uint32_t hidden) {
    const uint32_t idle = device_sm_count() / filter_tiles(tokens), blocks = (hidden + kFilterColumns - 1u) / kFilterColumns;
    const uint32_t most = blocks / 4u < kFilterSplits ? blocks / 4u : kFilterSplits;
    return idle < most ? (idle > 1u ? idle : 1u) : (most > 1u ? most : 1u);
}

static uint32_t router_filter_width(uint32_t outputs) { return (outputs + 15u) / 16u * 16u; }

// Splits x tokens of any call of up to so many tokens.
static size_t filter_rows(uint32_t max_tokens) {
    const size_t split = (size_t)kFilterSplits * max_tokens, filled = device_sm_count() * (size_t)kFilterTokens;
    return max_tokens > (split < filled ? split : filled) ? max_tokens : (split < filled ? split : filled);
}
size_t router_filter_floats(uint32_t max_tokens, uint32_t experts) { return filter_rows(max_tokens) * (router_filter_width(experts) + 1u) + experts; }

struct Scratch {
    float* w_norm;
    float* x_norm2;
    float* product;
};
static Scratch scratch_of(const RouterFilter& f, uint32_t tokens, uint32_t experts) {
    const size_t rows = (size_t)filter_splits(tokens, f.hidden) * tokens, width = router_filter_width(experts);
    return Scratch{f.scratch + rows * (width + 1u), f.scratch + rows * width, f.scratch};
}

bool launch_router_filter(const RouterLaunch& router, const RouterFilter& f, cudaStream_t stream) {
    const uint32_t E = router.g.routed_experts, n = router_filter_width(E);
    CUtensorMap x_map, w_map;
    if (!tc_encode_bf16_map(&x_map, f.x, router.tokens, f.hidden, kFilterColumns, kFilterTokens) || !tc_encode_bf16_map(&w_map, f.w, E, f.hidden, kFilterColumns, n)) return false;
    FilterKernel k{};
    k.w = f.w;
    const Scratch scratch = scratch_of(f, router.tokens, E);
    k.product = scratch.product;
    k.x_norm2 = scratch.x_norm2;
    k.w_norm = scratch.w_norm;
    k.status = router.status;
    k.tokens = router.tokens;
    k.hidden = f.hidden;
    k.outputs = E;
    k.n = n;
    k.slots = kFilterSmem / (kFilterTokens * 128u + n * 128u);
    if (k.slots > kFilterMaxSlots) k.slots = kFilterMaxSlots;
    k.tmem_columns = 32u;
    while (k.tmem_columns < 2u * n) k.tmem_columns *= 2u;
    k.wait_cycles = f.wait_cycles;
    k.withhold = f.withhold;
    k.start = f.start;
    launch_chained(router_filter_kernel, dim3(filter_tiles(router.tokens), filter_splits(router.tokens, f.hidden)), dim3(kFilterThreads),
                   (size_t)k.slots * (kFilterTokens * 128u + n * 128u) + 1024u, stream, x_map, w_map, k);
    return true;
}

// The bound, of |x| |w| (a fiftieth for the roundings of the norms and of the bound itself, two units for those of the interval's ends).
static float router_filter_relative(uint32_t hidden, uint32_t splits) {
    const double chain = hidden / 64.0 + 6.0, steps = kFlushBlocks * (kFilterColumns / 16u) * kStepUnits;
    const double flushes = (double)(hidden + kFlushBlocks * kFilterColumns - 1u) / (kFlushBlocks * kFilterColumns) + 2.0 * splits;
    return (float)(1.02 * (chain + steps + flushes + 2.0) / (1 << 24));
}

RouterProduct router_product_of(const RouterFilter& f, uint32_t tokens, uint32_t experts) {
    const Scratch scratch = scratch_of(f, tokens, experts);
    const uint32_t splits = filter_splits(tokens, f.hidden);
    return RouterProduct{scratch.product, scratch.x_norm2, scratch.w_norm, splits, router_filter_width(experts), router_filter_relative(f.hidden, splits)};
}

void launch_router_refine(const RouterLaunch& router, const RouterFilter& f, cudaStream_t stream) {
    const uint32_t E = router.g.routed_experts;
    RefineKernel r{};
    r.router = router;
    r.x = f.x;
    r.w = f.w;
    r.logit_bias = f.logit_bias;
    const Scratch scratch = scratch_of(f, router.tokens, E);
    r.product = scratch.product;
    r.x_norm2 = scratch.x_norm2;
    r.w_norm = scratch.w_norm;
    r.hidden = f.hidden;
    r.splits = filter_splits(router.tokens, f.hidden);
    r.n = router_filter_width(E);
    r.relative = router_filter_relative(f.hidden, r.splits);
    const dim3 grid((router.tokens + kRefineWarps - 1u) / kRefineWarps), block(32u * kRefineWarps);
    const bool groups = router.g.n_group != 0u;
    const auto kernel = groups ? (E <= 32u ? router_refine_kernel<1, true> : E <= 128u ? router_refine_kernel<4, true> : router_refine_kernel<8, true>)
                               : (E <= 32u ? router_refine_kernel<1, false> : E <= 128u ? router_refine_kernel<4, false> : router_refine_kernel<8, false>);
    launch_chained(kernel, grid, block, 0, stream, r);
}

void configure_router_filter() {
    cudaFuncSetAttribute(router_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kFilterSmem + 1024u));
}

}  // namespace nvmoe
