// Weighted combine of the per-route expert outputs.
//
//   runtime-rs/shaders/moe_reduce_batch1_bf16.comp.template:29-55
//
// The route weight is already inside each per-route row (the down stage applied it), so the
// combine is a sum over the K routes of a token in route order — ascending expert id — with a
// bf16 rounding after every add, then one multiply by ROUTED_SCALE and a final rounding.  That
// order and those roundings are the reference's and are reproduced exactly.
#include "common.cuh"

namespace nvmoe {
namespace {

__global__ void __launch_bounds__(256) reduce_kernel(const uint32_t* __restrict__ expert_outputs,
                                                    uint32_t* __restrict__ output, uint32_t tokens, uint32_t K,
                                                    uint32_t hidden_words, float routed_scale,
                                                    const uint32_t* __restrict__ computed, CallClock* clock) {
    grid_dependency_sync();
    const uint64_t total = (uint64_t)tokens * hidden_words;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = (uint32_t)(i / hidden_words), word = (uint32_t)(i % hidden_words);
        const uint32_t* in = expert_outputs + (size_t)t * K * hidden_words + word;
        float lo = 0.0f, hi = 0.0f;
        for (uint32_t r = 0; r < K; r++) {
            // a route the down stage skipped (computed[route] says "nowhere") counts as a row of zeros
            const uint32_t c = (computed && computed[(size_t)t * K + r] == kUnboundSlot) ? 0u : in[(size_t)r * hidden_words];
            lo = nvmoe_round_bf16(__fadd_rn(lo, nvmoe_bf16_to_f32(c)));
            hi = nvmoe_round_bf16(__fadd_rn(hi, nvmoe_bf16_to_f32(c >> 16)));
        }
        output[i] = pack_bf16x2(__fmul_rn(lo, routed_scale), __fmul_rn(hi, routed_scale));
    }
    note_end(clock);
}

// Two columns of a sum, rounded to bf16: as the f32 sum rounded, since 24 bits are more than twice 8 and two.
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ bool either_is_nan(uint32_t pair) { return (pair & 0x7fffu) > 0x7f80u || (pair & 0x7fff0000u) > 0x7f800000u; }

// One word of a token's sum as reduce_kernel takes it, for words in which a NaN turns up (its bits are those of the f32 sums rounded).
__device__ __noinline__ uint32_t combine_word(const uint32_t* in, const uint32_t* marks, uint32_t K, uint32_t hidden_words, float routed_scale) {
    float lo = 0.0f, hi = 0.0f;
    for (uint32_t r = 0; r < K; r++) {
        const uint32_t c = (marks && marks[r] == kUnboundSlot) ? 0u : in[(size_t)r * hidden_words];
        lo = nvmoe_round_bf16(__fadd_rn(lo, nvmoe_bf16_to_f32(c)));
        hi = nvmoe_round_bf16(__fadd_rn(hi, nvmoe_bf16_to_f32(c >> 16)));
    }
    return pack_bf16x2(__fmul_rn(lo, routed_scale), __fmul_rn(hi, routed_scale));
}

// The same sum over 16-byte pieces (eight columns a thread) for rows that allow it: the order of the adds
// of a column and every rounding are unchanged. Bound by memory: DEPTH routes are fetched together, in small calls with their marks
// (EARLY), which then only choose what is added, else after their marks, so that rows of skipped routes are not read.
// Four at a time, except for nine routes, which then take one step where fours would take three (with adds in f32, 4096 tokens of
// 4096 columns 67.8 against 72.4 us). A deeper step that fours need only two for, or that ends in a second one, costs more in
// registers than it saves (with adds in f32, nine against four at a time 62.1 / 61.4 us for 8 routes, 84.0 / 77.4 for 10, 58.1 /
// 54.6 for 16 of 2048 columns).
// Adds in pairs of columns and whole-number arithmetic in 32 bits, before / after: 4096 tokens of four
// routes of 2880 columns 25.8 / 21.0 us, 16384 93.1 / 76.2, 96 of nine of 7168 6.3 / 4.1, 16384 434 / 341 (6.9 TB/s). A grid of the
// resident blocks, 4 or 6 per SM, 74.8 and 344; a thread a piece 76.2 and 337, but 11.5 against 10.5 at 2048 tokens.
template <uint32_t DEPTH, bool EARLY>
__global__ void __launch_bounds__(256) reduce_vec_kernel(const uint4* __restrict__ expert_outputs, uint4* __restrict__ output,
                                                        uint32_t total, uint32_t K, uint32_t hidden_vecs, float routed_scale,
                                                        const uint32_t* __restrict__ computed, CallClock* clock) {
    grid_dependency_sync();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const uint32_t t = i / hidden_vecs, vec = i - t * hidden_vecs;
        const uint4* in = expert_outputs + (size_t)t * K * hidden_vecs + vec;
        const uint32_t* marks = computed ? computed + (size_t)t * K : nullptr;
        uint32_t acc[4] = {0u, 0u, 0u, 0u};
        // (the adds keep the route order)
        for (uint32_t r0 = 0; r0 < K; r0 += DEPTH) {
            bool skipped[DEPTH];
            uint4 c[DEPTH];
#pragma unroll
            for (uint32_t u = 0; u < DEPTH; u++)
                // a route the down stage skipped (computed[route] says "nowhere") counts as a row of zeros
                skipped[u] = r0 + u >= K || (marks && __ldg(marks + r0 + u) == kUnboundSlot);
#pragma unroll
            for (uint32_t u = 0; u < DEPTH; u++)
                c[u] = (EARLY ? r0 + u >= K : skipped[u]) ? make_uint4(0u, 0u, 0u, 0u) : __ldg(in + (size_t)(r0 + u) * hidden_vecs);
#pragma unroll
            for (uint32_t u = 0; u < DEPTH; u++) {
                if (r0 + u >= K) break;
                const uint32_t w[4] = {c[u].x, c[u].y, c[u].z, c[u].w};
#pragma unroll
                for (int j = 0; j < 4; j++) acc[j] = add_bf16x2(acc[j], EARLY && skipped[u] ? 0u : w[j]);
            }
        }
        uint32_t out[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            out[j] = pack_bf16x2(__fmul_rn(nvmoe_bf16_to_f32(acc[j]), routed_scale), __fmul_rn(nvmoe_bf16_to_f32(acc[j] >> 16), routed_scale));
            if (either_is_nan(acc[j])) out[j] = combine_word(reinterpret_cast<const uint32_t*>(in) + j, marks, K, 4u * hidden_vecs, routed_scale);
        }
        output[i] = make_uint4(out[0], out[1], out[2], out[3]);
    }
    note_end(clock);
}

// The combine of an expert-parallel step read straight from the rows that came back from the owners:
// route (t, r) lies at row gather[t * K + r] of `rows` (all-ones: the route was left out and counts as a row
// of zeros). The same adds in the same order with the same roundings as reduce_vec_kernel; only where a row is
// read from differs, which saves the pass that would put the rows back into [T][K][H] order first.
__global__ void __launch_bounds__(256) reduce_gather_kernel(const uint4* __restrict__ rows, const uint32_t* __restrict__ gather,
                                                           uint4* __restrict__ output, uint32_t tokens, uint32_t K,
                                                           uint32_t hidden_vecs, float routed_scale) {
    grid_dependency_sync();
    const uint64_t total = (uint64_t)tokens * hidden_vecs;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = (uint32_t)(i / hidden_vecs), vec = (uint32_t)(i % hidden_vecs);
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] = 0.0f;
        // four routes at a time, as in reduce_vec_kernel: the row numbers together, then the rows together
        for (uint32_t r0 = 0; r0 < K; r0 += 4u) {
            uint32_t row[4];
            uint4 c[4];
#pragma unroll
            for (uint32_t u = 0; u < 4u; u++) row[u] = r0 + u < K ? __ldg(gather + (size_t)t * K + r0 + u) : kUnboundSlot;
#pragma unroll
            for (uint32_t u = 0; u < 4u; u++)
                c[u] = row[u] == kUnboundSlot ? make_uint4(0u, 0u, 0u, 0u) : rows[(size_t)row[u] * hidden_vecs + vec];
#pragma unroll
            for (uint32_t u = 0; u < 4u; u++) {
                if (r0 + u >= K) break;
                const uint32_t w[4] = {c[u].x, c[u].y, c[u].z, c[u].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[2 * j] = nvmoe_round_bf16(__fadd_rn(acc[2 * j], nvmoe_bf16_to_f32(w[j])));
                    acc[2 * j + 1] = nvmoe_round_bf16(__fadd_rn(acc[2 * j + 1], nvmoe_bf16_to_f32(w[j] >> 16)));
                }
            }
        }
        uint4 out;
        out.x = pack_bf16x2(__fmul_rn(acc[0], routed_scale), __fmul_rn(acc[1], routed_scale));
        out.y = pack_bf16x2(__fmul_rn(acc[2], routed_scale), __fmul_rn(acc[3], routed_scale));
        out.z = pack_bf16x2(__fmul_rn(acc[4], routed_scale), __fmul_rn(acc[5], routed_scale));
        out.w = pack_bf16x2(__fmul_rn(acc[6], routed_scale), __fmul_rn(acc[7], routed_scale));
        output[i] = out;
    }
}

// The finaliser of a tensor-parallel expert stage
// (runtime-rs/shaders/distributed_sum_f32_scale_packed_bf16_to_bf16.comp:44-66): the participants' f32
// partial planes are added in participant order, the sum is scaled by a bf16 taken from a packed word
// (the route weight in the upper half of a route word) and rounded to bf16 once.
__global__ void __launch_bounds__(256) sum_f32_scale_packed_bf16_kernel(const float* __restrict__ partials,
                                                                       const uint32_t* __restrict__ scales,
                                                                       uint32_t* __restrict__ output, uint32_t element_count,
                                                                       uint32_t participant_count, uint32_t lane_count,
                                                                       uint32_t elements_per_scale, uint32_t scale_bit_offset) {
    grid_dependency_sync();
    const uint32_t words = element_count / 2u, scales_per_lane = element_count / elements_per_scale;
    const uint64_t total = (uint64_t)lane_count * words;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t lane = (uint32_t)(i / words), element = (uint32_t)(i % words) * 2u;
        float lo = 0.0f, hi = 0.0f;
        for (uint32_t part = 0; part < participant_count; part++) {
            const float2 v = *reinterpret_cast<const float2*>(partials + ((size_t)part * lane_count + lane) * element_count + element);
            lo = __fadd_rn(lo, v.x);
            hi = __fadd_rn(hi, v.y);
        }
        const float slo = nvmoe_bf16_to_f32(scales[(size_t)lane * scales_per_lane + element / elements_per_scale] >> scale_bit_offset);
        const float shi = nvmoe_bf16_to_f32(scales[(size_t)lane * scales_per_lane + (element + 1u) / elements_per_scale] >> scale_bit_offset);
        output[i] = pack_bf16x2(__fmul_rn(lo, slo), __fmul_rn(hi, shi));
    }
}

// Rows of a small call from page-locked host memory, sixteen bytes a thread: bound by the latency of the bus. The copy engine takes as
// long for a few hundred kilobytes, and some microseconds more to hand over to the kernel after it (host call of a tiny layer, 64
// tokens, with the combine storing its rows to host memory too: 51.3 us by copies, 46.4).
__global__ void __launch_bounds__(256) fetch_host_kernel(const uint4* host, uint4* device, uint32_t pieces) {
    grid_dependency_sync();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i < pieces) device[i] = __ldcv(host + i);
}

}  // namespace

void launch_fetch_host(const void* host, void* device, size_t bytes, cudaStream_t stream) {
    const uint32_t pieces = (uint32_t)(bytes / 16u);
    launch_chained(fetch_host_kernel, dim3((pieces + 255u) / 256u), dim3(256), 0, stream, static_cast<const uint4*>(host), static_cast<uint4*>(device), pieces);
}

void launch_sum_f32_scale_packed_bf16(const float* partials, const uint32_t* scales, uint32_t* output, uint32_t element_count,
                                      uint32_t participant_count, uint32_t lane_count, uint32_t elements_per_scale,
                                      uint32_t scale_bit_offset, cudaStream_t stream) {
    const uint64_t total = (uint64_t)lane_count * (element_count / 2u);
    uint64_t blocks = (total + 255u) / 256u;
    if (blocks > 148u * 16u) blocks = 148u * 16u;
    if (blocks == 0u) return;
    launch_chained(sum_f32_scale_packed_bf16_kernel, dim3((uint32_t)blocks), dim3(256), 0, stream, partials, scales, output,
                   element_count, participant_count, lane_count, elements_per_scale, scale_bit_offset);
}

bool launch_reduce_gather(const uint16_t* rows, const uint32_t* gather, uint16_t* output, uint32_t tokens, uint32_t K,
                          uint32_t hidden, float routed_scale, cudaStream_t stream) {
    if (hidden % 8u != 0u || ((reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(output)) & 15u) != 0u) return false;
    const uint64_t vecs = (uint64_t)tokens * (hidden / 8u);
    uint64_t blocks = (vecs + 255u) / 256u;
    if (blocks > 148u * 16u) blocks = 148u * 16u;
    if (blocks == 0u) return true;
    launch_chained(reduce_gather_kernel, dim3((uint32_t)blocks), dim3(256), 0, stream, reinterpret_cast<const uint4*>(rows), gather,
                   reinterpret_cast<uint4*>(output), tokens, K, hidden / 8u, routed_scale);
    return true;
}

void launch_reduce(const uint16_t* expert_outputs, uint16_t* output, uint32_t tokens, uint32_t K, uint32_t hidden,
                   float routed_scale, const uint32_t* computed, CallClock* clock, cudaStream_t stream) {
    if (tokens == 0u) return;
    const uint64_t vecs = (uint64_t)tokens * (hidden / 8u);
    if (hidden % 8u == 0u && ((reinterpret_cast<uintptr_t>(expert_outputs) | reinterpret_cast<uintptr_t>(output)) & 15u) == 0u && vecs < (1ull << 31)) {
        // Up to two blocks per SM (one with nine routes) the latency of the marks counts, beyond it what is read. Layers of 2880 x 256, 32 experts, rows with their marks /
        // after them, us, all experts resident and an eighth of them: 1 token 28.5 / 28.7, 19.9 / 19.8, 64 (90 blocks) 35.5 / 35.7, 31.5 / 31.7,
        // 200 (282) 45.4 / 45.7, 39.7 / 39.3, 1024 87.5 / 87.6, 58.9 / 55.9, 8192 353.5 / 353.5, 189.8 / 166.6; nine routes of 4096 columns,
        // 64 experts, 96 tokens (192) 69.2 / 68.7, 49.2 / 48.2, 4096 494 / 491, 235 / 192.
        uint64_t vec_blocks = (vecs + 255u) / 256u;
        const bool early = vec_blocks <= (K == 9u ? 148u : 2u * 148u);
        if (vec_blocks > 148u * 16u) vec_blocks = 148u * 16u;
        const auto kernel = K == 9u ? (early ? reduce_vec_kernel<9u, true> : reduce_vec_kernel<9u, false>)
                                    : (early ? reduce_vec_kernel<4u, true> : reduce_vec_kernel<4u, false>);
        launch_chained(kernel, dim3((uint32_t)vec_blocks), dim3(256), 0, stream,
                       reinterpret_cast<const uint4*>(expert_outputs), reinterpret_cast<uint4*>(output), (uint32_t)vecs, K, hidden / 8u,
                       routed_scale, computed, clock);
        return;
    }
    const uint64_t total = (uint64_t)tokens * (hidden / 2u);
    uint64_t blocks = (total + 255u) / 256u;
    if (blocks > 148u * 8u) blocks = 148u * 8u;
    launch_chained(reduce_kernel, dim3((uint32_t)blocks), dim3(256), 0, stream,
                   reinterpret_cast<const uint32_t*>(expert_outputs), reinterpret_cast<uint32_t*>(output), tokens, K,
                   hidden / 2u, routed_scale, computed, clock);
}

}  // namespace nvmoe
