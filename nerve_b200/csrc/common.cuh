// Shared declarations of the CUDA MoE backend: launch parameter blocks, the resolved expert
// pointer table, fail-closed status bits and small device helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nerve_cuda_moe.h"
#include "../../include/nvmoe_math.h"

namespace nvmoe {

constexpr uint32_t kUnboundSlot = 0xffffffffu;
constexpr uint32_t kRecordWords = 8u;
constexpr uint32_t kMaxTopK = 64u;       // routed_k + always_count
constexpr uint32_t kMaxExperts = 4096u;  // ids travel in the low 16 bits of a route word
// Programmatic dependent launch: a kernel launched with launch_chained may start (and run whatever
// precedes its grid_dependency_sync) while the kernel before it in the stream is still running;
// grid_dependency_sync returns once that kernel has completed and its writes are visible, and lets
// the next kernel in the stream start in the same way. Every thread of a chained kernel calls it
// before any return, so completion still implies that all earlier kernels have completed, and before
// touching global memory that the launch ahead of it may write or read. What stands before the call may
// rely on the launches before that one: the kernel ahead let this one start after its own wait, when they
// had completed. (Tensor maps and expert tables are read there, place_operands_kernel reads the tokens, experts_layer.cu claims its first work
// from a counter that an earlier launch of the call cleared.) One kernel lets the next start before its wait and does all of its work ahead of
// it: small_schedule_kernel, right behind place_operands_kernel. Whatever it reads, and whatever the kernel behind it reads or counts before its own
// wait, has to stand from launches before place_operands_kernel, which may still be running then, as the schedule may. No other kernel may let the next
// start before its wait. Launched the ordinary way, the same kernels run unchanged.
#ifdef __CUDACC__
__device__ __forceinline__ void grid_dependency_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  Args&&... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}
#endif

constexpr uint32_t kSortChunk = 256u;    // routes per block in the multi-block counting sort

// Weight pointers of one expert after the address/slot tables were validated
// (address_record_is_resident + dynamic_expert_is_valid of
// runtime-rs/shaders/independent_sparse_moe_gate_up_batch1_mxfp4.comp.template:120-228).
// A null w pointer means "not resident": every route to that expert is skipped.
enum : uint32_t {
    kFormatCompact = 0u,   // packaged MXFP4: E2M1 codes two per byte, E8M0 scale per 32 columns
    kFormatExpanded = 1u,  // the same matrix pre-expanded to one E4M3 byte per element, same scales
    kFormatNativeFp8 = 2u  // E4M3 bytes with one E8M0 scale per 128 x 128 block
};
struct ExpertPtrs {
    const uint8_t* w[2];   // gate/up: w1, w3;  down: w2, unused
    const uint8_t* s[2];   // matching E8M0 scales as packaged: [rows][cols/32], or [rows/128][cols/128] (native FP8)
    const uint8_t* ts[2];  // derived copy of the scales, tiled for tcgen05.cp: [row tile][K block][512 bytes]
    uint64_t gen[2];       // generation word of the scale records (what the derived copy is keyed on)
    uint32_t format;       // kFormat* of the expert's matrices
    uint32_t reserved;
};

// The E8M0 scales of an operand matrix: a word of four bytes per row and K block of 128 columns. The words of a row lie side
// by side for the kernels of one CTA (a row's next word is then in the cache when its next K block is fetched) and those of a
// K block for CTA pairs (the scales of a token tile are then one copy).
struct ScaleWords {
    uint32_t* words;
    uint32_t row_stride, block_stride;
    __device__ __forceinline__ uint32_t* at(uint32_t row, uint32_t block) const {
        return words + (size_t)row * row_stride + (size_t)block * block_stride;
    }
    __device__ __forceinline__ uint8_t* byte_at(uint32_t row, uint32_t group) const {  // of columns 32 group ..
        return reinterpret_cast<uint8_t*>(at(row, group / 4u)) + group % 4u;
    }
};

// Everything a grouped expert kernel needs to find its work, produced by group_slots().
struct GroupedWork {
    const uint32_t* grouped_routes;   // route indices (t*K + r) sorted by expert, stable
    const uint32_t* expert_offsets;   // [num_experts + 1] into grouped_routes
    const ExpertPtrs* experts;        // [num_experts]
    uint32_t num_experts;
};

// When a layer call ran, by the device's clock in ns: its first kernel notes when it starts, every block of its last one when it
// ends. Events around the call would do, but stand between its kernels and those of the calls before and after it, which then
// do not start while the kernel ahead still runs: tiny layer of 64 tokens 32.8 us, 25.2 without them. Null: not noted.
struct CallClock {
    unsigned long long begin, end;
};
__device__ __forceinline__ unsigned long long device_clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// What a layer call's first kernel does beside its own work: it notes the time (clock null: not), and zeroes words that a later kernel of the
// call counts in, where that one counts before the launch ahead of it is through.
struct CallStart {
    CallClock* clock;
    uint32_t* clear;
    uint32_t clear_words;
};
__device__ __forceinline__ void begin_call(const CallStart& start) {
    if ((blockIdx.x | blockIdx.y) != 0u) return;
    for (uint32_t w = threadIdx.x; w < start.clear_words; w += blockDim.x) start.clear[w] = 0u;
    if (start.clock == nullptr || threadIdx.x != 0u) return;
    start.clock->begin = device_clock_ns();
    start.clock->end = 0u;
}
__device__ __forceinline__ void note_end(CallClock* clock) {
    if (clock != nullptr && threadIdx.x == 0u) atomicMax(&clock->end, device_clock_ns());
}

__device__ __forceinline__ void raise_status(uint32_t* status, uint32_t bit) {
    if (status) atomicOr(status, bit);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    return nvmoe_f32_to_bf16(lo) | (nvmoe_f32_to_bf16(hi) << 16);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// xor-butterfly sum: every lane ends with the same bits; the order is part of the numeric contract
__device__ __forceinline__ float warp_butterfly_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---- kernels launched by capi.cu (defined in the .cu file named in the comment) ------------

struct RouterLaunch {  // router.cu
    const uint32_t* logits;
    const void* bias;
    uint32_t* routes;
    uint32_t* telemetry;
    uint32_t* status;
    uint32_t tokens;
    nvmoe_geometry g;
};
void configure_router_kernels();
void launch_router(const RouterLaunch& p, cudaStream_t stream);
bool router_is_small(const RouterLaunch& p);  // at most 128 experts, 32 selections, no groups: route_token covers it
void launch_router_linear(const uint16_t* x, const uint16_t* w, const uint16_t* bias, uint32_t* logits,
                          uint32_t tokens, uint32_t hidden, uint32_t outputs, bool beside, const CallStart& start, cudaStream_t stream);  // (beside: see there)

uint32_t device_sm_count();  // of the current device

// router_filter.cu: projection and routing of a large call, of which only the logits that matter are made exactly.
struct RouterFilter {
    const uint16_t* x;
    const uint16_t* w;
    const uint16_t* logit_bias;  // or null
    float* scratch;              // router_filter_floats of them
    uint32_t hidden;
    long long wait_cycles;
    bool withhold;  // (debug) one stage is left out
    CallStart start;
};
void configure_router_filter();
bool router_filter_form(const nvmoe_geometry& g);  // whether it can
bool router_filter_takes(const nvmoe_geometry& g, uint32_t tokens);  // ... and does take the call, if its buffers lie on the 16-byte grid
size_t router_filter_floats(uint32_t max_tokens, uint32_t experts);  // scratch of calls of up to so many tokens
bool launch_router_filter(const RouterLaunch& router, const RouterFilter& f, cudaStream_t stream);  // false: no tensor maps here
void launch_router_refine(const RouterLaunch& router, const RouterFilter& f, cudaStream_t stream);
struct RouterProduct {  // what the refinement reads (diagnostics)
    const float* product;  // [splits][tokens][width]
    const float* x_norm2;  // [splits][tokens]
    const float* w_norm;   // [experts]
    uint32_t splits, width;
    float relative;
};
RouterProduct router_product_of(const RouterFilter& f, uint32_t tokens, uint32_t experts);

struct SortScratch {  // schedule.cu: scratch of the counting sort, sized for max_tokens
    uint32_t* block_hist;      // [blocks][buckets]
    uint32_t* bucket_totals;   // [buckets]
    uint32_t blocks_capacity;
    uint32_t buckets_capacity;
};
// moe_route_compact_batch1 / moe_route_count_batch1
void launch_route_compact(const uint32_t* routes, uint32_t* intermediates, const uint32_t* slots,
                          uint32_t slot_words, uint32_t params_per_resource, uint32_t* control,
                          uint32_t max_tokens, uint32_t K, uint32_t intermediate_size,
                          uint32_t tiles_per_route, uint32_t num_experts, const SortScratch& scratch,
                          cudaStream_t stream);
void launch_route_count(const uint32_t* routes, const uint32_t* slots, uint32_t slot_words,
                        uint32_t params_per_resource, uint32_t* control, uint32_t max_tokens, uint32_t K,
                        uint32_t tiles_per_route, cudaStream_t stream);
// (expert, token tile) list of the tensor-core expert kernels; the list holds routes / 16 + experts + 1 entries: enough for
// any token tile size. list null: none
struct TileOut {
    uint32_t* list;
    uint32_t* count;
    uint32_t n_tile;
};
// Schedule of a whole layer call in one launch, or three for large T*K (layer_schedule_is_fused): control words,
// compact list, owned count, and per expert stage [gate/up, down] the grouped routes, expert offsets
// and (when tiles[stage] is set) the tile list. experts[stage] must already be resolved.
struct LayerSchedule {
    const uint32_t* routes;
    uint32_t* intermediates;
    const uint32_t* slots[2];
    uint32_t slot_words[2];
    uint32_t* control[2];
    const ExpertPtrs* experts[2];
    uint32_t* grouped[2];
    uint32_t* offsets[2];
    uint32_t* position[2];  // optional inverse of grouped: position[stage][route] (0xffffffff if dropped)
    uint32_t* tiles[2];
    uint32_t* tile_count[2];
    uint32_t* status;
    uint32_t tokens, expert_start, expert_count, K, I, tiles_per_route[2], num_experts, n_tile[2];
    uint32_t* clear;       // words that a later kernel of the call counts in, to be zeroed
    uint32_t clear_words;
};
// The down stage's operand rows, of which those of routes that only the down stage keeps are set to zero (q null: none).
struct DownRows {
    const uint32_t* position;  // [route] (null where the places come from elsewhere)
    uint8_t* q;
    ScaleWords scales;
    uint32_t cols;
};
// The gate/up operands of a small call, made ahead of its schedule: a launch that counts the places of its rows itself.
struct OperandRows {
    const uint16_t* input;  // [tokens][cols]
    uint32_t cols, chunks;  // (chunks of 512 columns a row)
    uint8_t* q;
    ScaleWords scales;
    DownRows down;
    bool early;             // the launch ahead has waited for whatever writes the input
};
bool places_operands(const LayerSchedule& s, bool routed, const OperandRows& o, uint32_t block);  // whether a call's are
// (router: the tokens are routed here too, else by a launch ahead)
void launch_place_operands(const RouterLaunch* router, const LayerSchedule& s, const OperandRows& o, uint32_t block, cudaStream_t stream);
// ... and, right behind it, what the later kernels of the call read of its schedule: offsets, grouped routes, positions and tiles of both
// stages, but neither the compact list nor the control words. (tiles, position and so on are all set)
void launch_small_schedule(const RouterLaunch* router, const LayerSchedule& s, cudaStream_t stream);
bool layer_schedule_is_fused(uint32_t tokens, uint32_t K, uint32_t num_experts, bool partitioned);
// the router and the schedule of a call of up to 16 tokens (32 of up to 32 experts) in one launch
bool layer_routes_in_schedule(const RouterLaunch& router, uint32_t K, uint32_t num_experts);
void launch_route_schedule(const RouterLaunch& router, const LayerSchedule& s, cudaStream_t stream);
uint32_t launch_layer_schedule(const LayerSchedule& s, const SortScratch& scratch, cudaStream_t stream);  // returns its launches
// validates the address/slot tables of every expert once per call
// (rows, cols: logical shape of one matrix; experts from native_start on hold native FP8; with
// whole_blocks_only an FP8-form matrix whose columns are not whole 128-blocks is treated as not resident:
// the tensor path stages such a tail for the compact form only)
void launch_resolve_experts(const uint32_t* addresses, uint32_t address_words, const uint32_t* slots,
                            uint32_t slot_words, uint32_t params_per_resource, uint32_t num_experts,
                            uint32_t rows, uint32_t cols, uint32_t native_start, bool whole_blocks_only,
                            uint8_t* derived_scales, size_t derived_matrix_bytes, ExpertPtrs* out, cudaStream_t stream);
// groups the compact slots the expert shaders would visit by expert (stable), skipping what the
// shaders skip; writes grouped_routes and expert_offsets and, if `position` is given, the inverse
// position[route] = place in grouped_routes (0xffffffff for routes that were skipped) and the tile list; returns its launches
uint32_t launch_group_slots(const uint32_t* routes, const uint32_t* intermediates, const uint32_t* control,
                        const ExpertPtrs* experts, uint32_t num_experts, uint32_t max_tokens, uint32_t K,
                        uint32_t intermediate_size, uint32_t* grouped_routes, uint32_t* expert_offsets,
                        uint32_t* position, const TileOut& tiles, uint32_t* status, const SortScratch& scratch,
                        cudaStream_t stream);

// expert-parallel dispatch (schedule.cu): routes grouped by the rank owning their expert, stable
// in source order; send_index[i] = position of source route i (kUnboundSlot if dropped),
// send_source[pos] = source route; hidden rows are gathered into send_rows in that order
void launch_ep_pack(const uint16_t* hidden, const uint32_t* routes, const uint32_t* owner, uint32_t tokens,
                    uint32_t K, uint32_t hidden_size, uint32_t num_experts, uint32_t world, uint32_t self,
                    uint16_t* send_rows, uint32_t* send_routes, uint32_t* send_index, uint32_t* send_source,
                    uint32_t* dest_counts, uint32_t* total, uint32_t segment_rows, uint32_t* contiguous_routes,
                    uint32_t* status, const SortScratch& scratch, cudaStream_t stream);
void launch_ep_unpack(const uint16_t* returned_rows, const uint32_t* send_index, uint32_t tokens, uint32_t K,
                      uint32_t hidden_size, uint16_t* expert_outputs, cudaStream_t stream);

// quantize.cu: bf16 rows -> E4M3 bytes + per-block power-of-two scales.
// scales_f32 is [rows][cols/block].
void launch_quantize(const uint16_t* input, uint32_t rows, uint32_t cols, uint32_t block,
                     size_t input_row_stride, uint8_t* q, float* scales_f32, cudaStream_t stream);
// The tensor path's operand form: row `pos` of the output is the quantised source row of route
// grouped_routes[pos] (the token's hidden row when frames is false: source row = route / K of
// `input` with `cols` columns; the route's own row of the intermediates frames otherwise), for pos below
// expert_offsets[num_experts]. Scales as E8M0 words only. Expert-grouped rows are what a tiled TMA
// load can fetch as one box per (expert, token tile). `written` (optional, [route]): a route marked 0xffffffff there has
// no frame of this call and gives a row of zeros.
void launch_quantize_grouped(const void* input, bool frames, const uint32_t* grouped_routes,
                             const uint32_t* expert_offsets, uint32_t num_experts, uint32_t max_routes, uint32_t K,
                             uint32_t cols, uint32_t intermediate_size, uint32_t block, uint8_t* q,
                             const ScaleWords& scales, const uint32_t* written, cudaStream_t stream);
// The same gate/up operands from the inverse list: position[token * K + r] = row of that route (0xffffffff: skipped),
// valid for every route of the call; `down` (position null: nothing). False when the shape needs the form above (blocks other than
// 32 or 128 columns, input not 16-byte aligned).
bool launch_quantize_tokens(const void* input, const uint32_t* position, uint32_t tokens, uint32_t K, uint32_t cols, uint32_t block,
                            uint8_t* q, const ScaleWords& scales, const DownRows& down, cudaStream_t stream);
// the same for the K rows of every intermediates frame (skips the schedule words)
void launch_quantize_frames(const uint32_t* intermediates, uint32_t tokens, uint32_t K,
                            uint32_t intermediate_size, uint32_t block, uint8_t* q, float* scales_f32,
                            const uint32_t* written, cudaStream_t stream);
struct ExpertLaunch {  // experts_simt.cu and experts_tc.cu
    GroupedWork work;
    const uint8_t* act_q;        // [rows][K_dim] E4M3; row = token (gate/up) or route index (down)
    const float* act_scales;     // [rows][K_dim/act_block] f32
    ScaleWords act_e8m0;         // packed E8M0 (tensor path)
    const uint32_t* routes;      // route words (down: weights)
    uint32_t* intermediates;     // gate/up output frames (tensor path with q_out: may be null)
    uint16_t* outputs;           // down output [T][K][H]
    float* partial_outputs;      // down, tensor-parallel form: raw f32 sums [T][K][H] instead of `outputs` (no route weight, no rounding)
    uint32_t* status;
    const uint8_t* tmaps;        // tensor path: tensor maps [expert][matrix][kWeightMaps][128 bytes], then that of the derived scales;
                                 // null = move weights with cp.async
    // tensor path: act_q / act_e8m0 hold expert-grouped rows (row = position in grouped_routes);
    // act_tmap is the tensor map of act_q with a box of [token tile][128 bytes] (null: fetch rows with cp.async); for CTA
    // pairs the first of those of half tiles
    const uint8_t* act_tmap;
    // tensor path, gate/up only: where the down stage's grouping puts each route (its operand row)
    const uint32_t* down_position;
    // tensor path, gate/up only, optional: the down stage's activation quantisation done in the epilogue
    // (E4M3 bytes [down_position][I] and their scales); needs act_block 32 or 128
    uint8_t* q_out;
    ScaleWords q_e8m0;
    uint32_t token_rows;         // tensor path: rows of the operand matrix per token tile of the list
    bool pairs;                  // tensor path: by CTA pairs
    uint8_t* scale_base;         // tensor path: the derived scale copy of the whole expert set (null: no map of it is needed)
    uint64_t* cta_trace;         // tensor path diagnostics: [2][grid][4] words per CTA, or null
    uint64_t* scale_stamps;      // tensor path: {scale pointer, generation} the derived tiles were built from
    uint32_t* tile_list;         // tensor path scratch: routes / 16 + experts + 1 words
    uint32_t tile_capacity;      // ... of which so many may be read
    bool fresh_maps;             // tensor path: the launch right before this one wrote the tensor maps
    const void* dense_maps;      // CTA pairs, down, one matrix: its tensor maps on the host (boxes of one K block and of two), rows in order
    uint32_t* tile_count;        // tensor path scratch: one word
    uint32_t tokens;             // upper bound (max over what control may hold)
    long long wait_cycles;       // tensor path: clock cycles after which a bounded in-kernel wait gives up
    uint32_t debug_flags;        // tensor path: bit n = CTA n (0 or 1) leaves out its first stage arrival (exercises the give-up path); bit 2: RouterFilter.withhold; from bit 8 on always zero
    nvmoe_geometry g;
};
void configure_simt_kernels();
void launch_gate_up_simt(const ExpertLaunch& p, cudaStream_t stream);
void launch_down_simt(const ExpertLaunch& p, cudaStream_t stream);

// ffn_tail.cu: the nodes either side of the MoE chain and the token-id table routing
void launch_rms_norm(const uint16_t* input, const uint16_t* weight, uint16_t* output, uint32_t rows, uint32_t hidden, float eps,
                     float weight_offset, cudaStream_t stream);
void launch_silu_multiply(const uint16_t* gate, const uint16_t* up, uint16_t* out, size_t elements, float limit, cudaStream_t stream);
void launch_add_bf16(const uint16_t* a, const uint16_t* b, uint16_t* out, size_t elements, cudaStream_t stream);
void launch_preselect_table(const uint32_t* token_ids, const uint32_t* table, uint32_t word_stride, uint32_t vocab, uint32_t routed,
                            uint32_t k, uint32_t always, uint32_t tokens, uint32_t* selections, uint32_t* telemetry, uint32_t* status,
                            cudaStream_t stream);
void launch_route_preselected(const uint32_t* logits, const uint32_t* selections, uint32_t tokens, uint32_t* routes, uint32_t* status,
                              const nvmoe_geometry& g, cudaStream_t stream);
// reduce.cu: the same combine with route (t, r) read from row gather[t * K + r] of `rows` (all-ones = a row of
// zeros); false when the shape needs the plain form (hidden not a multiple of 8, unaligned buffers)
bool launch_reduce_gather(const uint16_t* rows, const uint32_t* gather, uint16_t* output, uint32_t tokens, uint32_t K,
                          uint32_t hidden, float routed_scale, cudaStream_t stream);
// reduce.cu: distributed_sum_f32_scale_packed_bf16_to_bf16: out[lane][e] = bf16(sum over participants of
// partials[participant][lane][e] * bf16(scales[lane * (elements / elements_per_scale) + e / elements_per_scale] >> bit_offset))
void launch_sum_f32_scale_packed_bf16(const float* partials, const uint32_t* scales, uint32_t* output, uint32_t element_count,
                                      uint32_t participant_count, uint32_t lane_count, uint32_t elements_per_scale,
                                      uint32_t scale_bit_offset, cudaStream_t stream);

// ffn_tail.cu: most (zeroed) receives by how many units the fast SiLU differs from the pinned one, of which it allows silu_units_bound
void launch_silu_units(uint32_t* most, cudaStream_t stream);
uint32_t silu_units_bound();

// probe.cu: a run of `groups` x 8 block-scaled MMAs (128 x n_tile x 32, two alternating accumulators)
// on every one of `ctas` CTAs; cycles[cta] = clock cycles from first issue to completion
cudaError_t launch_mma_rate_probe(uint32_t n_tile, uint32_t groups, uint32_t ctas, long long* cycles, uint32_t* status,
                                  cudaStream_t stream);

// reduce.cu: `bytes` (a multiple of 16, both addresses 16-byte aligned) from page-locked host memory, at its device address
void launch_fetch_host(const void* host, void* device, size_t bytes, cudaStream_t stream);
// reduce.cu: moe_reduce_batch1_bf16. `computed` (optional, [tokens * K]) marks with 0xffffffff the routes
// whose rows were never written: they count as zeros, so the rows need no clearing beforehand.
void launch_reduce(const uint16_t* expert_outputs, uint16_t* output, uint32_t tokens, uint32_t K,
                   uint32_t hidden, float routed_scale, const uint32_t* computed, CallClock* clock, cudaStream_t stream);

}  // namespace nvmoe
