// Route scheduling: the reference's compact/count stages and the expert grouping the grouped
// expert kernels consume.
//
//   route_compact   runtime-rs/shaders/moe_route_compact_batch1.comp.template:26-105
//   route_count     runtime-rs/shaders/moe_route_count_batch1.comp.template:21-58
//
// The reference ranks every (token, route) against every other one — quadratic in T*K.  The
// rank it computes, #{c : expert(c) < expert(s) or (expert(c) == expert(s) and c < s)}, is the
// position of s in a STABLE sort by expert id, so the same list comes out of a counting sort:
// per-block histograms, an exclusive scan over (expert, block), and a scatter in which equal
// experts keep source order (warp match + popcount of lower lanes, warps taken in order).
// Route ids at or above the expert count cannot be produced by the routers here; they are placed
// after every valid id in source order (the reference would order them by id).
#include "quantize.cuh"
#include "router_reg.cuh"

namespace nvmoe {
namespace {

// ---- generic stable counting sort over `count` keys ------------------------------------------
// KeyFn(i) -> bucket in [0, buckets) or kUnboundSlot to drop item i.  EmitFn(rank, i) stores it.

template <class KeyFn>
__device__ void block_histogram(uint32_t begin, uint32_t end, uint32_t buckets, uint32_t* hist, KeyFn key) {
    for (uint32_t b = threadIdx.x; b < buckets; b += blockDim.x) hist[b] = 0u;
    __syncthreads();
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        uint32_t kb = key(i);
        if (kb != kUnboundSlot) atomicAdd(hist + kb, 1u);
    }
    __syncthreads();
}

// Stable scatter of items [begin, end) given running[b] = rank of the next item of bucket b.
// blockDim.x must be a multiple of 32; warps take turns so that source order is kept.
template <class KeyFn, class EmitFn>
__device__ void block_stable_scatter(uint32_t begin, uint32_t end, uint32_t* running, KeyFn key, EmitFn emit) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint32_t base = begin; base < end; base += blockDim.x) {
        uint32_t i = base + threadIdx.x;
        uint32_t kb = i < end ? key(i) : kUnboundSlot;
        for (uint32_t w = 0; w < warps; w++) {
            if (w == warp) {
                uint32_t peers = __match_any_sync(0xffffffffu, kb);
                if (kb != kUnboundSlot) {
                    uint32_t before = __popc(peers & ((1u << lane) - 1u));
                    uint32_t leader = __ffs(peers) - 1u;
                    uint32_t start = 0u;
                    if (lane == leader) {
                        start = running[kb];
                        running[kb] = start + __popc(peers);
                    }
                    start = __shfl_sync(peers, start, leader);
                    emit(start + before, i);
                }
            }
            __syncthreads();
        }
    }
}

// One block does the whole sort (small inputs: one launch instead of three).
template <class KeyFn, class EmitFn, class DoneFn>
__device__ void sort_single_block(uint32_t count, uint32_t buckets, uint32_t* smem_hist, KeyFn key,
                                  EmitFn emit, DoneFn done) {
    block_histogram(0u, count, buckets, smem_hist, key);
    // exclusive scan over buckets by one warp (buckets <= 4097)
    if (threadIdx.x < 32u) {
        uint32_t carry = 0u;
        for (uint32_t b0 = 0; b0 < buckets; b0 += 32u) {
            uint32_t b = b0 + threadIdx.x;
            uint32_t v = b < buckets ? smem_hist[b] : 0u;
            uint32_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += n;
            }
            if (b < buckets) smem_hist[b] = carry + incl - v;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0u) smem_hist[buckets] = carry;
    }
    __syncthreads();
    done(smem_hist);  // bucket bases (exclusive) with the total at [buckets]
    __syncthreads();
    block_stable_scatter(0u, count, smem_hist, key, emit);
}

// out[b] <- sum of value(0 .. b-1) for b <= buckets, by one warp
template <class ValueFn>
__device__ __forceinline__ void warp_exclusive_scan(uint32_t buckets, uint32_t* out, ValueFn value) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t carry = 0u;
    for (uint32_t b0 = 0; b0 < buckets; b0 += 32u) {
        const uint32_t b = b0 + lane;
        const uint32_t v = b < buckets ? value(b) : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += n;
        }
        if (b < buckets) out[b] = carry + incl - v;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0u) out[buckets] = carry;
}

// The same sort of at most an item a thread: every key is found once, a warp ranks its items by match_any and leaves its counts per
// bucket in a table [warp][bucket], columns of which are summed; where a warp's turn would come after those of all warps before it,
// everything is done side by side. Bound by the latency of the keys' dependent loads and four block barriers. `done` gets the bucket
// bases (total at [buckets]) and the same of tiles of n_tile items. Node chains, us, by turns / this way: 45 tokens of 32 experts 147.2 / 143.1, 16
// of 128 191.6 / 187.6, 90 of 128 342.8 / 327.8.
__host__ __device__ inline size_t rank_block_words(uint32_t threads, uint32_t buckets) {
    return (size_t)buckets + 2u * (buckets + 1u) + ((size_t)threads / 32u * buckets + 1u) / 2u;
}
// Shared memory that a launch may ask for beside the static arrays of the one-block kernels (144 bytes, the tile list's): together 48 KB.
constexpr size_t kOneBlockBytes = 48u * 1024u - 256u;
__host__ __device__ inline bool rank_block_fits(uint32_t threads, uint32_t buckets) { return rank_block_words(threads, buckets) * 4u <= kOneBlockBytes; }
template <class KeyFn, class EmitFn, class DoneFn>
__device__ void rank_single_block(uint32_t count, uint32_t buckets, uint32_t* words, uint32_t n_tile, KeyFn key, EmitFn emit, DoneFn done) {
    uint32_t* total = words;
    uint32_t* base = total + buckets;
    uint32_t* tile_base = base + buckets + 1u;
    uint16_t* table = reinterpret_cast<uint16_t*>(tile_base + buckets + 1u);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, rows = (count + 31u) / 32u, i = threadIdx.x;
    for (uint32_t w = threadIdx.x; w < (rows * buckets + 1u) / 2u; w += blockDim.x) reinterpret_cast<uint32_t*>(table)[w] = 0u;
    const uint32_t kb = i < count ? key(i) : kUnboundSlot;
    __syncthreads();
    const uint32_t peers = __match_any_sync(0xffffffffu, kb), before = __popc(peers & ((1u << lane) - 1u));
    if (kb != kUnboundSlot && before == 0u) table[warp * buckets + kb] = (uint16_t)__popc(peers);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < buckets; b += blockDim.x) {
        uint32_t running = 0u;
        for (uint32_t r = 0; r < rows; r++) {
            const uint32_t here = table[r * buckets + b];
            table[r * buckets + b] = (uint16_t)running;
            running += here;
        }
        total[b] = running;
    }
    __syncthreads();
    if (warp == 0u) warp_exclusive_scan(buckets, base, [&](uint32_t b) { return total[b]; });
    if (warp == 1u) warp_exclusive_scan(buckets, tile_base, [&](uint32_t b) { return (total[b] + n_tile - 1u) / n_tile; });
    __syncthreads();
    done(base, tile_base);
    if (kb != kUnboundSlot) emit(base[kb] + table[warp * buckets + kb] + before, i);
}

// ---- keys ----------------------------------------------------------------------------------

struct RouteKey {  // compact: rank all T*K routes by expert id
    const uint32_t* routes;
    uint32_t num_experts;
    __device__ uint32_t operator()(uint32_t i) const {
        uint32_t e = routes[i] & 0xffffu;
        return e < num_experts ? e : num_experts;
    }
};

__device__ __forceinline__ bool resource_is_local(const uint32_t* slots, uint32_t slot_words,
                                                  uint32_t params, uint32_t expert) {
    if (!slots) return true;
    uint64_t index = (uint64_t)expert * params;
    if (index >= slot_words) return false;
    return slots[index] != kUnboundSlot;
}

struct OwnedKey {  // partitioned compact: keep owned routes, in source order (one bucket)
    const uint32_t* routes;
    const uint32_t* slots;
    uint32_t slot_words, params, start, end;
    __device__ uint32_t operator()(uint32_t i) const {
        uint32_t e = routes[i] & 0xffffu;
        if (e < start || e >= end || !resource_is_local(slots, slot_words, params, e)) return kUnboundSlot;
        return 0u;
    }
};

struct ScheduleEmit {  // writes the compact list into the schedule words of the frames
    uint32_t* intermediates;
    uint32_t K, frame_words, data_words;
    uint32_t* copy = nullptr;  // optional second, flat copy of the list
    __device__ void operator()(uint32_t rank, uint32_t i) const {
        intermediates[(size_t)(rank / K) * frame_words + data_words + rank % K] = i;
        if (copy) copy[rank] = i;
    }
};

// the slot the expert shaders read for compact position c, or kUnboundSlot when they return early
struct SlotKey {
    const uint32_t* routes;
    const uint32_t* intermediates;
    const ExpertPtrs* experts;
    uint32_t* status;
    uint32_t num_experts, K, frame_words, data_words, capacity;
    const uint8_t* resident = nullptr;  // optional per-expert copy of "experts[e].w[0] != nullptr" (a faster place)
    __device__ uint32_t route_index(uint32_t c) const {
        return intermediates[(size_t)(c / K) * frame_words + data_words + c % K];
    }
    __device__ uint32_t operator()(uint32_t c) const {
        uint32_t ri = route_index(c);
        if (ri >= capacity) {
            raise_status(status, NVMOE_STATUS_ROUTE_OUT_OF_RANGE);
            return kUnboundSlot;
        }
        uint32_t e = routes[ri] & 0xffffu;
        if (e >= num_experts) {
            raise_status(status, NVMOE_STATUS_ROUTE_OUT_OF_RANGE);
            return kUnboundSlot;
        }
        if (resident ? resident[e] == 0u : experts[e].w[0] == nullptr) {
            raise_status(status, NVMOE_STATUS_EXPERT_NOT_RESIDENT);
            return kUnboundSlot;
        }
        return e;
    }
};

struct GroupEmit {
    const SlotKey key;
    uint32_t* grouped;
    uint32_t* position;  // optional inverse: position[route] = its place in `grouped`
    __device__ void operator()(uint32_t rank, uint32_t c) const {
        const uint32_t ri = key.route_index(c);
        grouped[rank] = ri;
        if (position) position[ri] = rank;
    }
};

// ---- kernels ---------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t min_u32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// Single-block compact (T*K small).  `control` is read for batch_width / expert range and the
// owned count and indirect-dispatch words are written back exactly as the shader does.
__device__ void compact_small_body(const uint32_t* routes, uint32_t* intermediates, const uint32_t* slots,
                                   uint32_t slot_words, uint32_t params, uint32_t* control, uint32_t max_tokens,
                                   uint32_t K, uint32_t I, uint32_t tiles_per_route, uint32_t num_experts,
                                   uint32_t* hist, uint32_t* list_copy = nullptr) {
    const uint32_t T = min_u32(control[0], max_tokens);
    const uint32_t count = T * K;
    const uint32_t data_words = K * (I / 2u);
    ScheduleEmit emit{intermediates, K, data_words + K, data_words, list_copy};
    if (control[2] != 0u) {
        OwnedKey key{routes, slots, slot_words, params, control[1], control[1] + control[2]};
        sort_single_block(count, 1u, hist, key, emit, [&](const uint32_t* base) {
            if (threadIdx.x == 0u) {
                control[3] = base[1];
                control[4] = base[1] * tiles_per_route;
                control[5] = 1u;
                control[6] = 1u;
            }
        });
    } else {
        RouteKey key{routes, num_experts};
        sort_single_block(count, num_experts + 1u, hist, key, emit, [&](const uint32_t*) {
            if (threadIdx.x == 0u) {
                control[3] = count;
                control[4] = K * tiles_per_route;
                control[5] = T;
                control[6] = 1u;
            }
        });
    }
}

// The same by rank_single_block, for at most a route a thread.
__device__ void compact_rank_body(const uint32_t* routes, uint32_t* intermediates, const uint32_t* slots, uint32_t slot_words, uint32_t params,
                                  uint32_t* control, uint32_t T, uint32_t K, uint32_t I, uint32_t tiles_per_route, uint32_t num_experts,
                                  uint32_t* words) {
    const uint32_t count = T * K, data_words = K * (I / 2u), start = control[1], owned = control[2];
    ScheduleEmit emit{intermediates, K, data_words + K, data_words, nullptr};
    auto done = [&](const uint32_t* base, const uint32_t*) {
        if (threadIdx.x != 0u) return;
        const uint32_t listed = owned != 0u ? base[1] : count;
        control[3] = listed;
        control[4] = (owned != 0u ? listed : K) * tiles_per_route;
        control[5] = owned != 0u ? 1u : T;
        control[6] = 1u;
    };
    if (owned != 0u) {
        rank_single_block(count, 1u, words, 1u, OwnedKey{routes, slots, slot_words, params, start, start + owned}, emit, done);
    } else {
        rank_single_block(count, num_experts + 1u, words, 1u, RouteKey{routes, num_experts}, emit, done);
    }
}

__global__ void __launch_bounds__(1024) compact_small_kernel(const uint32_t* routes, uint32_t* intermediates,
                                                            const uint32_t* slots, uint32_t slot_words,
                                                            uint32_t params, uint32_t* control,
                                                            uint32_t max_tokens, uint32_t K, uint32_t I,
                                                            uint32_t tiles_per_route, uint32_t num_experts) {
    extern __shared__ uint32_t hist[];
    grid_dependency_sync();
    const uint32_t T = min_u32(control[0], max_tokens);
    if (rank_block_fits(blockDim.x, num_experts + 1u) && T * K <= blockDim.x) {
        compact_rank_body(routes, intermediates, slots, slot_words, params, control, T, K, I, tiles_per_route, num_experts, hist);
        return;
    }
    compact_small_body(routes, intermediates, slots, slot_words, params, control, max_tokens, K, I, tiles_per_route,
                       num_experts, hist);
}

// Multi-block sort, phase 1: per-block histograms.
template <class KeyFn>
__device__ void phase_hist(uint32_t count, uint32_t buckets, uint32_t* block_hist, KeyFn key) {
    extern __shared__ uint32_t hist[];
    uint32_t begin = blockIdx.x * kSortChunk;
    if (begin >= count) {
        for (uint32_t b = threadIdx.x; b < buckets; b += blockDim.x) block_hist[(size_t)blockIdx.x * buckets + b] = 0u;
        return;
    }
    uint32_t end = min_u32(begin + kSortChunk, count);
    block_histogram(begin, end, buckets, hist, key);
    for (uint32_t b = threadIdx.x; b < buckets; b += blockDim.x) block_hist[(size_t)blockIdx.x * buckets + b] = hist[b];
}

// phase 2: block_hist[blk][b] <- rank, within bucket b, of the first item of block blk; totals[b] <- items of bucket b.
// A block of 32 warps owns 32 buckets: a lane is a bucket (a warp reads 128 neighbouring bytes of a row of counts), a
// warp is a run of rows, which it sums, and writes back once it knows what the runs before it hold. Bound by the latency
// of the few dependent loads. One block for all buckets with a warp walking each column read every count from a sector
// of its own: 576 x 257 counts took 120 us.
__global__ void __launch_bounds__(1024) phase_scan_kernel(uint32_t* block_hist, uint32_t* totals, uint32_t blocks, uint32_t buckets) {
    __shared__ uint32_t part[32][32];
    grid_dependency_sync();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b = blockIdx.x * 32u + lane;
    const uint32_t per = (blocks + 31u) / 32u;
    const uint32_t begin = min_u32(warp * per, blocks), end = min_u32(begin + per, blocks);
    uint32_t sum = 0u;
    if (b < buckets) {
#pragma unroll 8
        for (uint32_t r = begin; r < end; r++) sum += block_hist[(size_t)r * buckets + b];
    }
    part[warp][lane] = sum;
    __syncthreads();
    uint32_t running = 0u;
    for (uint32_t w = 0; w < warp; w++) running += part[w][lane];
    if (b >= buckets) return;
    if (warp == 31u) totals[b] = running + sum;
#pragma unroll 8
    for (uint32_t r = begin; r < end; r++) {
        const uint32_t here = block_hist[(size_t)r * buckets + b];
        block_hist[(size_t)r * buckets + b] = running;
        running += here;
    }
}

// phase 3: every block scans the bucket totals itself (`bases`, if given, receives the scan, total at [buckets]) and
// places its items. Needs buckets + 1 words of dynamic shared memory.
template <class KeyFn, class EmitFn>
__device__ void phase_scatter(uint32_t count, uint32_t buckets, const uint32_t* block_hist, const uint32_t* totals,
                              KeyFn key, EmitFn emit, uint32_t* bases = nullptr) {
    extern __shared__ uint32_t running[];
    if (threadIdx.x < 32u) warp_exclusive_scan(buckets, running, [&](uint32_t b) { return totals[b]; });
    __syncthreads();
    if (bases && blockIdx.x == 0u)
        for (uint32_t b = threadIdx.x; b <= buckets; b += blockDim.x) bases[b] = running[b];
    uint32_t begin = blockIdx.x * kSortChunk;
    if (begin >= count) return;
    uint32_t end = min_u32(begin + kSortChunk, count);
    if (bases) __syncthreads();
    for (uint32_t b = threadIdx.x; b < buckets; b += blockDim.x) running[b] += block_hist[(size_t)blockIdx.x * buckets + b];
    __syncthreads();
    block_stable_scatter(begin, end, running, key, emit);
}

__global__ void __launch_bounds__(256) compact_hist_kernel(const uint32_t* routes, const uint32_t* slots,
                                                          uint32_t slot_words, uint32_t params,
                                                          const uint32_t* control, uint32_t max_tokens,
                                                          uint32_t K, uint32_t num_experts, uint32_t* block_hist) {
    const uint32_t count = min_u32(control[0], max_tokens) * K;
    if (control[2] != 0u) {
        OwnedKey key{routes, slots, slot_words, params, control[1], control[1] + control[2]};
        phase_hist(count, num_experts + 1u, block_hist, key);  // one bucket used, same stride
    } else {
        RouteKey key{routes, num_experts};
        phase_hist(count, num_experts + 1u, block_hist, key);
    }
}

__global__ void __launch_bounds__(256) compact_scatter_kernel(const uint32_t* routes, uint32_t* intermediates,
                                                             const uint32_t* slots, uint32_t slot_words,
                                                             uint32_t params, uint32_t* control,
                                                             uint32_t max_tokens, uint32_t K, uint32_t I,
                                                             uint32_t tiles_per_route, uint32_t num_experts,
                                                             const uint32_t* block_hist, const uint32_t* totals) {
    const uint32_t T = min_u32(control[0], max_tokens);
    const uint32_t count = T * K;
    const uint32_t data_words = K * (I / 2u);
    ScheduleEmit emit{intermediates, K, data_words + K, data_words};
    const bool partitioned = control[2] != 0u;
    // every block has read what it needs from control[0..2]; block 0 publishes the command words
    if (partitioned) {
        OwnedKey key{routes, slots, slot_words, params, control[1], control[1] + control[2]};
        phase_scatter(count, num_experts + 1u, block_hist, totals, key, emit);
        if (blockIdx.x == 0u && threadIdx.x == 0u) {
            uint32_t owned = totals[0];
            control[3] = owned;
            control[4] = owned * tiles_per_route;
            control[5] = 1u;
            control[6] = 1u;
        }
    } else {
        RouteKey key{routes, num_experts};
        phase_scatter(count, num_experts + 1u, block_hist, totals, key, emit);
        if (blockIdx.x == 0u && threadIdx.x == 0u) {
            control[3] = count;
            control[4] = K * tiles_per_route;
            control[5] = T;
            control[6] = 1u;
        }
    }
}

// moe_route_count: the owned count only (one block; a grid-stride count is plenty here)
// (every thread of the block calls it; the branch is uniform)
__device__ void route_count_body(const uint32_t* routes, const uint32_t* slots, uint32_t slot_words, uint32_t params,
                                 uint32_t* control, uint32_t max_tokens, uint32_t K, uint32_t tiles_per_route) {
    __shared__ uint32_t owned;
    const uint32_t T = min_u32(control[0], max_tokens);
    const uint32_t start = control[1], owned_experts = control[2];
    __syncthreads();  // every thread has read the control words before one of them rewrites the tail
    if (owned_experts == 0u) {
        if (threadIdx.x == 0u) {
            control[3] = T * K;
            control[4] = K * tiles_per_route;
            control[5] = T;
            control[6] = 1u;
        }
        return;
    }
    if (threadIdx.x == 0u) owned = 0u;
    __syncthreads();
    const uint32_t end = start + owned_experts;
    uint32_t mine = 0u;
    for (uint32_t i = threadIdx.x; i < T * K; i += blockDim.x) {
        uint32_t e = routes[i] & 0xffffu;
        if (e >= start && e < end && resource_is_local(slots, slot_words, params, e)) mine++;
    }
    atomicAdd(&owned, mine);
    __syncthreads();
    if (threadIdx.x == 0u) {
        control[3] = owned;
        control[4] = owned * tiles_per_route;
        control[5] = 1u;
        control[6] = 1u;
    }
}

__global__ void __launch_bounds__(1024) route_count_kernel(const uint32_t* routes, const uint32_t* slots,
                                                          uint32_t slot_words, uint32_t params, uint32_t* control,
                                                          uint32_t max_tokens, uint32_t K, uint32_t tiles_per_route) {
    grid_dependency_sync();
    route_count_body(routes, slots, slot_words, params, control, max_tokens, K, tiles_per_route);
}

// address_record_is_resident + dynamic_parameter_record_is_valid for every expert, once per call
// (dynamic_expert_is_valid of independent_sparse_moe_gate_up_batch1_mxfp4.comp.template:166-228: a weight record's
// representation word is 0 (compact) or 1 (pre-expanded FP8), the same for both matrices of a pair; resources
// from native_start on are native FP8 and must say 0)
__global__ void resolve_experts_kernel(const uint32_t* addresses, uint32_t address_words, const uint32_t* slots,
                                       uint32_t slot_words, uint32_t params, uint32_t num_experts,
                                       uint32_t rows, uint32_t cols, uint32_t native_start, bool whole_blocks_only,
                                       uint8_t* derived_scales, size_t derived_matrix_bytes, ExpertPtrs* out) {
    uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num_experts) return;
    ExpertPtrs r{{nullptr, nullptr}, {nullptr, nullptr}, {nullptr, nullptr}, {0u, 0u}, kFormatCompact, 0u};
    bool ok = true;
    const uint8_t* ptrs[4] = {nullptr, nullptr, nullptr, nullptr};
    uint64_t gens[4] = {0u, 0u, 0u, 0u};
    const bool native = e >= native_start;
    // the form of the expert's matrices: the representation word of its first weight record
    uint32_t format = native ? kFormatNativeFp8 : kFormatCompact;
    if (!native && (uint64_t)e * params < slot_words) {
        const uint32_t slot = slots[(uint64_t)e * params];
        if (slot != kUnboundSlot && slot < address_words / kRecordWords && addresses[(size_t)slot * kRecordWords + 7u] == 1u)
            format = kFormatExpanded;
    }
    if (format != kFormatCompact && whole_blocks_only && cols % 128u != 0u) ok = false;
    const uint64_t weight_bytes = format == kFormatCompact ? (uint64_t)rows * (cols / 2u) : (uint64_t)rows * cols;
    const uint64_t scale_bytes = format == kFormatNativeFp8 ? (uint64_t)((rows + 127u) / 128u) * ((cols + 127u) / 128u)
                                                            : (uint64_t)rows * (cols / 32u);
    for (uint32_t j = 0; j < params && ok; j++) {
        uint64_t index = (uint64_t)e * params + j;
        if (index >= slot_words) {
            ok = false;
            break;
        }
        uint32_t slot = slots[index];
        if (slot == kUnboundSlot || slot >= address_words / kRecordWords) {
            ok = false;
            break;
        }
        const uint32_t* rec = addresses + (size_t)slot * kRecordWords;
        uint64_t address = (uint64_t)rec[0] | ((uint64_t)rec[1] << 32);
        uint64_t bytes = (uint64_t)rec[2] | ((uint64_t)rec[3] << 32);
        uint64_t required = (j & 1u) ? scale_bytes : weight_bytes;
        // what the record must say about its form: weights of a compact or native resource 0, of a pre-expanded one 1
        // (a pair that disagrees fails closed); scale records are not looked at, as in the shader
        const uint32_t expected = format == kFormatExpanded ? 1u : 0u;
        // the kernels read rows with 16-byte loads and TMA boxes, so the shader's 4-byte address rule becomes 32
        // (native FP8 scale blocks are read byte by byte: 4 as in the shader)
        const uint64_t align_mask = ((j & 1u) && format == kFormatNativeFp8) ? 3u : 31u;
        if (address == 0u || (address & align_mask) != 0u || bytes < required || (rec[4] | rec[5]) == 0u ||
            rec[6] != 1u || (!(j & 1u) && rec[7] != expected)) {
            ok = false;
            break;
        }
        ptrs[j] = reinterpret_cast<const uint8_t*>(address);
        gens[j] = (uint64_t)rec[4] | ((uint64_t)rec[5] << 32);
    }
    if (ok) {
        const uint32_t matrices = params / 2u;
        r.w[0] = ptrs[0];
        r.s[0] = ptrs[1];
        r.gen[0] = gens[1];
        r.w[1] = params == 4u ? ptrs[2] : nullptr;
        r.s[1] = params == 4u ? ptrs[3] : nullptr;
        r.gen[1] = params == 4u ? gens[3] : 0u;
        r.format = format;
        if (derived_scales) {
            r.ts[0] = derived_scales + ((size_t)e * matrices) * derived_matrix_bytes;
            // gate and up blocks of the same (row tile, K block) lie side by side, 512 bytes each: one copy brings both
            r.ts[1] = params == 4u ? r.ts[0] + 512u : nullptr;
        }
    }
    out[e] = r;
}

__device__ __forceinline__ uint32_t slot_count(const uint32_t* control, uint32_t max_tokens, uint32_t K) {
    const uint32_t T = min_u32(control[0], max_tokens);
    // route-native calls visit owned_route_count slots, the others every (batch, route) position
    return control[2] != 0u ? min_u32(control[3], T * K) : T * K;
}

__device__ void group_small_body(SlotKey key, const uint32_t* control, uint32_t max_tokens, uint32_t* grouped,
                                 uint32_t* expert_offsets, uint32_t* position, uint32_t* hist) {
    const uint32_t T = min_u32(control[0], max_tokens);
    key.capacity = T * key.K;
    const uint32_t count = slot_count(control, max_tokens, key.K);
    if (position) {  // routes the grouping drops keep "nowhere"
        for (uint32_t i = threadIdx.x; i < key.capacity; i += blockDim.x) position[i] = kUnboundSlot;
        __syncthreads();
    }
    GroupEmit emit{key, grouped, position};
    const uint32_t buckets = key.num_experts;
    sort_single_block(count, buckets, hist, key, emit, [&](const uint32_t* base) {
        for (uint32_t b = threadIdx.x; b <= buckets; b += blockDim.x) expert_offsets[b] = base[b];
    });
}

// (expert, token tile) pairs in expert order for the tensor-core expert kernels: entry =
// (expert << 16) | token tile within the expert; every thread of one block calls it
__device__ void build_tiles_body(const uint32_t* expert_offsets, uint32_t num_experts, uint32_t n_tile,
                                 uint32_t* tiles, uint32_t* count) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0u) carry = 0u;
    __syncthreads();
    for (uint32_t base = 0; base < num_experts; base += blockDim.x) {
        const uint32_t e = base + threadIdx.x;
        uint32_t mine = 0u;
        if (e < num_experts) mine = (expert_offsets[e + 1u] - expert_offsets[e] + n_tile - 1u) / n_tile;
        // block-wide exclusive scan
        uint32_t incl = mine;
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += n;
        }
        if (lane == 31u) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 0u) {
            uint32_t v = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0u;
            uint32_t sum = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t n = __shfl_up_sync(0xffffffffu, sum, o);
                if ((int)lane >= o) sum += n;
            }
            warp_sums[lane] = sum - v;
        }
        __syncthreads();
        const uint32_t start = carry + warp_sums[warp] + incl - mine;
        for (uint32_t j = 0; j < mine; j++) tiles[start + j] = (e << 16) | j;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1u) carry = start + mine;
        __syncthreads();
    }
    if (threadIdx.x == 0u) *count = carry;
}

__global__ void __launch_bounds__(1024) build_tiles_kernel(const uint32_t* expert_offsets, uint32_t num_experts,
                                                          uint32_t n_tile, uint32_t* tiles, uint32_t* count) {
    grid_dependency_sync();
    build_tiles_body(expert_offsets, num_experts, n_tile, tiles, count);
}

// one block groups the slots of a stage and, for the tensor path, lists its tiles
__global__ void __launch_bounds__(1024) group_small_kernel(SlotKey key, const uint32_t* control,
                                                          uint32_t max_tokens, uint32_t* grouped,
                                                          uint32_t* expert_offsets, uint32_t* position, TileOut tiles) {
    extern __shared__ uint32_t hist[];
    grid_dependency_sync();
    const uint32_t T = min_u32(control[0], max_tokens), buckets = key.num_experts;
    const uint32_t slots = slot_count(control, max_tokens, key.K);
    if (rank_block_fits(blockDim.x, buckets) && slots <= blockDim.x) {
        key.capacity = T * key.K;
        if (position)  // routes the grouping drops keep "nowhere" (the barriers of the ranking stand between this and the places)
            for (uint32_t i = threadIdx.x; i < key.capacity; i += blockDim.x) position[i] = kUnboundSlot;
        GroupEmit emit{key, grouped, position};
        rank_single_block(slots, buckets, hist, tiles.list ? tiles.n_tile : 1u, key, emit, [&](const uint32_t* base, const uint32_t* tile_base) {
            for (uint32_t b = threadIdx.x; b <= buckets; b += blockDim.x) {
                expert_offsets[b] = base[b];
                if (!tiles.list) continue;
                if (b == buckets) {
                    *tiles.count = tile_base[b];
                } else {
                    for (uint32_t t = tile_base[b]; t < tile_base[b + 1u]; t++) tiles.list[t] = (b << 16) | (t - tile_base[b]);
                }
            }
        });
        return;
    }
    group_small_body(key, control, max_tokens, grouped, expert_offsets, position, hist);
    if (tiles.list) {
        __syncthreads();
        build_tiles_body(expert_offsets, key.num_experts, tiles.n_tile, tiles.list, tiles.count);
    }
}

// The whole schedule of one layer call in one block (T*K small): the control words the host of the
// reference writes, the compact list in front of gate/up, the owned count in front of down, and for
// each of the two expert stages the expert-grouped route list and the tensor-path tile list.
// Shared memory of the fused schedule: sort histogram, then copies of what the five passes would otherwise
// fetch from global memory through chains of dependent loads: the route words, the compact list, and
// per stage whether each expert is resident.
__host__ __device__ inline size_t layer_schedule_smem_bytes(uint32_t count, uint32_t num_experts) {
    return ((size_t)num_experts + 2u + 2u * count) * sizeof(uint32_t) + 2u * (size_t)num_experts;
}

__global__ void __launch_bounds__(1024) layer_schedule_small_kernel(LayerSchedule s) {
    extern __shared__ uint32_t hist[];
    const uint32_t count = s.tokens * s.K;
    uint32_t* route_words = hist + s.num_experts + 2u;
    uint32_t* compact_list = route_words + count;
    uint8_t* resident = reinterpret_cast<uint8_t*>(compact_list + count);
    grid_dependency_sync();
    for (uint32_t w = threadIdx.x; w < s.clear_words; w += blockDim.x) s.clear[w] = 0u;
    if (threadIdx.x < 14u) {
        const uint32_t j = threadIdx.x % 7u;
        s.control[threadIdx.x / 7u][j] = j == 0u ? s.tokens : j == 1u ? s.expert_start : j == 2u ? s.expert_count : 0u;
    }
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
        route_words[i] = s.routes[i];
        compact_list[i] = kUnboundSlot;  // positions past the owned count stay out of range
    }
    for (uint32_t e = threadIdx.x; e < 2u * s.num_experts; e += blockDim.x)
        resident[e] = s.experts[e / s.num_experts][e % s.num_experts].w[0] != nullptr ? 1u : 0u;
    __syncthreads();
    compact_small_body(route_words, s.intermediates, s.slots[0], s.slot_words[0], 4u, s.control[0], s.tokens, s.K, s.I,
                       s.tiles_per_route[0], s.num_experts, hist, compact_list);
    __syncthreads();
    route_count_body(route_words, s.slots[1], s.slot_words[1], 2u, s.control[1], s.tokens, s.K, s.tiles_per_route[1]);
    __syncthreads();
    for (uint32_t stage = 0; stage < 2u; stage++) {
        // the flat copy of the compact list stands in for the schedule words of the frames: frame = K words, no data
        SlotKey key{route_words, compact_list, s.experts[stage], s.status, s.num_experts, s.K, s.K, 0u, 0u,
                    resident + stage * s.num_experts};
        group_small_body(key, s.control[stage], s.tokens, s.grouped[stage], s.offsets[stage], s.position[stage], hist);
        __syncthreads();
        if (s.tiles[stage]) build_tiles_body(s.offsets[stage], s.num_experts, s.n_tile[stage], s.tiles[stage], s.tile_count[stage]);
        __syncthreads();
    }
}

// The same schedule from one pass over the routes.  The compact list and both expert groupings are one
// stable sort of the routes by expert id seen through different filters: the rank r of a route among the
// listed routes of its expert is found once, and every list position is a per-list bucket base plus r.
// Rank: a warp ranks its 32 routes with match_any and leaves its per-bucket counts in a table
// [warp][bucket]; a column-wise running sum turns the counts into the ranks where each warp's routes start.
// The partitioned call (expert_count != 0) lists only owned routes, in source order (one more table column
// counts them per warp), and its down stage visits the first owned-by-the-down-table-count of them.
// One round trip to global memory, five block barriers.
constexpr uint32_t kRankChunks = 16u;  // routes per thread at most (count <= 16 * blockDim); the kernel is built for 1, 4 and 16
constexpr uint32_t kWideScheduleRoutes = 1280u;
constexpr uint32_t kNotListed = 0xffffu;  // bucket field of a route that is in no list

__host__ __device__ inline uint32_t layer_schedule_rank_threads(uint32_t count) { return count <= 256u ? 256u : 1024u; }

__host__ __device__ inline size_t layer_schedule_rank_smem_bytes(uint32_t count, uint32_t num_experts) {
    const size_t columns = (size_t)num_experts + 2u;  // experts, out-of-range ids, owned routes
    const size_t warps = ((size_t)count + 31u) / 32u;
    // table (u16, rounded to words); hist, hist_down, base_all, gbase[2], tile_base[2] (columns + 1 words each);
    // two totals; kept[2] (a byte per column)
    return ((warps * columns + 1u) / 2u + 7u * (columns + 1u) + 2u) * sizeof(uint32_t) + 2u * columns;
}

// words for the places of the routes of the tokens that a block of so many warps, each with one of a token's `chunks` of columns, can meet
__host__ __device__ inline uint32_t place_words(uint32_t warps, uint32_t chunks, uint32_t K) { return ((warps + chunks - 2u) / chunks + 1u) * K; }

// `before` runs once the table has been cleared: the wait for the kernel before this one, or that and the routing.
template <uint32_t CHUNKS, class BeforeFn>
__device__ __forceinline__ void layer_schedule_rank_body(const LayerSchedule& s, BeforeFn before) {
    extern __shared__ uint32_t smem_words[];
    const uint32_t count = s.tokens * s.K;
    const uint32_t E = s.num_experts;
    const uint32_t B = E + 1u;   // bucket E collects out-of-range expert ids
    const uint32_t C = E + 2u;   // column B counts the owned routes of a warp (partitioned calls)
    const uint32_t V = (count + 31u) / 32u;
    const uint32_t table_words = (V * C + 1u) / 2u;
    uint16_t* table = reinterpret_cast<uint16_t*>(smem_words);
    uint32_t* hist = smem_words + table_words;  // listed routes per bucket
    uint32_t* hist_down = hist + (C + 1u);      // of which the down stage visits
    uint32_t* base_all = hist + 2u * (C + 1u);
    uint32_t* gbase[2] = {hist + 3u * (C + 1u), hist + 4u * (C + 1u)};
    uint32_t* tile_base[2] = {hist + 5u * (C + 1u), hist + 6u * (C + 1u)};
    uint32_t* totals = hist + 7u * (C + 1u);  // owned routes under the gate/up and the down slot table
    uint8_t* kept = reinterpret_cast<uint8_t*>(totals + 2u);  // [2][C]: the stage keeps routes of this bucket
    const uint32_t lane = threadIdx.x & 31u;
    const bool partitioned = s.expert_count != 0u;
    const uint32_t owned_end = s.expert_start + s.expert_count;

    for (uint32_t w = threadIdx.x; w < table_words; w += blockDim.x) smem_words[w] = 0u;
    if (threadIdx.x < 2u) totals[threadIdx.x] = 0u;
    before();
    for (uint32_t w = threadIdx.x; w < s.clear_words; w += blockDim.x) s.clear[w] = 0u;
    // residency of every expert for both stages (bucket E is never kept)
    // (the two stages are unrolled throughout: pointers picked by a run-time stage would live in local memory)
    for (uint32_t b = threadIdx.x; b < C; b += blockDim.x) {
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++) kept[stage * C + b] = (b < E && s.experts[stage][b].w[0] != nullptr) ? 1u : 0u;
    }
    // per route: bucket (16 bits) | routes of the same bucket before it in its warp (8) | owned routes before it (8)
    uint32_t state[CHUNKS];
    __syncthreads();
#pragma unroll
    for (uint32_t c = 0; c < CHUNKS; c++) {
        const uint32_t i = c * blockDim.x + threadIdx.x;
        state[c] = kNotListed;
        if (c * blockDim.x < count) {  // uniform over the block: whole warps take part in the votes
            bool listed = i < count, owned_down = false;
            uint32_t e = 0u;
            if (listed) e = s.routes[i] & 0xffffu;
            if (partitioned) {
                const bool in_range = listed && e >= s.expert_start && e < owned_end;
                listed = in_range && resource_is_local(s.slots[0], s.slot_words[0], 4u, e);
                owned_down = in_range && resource_is_local(s.slots[1], s.slot_words[1], 2u, e);
                const uint32_t owners = __ballot_sync(0xffffffffu, listed);
                const uint32_t owners_down = __ballot_sync(0xffffffffu, owned_down);
                state[c] |= (uint32_t)__popc(owners & ((1u << lane) - 1u)) << 24;
                if (lane == 0u) {
                    if (owners) {  // a warp past the end of the routes has no row in the table
                        table[(size_t)(i >> 5) * C + B] = (uint16_t)__popc(owners);
                        atomicAdd(totals + 0, (uint32_t)__popc(owners));
                    }
                    if (owners_down) atomicAdd(totals + 1, (uint32_t)__popc(owners_down));
                }
            }
            const uint32_t bucket = listed ? min_u32(e, E) : kNotListed;
            const uint32_t peers = __match_any_sync(0xffffffffu, bucket);
            state[c] = (state[c] & 0xff000000u) | ((uint32_t)__popc(peers & ((1u << lane) - 1u)) << 16) | bucket;
            if (listed && lane == (uint32_t)__ffs(peers) - 1u) table[(size_t)(i >> 5) * C + bucket] = (uint16_t)__popc(peers);
        }
    }
    __syncthreads();
    // the down stage of a partitioned call visits the first totals[1] entries of the compact list
    const uint32_t listed_total = partitioned ? totals[0] : count;
    const uint32_t down_total = partitioned ? totals[1] : count;
    const bool cut = down_total < listed_total;
    for (uint32_t b = threadIdx.x; b < C; b += blockDim.x) {
        uint32_t running = 0u;
        for (uint32_t v = 0; v < V; v++) {
            const uint32_t here = table[(size_t)v * C + b];
            table[(size_t)v * C + b] = (uint16_t)running;
            running += here;
        }
        hist[b] = running;
        hist_down[b] = cut ? 0u : running;
    }
    __syncthreads();
    if (cut) {
        // the entries cut off are the last in source order, so the ranks of the others stand; only the counts change
#pragma unroll
        for (uint32_t c = 0; c < CHUNKS; c++) {
            const uint32_t i = c * blockDim.x + threadIdx.x;
            const uint32_t bucket = state[c] & 0xffffu;
            if (i < count && bucket != kNotListed && table[(size_t)(i >> 5) * C + B] + (state[c] >> 24) < down_total)
                atomicAdd(hist_down + bucket, 1u);
        }
        __syncthreads();
    }
    // five exclusive scans over the buckets, a warp each: the compact list of an unpartitioned call, and per
    // stage the grouped list and the tile list
    const uint32_t warp = threadIdx.x >> 5;
    if (warp < 5u) {
        const uint32_t stage = warp == 0u ? 0u : (warp - 1u) & 1u;
        const bool tiles = warp >= 3u;
        const uint32_t* counts = stage == 1u ? hist_down : hist;
        const uint32_t n_tile = stage == 0u ? s.n_tile[0] : s.n_tile[1];
        warp_exclusive_scan(B, base_all + warp * (C + 1u), [&](uint32_t b) {  // (the arrays lie in the warps' order)
            const uint32_t v = counts[b];
            if (warp == 0u) return v;
            if (!kept[stage * C + b]) return 0u;
            return tiles ? (v + n_tile - 1u) / n_tile : v;
        });
    }
    __syncthreads();
#pragma unroll
    for (uint32_t stage = 0; stage < 2u; stage++) {
        const uint32_t j = threadIdx.x, visited = stage == 0u ? listed_total : down_total;
        if (j < 7u)
            s.control[stage][j] = j == 0u ? s.tokens : j == 1u ? s.expert_start : j == 2u ? s.expert_count : j == 3u ? visited
                                  : j == 4u ? (partitioned ? visited : s.K) * s.tiles_per_route[stage]
                                  : j == 5u && !partitioned ? s.tokens : 1u;
    }
    // a down count beyond the compact list makes the down stage read entries that were never written
    if (threadIdx.x == 0u && down_total > listed_total) raise_status(s.status, NVMOE_STATUS_ROUTE_OUT_OF_RANGE);
    const uint32_t data_words = s.K * (s.I / 2u), frame_words = data_words + s.K;
#pragma unroll
    for (uint32_t c = 0; c < CHUNKS; c++) {
        const uint32_t i = c * blockDim.x + threadIdx.x;
        if (i >= count) continue;
        const uint32_t b = state[c] & 0xffffu;
        const bool listed = b != kNotListed;
        uint32_t rank = 0u, at = 0u;
        if (listed) {
            rank = table[(size_t)(i >> 5) * C + b] + ((state[c] >> 16) & 0xffu);
            at = partitioned ? table[(size_t)(i >> 5) * C + B] + (state[c] >> 24) : base_all[b] + rank;
            s.intermediates[(size_t)(at / s.K) * frame_words + data_words + at % s.K] = i;
        }
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++) {
            uint32_t place = kUnboundSlot;
            if (listed && (stage == 0u || at < down_total)) {
                if (kept[stage * C + b]) {
                    place = gbase[stage][b] + rank;
                    s.grouped[stage][place] = i;
                } else {
                    raise_status(s.status, b == E ? NVMOE_STATUS_ROUTE_OUT_OF_RANGE : NVMOE_STATUS_EXPERT_NOT_RESIDENT);
                }
            }
            if (s.position[stage]) s.position[stage][i] = place;
        }
    }
#pragma unroll
    for (uint32_t stage = 0; stage < 2u; stage++) {
        for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) {
            // bucket E is never kept, so gbase[stage][E] is already the total the offsets end with
            s.offsets[stage][b] = gbase[stage][b];
            if (s.tiles[stage] && b < E) {
                const uint32_t first = tile_base[stage][b], n = tile_base[stage][b + 1u] - first;
                for (uint32_t j = 0; j < n; j++) s.tiles[stage][first + j] = (b << 16) | j;
            }
            if (s.tiles[stage] && b == E) *s.tile_count[stage] = tile_base[stage][E];
        }
    }
}

template <uint32_t CHUNKS>
__global__ void __launch_bounds__(1024) layer_schedule_rank_kernel(LayerSchedule s) {
    layer_schedule_rank_body<CHUNKS>(s, [] { grid_dependency_sync(); });
}

// Router and schedule of a handful of tokens in one block: a warp routes a token, the block barrier inside the schedule
// stands where the next launch would. Each of the two is a few microseconds of latency, so is the hand-over between them.
template <int EPL>
__global__ void __launch_bounds__(1024) route_schedule_kernel(RouterLaunch router, LayerSchedule s) {
    layer_schedule_rank_body<1u>(s, [&] {
        grid_dependency_sync();
        const uint32_t token = threadIdx.x >> 5;
        if (token < router.tokens) route_token<false, EPL, false>(router, token);
    });
}

// ---- small calls: operands and schedule side by side -------------------------------------------------------
// A layer call of at most 1024 routes of all experts, a route a thread, of not too many a token (places_operands): the gate/up operands (place_operands_kernel) are made ahead of the
// schedule (small_schedule_kernel) instead of behind it, and the two run at the same time.
//
// What a block of operands has to know of the schedule are the places of its own tokens' routes, which it counts itself: a place is the number
// of kept routes that come before by (expert, route index). The rows are read and quantised before the wait where the launches ahead allow it
// (`early`); after it a block loads the route words, counts and stores. Where the call's tokens are routed here too (EPL != 0), every block
// selects the experts of all of them from the logits, and the first one also writes the route words.
//
// Both are bound by latency. In turn, the quantisation added a hand-over, two dependent loads and the rows' fetch to the schedule. Layers, us,
// in turn / side by side: 64 tokens of the tiny layer 24.4 / 23.1; 32 experts of 2880 x 2880, one token 37.0 / 35.0, seven 67.1 / 63.7, 64 94.8 / 92.1, 32 from
// host buffers 121.0 / 118.0; 96 of 257 of 7168 x 2048 749 / 737.
template <int EPL, uint32_t LANES>
__global__ void __launch_bounds__(1024) place_operands_kernel(const __grid_constant__ RouterLaunch router, const __grid_constant__ LayerSchedule s, const __grid_constant__ OperandRows o) {
    extern __shared__ uint32_t smem_words[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t count = s.tokens * s.K, first = blockIdx.x * warps, item = first + warp;
    const uint32_t token = item / o.chunks, col = (item % o.chunks) * 512u + lane * 16u;
    const bool active = token < s.tokens && col < o.cols;  // (columns come in whole blocks: the lanes of a block agree)
    uint32_t out[4], word;
    if (o.early) quantize_sixteen<LANES>(o.input + (size_t)token * o.cols + col, active, lane, out, word);
    // per stage (expert << 16 | route) of every route that the stage keeps, all ones above the route of the others: their order is the grouping's
    uint32_t* keys[2] = {smem_words, smem_words + count};
    uint32_t* places[2] = {smem_words + 2u * count, smem_words + 2u * count + place_words(warps, o.chunks, s.K)};
    auto list_route = [&](uint32_t i, uint32_t e) {
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++)
            keys[stage][i] = (e < s.num_experts && s.experts[stage][e].w[0] != nullptr ? e << 16 : 0xffff0000u) | i;
    };
    grid_dependency_sync();
    if (EPL != 0) {
        if (warp < router.tokens) {
            uint32_t e, rank;
            float v;
            const bool found = select_experts<true, EPL == 0 ? 1 : EPL, false>(router, warp, e, v);
            if (blockIdx.x == 0u) {
                finish_token<true>(router, counts_of(router), warp, found, e, v, rank);
            } else {
                order_token(router, found, e, rank);
            }
            if (lane < s.K) list_route(warp * s.K + rank, e);
        }
    } else {
#pragma unroll 1
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) list_route(i, __ldg(s.routes + i) & 0xffffu);
    }
    if (!o.early) quantize_sixteen<LANES>(o.input + (size_t)token * o.cols + col, active, lane, out, word);
    __syncthreads();
    const uint32_t token0 = first / o.chunks, token1 = min_u32((first + warps - 1u) / o.chunks + 1u, s.tokens);
#pragma unroll 1
    for (uint32_t n = warp; n < (token1 - token0) * s.K; n += warps) {
        const uint32_t i = token0 * s.K + n;
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++) {
            if (stage == 1u && keys[0][i] < 0xffff0000u) continue;  // (uniform) the down place is asked for only where gate/up skips the route
            const uint32_t mine = keys[stage][i];
            uint32_t before = 0u;
#pragma unroll 4
            for (uint32_t j = lane; j < count; j += 32u) before += keys[stage][j] < mine ? 1u : 0u;
            before = __reduce_add_sync(0xffffffffu, before);
            if (lane == 0u) places[stage][n] = mine < 0xffff0000u ? before : kUnboundSlot;
        }
    }
    __syncthreads();
    if (token >= s.tokens) return;
#pragma unroll 1
    for (uint32_t r = 0; r < s.K; r++) {
        const uint32_t n = (token - token0) * s.K + r, row = places[0][n];
        if (row == kUnboundSlot) {  // a route that gate/up skips: zeros for the down stage, if that keeps it
            if (o.down.q == nullptr || item % o.chunks != 0u || places[1][n] == kUnboundSlot) continue;
            zero_down_row(o.down, places[1][n], lane);
            continue;
        }
        if (!active) continue;
        *reinterpret_cast<uint4*>(o.q + (size_t)row * o.cols + col) = make_uint4(out[0], out[1], out[2], out[3]);
        if ((lane & 7u) == 0u) *o.scales.at(row, col / 128u) = word;
    }
}

// What the expert kernels and the combine read of a schedule (layer_schedule_rank_body makes the reference's lists too), by one block.
// place_operands_kernel, the launch ahead, writes nothing that this one touches but at most the route words, which it then selects itself (EPL !=
// 0), reads nothing that this one writes, and let it start once all launches before it had completed: the work stands before the wait,
// which is there so that who waits for this launch has waited for both. The next one may start at once: what it does before its wait relies on
// launches before place_operands_kernel. (That the code is short counts: a block of this kind runs it once, and waits for each line of
// it. The end of the general form, with the lists, took 1.6 to 2.6 us of its 3.4 to 7.8.)
__host__ __device__ inline size_t small_schedule_words(uint32_t count, uint32_t num_experts) {
    // per route its expert; per stage and expert the routes before it << 16 | tiles before it within its 32 experts, and its own; the sums of
    // the 32s; [warp][expert] counts (u16)
    return (size_t)count + 4u * (size_t)num_experts + 2u * ((num_experts + 31u) / 32u) + ((size_t)(count + 31u) / 32u * num_experts + 1u) / 2u;
}
template <int EPL>
__global__ void __launch_bounds__(1024) small_schedule_kernel(const __grid_constant__ RouterLaunch router, const __grid_constant__ LayerSchedule s) {
    extern __shared__ uint32_t smem_words[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t E = s.num_experts, count = s.tokens * s.K, groups = (E + 31u) / 32u, rows = (count + 31u) / 32u;
    uint32_t* ids = smem_words;
    uint32_t* before_expert = ids + count;           // [stage][expert]
    uint32_t* of_expert = before_expert + 2u * E;    // [stage][expert]
    uint32_t* of_group = of_expert + 2u * E;         // [stage][32 experts]
    uint16_t* table = reinterpret_cast<uint16_t*>(of_group + 2u * groups);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, i = threadIdx.x;
#pragma unroll 1
    for (uint32_t w = threadIdx.x; w < (rows * E + 1u) / 2u; w += blockDim.x) reinterpret_cast<uint32_t*>(table)[w] = 0u;
#pragma unroll 1
    for (uint32_t w = threadIdx.x; w < s.clear_words; w += blockDim.x) s.clear[w] = 0u;
#pragma unroll 1
    for (uint32_t b = threadIdx.x; b < 2u * E; b += blockDim.x)  // (for now whether the stage has the expert)
        of_expert[b] = (b < E ? s.experts[0][b] : s.experts[1][b - E]).w[0] != nullptr ? 1u : 0u;
    uint32_t e = kUnboundSlot;
    if (EPL != 0) {
        if (warp < router.tokens) {
            uint32_t mine, rank;
            float v;
            order_token(router, select_experts<true, EPL == 0 ? 1 : EPL, false>(router, warp, mine, v), mine, rank);
            if (lane < s.K) ids[warp * s.K + rank] = mine;
        }
        __syncthreads();
        if (i < count) e = ids[i];
    } else {
        if (i < count) e = __ldg(s.routes + i) & 0xffffu;
        __syncthreads();
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, e), before = __popc(peers & ((1u << lane) - 1u));
    if (e < E && before == 0u) table[warp * E + e] = (uint16_t)__popc(peers);
    __syncthreads();
#pragma unroll 1
    for (uint32_t b = threadIdx.x; (b & ~31u) < E; b += blockDim.x) {
        uint32_t total = 0u;
        if (b < E) {
            for (uint32_t r = 0; r < rows; r++) {
                const uint32_t here = table[r * E + b];
                table[r * E + b] = (uint16_t)total;
                total += here;
            }
        }
#pragma unroll 1
        for (uint32_t stage = 0; stage < 2u; stage++) {
            const uint32_t n_tile = s.n_tile[stage];
            const uint32_t own = b < E && of_expert[stage * E + b] != 0u ? total << 16 | (total + n_tile - 1u) / n_tile : 0u;
            uint32_t sum = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t n = __shfl_up_sync(0xffffffffu, sum, o);
                if ((int)lane >= o) sum += n;
            }
            if (b < E) {
                before_expert[stage * E + b] = sum - own;
                of_expert[stage * E + b] = own;
            }
            if (lane == 31u) of_group[stage * groups + b / 32u] = sum;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t stage = 0; stage < 2u; stage++) {
        auto base_of = [&](uint32_t b) {
            uint32_t sum = before_expert[stage * E + b];
#pragma unroll 1
            for (uint32_t w = 0; w < b / 32u; w++) sum += of_group[stage * groups + w];
            return sum;
        };
        if (i < count) {
            uint32_t place = kUnboundSlot;
            if (e < E && of_expert[stage * E + e] != 0u) {
                place = (base_of(e) >> 16) + table[warp * E + e] + before;
                s.grouped[stage][place] = i;
            } else {
                raise_status(s.status, e >= E ? NVMOE_STATUS_ROUTE_OUT_OF_RANGE : NVMOE_STATUS_EXPERT_NOT_RESIDENT);
            }
            s.position[stage][i] = place;
        }
#pragma unroll 1
        for (uint32_t b = threadIdx.x; b < E; b += blockDim.x) {
            const uint32_t base = base_of(b), own = of_expert[stage * E + b], first = base & 0xffffu;
            const uint32_t tiles = own & 0xffffu;
            s.offsets[stage][b] = base >> 16;
#pragma unroll 1
            for (uint32_t t = 0; t < tiles; t++) s.tiles[stage][first + t] = b << 16 | t;
            if (b + 1u == E) {
                s.offsets[stage][E] = (base + own) >> 16;
                *s.tile_count[stage] = first + tiles;
            }
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The same schedule for more routes than one block ranks well: 256 routes a block, in three launches. As above, one
// stable sort of the routes by expert id serves all lists: the counts per (block, bucket) are taken once (a histogram
// launch, then phase_scan_kernel), and the last launch turns them into places in the compact list and in both
// groupings at once. Every block scans the bucket totals itself; block 0 also writes what is per call. Unpartitioned
// calls only: the owned-route form lists routes in source order, which is another sort.
// Bound by the latency of three short dependent kernels. The thirteen launches of one sort per list took 413 us for
// 147456 routes of 257 experts, and the one-block form 44 us for 16384 of 32.
__global__ void __launch_bounds__(256) layer_schedule_hist_kernel(LayerSchedule s, uint32_t* block_hist) {
    grid_dependency_sync();
    phase_hist(s.tokens * s.K, s.num_experts + 1u, block_hist, RouteKey{s.routes, s.num_experts});
}

__host__ __device__ inline size_t layer_schedule_wide_smem_bytes(uint32_t num_experts) {
    // the compact list's, two groupings' and two tile lists' bases; ranks of this block; totals; [warp][bucket] counts (u16); kept[2]
    const size_t buckets = (size_t)num_experts + 1u;
    return (5u * (buckets + 1u) + 2u * buckets) * sizeof(uint32_t) + (8u * buckets + 1u) / 2u * 4u + 2u * buckets;
}

__global__ void __launch_bounds__(256) layer_schedule_scatter_kernel(LayerSchedule s, const uint32_t* __restrict__ block_hist,
                                                                    const uint32_t* __restrict__ totals) {
    extern __shared__ uint32_t smem_words[];
    const uint32_t count = s.tokens * s.K, E = s.num_experts, B = E + 1u;  // bucket E collects out-of-range expert ids
    uint32_t* base_all = smem_words;
    uint32_t* gbase[2] = {base_all + (B + 1u), base_all + 2u * (B + 1u)};
    uint32_t* tile_base[2] = {base_all + 3u * (B + 1u), base_all + 4u * (B + 1u)};
    uint32_t* first = base_all + 5u * (B + 1u);
    uint32_t* total = first + B;
    uint32_t* table_words = total + B;
    uint16_t* table = reinterpret_cast<uint16_t*>(table_words);
    uint8_t* kept = reinterpret_cast<uint8_t*>(table_words + (8u * B + 1u) / 2u);  // [2][B]: the stage keeps routes of this bucket
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (uint32_t w = threadIdx.x; w < (8u * B + 1u) / 2u; w += blockDim.x) table_words[w] = 0u;
    grid_dependency_sync();
    if (blockIdx.x == 0u)
        for (uint32_t w = threadIdx.x; w < s.clear_words; w += blockDim.x) s.clear[w] = 0u;
    const uint32_t i = blockIdx.x * kSortChunk + threadIdx.x;
    uint32_t bucket = kNotListed;
    if (i < count) bucket = min_u32(__ldg(s.routes + i) & 0xffffu, E);
    for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) {
        first[b] = __ldg(block_hist + (size_t)blockIdx.x * B + b);
        total[b] = __ldg(totals + b);
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++) kept[stage * B + b] = (b < E && s.experts[stage][b].w[0] != nullptr) ? 1u : 0u;
    }
    __syncthreads();
    const uint32_t peers = __match_any_sync(0xffffffffu, bucket);
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    if (bucket != kNotListed && before == 0u) table[warp * B + bucket] = (uint16_t)__popc(peers);
    if (warp < 5u) {  // five scans, a warp each
        const uint32_t stage = warp == 0u ? 0u : (warp - 1u) & 1u;
        const uint32_t n_tile = stage == 0u ? s.n_tile[0] : s.n_tile[1];
        warp_exclusive_scan(B, base_all + warp * (B + 1u), [&](uint32_t b) {  // (the arrays lie in the warps' order)
            const uint32_t v = total[b];
            if (warp == 0u) return v;
            if (!kept[stage * B + b]) return 0u;
            return warp >= 3u ? (v + n_tile - 1u) / n_tile : v;
        });
    }
    __syncthreads();
    if (i < count) {
        uint32_t rank = first[bucket] + before;
        for (uint32_t w = 0; w < warp; w++) rank += table[w * B + bucket];
        const uint32_t at = base_all[bucket] + rank;
        const uint32_t data_words = s.K * (s.I / 2u);
        s.intermediates[(size_t)(at / s.K) * (data_words + s.K) + data_words + at % s.K] = i;
#pragma unroll
        for (uint32_t stage = 0; stage < 2u; stage++) {
            uint32_t place = kUnboundSlot;
            if (kept[stage * B + bucket]) {
                place = gbase[stage][bucket] + rank;
                s.grouped[stage][place] = i;
            } else {
                raise_status(s.status, bucket == E ? NVMOE_STATUS_ROUTE_OUT_OF_RANGE : NVMOE_STATUS_EXPERT_NOT_RESIDENT);
            }
            if (s.position[stage]) s.position[stage][i] = place;
        }
    }
    // tile lists: a warp per expert, its tiles side by side, the experts shared out over the blocks (by block 0 alone the
    // lists of 257 experts took 20 us)
#pragma unroll
    for (uint32_t stage = 0; stage < 2u; stage++) {
        if (!s.tiles[stage]) continue;
        for (uint32_t b = blockIdx.x * 8u + warp; b < E; b += gridDim.x * 8u) {
            const uint32_t at = tile_base[stage][b], n = tile_base[stage][b + 1u] - at;
            for (uint32_t j = lane; j < n; j += 32u) s.tiles[stage][at + j] = (b << 16) | j;
        }
    }
    if (blockIdx.x != 0u) return;
#pragma unroll
    for (uint32_t stage = 0; stage < 2u; stage++) {
        const uint32_t j = threadIdx.x;
        if (j < 7u)
            s.control[stage][j] = j == 0u || j == 5u ? s.tokens : j == 1u ? s.expert_start : j == 2u ? 0u : j == 3u ? count
                                  : j == 4u ? s.K * s.tiles_per_route[stage] : 1u;
        for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) s.offsets[stage][b] = gbase[stage][b];  // bucket E is never kept: the total
        if (s.tiles[stage] && threadIdx.x == 0u) *s.tile_count[stage] = tile_base[stage][E];
    }
}

__global__ void __launch_bounds__(256) group_hist_kernel(SlotKey key, const uint32_t* control,
                                                        uint32_t max_tokens, uint32_t* block_hist, uint32_t* position) {
    key.capacity = min_u32(control[0], max_tokens) * key.K;
    key.status = nullptr;  // raised once, by the scatter pass
    if (position)  // routes the grouping drops keep "nowhere"; the scatter pass (a later launch) fills the rest
        for (uint32_t i = blockIdx.x * kSortChunk + threadIdx.x; i < min_u32(key.capacity, (blockIdx.x + 1u) * kSortChunk); i += blockDim.x)
            position[i] = kUnboundSlot;
    phase_hist(slot_count(control, max_tokens, key.K), key.num_experts, block_hist, key);
}

__global__ void __launch_bounds__(256) group_scatter_kernel(SlotKey key, const uint32_t* control,
                                                           uint32_t max_tokens, uint32_t* grouped,
                                                           uint32_t* expert_offsets, const uint32_t* block_hist,
                                                           const uint32_t* totals, uint32_t* position) {
    key.capacity = min_u32(control[0], max_tokens) * key.K;
    GroupEmit emit{key, grouped, position};
    phase_scatter(slot_count(control, max_tokens, key.K), key.num_experts, block_hist, totals, key, emit, expert_offsets);
}

// ---- expert-parallel dispatch: group routes by the rank that owns their expert ------------------

struct DestKey {  // bucket = destination rank; kUnboundSlot in the owner table means "this rank"
    const uint32_t* routes;
    const uint32_t* owner;
    uint32_t num_experts, world, self;
    __device__ uint32_t operator()(uint32_t i) const {
        uint32_t e = routes[i] & 0xffffu;
        if (e >= num_experts) return kUnboundSlot;
        uint32_t r = owner[e];
        if (r == kUnboundSlot) r = self;
        return r < world ? r : kUnboundSlot;
    }
};

struct PackEmit {  // one warp-wide row copy per route would be faster; rows are copied by a second kernel
    const uint32_t* routes;
    uint32_t* send_routes;
    uint32_t* send_index;
    uint32_t* send_source;
    __device__ void operator()(uint32_t rank, uint32_t i) const {
        send_routes[rank] = routes[i];
        send_index[i] = rank;
        send_source[rank] = i;
    }
};

__global__ void __launch_bounds__(1024) ep_pack_small_kernel(DestKey key, PackEmit emit, uint32_t count,
                                                            uint32_t* dest_counts) {
    extern __shared__ uint32_t hist[];
    grid_dependency_sync();
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) emit.send_index[i] = kUnboundSlot;
    __syncthreads();
    sort_single_block(count, key.world, hist, key, emit, [&](const uint32_t* base) {
        for (uint32_t b = threadIdx.x; b < key.world; b += blockDim.x) dest_counts[b] = base[b + 1u] - base[b];
    });
}

__global__ void __launch_bounds__(256) ep_pack_hist_kernel(DestKey key, uint32_t count, uint32_t* block_hist,
                                                          uint32_t* send_index) {
    for (uint32_t i = blockIdx.x * kSortChunk + threadIdx.x; i < min_u32(count, (blockIdx.x + 1u) * kSortChunk); i += blockDim.x)
        send_index[i] = kUnboundSlot;
    phase_hist(count, key.world, block_hist, key);
}

__global__ void __launch_bounds__(256) ep_pack_scatter_kernel(DestKey key, PackEmit emit, uint32_t count,
                                                             const uint32_t* block_hist, const uint32_t* totals,
                                                             uint32_t* dest_counts) {
    phase_scatter(count, key.world, block_hist, totals, key, emit);
    if (blockIdx.x == 0u)
        for (uint32_t b = threadIdx.x; b < key.world; b += blockDim.x) dest_counts[b] = totals[b];
}

// send_rows[p] = hidden[token of route send_source[p]]; one warp per row, 16-byte pieces
__global__ void __launch_bounds__(256) ep_gather_rows_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                            const uint32_t* __restrict__ index, const uint32_t* total,
                                                            uint32_t max_rows, uint32_t divide, uint32_t row_vec) {
    grid_dependency_sync();
    const uint32_t rows = total ? min_u32(*total, max_rows) : max_rows;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31u;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
        const uint32_t s = index[r];
        if (s == kUnboundSlot) {
            for (uint32_t c = lane; c < row_vec; c += 32u) dst[(size_t)r * row_vec + c] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        const uint4* from = src + (size_t)(s / divide) * row_vec;
        uint4* to = dst + (size_t)r * row_vec;
        // eight loads in flight a lane (see ep_pad_kernel)
        for (uint32_t c0 = lane; c0 < row_vec; c0 += 256u) {
            uint4 piece[8];
#pragma unroll
            for (uint32_t u = 0; u < 8u; u++)
                if (c0 + 32u * u < row_vec) piece[u] = __ldg(from + c0 + 32u * u);
#pragma unroll
            for (uint32_t u = 0; u < 8u; u++)
                if (c0 + 32u * u < row_vec) to[c0 + 32u * u] = piece[u];
        }
    }
}

// Padded dispatch layout: destination rank d owns slots [d*cap, (d+1)*cap) of the send buffers, the
// first dest_counts[d] of them filled in source order, the others marked with an all-ones route word
// (expert id 0xffff: no scheduler keeps it). Every slot is written, so the buffers can be exchanged
// with equal splits and no count has to reach the host. One warp per slot.
__global__ void __launch_bounds__(256) ep_pad_kernel(const uint4* __restrict__ hidden, const uint32_t* __restrict__ routes,
                                                    const uint32_t* __restrict__ dest_counts,
                                                    const uint32_t* __restrict__ send_source, uint32_t world, uint32_t cap,
                                                    uint32_t K, uint32_t row_vec, uint4* __restrict__ rows_out,
                                                    uint32_t* __restrict__ routes_out, uint32_t* __restrict__ send_index,
                                                    uint32_t* status) {
    grid_dependency_sync();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31u;
    const uint32_t slots = world * cap;
    // a segment that cannot hold what is bound for its rank: the excess routes stay "nowhere" (send_index keeps
    // its all-ones mark, the combine counts their rows as zeros) and the caller is told
    if (blockIdx.x == 0u && threadIdx.x < world && dest_counts[threadIdx.x] > cap) raise_status(status, NVMOE_STATUS_EXCHANGE_OVERFLOW);
    for (uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; slot < slots; slot += warps) {
        const uint32_t d = slot / cap, j = slot % cap;
        if (j >= min_u32(dest_counts[d], cap)) {
            if (lane == 0u) routes_out[slot] = kUnboundSlot;
            continue;
        }
        uint32_t offset = 0u;
        for (uint32_t x = lane; x < d; x += 32u) offset += dest_counts[x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) offset += __shfl_xor_sync(0xffffffffu, offset, o);
        const uint32_t i = send_source[offset + j];
        if (lane == 0u) {
            routes_out[slot] = routes[i];
            send_index[i] = slot;
        }
        const uint4* from = hidden + (size_t)(i / K) * row_vec;
        uint4* to = rows_out + (size_t)slot * row_vec;
        // eight loads in flight a lane: a row copied piece by piece costs one memory round trip per piece
        for (uint32_t c0 = lane; c0 < row_vec; c0 += 256u) {
            uint4 piece[8];
#pragma unroll
            for (uint32_t u = 0; u < 8u; u++)
                if (c0 + 32u * u < row_vec) piece[u] = __ldg(from + c0 + 32u * u);
#pragma unroll
            for (uint32_t u = 0; u < 8u; u++)
                if (c0 + 32u * u < row_vec) to[c0 + 32u * u] = piece[u];
        }
    }
}

__global__ void sum_counts_kernel(const uint32_t* counts, uint32_t n, uint32_t* total) {
    if (threadIdx.x == 0u && blockIdx.x == 0u) {
        uint32_t s = 0u;
        for (uint32_t i = 0; i < n; i++) s += counts[i];
        *total = s;
    }
}

constexpr uint32_t kSmallSortLimit = 4096u;

void launch_phase_scan(const SortScratch& scratch, uint32_t blocks, uint32_t buckets, cudaStream_t stream) {
    launch_chained(phase_scan_kernel, dim3((buckets + 31u) / 32u), dim3(1024), 0, stream, scratch.block_hist, scratch.bucket_totals,
                   blocks, buckets);
}

}  // namespace

void launch_ep_pack(const uint16_t* hidden, const uint32_t* routes, const uint32_t* owner, uint32_t tokens,
                    uint32_t K, uint32_t hidden_size, uint32_t num_experts, uint32_t world, uint32_t self,
                    uint16_t* send_rows, uint32_t* send_routes, uint32_t* send_index, uint32_t* send_source,
                    uint32_t* dest_counts, uint32_t* total, uint32_t segment_rows, uint32_t* contiguous_routes,
                    uint32_t* status, const SortScratch& scratch, cudaStream_t stream) {
    const uint32_t count = tokens * K;
    DestKey key{routes, owner, num_experts, world, self};
    // the padded form packs positions only; its route words and rows are placed by ep_pad_kernel
    PackEmit emit{routes, segment_rows ? contiguous_routes : send_routes, send_index, send_source};
    if (count <= kSmallSortLimit) {
        launch_chained(ep_pack_small_kernel, dim3(1), dim3(count <= 256u ? 256u : 1024u), (world + 1u) * sizeof(uint32_t),
                       stream, key, emit, count, dest_counts);
    } else {
        const uint32_t blocks = (count + kSortChunk - 1u) / kSortChunk;
        ep_pack_hist_kernel<<<blocks, 256, world * sizeof(uint32_t), stream>>>(key, count, scratch.block_hist, send_index);
        launch_phase_scan(scratch, blocks, world, stream);
        ep_pack_scatter_kernel<<<blocks, 256, (world + 1u) * sizeof(uint32_t), stream>>>(key, emit, count, scratch.block_hist,
                                                                                        scratch.bucket_totals, dest_counts);
    }
    const uint32_t row_vec = hidden_size / 8u;  // uint4 per bf16 row
    if (segment_rows) {
        uint32_t pad_blocks = (world * segment_rows + 7u) / 8u;
        if (pad_blocks > 148u * 8u) pad_blocks = 148u * 8u;
        launch_chained(ep_pad_kernel, dim3(pad_blocks), dim3(256), 0, stream, reinterpret_cast<const uint4*>(hidden), routes,
                       dest_counts, send_source, world, segment_rows, K, row_vec, reinterpret_cast<uint4*>(send_rows),
                       send_routes, send_index, status);
        return;
    }
    sum_counts_kernel<<<1, 32, 0, stream>>>(dest_counts, world, total);
    uint32_t blocks = (count + 7u) / 8u;
    if (blocks > 148u * 8u) blocks = 148u * 8u;
    ep_gather_rows_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uint4*>(hidden), reinterpret_cast<uint4*>(send_rows),
                                                      send_source, total, count, K, row_vec);
}

void launch_ep_unpack(const uint16_t* returned_rows, const uint32_t* send_index, uint32_t tokens, uint32_t K,
                      uint32_t hidden_size, uint16_t* expert_outputs, cudaStream_t stream) {
    const uint32_t count = tokens * K;
    uint32_t blocks = (count + 7u) / 8u;
    if (blocks > 148u * 8u) blocks = 148u * 8u;
    // expert_outputs[t][r] = returned_rows[send_index[t*K + r]]; routes that were dropped give zeros
    launch_chained(ep_gather_rows_kernel, dim3(blocks), dim3(256), 0, stream, reinterpret_cast<const uint4*>(returned_rows),
                   reinterpret_cast<uint4*>(expert_outputs), send_index, (const uint32_t*)nullptr, count, 1u, hidden_size / 8u);
}

void launch_route_compact(const uint32_t* routes, uint32_t* intermediates, const uint32_t* slots,
                          uint32_t slot_words, uint32_t params_per_resource, uint32_t* control,
                          uint32_t max_tokens, uint32_t K, uint32_t intermediate_size,
                          uint32_t tiles_per_route, uint32_t num_experts, const SortScratch& scratch,
                          cudaStream_t stream) {
    const uint32_t count = max_tokens * K;
    const uint32_t buckets = num_experts + 1u;
    if (count <= kSmallSortLimit) {
        uint32_t threads = count <= 256u ? 256u : 1024u;
        const size_t words = rank_block_fits(threads, buckets) ? rank_block_words(threads, buckets) : buckets + 1u;
        launch_chained(compact_small_kernel, dim3(1), dim3(threads), words * sizeof(uint32_t), stream, routes, intermediates, slots,
                       slot_words, params_per_resource, control, max_tokens, K, intermediate_size, tiles_per_route, num_experts);
        return;
    }
    const uint32_t blocks = (count + kSortChunk - 1u) / kSortChunk;
    compact_hist_kernel<<<blocks, 256, buckets * sizeof(uint32_t), stream>>>(
        routes, slots, slot_words, params_per_resource, control, max_tokens, K, num_experts, scratch.block_hist);
    // the partitioned form uses one bucket; scanning all of them costs nothing and needs no host read
    launch_phase_scan(scratch, blocks, buckets, stream);
    compact_scatter_kernel<<<blocks, 256, (buckets + 1u) * sizeof(uint32_t), stream>>>(
        routes, intermediates, slots, slot_words, params_per_resource, control, max_tokens, K,
        intermediate_size, tiles_per_route, num_experts, scratch.block_hist, scratch.bucket_totals);
}

static bool rank_schedule_fits(uint64_t count, uint32_t num_experts) {
    return count <= (uint64_t)kRankChunks * layer_schedule_rank_threads((uint32_t)count) && num_experts < kNotListed - 1u &&
           layer_schedule_rank_smem_bytes((uint32_t)count, num_experts) <= 48u * 1024u;
}

static bool three_sort_schedule_fits(uint64_t count, uint32_t num_experts) {
    return count <= kSmallSortLimit && layer_schedule_smem_bytes((uint32_t)count, num_experts) <= kOneBlockBytes;
}

// Beyond 1280 routes the three launches are cheaper than the one block's longer loop, unless it is a partitioned call or
// the tables of that many experts do not fit. Layer of 384 x 256, three launches / one, us: 1028 routes of 32 experts
// 48.1 / 47.4, 1200 of 128 61.3 / 60.5, 1440 of 129 (512 x 256) 72.8 / 73.0, 1600 of 16 49.3 / 48.6, of 128 60.6 / 61.5,
// 2048 of 32 50.4 / 51.6, 4096 of 128 72.6 / 80.5.
static bool wide_schedule_fits(uint64_t count, uint32_t num_experts, bool partitioned) {
    return count > kWideScheduleRoutes && !partitioned && num_experts < kNotListed - 1u &&
           layer_schedule_wide_smem_bytes(num_experts) <= 48u * 1024u;
}

bool layer_schedule_is_fused(uint32_t tokens, uint32_t K, uint32_t num_experts, bool partitioned) {
    const uint64_t count = (uint64_t)tokens * K;
    return wide_schedule_fits(count, num_experts, partitioned) || rank_schedule_fits(count, num_experts) ||
           three_sort_schedule_fits(count, num_experts);
}

// Calls whose tokens are routed, a warp each, in the blocks that make the operands and the schedule (place_operands_kernel, small_schedule_kernel), or else in
// the schedule's one block (route_schedule_kernel), without a launch of their own. That launch is about a microsecond; the router's own chain grows with the
// experts a lane holds, and the warps of an SM get in each other's way. Layers, us, in these blocks / by a launch of its own, operands beside the schedule: 384 x 256,
// 8 tokens of 32 experts 20.6 / 20.8, 16 20.9 / 20.9, 24 22.2 / 22.3, 32 23.6 / 22.8; 2880 x 2880 8 69.3 / 71.3, 16 80.5 / 81.4, 32 86.6 / 86.4; 12 of 64 22.1 /
// 23.1, 16 22.7 / 22.8, 24 24.4 / 23.7, 32 25.6 / 23.7; 2048 x 256, 8 routes, 16 33.7 / 34.4, 24 37.2 / 34.9; 16 of 128 25.3 / 26.9, 32 27.7 / 28.6. In the schedule's
// block alone: 8 tokens of 32 33.0 / 34.0, 16 34.2 / 35.4, 24 36.4 / 36.1, 32 37.2 / 37.1; 16 of 128 41.9 / 41.8, 24 of 64 39.6 / 38.7, 32 of 128 46.0 / 44.8.
bool layer_routes_in_schedule(const RouterLaunch& router, uint32_t K, uint32_t num_experts) {
    const uint64_t count = (uint64_t)router.tokens * K;
    return router.tokens <= (router.g.routed_experts <= 32u ? 32u : 16u) && router_is_small(router) && count <= 1024u && rank_schedule_fits(count, num_experts);
}

static uint32_t route_schedule_threads(const LayerSchedule& s) {
    const uint32_t count = s.tokens * s.K, warps = s.tokens > (count + 31u) / 32u ? s.tokens : (count + 31u) / 32u;
    return warps <= 8u ? 256u : warps <= 16u ? 512u : 1024u;
}

// A block of the operands' kernel has a warp for every token where it routes them, and as many threads as the schedule's otherwise.
static uint32_t place_operands_threads(const LayerSchedule& s, bool routed) {
    return routed ? route_schedule_threads(s) : layer_schedule_rank_threads(s.tokens * s.K);
}
static size_t place_operands_smem_bytes(const LayerSchedule& s, const OperandRows& o, bool routed) {
    return (2u * (size_t)s.tokens * s.K + 2u * place_words(place_operands_threads(s, routed) / 32u, o.chunks, s.K)) * sizeof(uint32_t);
}

// Which calls. A block ranks the routes of its own tokens, each by a pass over all routes, and a warp stores a piece of a row as often as its token has routes:
// with many routes a token and few pieces a row these take longer than what stands beside them. In turn, the schedule takes the longer the more experts there
// are. `steps` are a warp's passes, in 32 routes. Layers of 64 experts, us, in turn / beside: 16 routes a token 64 tokens of 512 columns (steps 512) 38.1 / 50.8, of 1024
// (288) 42.0 / 47.3, of 2880 (128) 59.6 / 59.7; 12 routes 66 tokens of 2048 (100) 47.1 / 47.4, of 2880 (75) 55.9 / 54.7; 8 routes 128 tokens of 512 (256) 35.6 / 38.6, of
// 1024 (160) 40.1 / 38.7; 4 routes 256 of 512 (128) 37.2 / 35.7; 2 routes 512 (64) 36.1 / 32.1. Of 192 experts: 12 routes 49 tokens of 512 (228) 53.5 / 56.2, 38 of 960 (105)
// 56.9 / 54.3, 20 routes 24 of 2048 (105) 70.4 / 66.9; of 256: 24 routes 9 of 384 (200) 65.3 / 67.5, 2 of 1280 (14) 55.7 / 49.6, 9 routes 90 of 768 (130) 57.2 / 50.8; of 8: 7 routes
// 45 of 512 (70) 27.0 / 28.1. Routed in the same blocks, 64 experts, 32 routes 8 of 512 (256) 38.8 / 44.7, 4 of 2048 (48) 44.2 / 43.4; 16 routes 16 of 512 (128) 33.0 / 34.8, of 1024 (72) 35.0 /
// 34.4; 128 experts, 20 routes 7 of 1472 (50) 42.0 / 39.2, 31 routes 2 of 320 (16) 36.8 / 38.3. Of 1920 layers drawn (1 to 32 routes, 8 to 256 experts, 256 to 4096 columns) the
// rule takes the slower way by more than 1.5 % in 44, at most 6 %. (1024 routes are what a block of the schedule has threads for, one each. 4 routes, 2880 columns, in turn /
// beside: 900 of 32 experts 48.6 / 44.5, 1024 49.7 / 45.1; 900 of 128 102.3 / 96.5, 1024 102.8 / 96.5; in turn 1100 55.7 and 102.1, 1500 61.8 and 105.4, 2000 66.8 and 110.7.)
static bool operands_gain(const LayerSchedule& s, const OperandRows& o, bool routed) {
    const uint32_t count = s.tokens * s.K, warps = place_operands_threads(s, routed) / 32u;
    const uint32_t most = place_words(warps, o.chunks, s.K), routes = most < count ? most : count;
    const uint32_t steps = (routes + warps - 1u) / warps * ((count + 31u) / 32u);
    if (routed) return steps + 2u * s.K <= 50u + s.num_experts / 2u;
    return steps + 6u * s.K <= 60u + s.num_experts + count / 16u;
}

bool places_operands(const LayerSchedule& s, bool routed, const OperandRows& o, uint32_t block) {
    const uint64_t count = (uint64_t)s.tokens * s.K;
    return s.expert_count == 0u && count <= 1024u && small_schedule_words((uint32_t)count, s.num_experts) <= 12u * 1024u &&
           (block == 32u || block == 128u) && o.cols % block == 0u && (reinterpret_cast<uintptr_t>(o.input) & 15u) == 0u &&
           place_operands_smem_bytes(s, o, routed) <= 48u * 1024u && operands_gain(s, o, routed);
}

void launch_place_operands(const RouterLaunch* router, const LayerSchedule& s, const OperandRows& o, uint32_t block, cudaStream_t stream) {
    const uint32_t threads = place_operands_threads(s, router != nullptr), warps = threads / 32u;
    const int epl = !router ? 0 : router->g.routed_experts <= 32u ? 1 : 4;
    const auto kernel = block == 32u ? (epl == 0 ? place_operands_kernel<0, 2u> : epl == 1 ? place_operands_kernel<1, 2u> : place_operands_kernel<4, 2u>)
                                     : (epl == 0 ? place_operands_kernel<0, 8u> : epl == 1 ? place_operands_kernel<1, 8u> : place_operands_kernel<4, 8u>);
    launch_chained(kernel, dim3((s.tokens * o.chunks + warps - 1u) / warps), dim3(threads), place_operands_smem_bytes(s, o, router != nullptr), stream,
                   router ? *router : RouterLaunch{}, s, o);
}

void launch_small_schedule(const RouterLaunch* router, const LayerSchedule& s, cudaStream_t stream) {
    const int epl = !router ? 0 : router->g.routed_experts <= 32u ? 1 : 4;
    launch_chained(epl == 0 ? small_schedule_kernel<0> : epl == 1 ? small_schedule_kernel<1> : small_schedule_kernel<4>, dim3(1),
                   dim3(place_operands_threads(s, router != nullptr)), small_schedule_words(s.tokens * s.K, s.num_experts) * sizeof(uint32_t), stream,
                   router ? *router : RouterLaunch{}, s);
}

void launch_route_schedule(const RouterLaunch& router, const LayerSchedule& s, cudaStream_t stream) {
    const uint32_t count = s.tokens * s.K;
    launch_chained(router.g.routed_experts <= 32u ? route_schedule_kernel<1> : route_schedule_kernel<4>, dim3(1),
                   dim3(route_schedule_threads(s)), layer_schedule_rank_smem_bytes(count, s.num_experts), stream, router, s);
}

uint32_t launch_layer_schedule(const LayerSchedule& s, const SortScratch& scratch, cudaStream_t stream) {
    const uint32_t count = s.tokens * s.K;
    if (wide_schedule_fits(count, s.num_experts, s.expert_count != 0u)) {
        const uint32_t blocks = (count + kSortChunk - 1u) / kSortChunk, buckets = s.num_experts + 1u;
        launch_chained(layer_schedule_hist_kernel, dim3(blocks), dim3(256), buckets * sizeof(uint32_t), stream, s, scratch.block_hist);
        launch_phase_scan(scratch, blocks, buckets, stream);
        launch_chained(layer_schedule_scatter_kernel, dim3(blocks), dim3(256), layer_schedule_wide_smem_bytes(s.num_experts), stream, s,
                       scratch.block_hist, scratch.bucket_totals);
        return 3u;
    }
    if (rank_schedule_fits(count, s.num_experts)) {
        const uint32_t threads = layer_schedule_rank_threads(count);
        const uint32_t chunks = (count + threads - 1u) / threads;
        auto kernel = chunks <= 1u ? layer_schedule_rank_kernel<1> : chunks <= 4u ? layer_schedule_rank_kernel<4>
                                                                                  : layer_schedule_rank_kernel<kRankChunks>;
        launch_chained(kernel, dim3(1), dim3(threads),
                       layer_schedule_rank_smem_bytes(count, s.num_experts), stream, s);
        return 1u;
    }
    launch_chained(layer_schedule_small_kernel, dim3(1), dim3(count <= 256u ? 256u : 1024u),
                   layer_schedule_smem_bytes(count, s.num_experts), stream, s);
    return 1u;
}

void launch_route_count(const uint32_t* routes, const uint32_t* slots, uint32_t slot_words,
                        uint32_t params_per_resource, uint32_t* control, uint32_t max_tokens, uint32_t K,
                        uint32_t tiles_per_route, cudaStream_t stream) {
    launch_chained(route_count_kernel, dim3(1), dim3(1024), 0, stream, routes, slots, slot_words, params_per_resource, control, max_tokens, K,
                   tiles_per_route);
}

void launch_resolve_experts(const uint32_t* addresses, uint32_t address_words, const uint32_t* slots,
                            uint32_t slot_words, uint32_t params_per_resource, uint32_t num_experts,
                            uint32_t rows, uint32_t cols, uint32_t native_start, bool whole_blocks_only,
                            uint8_t* derived_scales, size_t derived_matrix_bytes, ExpertPtrs* out, cudaStream_t stream) {
    resolve_experts_kernel<<<(num_experts + 127u) / 128u, 128, 0, stream>>>(
        addresses, address_words, slots, slot_words, params_per_resource, num_experts, rows, cols, native_start,
        whole_blocks_only, derived_scales, derived_matrix_bytes, out);
}

uint32_t launch_group_slots(const uint32_t* routes, const uint32_t* intermediates, const uint32_t* control,
                        const ExpertPtrs* experts, uint32_t num_experts, uint32_t max_tokens, uint32_t K,
                        uint32_t intermediate_size, uint32_t* grouped_routes, uint32_t* expert_offsets,
                        uint32_t* position, const TileOut& tiles, uint32_t* status, const SortScratch& scratch,
                        cudaStream_t stream) {
    const uint32_t data_words = K * (intermediate_size / 2u);
    SlotKey key{routes, intermediates, experts, status, num_experts, K, data_words + K, data_words, 0u};
    const uint32_t count = max_tokens * K;
    if (count <= kSmallSortLimit) {
        uint32_t threads = count <= 256u ? 256u : 1024u;
        const size_t words = rank_block_fits(threads, num_experts) ? rank_block_words(threads, num_experts) : num_experts + 1u;
        launch_chained(group_small_kernel, dim3(1), dim3(threads), words * sizeof(uint32_t), stream, key, control, max_tokens,
                       grouped_routes, expert_offsets, position, tiles);
        return 1u;
    }
    const uint32_t blocks = (count + kSortChunk - 1u) / kSortChunk;
    group_hist_kernel<<<blocks, 256, num_experts * sizeof(uint32_t), stream>>>(key, control, max_tokens,
                                                                               scratch.block_hist, position);
    launch_phase_scan(scratch, blocks, num_experts, stream);
    group_scatter_kernel<<<blocks, 256, (num_experts + 1u) * sizeof(uint32_t), stream>>>(
        key, control, max_tokens, grouped_routes, expert_offsets, scratch.block_hist, scratch.bucket_totals, position);
    if (!tiles.list) return 3u;
    launch_chained(build_tiles_kernel, dim3(1), dim3(1024), 0, stream, expert_offsets, num_experts, tiles.n_tile, tiles.list, tiles.count);
    return 4u;
}

}  // namespace nvmoe
