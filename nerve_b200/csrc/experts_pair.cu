// The grouped expert projections by CTA pairs (tcgen05 cta_group::2), for calls with many tokens per expert.
//
// Arithmetic, operands and results are those of experts_tc.cu. What differs is the tile: two CTAs of a cluster work on one
// D[256 weight rows x up to 240 tokens], each with 128 of the rows and half of the tokens in its shared memory; the tensor
// cores of both read the other's token rows through the pair. What bounds the one-CTA kernel with large batches is its
// shared memory: for 256 rows x 128 tokens x 128 columns the MMAs read 64 KB and the copies write 48 KB (the 4-bit codes take
// a byte each), 900 cycles at 128 bytes a clock beside 512 cycles of MMAs. A CTA of a pair does the same work with 32 KB
// read and 32 KB written, and fetches 25 KB from L2 instead of 33.5.
//
// Gate/up: CTA 0 holds gate rows, CTA 1 the up rows of the same index; each takes half of the tokens through the activation
// and sends the other half of its accumulators, rounded to bf16 as the activation reads them, to the other CTA's shared
// memory. Down: the CTAs hold neighbouring 128-row tiles and have nothing to exchange.
//
// 240 columns: two accumulators of them and two sets of scales are 504 of the 512 columns of tensor memory. (256 columns,
// with accumulators that share some, stop the MMAs at the end of every tile until the shared columns have been read.) A tile
// with fewer tokens runs with fewer columns.
//
// A stage is two K blocks, four copies: with one block a stage the lane that issues them and the one that issues the MMAs take
// longer for a stage than the tensor cores. All operands come by TMA, a trailing half K block too (a stage of its own: a
// whole block that ends with the row, of which only the second half is multiplied), credited to the barrier of CTA 0, whose
// MMA thread feeds both. Only the token scales pass through
// a warp: they lie as [K block][row], a tile's start at any row, and the 32 x 16-byte block that tcgen05.cp expands wants
// four tokens, 32 apart, side by side; a warp of either CTA puts them there, in place, and arrives at CTA 0. All waits are
// bounded (tcgen05.cuh); a CTA leaves only when both are done.
#include <cuda.h>
#include <cuda_fp8.h>

#include <cstddef>
#include <cstring>

#include "experts_device.cuh"
#include "experts_tc.cuh"
#include "quantize.cuh"
#include "tcgen05.cuh"

namespace nvmoe {
namespace {

using namespace tc;

constexpr uint32_t kPairEpilogueGroups = 4u;                            // of four warps, one per quadrant of tensor-memory lanes
constexpr uint32_t kPairEpilogueWarps = 4u * kPairEpilogueGroups;
constexpr uint32_t kPairMmaWarp = kPairEpilogueWarps, kPairTmaWarp = kPairMmaWarp + 1u, kPairInfoWarp = kPairTmaWarp + 1u;
constexpr uint32_t kPairScaleWarp = kPairInfoWarp + 1u;
constexpr uint32_t kPairThreads = 32u * (kPairScaleWarp + 1u);
constexpr uint32_t kPairWatchWarp = 2u;                                 // polls for a finished accumulator (shares no scheduler with MMA and TMA)
constexpr uint32_t kPairColumns = kPairTokens;
// Slots of the ring: three of 240 columns; four of 128 where nothing is exchanged, for calls whose list has no wider tiles (a
// slot is held for about two microseconds, most of it latency, so that the narrower stages wait for the ring: dense block of
// 777 rows of 7168 x 2048 98.7 us with three, 94.7 with four, of 100 rows 68.8 / 63.4; 2000 rows, wider tiles, 155.9 / 156.4).
constexpr uint32_t kPairStages = 3u, kPairNarrowStages = 4u, kPairNarrowTokens = 128u;
constexpr uint32_t kPairBlocks = 2u;                                     // K blocks a stage
constexpr uint32_t kPairTokenBytes = kPairColumns / 2u * 128u;          // token rows of one K block in one CTA
// a stage's weight scales, then its token scales: as they come, 244 words a K block, then as two blocks of 512 bytes each
constexpr uint32_t kPairScaleBytes = kPairBlocks * 3u * kScaleBlockBytes;
constexpr uint32_t kPairScaleWords = kPairTokens + 4u;
static_assert(kPairTokenBytes % 1024u == 0u, "operand tiles keep their alignment");
constexpr uint32_t kPairScaleColumn = 2u * kPairColumns, kPairScaleColumns = 12u;  // of either set: 4 for the weights, 8 for the tokens
constexpr uint32_t kPairTmemColumns = 512u;
static_assert(kPairScaleColumn + 2u * kPairScaleColumns <= kPairTmemColumns, "tensor memory");

struct PairBarriers {
    uint64_t full[kPairNarrowStages];    // CTA 0's count
    uint64_t empty[kPairNarrowStages];
    uint64_t staged[kPairNarrowStages];  // the token scales of a slot are there, as they lie in memory
    uint64_t acc_full[2];
    uint64_t acc_empty[2];         // CTA 0's
    uint64_t info_full[2];         // what the epilogue has to know of a tile is there
    uint64_t info_empty[2];
    uint64_t drain;
    uint64_t sent[kPairEpilogueWarps];    // the other CTA's warp has written its chunk
    uint64_t taken[kPairEpilogueWarps];   // ... has read the chunk this warp sent
    uint32_t tmem_base;
    uint32_t abort;
    uint32_t stage_info[kPairNarrowStages];     // of the tile whose operands a slot holds: format << 16 | first row % 4 << 12 | columns
    uint32_t acc_ready[2];
    // per tile, alternating: its tokens, its row tile, and per column the route (0xffffffff: no token) with its down row
    // (gate/up) or its weight (down)
    uint32_t tile_tokens[2], tile_rows[2];
    __align__(16) uint32_t route[2][256];
    __align__(16) uint32_t extra[2][256];
    uint32_t maxima[kPairEpilogueGroups][2][4][8];  // [group][chunk, alternating][lane quadrant][tokens in pairs], bf16
};
constexpr uint32_t kPairExchangeBytes = kPairEpilogueWarps * 1024u;     // 16 columns x 32 rows of bf16 a warp
constexpr uint32_t kPairExchangeRegion = kPairStages * (kPairBlocks * (kATileBytes + kPairTokenBytes) + kPairScaleBytes);
constexpr uint32_t kPairBarrierRegion = kPairExchangeRegion + kPairExchangeBytes;
constexpr uint32_t kPairSmemBytes = kPairBarrierRegion + sizeof(PairBarriers) + 1024u;  // (the round-up to a 1024-byte boundary)
static_assert(kPairSmemBytes <= 227u * 1024u && kPairBarrierRegion % 128u == 0u, "shared memory");
static_assert(kPairNarrowStages * (kPairBlocks * (kATileBytes + kPairNarrowTokens / 2u * 128u) + kPairScaleBytes) <= kPairBarrierRegion, "narrow slots");

__device__ __forceinline__ uint32_t bf16x2_bits(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {  // (the number where the other is none)
    const __nv_bfloat162 v = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float low_bf16(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float high_bf16(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }

// Columns the MMAs take for a tile of that many tokens, in sixteens: what the tensor cores draw bounds large calls (the clock stands at
// 1.25 to 1.6 GHz in them, also in a call by itself). In 64s with 240 the last step: 8192 tokens of 128 experts 1.7 % more, 4096 of 32 and
// 16384 of 256 half a percent. And the tokens that are fetched: the tensor maps of the token rows have boxes of half of 64, 128, 192, 240.
__device__ __forceinline__ uint32_t columns_for(uint32_t tokens) { return tokens <= 32u ? 32u : (tokens + 15u) & ~15u; }
__device__ __forceinline__ uint32_t fetched_for(uint32_t columns) { return columns <= 64u ? 64u : columns <= 128u ? 128u : columns <= 192u ? 192u : kPairColumns; }

// DENSE: one matrix, whose tensor maps come with the launch and whose tiles follow from its sizes, so that nothing has to be acquired or looked up
// when the launch ahead (which quantises the tokens and re-tiles the scales) is through: its SMs are taken over by CTAs that have all of their set-up still
// to do, and the first stage came 4.2 us after their start, of which the maps 1.0 and the list 0.7. The weights of the first stages are asked for before the
// wait, while tensor memory is allocated. With that, barriers that the lanes of a warp set up and sums stored two rows at a time (below), us a call before / after: 100
// rows of 7168 columns to 2048 18.0 / 17.1, 777 24.1 / 22.9, 4096 68.6 / 64.3; of 2048 to 7168 11.7 / 10.6, 23.1 / 19.1, 70.7 / 55.2.
template <bool DENSE>
struct PairMaps {};
template <>
struct PairMaps<true> {
    CUtensorMap weights[2];  // boxes of one K block, of two
};
template <bool GATE_UP, bool DENSE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1) experts_pair_kernel(ExpertLaunch p, TileList list, const __grid_constant__ PairMaps<DENSE> maps) {
    const uint8_t* const dense_maps = DENSE ? reinterpret_cast<const uint8_t*>(&maps) : nullptr;
    const long long wait_limit = p.wait_cycles;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    PairBarriers* bars = reinterpret_cast<PairBarriers*>(smem + kPairBarrierRegion);
    volatile uint32_t* abort_flag = &bars->abort;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = cluster_rank();
    const uint32_t pair_id = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t H = p.g.hidden_size, I = p.g.intermediate_size;
    const uint32_t K = p.g.routed_k + p.g.always_count;
    const uint32_t k_dim = GATE_UP ? H : I;
    const uint32_t out_rows = GATE_UP ? I : H;
    const uint32_t k_blocks = (k_dim + kBlockK - 1u) / kBlockK;
    const uint32_t row_tiles = (out_rows + kBlockM - 1u) / kBlockM;
    // stages of a tile: two whole K blocks each, then a whole one and a trailing half one by themselves
    const uint32_t doubles = k_dim / kBlockK / 2u, stages = doubles + (k_blocks - 2u * doubles);
    const uint32_t m_tiles = GATE_UP ? row_tiles : (row_tiles + 1u) / 2u;
    constexpr uint32_t kSources = GATE_UP ? 2u : 1u;

    // the ring: weight tiles, token tiles, scales, each an array over (slot, K block)
    const bool narrow = !GATE_UP && p.token_rows <= kPairNarrowTokens;
    const uint32_t slots = narrow ? kPairNarrowStages : kPairStages;
    const uint32_t token_bytes = narrow ? kPairNarrowTokens / 2u * 128u : kPairTokenBytes;
    const uint32_t token_region = slots * kPairBlocks * kATileBytes, scale_region = token_region + slots * kPairBlocks * token_bytes;

    // ---- one-time setup (the barriers by the lanes of a warp: one after the other they took half a microsecond) -----------------
    if (warp == 0u) {
        uint64_t* all = bars->full;
        constexpr uint32_t kSlots = kPairNarrowStages, kAcc = 3u * kSlots, kDrain = kAcc + 8u, kCount = kDrain + 1u + 2u * kPairEpilogueWarps;
        static_assert(offsetof(PairBarriers, tmem_base) == kCount * 8u, "the barriers come first and in this order");
        for (uint32_t i = lane; i < kCount; i += 32u) {
            uint32_t arrivals = 1u;
            if (i < kSlots) arrivals = 3u;                                               // full: the announcement of the copies, the scale warps of both CTAs
            if (i >= kAcc + 2u && i < kAcc + 4u) arrivals = 2u * kPairEpilogueWarps;     // acc_empty
            if (i >= kAcc + 4u && i < kAcc + 6u) arrivals = 32u;                         // info_full
            if (i >= kAcc + 6u && i < kDrain) arrivals = kPairEpilogueWarps;             // info_empty
            mbar_init(all + i, arrivals);
        }
        if (lane == 0u) bars->abort = 0u;
        fence_mbar_init();
    }
    __syncwarp();
    cluster_sync();  // the barriers of both CTAs are up before either arrives on the other's
    // a stage's weights; CTA 0 announces with them what both CTAs fetch for it
    auto load_weights = [&](uint32_t st, uint32_t into, const uint8_t* weight_map, int row0, uint32_t bytes) {
        const bool two = st < doubles;
        const uint32_t kb = two ? 2u * st : doubles + st, at = smem_u32(smem) + into * kPairBlocks * kATileBytes, bar = map_shared(smem_u32(&bars->full[into]), 0u);
        if (rank == 0u) mbar_arrive_expect_tx(&bars->full[into], (two ? 2u * bytes : bytes) + 2u * kPairBlocks * kScaleBlockBytes);
        if (two) {
            tma_load_3d_pair(at, weight_map + 128u, 0, row0, (int)kb, bar);
        } else {
            tma_load_3d_pair(at, weight_map, 0, (int)min(2u * kb, k_dim / 64u - 2u), row0, bar);  // in units of 64 columns: a trailing half block ends with the row
        }
    };
    // DENSE: stages of the first tile whose weights are on their way before the wait
    const uint32_t dense_tiles = DENSE ? (p.tokens + p.token_rows - 1u) / p.token_rows * m_tiles : 0u;
    const uint32_t ahead = pair_id < dense_tiles ? min(slots, stages) : 0u;
    const bool withheld = blockIdx.x < 2u && ((p.debug_flags >> blockIdx.x) & 1u) != 0u;  // (debug) the first stage is left out
    if (DENSE && warp == kPairTmaWarp && lane == 0u && ahead != 0u) {
        const uint32_t first = pair_id / m_tiles * p.token_rows, columns = columns_for(min(p.token_rows, p.tokens - first));
        for (uint32_t st = withheld ? 1u : 0u; st < ahead; st++)
            load_weights(st, st, dense_maps, (int)((2u * (pair_id % m_tiles) + rank) * kBlockM), 2u * (kTmaBoxBytes + fetched_for(columns) / 2u * 128u));
    }
    __syncwarp();
    if (warp == kPairMmaWarp) {
        tmem_alloc_pair(&bars->tmem_base, kPairTmemColumns);
        tmem_relinquish_pair();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t tmem_scales = tmem_base + kPairScaleColumn;
    auto acquire_maps = [&] {  // (a tensor map written by an earlier kernel is acquired once per block before the TMA unit gets it)
        // (13 to 29 ns a map, one after the other: of gate and up the CTA's own, of the maps of two K blocks and of one those that a row has. Layers, us, all /
        // these: 8192 tokens of 256 experts of 2048 x 512 313.4 / 294.5, of 128 of 1024 x 1024 232.6 / 224.7, 6000 of 128 of 2048 x 2048 396.6 / 391.5)
        for (uint32_t m = threadIdx.x; m < p.work.num_experts; m += blockDim.x) {
            const uint8_t* maps = p.tmaps + (size_t)(GATE_UP ? 2u * m + rank : m) * kWeightMaps * 128u;
            if (doubles != 0u) tensormap_acquire(maps + 128u);
            if (stages != doubles) tensormap_acquire(maps);
        }
        if (threadIdx.x == kActMaps) tensormap_acquire(p.tmaps + (size_t)p.work.num_experts * kSources * kWeightMaps * 128u);  // the derived scales'
        if (threadIdx.x < kActMaps - 1u) tensormap_acquire(p.act_tmap + threadIdx.x * 128u);
        __syncthreads();
    };
    if (DENSE) {  // (those that stand)
        if (threadIdx.x < kActMaps - 1u) tensormap_acquire(p.act_tmap + threadIdx.x * 128u);
        if (threadIdx.x == kActMaps) tensormap_acquire(p.tmaps + (size_t)kWeightMaps * 128u);
        __syncthreads();
    } else if (!p.fresh_maps) {
        acquire_maps();  // as in experts_tc.cu: while the kernel ahead still runs
    }
    grid_dependency_sync();
    const uint32_t first_entry = !DENSE && warp == kPairTmaWarp ? __ldg(list.tiles + min(pair_id / m_tiles, p.tile_capacity - 1u)) : 0u;
    const uint32_t tile_count = DENSE ? dense_tiles : *list.count * m_tiles;
    if (!DENSE && p.fresh_maps) acquire_maps();

    // first row of a tile in the operand matrix, and how many rows it has
    auto first_row_of = [&](uint32_t n_tile, uint32_t e_begin) { return e_begin + n_tile * p.token_rows; };

    if (warp == kPairTmaWarp) {
        // ===== TMA issue (one lane of each CTA) =====
        if (lane == 0u) {
            // the list entry of a tile is fetched two tiles ahead, what hangs on it one tile ahead (loads only: a thread
            // stalls at the first instruction that needs a result)
            struct Meta {
                uint32_t pair, m_tile, e_begin, e_end, format;
            };
            auto entry_of = [&](uint32_t tile) { return !DENSE && tile < tile_count ? __ldg(list.tiles + tile / m_tiles) : 0u; };
            auto meta_of = [&](uint32_t tile, uint32_t pair, Meta& m) {
                m.pair = DENSE ? tile / m_tiles : pair;
                m.m_tile = tile % m_tiles;
                if (DENSE) {
                    m.e_begin = 0u;
                    m.e_end = p.tokens;
                    m.format = kFormatCompact;
                    return;
                }
                m.e_begin = __ldg(p.work.expert_offsets + (pair >> 16));
                m.e_end = __ldg(p.work.expert_offsets + (pair >> 16) + 1u);
                m.format = p.work.experts[pair >> 16].format;
            };
            const uint64_t begin = p.cta_trace ? global_timer_ns() : 0u;
            const uint32_t smem_base = smem_u32(smem), full0 = map_shared(smem_u32(&bars->full[0]), 0u);
            const uint8_t* scale_map = p.tmaps + (size_t)p.work.num_experts * kSources * kWeightMaps * 128u;
            const uint8_t* token_scale_map = p.act_tmap + (kTokenScaleMap - 1u) * 128u;
            uint32_t slot = 0u, empty_parity = 1u, stage_it = 0u;
            bool alive = true, withhold = withheld;
            Meta cur{}, nxt{};
            if (pair_id < tile_count) meta_of(pair_id, first_entry, cur);
            uint32_t pair_nxt = entry_of(pair_id + pairs);
            for (uint32_t tile = pair_id; tile < tile_count && alive; tile += pairs) {
                const uint32_t pair_nxt2 = entry_of(tile + 2u * pairs);
                if (tile + pairs < tile_count) meta_of(tile + pairs, pair_nxt, nxt);
                const uint32_t expert = DENSE ? 0u : cur.pair >> 16;
                const uint32_t first = first_row_of(DENSE ? cur.pair : cur.pair & 0xffffu, cur.e_begin);
                const uint32_t columns = columns_for(min(p.token_rows, cur.e_end - first));
                const uint8_t* weight_map = DENSE ? dense_maps : p.tmaps + (size_t)(GATE_UP ? 2u * expert + rank : expert) * kWeightMaps * 128u;
                const uint8_t* token_map = p.act_tmap + (columns - 1u) / 64u * 128u;
                const int row0 = (int)(GATE_UP ? cur.m_tile * kBlockM : (2u * cur.m_tile + rank) * kBlockM);
                // (a second tile past the last rows borrows the first's scale blocks: its weights arrive as zeros)
                const uint32_t row_tile = GATE_UP ? cur.m_tile : min(2u * cur.m_tile + rank, row_tiles - 1u);
                const int scale0 = (int)((expert * row_tiles + row_tile) * k_blocks), source = GATE_UP ? (int)rank : 0;
                const int token_row = (int)(first + rank * columns / 2u);
                const uint32_t box_bytes = cur.format == kFormatCompact ? kTmaBoxBytes : 2u * kTmaBoxBytes;
                const uint32_t block_bytes = 2u * (box_bytes + fetched_for(columns) / 2u * 128u);  // of both CTAs
                const uint32_t info = (cur.format << 16) | (first & 3u) << 12 | columns;
                for (uint32_t st = 0; st < stages; st++) {
                    if (!mbar_wait(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    const bool two = st < doubles;
                    const uint32_t kb = two ? 2u * st : doubles + st;
                    const uint32_t bar = full0 + slot * 8u;
                    *reinterpret_cast<volatile uint32_t*>(&bars->stage_info[slot]) = info;
                    if (!withhold) {
                        const uint32_t b = smem_base + token_region + slot * kPairBlocks * token_bytes;
                        const uint32_t sf = smem_base + scale_region + slot * kPairScaleBytes;
                        // the token scales first, which have the longest way to go (of one block, too, the scales of two are
                        // fetched: zeros, or the next row tile's, that nothing uses)
                        mbar_arrive_expect_tx(&bars->staged[slot], kPairBlocks * kPairScaleWords * 4u);
                        tma_load_2d(sf + kPairBlocks * kScaleBlockBytes, token_scale_map, (int)(first & ~3u), (int)kb, &bars->staged[slot]);
                        if (tile != pair_id || st >= ahead) load_weights(st, slot, weight_map, row0, block_bytes);
                        if (two) {
                            tma_load_3d_pair(b, token_map + kTokenMaps * 128u, 0, token_row, (int)kb, bar);
                        } else {
                            // in units of 64 columns: a trailing half block ends with the row
                            tma_load_2d_pair(b, token_map, (int)(min(2u * kb, k_dim / 64u - 2u) * 64u), token_row, bar);
                        }
                        tma_load_3d_pair(sf, scale_map, 0, source, scale0 + (int)kb, bar);
                    }
                    withhold = false;
                    stage_it++;
                    if (++slot == slots) {
                        slot = 0u;
                        empty_parity ^= 1u;
                    }
                }
                cur = nxt;
                pair_nxt = pair_nxt2;
            }
            if (p.cta_trace) {  // per-CTA diagnostics: loop begin, loop end, stages, SM id
                uint32_t smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                uint64_t* mine = p.cta_trace + (size_t)((GATE_UP ? 0u : gridDim.x) + blockIdx.x) * 4u;
                mine[0] = begin;
                mine[1] = global_timer_ns();
                mine[2] = stage_it;
                mine[3] = smid;
            }
        }
        __syncwarp();
    } else if (warp == kPairMmaWarp) {
        // ===== MMA issue (one lane of CTA 0, for both) =====
        if (rank == 0u && elect_one()) {
            constexpr uint32_t kIdescCompact = idesc_mxf8f6f4(kFmtE2M1, kFmtE4M3, 2u * kBlockM, 0u);
            constexpr uint32_t kIdescBytes = idesc_mxf8f6f4(kFmtE4M3, kFmtE4M3, 2u * kBlockM, 0u);
            const uint32_t base = smem_u32(smem);
            const uint64_t a_desc0 = desc_k_major_sw128(base);
            const uint64_t b_desc0 = desc_k_major_sw128(base + token_region);
            const uint64_t sf_desc0 = desc_scale_block(base + scale_region);
            const uint32_t tail_groups = (k_dim % kBlockK) / 32u;  // K steps of a trailing partial block, 0 = none
            uint32_t acc_it = 0u, slot = 0u, full_parity = 0u;
            bool alive = true;
            for (uint32_t tile = pair_id; tile < tile_count && alive; tile += pairs, acc_it++) {
                const uint32_t acc = acc_it & 1u;
                if (!mbar_wait(&bars->acc_empty[acc], ((acc_it >> 1) & 1u) ^ 1u, abort_flag, wait_limit)) break;
                const uint32_t d_tmem = tmem_base + acc * kPairColumns;
                for (uint32_t st = 0; st < stages; st++) {
                    if (!mbar_wait(&bars->full[slot], full_parity, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    const uint32_t info = *reinterpret_cast<volatile uint32_t*>(&bars->stage_info[slot]);
                    const uint32_t columns = info & 0xfffu;
                    tc_fence_after();
                    const uint32_t idesc = ((info >> 16) == kFormatCompact ? kIdescCompact : kIdescBytes) | (columns >> 3) << 17;
                    // (a trailing half block lies in the second half of its operand tiles; its scales come first in their words)
                    const uint32_t groups = st + 1u == stages && tail_groups != 0u ? tail_groups : 4u;
                    const uint32_t first = 2u * (4u - groups);  // a K step of 32 elements is two 16-byte units of the start address
#pragma unroll
                    for (uint32_t sub = 0; sub < kPairBlocks; sub++) {
                        if (sub != 0u && st >= doubles) break;
                        const uint32_t sfa = tmem_scales + sub * kPairScaleColumns, sfb = sfa + 4u;
                        const uint64_t sf_desc = sf_desc0 + (uint64_t)(slot * (kPairScaleBytes >> 4));
                        const uint64_t sfb_desc = sf_desc + (kPairBlocks + 2u * sub) * (kScaleBlockBytes >> 4);
                        tc_copy_scales_pair(sfa, sf_desc + sub * (kScaleBlockBytes >> 4));
                        tc_copy_scales_pair(sfb, sfb_desc);
                        if (columns > 128u) tc_copy_scales_pair(sfb + 4u, sfb_desc + (kScaleBlockBytes >> 4));
                        const uint64_t a_desc = a_desc0 + (uint64_t)((slot * kPairBlocks + sub) * (kATileBytes >> 4) + first);
                        const uint64_t b_desc = b_desc0 + (uint64_t)(slot * kPairBlocks * (token_bytes >> 4) + sub * (fetched_for(columns) << 2) + first);
#pragma unroll
                        for (uint32_t j = 0; j < 4u; j++) {
                            if (j < groups)
                                tc_mma_block_scaled_pair(d_tmem, a_desc + 2u * j, b_desc + 2u * j, idesc | (j << 4) | (j << 29), sfa, sfb,
                                                         j == 0u && sub == 0u ? (st != 0u ? 1u : 0u) : 1u);
                        }
                    }
                    tc_commit_pair_both(&bars->empty[slot]);
                    if (++slot == slots) {
                        slot = 0u;
                        full_parity ^= 1u;
                    }
                }
                if (alive) tc_commit_pair_both(&bars->acc_full[acc]);
            }
            // (nothing may still be reading either CTA's shared memory or using tensor memory when they are released)
            tc_commit_pair(&bars->drain);
            mbar_wait_winddown(&bars->drain, 0u, kWinddownCycles);
        }
        __syncwarp();
    } else if (warp == kPairScaleWarp) {
        // ===== token scales: in place, from row order to the two 32 x 16-byte blocks =====
        const uint32_t full0 = map_shared(smem_u32(&bars->full[0]), 0u);
        uint32_t slot = 0u, parity = 0u;
        bool alive = true;
        for (uint32_t tile = pair_id; tile < tile_count && alive; tile += pairs) {
            for (uint32_t st = 0; st < stages; st++) {
                if (!mbar_wait_warp(&bars->staged[slot], parity, abort_flag, wait_limit)) {
                    alive = false;
                    break;
                }
                uint32_t* words = reinterpret_cast<uint32_t*>(smem + scale_region + slot * kPairScaleBytes + kPairBlocks * kScaleBlockBytes);
                const uint32_t info = *reinterpret_cast<volatile uint32_t*>(&bars->stage_info[slot]);
                const volatile uint32_t* mine = words + ((info >> 12) & 3u) + lane;
                uint32_t w[kPairBlocks][8];
#pragma unroll
                for (uint32_t sub = 0; sub < kPairBlocks; sub++) {
#pragma unroll
                    for (uint32_t i = 0; i < 8u; i++) w[sub][i] = mine[sub * kPairScaleWords + 32u * i];  // (past the columns: not multiplied with)
                }
                __syncwarp();
#pragma unroll
                for (uint32_t sub = 0; sub < kPairBlocks; sub++) {
                    reinterpret_cast<uint4*>(words)[64u * sub + lane] = make_uint4(w[sub][0], w[sub][1], w[sub][2], w[sub][3]);
                    reinterpret_cast<uint4*>(words)[64u * sub + 32u + lane] = make_uint4(w[sub][4], w[sub][5], w[sub][6], w[sub][7]);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0u) mbar_arrive_cluster(full0 + slot * 8u);
                if (++slot == slots) {
                    slot = 0u;
                    parity ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == kPairInfoWarp) {
        // ===== what the epilogue has to know of a tile: fetched a tile ahead, the chain of four dependent loads (list entry,
        // expert offsets, route, its weight or row) would otherwise be the longest part of an epilogue =====
        uint32_t acc_it = 0u;
        for (uint32_t tile = pair_id; tile < tile_count; tile += pairs, acc_it++) {
            const uint32_t buffer = acc_it & 1u;
            const uint32_t pair = DENSE ? tile / m_tiles : __ldg(list.tiles + tile / m_tiles), expert = pair >> 16;
            const uint32_t first = DENSE ? first_row_of(pair, 0u) : first_row_of(pair & 0xffffu, __ldg(p.work.expert_offsets + expert));
            const uint32_t tokens = min(p.token_rows, (DENSE ? p.tokens : __ldg(p.work.expert_offsets + expert + 1u)) - first);
            uint32_t route[8], extra[8];
#pragma unroll
            for (uint32_t i = 0; i < 8u; i++)
                route[i] = 32u * i + lane < tokens ? (DENSE ? first + 32u * i + lane : __ldg(p.work.grouped_routes + first + 32u * i + lane)) : kUnboundSlot;
#pragma unroll
            for (uint32_t i = 0; i < 8u; i++) {
                extra[i] = DENSE ? 0x3f800000u : kUnboundSlot;
                if (DENSE || route[i] == kUnboundSlot) continue;
                if (GATE_UP) {
                    if (p.q_out != nullptr) extra[i] = __ldg(p.down_position + route[i]);
                } else {
                    extra[i] = __ldg(p.routes + route[i]) & 0xffff0000u;  // the bf16 weight as f32
                }
            }
            if (!mbar_wait_warp(&bars->info_empty[buffer], ((acc_it >> 1) & 1u) ^ 1u, abort_flag, wait_limit)) break;
#pragma unroll
            for (uint32_t i = 0; i < 8u; i++) {
                bars->route[buffer][32u * i + lane] = route[i];
                bars->extra[buffer][32u * i + lane] = extra[i];
            }
            if (lane == 0u) {
                bars->tile_tokens[buffer] = tokens;
                bars->tile_rows[buffer] = tile % m_tiles;
            }
            mbar_arrive(&bars->info_full[buffer]);
        }
        __syncwarp();
    } else {
        // ===== epilogue: TMEM -> registers -> global =============================================
        // Sixteen tokens at a time go through each step together, without a branch, so that the latencies of their
        // instructions overlap: columns without a token hold zeros or what is left of others and are only not stored.
        const uint32_t quad = warp & 3u, group = warp >> 2;
        const uint32_t frame_words = K * (I / 2u) + K;
        const bool whole_block = GATE_UP && p.g.act_block == 128u;
        const bool quantise = GATE_UP && p.q_out != nullptr;             // host: only with scale blocks of 32 or 128 rows
        const bool store_rows = !GATE_UP || p.intermediates != nullptr;
        const bool words_of_rows = !GATE_UP && p.partial_outputs == nullptr && ((reinterpret_cast<uintptr_t>(p.outputs) | (2u * H)) & 3u) == 0u;  // (uniform)
        uint32_t acc_it = 0u, sends = 0u, receipts = 0u, set_it = 0u;
        // this warp's place in the exchange: its own (read) and the same place of the other CTA's warp (written)
        const uint4* inbox = reinterpret_cast<const uint4*>(smem + kPairExchangeRegion + warp * 1024u) + lane;
        const uint32_t outbox = map_shared(smem_u32(inbox), rank ^ 1u);
        const uint32_t peer_sent = map_shared(smem_u32(&bars->sent[warp]), rank ^ 1u);
        const uint32_t peer_taken = map_shared(smem_u32(&bars->taken[warp]), rank ^ 1u);
        if (GATE_UP && lane == 0u) mbar_arrive_expect_tx(&bars->sent[warp], 1024u);  // the first chunk's
        for (uint32_t tile = pair_id; tile < tile_count; tile += pairs, acc_it++) {
            const uint32_t acc = acc_it & 1u;
            // (one warp polls, the others sleep on a hardware barrier; every warp reaches it in every round)
            if (warp == kPairWatchWarp) {
                const bool ready = mbar_wait_warp(&bars->info_full[acc], (acc_it >> 1) & 1u, abort_flag, wait_limit) &&
                                   mbar_wait_warp(&bars->acc_full[acc], (acc_it >> 1) & 1u, abort_flag, wait_limit);
                if (lane == 0u) *reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc]) = ready ? 1u : 0u;
                __threadfence_block();
            }
            named_barrier(1u, 32u * kPairEpilogueWarps);
            if (*reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc]) == 0u) break;
            tc_fence_after();
            const uint32_t tokens = bars->tile_tokens[acc], m_tile = bars->tile_rows[acc];
            const uint32_t first_row = (GATE_UP ? m_tile : 2u * m_tile + rank) * kBlockM + quad * 32u;
            const uint32_t row = first_row + lane;
            const bool row_ok = row < out_rows;
            const uint32_t lane_addr = tmem_base + ((quad * 32u) << 16) + acc * kPairColumns;
            const uint32_t chunks = (tokens + 15u) / 16u;                // of sixteen columns, with a token in them
            const uint32_t half = GATE_UP ? (chunks + 1u) / 2u : chunks; // gate/up: CTA 0 takes these, CTA 1 the others
            // the other CTA's i-th chunk, to its shared memory
            auto send = [&](uint32_t i) {
                const uint32_t c = rank == 0u ? half + i : i;
                if (i >= half || c >= chunks) return;
                uint32_t s[16];
                tmem_ld16(lane_addr + 16u * c, s);
                // (the place is free again once the other warp has taken what was sent last; a wait that gives up leaves rubbish
                // there, which the call reports: bytes that nobody announced keep the other warp's next wait from passing, no more)
                mbar_wait_cluster_warp(&bars->taken[warp], (sends & 1u) ^ 1u, abort_flag, wait_limit);
                tmem_ld_wait();
                uint32_t v[8];
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++) v[j] = bf16x2_bits(__uint_as_float(s[2u * j]), __uint_as_float(s[2u * j + 1u]));
                store_async_cluster(outbox, v[0], v[1], v[2], v[3], peer_sent);
                store_async_cluster(outbox + 512u, v[4], v[5], v[6], v[7], peer_sent);
                sends++;
            };
            if (GATE_UP) send(group);
            for (uint32_t i = group; i < half; i += kPairEpilogueGroups) {
                const uint32_t c = GATE_UP && rank == 1u ? half + i : i;
                const bool mine = c < chunks;
                uint32_t d[16], other[8];
                if (mine) tmem_ld16(lane_addr + 16u * c, d);
                if (GATE_UP && mine) {
                    const bool here = mbar_wait_cluster_warp(&bars->sent[warp], receipts & 1u, abort_flag, wait_limit);
                    const uint4 low = inbox[0], high = inbox[32];
                    other[0] = low.x, other[1] = low.y, other[2] = low.z, other[3] = low.w;
                    other[4] = high.x, other[5] = high.y, other[6] = high.z, other[7] = high.w;
                    // The place may be overwritten once the other warp hears that it was read, and an arrival there does not wait for loads that have only been
                    // issued (chunks whose successor was under way at once came out with eight tokens of it: layers of short K, where the other CTA waits
                    // for the place, differed from pass to pass). So its address depends on what was loaded: `none` is zero, which the compiler can't know.
                    const uint32_t none = __reduce_or_sync(0xffffffffu, low.x | low.y | low.z | low.w | high.x | high.y | high.z | high.w) & (p.debug_flags >> 8);
                    // (the announcement of a chunk only follows the arrival of the last: one more, on a barrier whose bytes are
                    // outstanding, would be one more than it counts)
                    if (here) {
                        if (lane == 0u) {
                            mbar_arrive_expect_tx(&bars->sent[warp], 1024u);
                            mbar_arrive_cluster(peer_taken + none);
                        }
                        receipts++;
                    }
                }
                tmem_ld_wait();
                if (GATE_UP) send(i + kPairEpilogueGroups);  // on its way while this chunk is worked on
                if (!mine) continue;
                const uint32_t* routes = &bars->route[acc][16u * c];
                const uint32_t* extras = &bars->extra[acc][16u * c];
                uint32_t v[8];  // the sixteen values as bf16, in pairs
                if (GATE_UP) {
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++) {
                        const uint32_t own = bf16x2_bits(__uint_as_float(d[2u * j]), __uint_as_float(d[2u * j + 1u]));
                        const uint32_t g = rank == 0u ? own : other[j], u = rank == 0u ? other[j] : own;
                        v[j] = bf16x2_bits(swiglu_approx(low_bf16(g), low_bf16(u), p.g.swiglu_limit, p.g.swiglu_alpha, p.g.swiglu_up_offset),
                                           swiglu_approx(high_bf16(g), high_bf16(u), p.g.swiglu_limit, p.g.swiglu_alpha, p.g.swiglu_up_offset));
                    }
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++)
                        v[j] = bf16x2_bits(__fmul_rn(__uint_as_float(d[2u * j]), __uint_as_float(extras[2u * j])),
                                           __fmul_rn(__uint_as_float(d[2u * j + 1u]), __uint_as_float(extras[2u * j + 1u])));
                }
                if (!GATE_UP && words_of_rows) {
                    // Neighbouring lanes (rows) hand each other one of two tokens, so that a lane stores two rows of a token at once: two bytes a lane
                    // a store took up the end of every tile (16384 tokens of 256 experts 7339 / 7142 us a layer, 4096 of 32 511.7 / 509.7).
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++) {
                        const uint32_t theirs = __shfl_xor_sync(0xffffffffu, v[j], 1), route = routes[2u * j + (lane & 1u)];
                        const uint32_t word = (lane & 1u) ? __byte_perm(theirs, v[j], 0x7632) : __byte_perm(v[j], theirs, 0x5410);
                        if (route != kUnboundSlot && row_ok) *reinterpret_cast<uint32_t*>(p.outputs + (size_t)route * H + (row & ~1u)) = word;
                    }
                } else if (store_rows) {
#pragma unroll
                    for (uint32_t j = 0; j < 16u; j++) {
                        const uint32_t route = routes[j];
                        if (route == kUnboundSlot || !row_ok) continue;
                        const uint16_t bits = (uint16_t)((j & 1u) ? v[j / 2u] >> 16 : v[j / 2u]);
                        if (GATE_UP) {
                            reinterpret_cast<uint16_t*>(p.intermediates + (size_t)(route / K) * frame_words)[(size_t)(route % K) * I + row] = bits;
                        } else if (p.partial_outputs != nullptr) {
                            // tensor-parallel form: the raw f32 sums over this participant's columns
                            p.partial_outputs[(size_t)route * H + row] = __uint_as_float(d[j]);
                        } else {
                            p.outputs[(size_t)route * H + row] = bits;
                        }
                    }
                }
                if (quantise) {
                    // the down stage's activation quantisation, as in experts_tc.cu: a power-of-two scale per 32 rows (this warp's)
                    // or per 128 (the four warps of the group, which hand their maxima round). The maxima of the sixteen tokens
                    // are folded over the lanes by halves, so that four lanes end with those of one pair of tokens and each
                    // token's scale is worked out once.
                    uint32_t m[8];
#pragma unroll
                    for (uint32_t j = 0; j < 8u; j++) m[j] = row_ok ? v[j] & 0x7fff7fffu : 0u;
#pragma unroll
                    for (uint32_t o = 16u, n = 4u; n > 0u; o >>= 1, n >>= 1) {
                        const bool upper = (lane & o) != 0u;
#pragma unroll
                        for (uint32_t j = 0; j < n; j++) {
                            const uint32_t kept = upper ? m[j + n] : m[j], given = upper ? m[j] : m[j + n];
                            m[j] = max_bf16x2(kept, __shfl_xor_sync(0xffffffffu, given, o));
                        }
                    }
                    uint32_t top = max_bf16x2(m[0], __shfl_xor_sync(0xffffffffu, m[0], 2));
                    top = max_bf16x2(top, __shfl_xor_sync(0xffffffffu, top, 1));
                    const uint32_t pair = lane >> 2;  // lane bits 4, 3, 2 chose the upper or lower four, two, one of the eight pairs
                    if (whole_block) {
                        // (a chunk's maxima are overwritten two chunks later, when every warp has passed the barrier between)
                        uint32_t(&quad_max)[4][8] = bars->maxima[group][set_it++ & 1u];
                        if ((lane & 3u) == 0u) quad_max[quad][pair] = top;
                        named_barrier(2u + group, 128u);
                        top = max_bf16x2(max_bf16x2(quad_max[0][pair], quad_max[1][pair]), max_bf16x2(quad_max[2][pair], quad_max[3][pair]));
                    }
                    // lanes 4 pair and 4 pair + 1: the two tokens of the pair
                    const uint32_t token = 2u * pair + (lane & 1u), my_row = extras[token];
                    const float scale = nvmoe_rounded_fp8_scale((lane & 1u) ? high_bf16(top) : low_bf16(top));
                    const float my_inv = __uint_as_float(0x7f000000u - __float_as_uint(scale));  // 1 / scale, exact (a power of two)
                    if ((lane & 2u) == 0u && my_row != kUnboundSlot && first_row < out_rows)
                        *p.q_e8m0.byte_at(my_row, first_row / 32u) = (uint8_t)(nvmoe_f32_bits(scale) >> 23);
                    // Four tokens' codes of a row are a word; four lanes (rows) turn their words round, so that each stores four rows of a token
                    // at once (a byte a lane a store: 0.2 to 1.2 % of the layers below more).
                    const uint32_t turn1 = (lane & 1u) ? 0x3715u : 0x6240u, turn2 = (lane & 2u) ? 0x3276u : 0x5410u;
#pragma unroll
                    for (uint32_t i = 0; i < 4u; i++) {
                        uint32_t word = 0u;
#pragma unroll
                        for (uint32_t h = 0; h < 2u; h++) {
                            const uint32_t j = 2u * i + h;
                            const float inv0 = __shfl_sync(0xffffffffu, my_inv, 4u * j), inv1 = __shfl_sync(0xffffffffu, my_inv, 4u * j + 1u);
                            word |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(low_bf16(v[j]) * inv0, high_bf16(v[j]) * inv1), __NV_SATFINITE, __NV_E4M3) << (16u * h);
                        }
                        word = __byte_perm(word, __shfl_xor_sync(0xffffffffu, word, 1), turn1);  // two rows of two tokens
                        word = __byte_perm(word, __shfl_xor_sync(0xffffffffu, word, 2), turn2);  // four rows of token 4 i + lane % 4
                        const uint32_t to = extras[4u * i + (lane & 3u)];
                        // (0xffffffff: columns without a token and routes the down stage skips)
                        if (to != kUnboundSlot && row_ok) *reinterpret_cast<uint32_t*>(p.q_out + (size_t)to * I + (row & ~3u)) = word;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0u) {
                mbar_arrive(&bars->info_empty[acc]);
                mbar_arrive_cluster(map_shared(smem_u32(&bars->acc_empty[acc]), 0u));
            }
        }
    }

    // ---- teardown: neither CTA leaves while the other may still reach into its shared memory -------------------
    __syncthreads();
    const bool gave_up = threadIdx.x == 0u && *abort_flag != 0u;
    if (gave_up) raise_status(p.status, NVMOE_STATUS_WAIT_EXPIRED);
    __syncwarp();
    cluster_sync();
    if (warp == kPairMmaWarp) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, kPairTmemColumns);
    }
    // A CTA that did not give up has seen every copy, store and commit that reaches its shared memory (each of its tiles was
    // finished); one that did may have some on their way that no role waited for, its own or, until the barrier above, the
    // other CTA's.
    if (gave_up) winddown_pause();
}

template <bool GATE_UP, bool DENSE>
void launch(const ExpertLaunch& p, int sms, const PairMaps<DENSE>& maps, cudaStream_t stream) {
    launch_chained(experts_pair_kernel<GATE_UP, DENSE>, dim3((uint32_t)sms & ~1u), dim3(kPairThreads), kPairSmemBytes, stream, p,
                   TileList{p.tile_list, p.tile_count}, maps);
}

}  // namespace

void pair_configure_kernels() {
    cudaFuncSetAttribute(experts_pair_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmemBytes);
    cudaFuncSetAttribute(experts_pair_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmemBytes);
    cudaFuncSetAttribute(experts_pair_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmemBytes);
}

void launch_experts_pair(const ExpertLaunch& p, bool gate_up, int sms, cudaStream_t stream) {
    if (gate_up) {
        launch<true, false>(p, sms, PairMaps<false>{}, stream);
    } else if (p.dense_maps != nullptr) {
        PairMaps<true> maps;
        std::memcpy(maps.weights, p.dense_maps, sizeof maps.weights);
        launch<false, true>(p, sms, maps, stream);
    } else {
        launch<false, false>(p, sms, PairMaps<false>{}, stream);
    }
}

}  // namespace nvmoe
