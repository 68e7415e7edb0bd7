// Gate/up and down of a layer call in one launch, by one CTA a tile: calls whose weights bound them.
//
// Arithmetic, operands, tiles and the pipeline are those of experts_tc.cu, and HBM bounds the loop as there. What two launches lose is
// their ends: the first waits for its slowest CTA and drains, the second sets up and fills its ring. Here a CTA goes from its
// gate/up tiles to its down tiles without a break: the copying lane runs ahead with down weights while the last gate/up sums are
// still worked on, and only the token rows of a down tile wait for what they are made from. Layers, two launches / one, us: 7
// tokens of 32 experts of 2880 x 2880 73.4 / 67.6, 64 tokens 102.5 / 93.8 (the two kernels 78.5, this one 73), 501 tokens of 128
// experts 362 / 349. Down tiles of 128 rows and two K blocks a stage instead of 256 rows and one: 97 -> 100 at 64 tokens, 360 ->
// 385 at 501. What the threads that issue copies do for a stage has to stay small: with the token rows issued by the warp of
// the token scales a stage took 80 ns more.
//
// Work.  The tiles of a phase are dealt to as many chunks as there are CTAs: chunk c takes tiles c, c + G, ... Chunks are claimed
// in order from a counter, all of gate/up before any of down, so that whoever waits for an expert's gate/up tiles waits for
// CTAs that are on the chip: no co-residency is needed, and every wait is bounded. A CTA claims its next chunk when the first
// token rows of the one at hand are on their way.
//
// Hand-over.  A gate/up epilogue warp counts itself into its expert's counter (release) when its part of the tile is stored; the
// warp that fetches a down tile's token rows and scales waits until the counter holds all of the expert's tiles (acquire, and a
// proxy fence: the rows are written by threads and read by the TMA unit). The call's projection or schedule clears the counters.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "experts_device.cuh"
#include "experts_tc.cuh"
#include "quantize.cuh"
#include "tcgen05.cuh"

namespace nvmoe {
namespace {

using namespace tc;

// Roles, as in experts_tc.cu: warps 0-3 and 8-15 epilogue, 4 MMA, 5 weights, 6 token scales, 7 token rows and the claims.
constexpr uint32_t kLayerThreads = 512u, kLayerGroups = 3u, kLayerEpilogueWarps = 4u * kLayerGroups;
// Who acquires the tensor maps of the weights: all threads ahead of the wait, an epilogue warp beside the first copies, or the lane that issues a tile's copies.
enum : uint32_t { kMapsAhead = 0u, kMapsBeside = 1u, kMapsByTile = 2u };
constexpr uint32_t kLayerMapWarp = 10u;   // the epilogue warp that does
constexpr uint32_t kLayerWatchWarp = 2u;  // the epilogue warp that polls (not on the MMA or TMA warp's scheduler)
constexpr uint32_t kLayerMaxSlots = 6u;
constexpr uint32_t kLayerMaxExperts = 2u * kLayerExperts;  // of both stages together

// A stage is one K block of 128 gate and 128 up rows, or of 256 neighbouring down rows.
template <uint32_t N_TILE>
struct LayerConfig {
    static constexpr uint32_t kABytes = 2u * kATileBytes, kBBytes = N_TILE * 128u;
    // (the scales of 16 tokens are half a block: the copy into tensor memory reads on into what follows, columns that do not exist)
    static constexpr uint32_t kTokenScaleBytes = N_TILE <= 16u ? kScaleBlockBytes / 2u : kScaleBlockBytes;
    static constexpr uint32_t kSfBytes = 2u * kScaleBlockBytes + kTokenScaleBytes;
    static constexpr uint32_t kStageBytes = kABytes + kBBytes + kSfBytes;
    static constexpr uint32_t kBarrierBytes = 512u + 64u * kLayerGroups;  // barriers, then the block maxima
    static constexpr uint32_t kSmemMax = 227u * 1024u;
    // (1024 bytes for the round-up to a boundary of as many: 6, 6, 5 and 4 slots, and leaving it out would buy none)
    static constexpr uint32_t kFit = (kSmemMax - kBarrierBytes - 1024u) / kStageBytes, kSlots = kFit > kLayerMaxSlots ? kLayerMaxSlots : kFit;
    static constexpr uint32_t kBRegion = kSlots * kABytes, kSfRegion = kBRegion + kSlots * kBBytes;
    static constexpr uint32_t kSmemBytes = kSlots * kStageBytes + 1024u + kBarrierBytes;
    static constexpr uint32_t kAccColumns = 2u * N_TILE, kScaleColumn0 = 2u * kAccColumns, kColumnsUsed = kScaleColumn0 + 12u;
    static constexpr uint32_t kTmemColumns = kColumnsUsed <= 128u ? 128u : kColumnsUsed <= 256u ? 256u : 512u;
    static_assert(kSlots >= 4u && kColumnsUsed <= 512u && kBBytes % 1024u == 0u, "layout");
};

struct LayerBarriers {
    uint64_t full[kLayerMaxSlots];
    uint64_t empty[kLayerMaxSlots];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t chunk_full[2];   // a claimed chunk is there
    uint64_t chunk_empty[2];  // ... has been read by the four that work by it
    uint64_t drain;
    uint64_t gate_maps;       // the tensor maps of the gate/up weights have been acquired
    uint64_t down_maps;       // those of the down weights
    uint32_t tmem_base;
    uint32_t abort;
    uint32_t format[kLayerMaxSlots];  // of the weights in a slot: 0 packed E2M1, 1 one byte an element
    uint32_t acc_ready[2];
    uint32_t chunk[2], epilogue_chunk[2];
    uint32_t bytes_form[kLayerMaxExperts / 32u];  // a bit per expert and stage: its weights are one byte an element
};
using BlockMaxima = uint16_t[2][4][4];

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_release(uint32_t* p, uint32_t v) { asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// What the roles have to know of a phase.
struct LayerPhase {
    uint32_t k_dim, out_rows, stages, m_tiles, row_tiles, tile_count;  // (a stage is a K block)
};
// The phase as a constant: the lane that issues the copies keeps up only with code that is made for it.
template <uint32_t P>
struct PhaseTag {
    static constexpr uint32_t value = P;
};

template <uint32_t N_TILE>
__global__ void __launch_bounds__(kLayerThreads, 1) experts_layer_kernel(const __grid_constant__ LayerLaunch p) {
    using C = LayerConfig<N_TILE>;
    const long long wait_limit = p.stage[0].wait_cycles;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    LayerBarriers* bars = reinterpret_cast<LayerBarriers*>(smem + C::kSlots * C::kStageBytes);
    static_assert(sizeof(LayerBarriers) <= 512u && sizeof(BlockMaxima) == 64u, "barrier block");
    BlockMaxima* maxima = reinterpret_cast<BlockMaxima*>(reinterpret_cast<unsigned char*>(bars) + 512u);
    volatile uint32_t* abort_flag = &bars->abort;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const nvmoe_geometry& g = p.stage[0].g;
    const uint32_t H = g.hidden_size, I = g.intermediate_size;
    const uint32_t G = gridDim.x;

    const uint32_t experts = p.stage[0].work.num_experts;
    const bool maps_beside = p.maps == kMapsBeside, maps_by_tile = p.maps == kMapsByTile;

    // ---- one-time setup ---------------------------------------------------------------------
    if (threadIdx.x >= 32u && threadIdx.x < 32u + kLayerMaxExperts / 32u) bars->bytes_form[threadIdx.x - 32u] = 0u;
    if (threadIdx.x == 0u) {
        for (uint32_t s = 0; s < C::kSlots; s++) {
            mbar_init(&bars->full[s], 3u);  // the announcements of the weights and of the token rows, the token scales
            mbar_init(&bars->empty[s], 1u);
        }
        for (uint32_t a = 0; a < 2u; a++) {
            mbar_init(&bars->acc_full[a], 1u);
            mbar_init(&bars->acc_empty[a], 32u * kLayerEpilogueWarps);
            mbar_init(&bars->chunk_full[a], 1u);
            mbar_init(&bars->chunk_empty[a], 4u);
        }
        mbar_init(&bars->drain, 1u);
        mbar_init(&bars->gate_maps, 32u);
        mbar_init(&bars->down_maps, maps_beside ? 32u : 32u * kLayerEpilogueWarps);
        bars->abort = 0u;
        fence_mbar_init();
    }
    __syncthreads();
    if (warp == 4u) {
        tmem_alloc(&bars->tmem_base, C::kTmemColumns);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    // What is read, and counted, before the wait: what stands since earlier calls, or since a launch of this one that had completed
    // when the kernel ahead let this one start: with the quantisation ahead all launches before that, the schedule, which cleared the counters, among
    // them; with the schedule of a small call ahead, which lets this one start before its own wait, those before place_operands_kernel, the
    // projection, which cleared them, among them. Where that schedule clears them itself, the claim follows the wait.
    uint32_t claimed = 0u;
    if (warp == 7u && lane == 0u && !p.claim_late) claimed = atomicAdd(p.sync, 1u);
    for (uint32_t m = threadIdx.x; m < 2u * experts; m += blockDim.x) {
        const bool bytes = (m < experts ? p.stage[0].work.experts[m].format : p.stage[1].work.experts[m - experts].format) != kFormatCompact;
        if (bytes) atomicOr(&bars->bytes_form[m / 32u], 1u << (m % 32u));
    }
    // (as in experts_tc.cu: a block acquires a tensor map once, while the kernel ahead still runs; 13 to 29 ns a map, one after the other, so that those of
    // the down weights are left to epilogue warps that have nothing to do yet. With many experts: layer_maps)
    if (p.maps == kMapsAhead)
        for (uint32_t m = threadIdx.x; m < 2u * experts; m += blockDim.x) tensormap_acquire(p.stage[0].tmaps + (size_t)m * kWeightMaps * 128u);
    if (threadIdx.x < 2u) tensormap_acquire(p.stage[threadIdx.x].act_tmap);
    __syncthreads();
    if (maps_beside && warp == kLayerMapWarp) {
#pragma unroll 1
        for (uint32_t m = lane; m < 2u * experts; m += 32u) tensormap_acquire(p.stage[0].tmaps + (size_t)m * kWeightMaps * 128u);
        mbar_arrive(&bars->gate_maps);
    }
    grid_dependency_sync();
    if (warp == 7u && lane == 0u && p.claim_late) claimed = atomicAdd(p.sync, 1u);
    const uint32_t entries[2] = {*p.stage[0].tile_count, *p.stage[1].tile_count};
    auto phase_of = [&](uint32_t phase) {
        LayerPhase s;
        s.k_dim = phase == 0u ? H : I;
        s.out_rows = phase == 0u ? I : H;
        s.stages = (s.k_dim + kBlockK - 1u) / kBlockK;
        s.row_tiles = (s.out_rows + kBlockM - 1u) / kBlockM;
        s.m_tiles = phase == 1u ? (s.row_tiles + 1u) / 2u : s.row_tiles;
        s.tile_count = (phase == 0u ? entries[0] : entries[1]) * s.m_tiles;
        return s;
    };
    // the k-th chunk of this CTA, for one thread of a role; 2 G and above: none is left (or a wait gave up)
    auto chunk_at = [&](uint32_t k) {
        if (!mbar_wait(&bars->chunk_full[k & 1u], (k >> 1) & 1u, abort_flag, wait_limit)) return 2u * G;
        const uint32_t id = *reinterpret_cast<volatile uint32_t*>(&bars->chunk[k & 1u]);
        mbar_arrive(&bars->chunk_empty[k & 1u]);
        return id;
    };

    if (warp == 5u) {
        // ===== weights and their scales (one lane) =====
        if (lane == 0u) {
            uint32_t slot = 0u, empty_parity = 1u;
            bool alive = true, maps_stand = !maps_beside;
            uint32_t acquired = kUnboundSlot;  // by tile: whose maps were last
            auto run = [&](auto tag, uint32_t id) {
                constexpr uint32_t phase = decltype(tag)::value;
                // (debug) leave out the very first arrival of chunk 0 or 1: its consumer's bounded wait must then give up
                bool withhold = id < 2u && ((p.stage[0].debug_flags >> id) & 1u) != 0u;
                const LayerPhase s = phase_of(phase);
                const ExpertLaunch& e = p.stage[phase];
                // (the list entry of a tile is fetched a tile ahead: a load only, a thread stalls at the first instruction that needs it)
                auto entry_of = [&](uint32_t tile) { return __ldg(e.tile_list + min(tile / s.m_tiles, e.tile_capacity - 1u)); };
                if (phase == 1u && !maps_by_tile && !mbar_wait(&bars->down_maps, 0u, abort_flag, wait_limit)) {
                    alive = false;
                    return;
                }
                const uint32_t scale_stride = phase == 0u ? 2u * kScaleBlockBytes : kScaleBlockBytes;
                const size_t expert_scales = (size_t)s.row_tiles * s.stages * scale_stride;  // derived bytes of an expert
                const uint32_t first_tile = id - phase * G;
                uint32_t entry_nxt = entry_of(first_tile);
                for (uint32_t tile = first_tile; tile < s.tile_count && alive; tile += G) {
                    const uint32_t expert = entry_nxt >> 16, m_tile = tile % s.m_tiles;
                    entry_nxt = entry_of(tile + G);
                    const uint32_t form = phase * experts + expert;
                    const uint32_t format = (bars->bytes_form[form / 32u] >> (form % 32u)) & 1u;
                    const uint32_t row_tile = phase == 1u ? 2u * m_tile : m_tile;
                    const int row0 = (int)(row_tile * kBlockM);
                    const uint8_t* scales = e.scale_base + expert * expert_scales + (size_t)row_tile * s.stages * scale_stride;
                    // (a second row tile past the last rows borrows the first's scales: its weights arrive as zeros)
                    const uint8_t* scales2 = row_tile + 1u < s.row_tiles ? scales + (size_t)s.stages * scale_stride : scales;
                    const uint8_t* maps = e.tmaps + (size_t)expert * (phase == 0u ? 2u : 1u) * kWeightMaps * 128u;
                    const uint32_t box_bytes = format == 0u ? kTmaBoxBytes : 2u * kTmaBoxBytes;
                    if (maps_by_tile ? form != acquired : phase == 0u && !maps_stand && !(maps_stand = mbar_test(&bars->gate_maps, 0u))) {
                        tensormap_acquire(phase == 0u ? maps : maps + 256u);
                        if (phase == 0u) tensormap_acquire(maps + kWeightMaps * 128u);
                        acquired = form;
                    }
                    for (uint32_t ks = 0; ks < s.stages; ks++) {
                        if (!mbar_wait(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                            alive = false;
                            break;
                        }
                        if (!withhold) {
                            const uint32_t a = smem_u32(smem) + slot * C::kABytes, sf = smem_u32(smem) + C::kSfRegion + slot * C::kSfBytes;
                            const uint32_t k64 = min(2u * ks, s.k_dim / 64u - 2u);  // in units of 64 columns, as in experts_tc.cu
                            *reinterpret_cast<volatile uint32_t*>(&bars->format[slot]) = format;
                            mbar_arrive_expect_tx(&bars->full[slot], 2u * (box_bytes + kScaleBlockBytes));
                            if (phase == 0u) {
                                tma_load_3d(a, maps, 0, (int)k64, row0, &bars->full[slot]);
                                tma_load_3d(a + kATileBytes, maps + kWeightMaps * 128u, 0, (int)k64, row0, &bars->full[slot]);
                                bulk_copy_g2s(sf, scales + (size_t)ks * scale_stride, 2u * kScaleBlockBytes, &bars->full[slot]);
                            } else {
                                tma_load_3d(a, maps + 256u, 0, (int)k64, row0, &bars->full[slot]);
                                bulk_copy_g2s(sf, scales + (size_t)ks * scale_stride, kScaleBlockBytes, &bars->full[slot]);
                                bulk_copy_g2s(sf + kScaleBlockBytes, scales2 + (size_t)ks * scale_stride, kScaleBlockBytes, &bars->full[slot]);
                            }
                        }
                        withhold = false;
                        if (++slot == C::kSlots) {
                            slot = 0u;
                            empty_parity ^= 1u;
                        }
                    }
                }
            };
            for (uint32_t k = 0; alive; k++) {
                const uint32_t id = chunk_at(k);
                if (id >= 2u * G) break;
                if (id < G) {
                    run(PhaseTag<0u>{}, id);
                } else {
                    run(PhaseTag<1u>{}, id);
                }
            }
        }
    } else if (warp == 6u || warp == 7u) {
        // ===== token scales (a lane per token, words fetched four stages ahead); token rows (one lane) and the claims =====
        // What hangs on a tile is fetched while the one before it streams, over the end of a chunk too: list entry, offsets and
        // counter would otherwise hold up the rows of every tile by 1.5 us.
        constexpr uint32_t kAhead = 4u, kPer = (N_TILE + 31u) / 32u;
        const bool rows = warp == 7u;
        struct Meta {
            uint32_t phase, tile, expert, first, valid, expected;
            bool ready;  // (lane 0) the counter has been seen to hold what is expected
        };
        uint32_t slot = 0u, empty_parity = 1u, chunk = 0u;
        bool alive = true;
        LayerPhase s = phase_of(0u);
        // The next chunk's first tile: kUnboundSlot if none is left, kEmptyChunk if it has none. In the middle of a tile one chunk
        // is asked for and no more: it is handed over once the other roles have read the one before the last, which the MMA
        // thread may only get to with the rows and scales of this tile.
        constexpr uint32_t kEmptyChunk = 0xfffffffeu;
        auto next_chunk = [&](Meta& m) {
            uint32_t id = 0u;
            if (lane == 0u) {
                if (!rows) {
                    id = chunk_at(chunk);
                } else {
                    id = min(chunk == 0u ? claimed : atomicAdd(p.sync, 1u), 2u * G);
                    if (mbar_wait(&bars->chunk_empty[chunk & 1u], ((chunk >> 1) & 1u) ^ 1u, abort_flag, wait_limit)) {
                        *reinterpret_cast<volatile uint32_t*>(&bars->chunk[chunk & 1u]) = id;
                        mbar_arrive(&bars->chunk_full[chunk & 1u]);
                    } else {
                        id = 2u * G;
                    }
                }
            }
            id = __shfl_sync(0xffffffffu, id, 0);
            chunk++;
            m.phase = id >= G ? 1u : 0u;
            m.tile = id < 2u * G ? id - m.phase * G : kUnboundSlot;
            if (m.tile != kUnboundSlot && m.tile >= phase_of(m.phase).tile_count) m.tile = kEmptyChunk;
        };
        auto load_meta = [&](Meta& m, uint32_t m_tiles) {
            const uint32_t entry = __ldg((m.phase == 0u ? p.stage[0].tile_list : p.stage[1].tile_list) + m.tile / m_tiles);
            const uint32_t* offsets = m.phase == 0u ? p.stage[0].work.expert_offsets : p.stage[1].work.expert_offsets;
            m.expert = entry >> 16;
            m.first = __ldg(offsets + m.expert) + (entry & 0xffffu) * N_TILE;
            m.valid = min(N_TILE, __ldg(offsets + m.expert + 1u) - m.first);
            m.expected = 0u;
            m.ready = true;
            if (m.phase == 1u) {  // what the tile reads is complete once every gate/up tile of the expert is
                const uint32_t routes = __ldg(p.stage[0].work.expert_offsets + m.expert + 1u) - __ldg(p.stage[0].work.expert_offsets + m.expert);
                m.expected = (routes + N_TILE - 1u) / N_TILE * ((I + kBlockM - 1u) / kBlockM) * kLayerEpilogueWarps;
                m.ready = lane == 0u && load_acquire(p.sync + 1u + m.expert) >= m.expected;
            }
        };
        Meta cur{}, nxt{};
        cur.tile = kEmptyChunk;
        while (alive) {
            if (cur.tile == kEmptyChunk) {
                while (cur.tile == kEmptyChunk) next_chunk(cur);
                if (cur.tile == kUnboundSlot) break;
                s = phase_of(cur.phase);
                load_meta(cur, s.m_tiles);
            }
            if (cur.phase == 1u) {
                uint32_t ok = 1u;
                if (lane == 0u) {
                    const long long start = clock64();
                    while (!cur.ready) {
                        cur.ready = load_acquire(p.sync + 1u + cur.expert) >= cur.expected;
                        if (!cur.ready && (*abort_flag || clock64() - start > wait_limit)) {
                            *abort_flag = 1u;
                            ok = 0u;
                            break;
                        }
                    }
                    if (rows) fence_proxy_async_all();
                }
                __syncwarp();  // what lane 0 has acquired is every lane's from here on (a shuffle orders no memory)
                if (__shfl_sync(0xffffffffu, ok, 0) == 0u) break;
            }
            nxt = cur;
            nxt.tile += G;
            auto look_ahead = [&] {
                uint32_t m_tiles = s.m_tiles;
                if (nxt.tile >= s.tile_count) {
                    next_chunk(nxt);
                    m_tiles = phase_of(nxt.phase).m_tiles;
                }
                if (nxt.tile < kEmptyChunk) load_meta(nxt, m_tiles);
            };
            auto run_rows = [&] {
                const uint8_t* map = cur.phase == 0u ? p.stage[0].act_tmap : p.stage[1].act_tmap;
                for (uint32_t ks = 0; ks < s.stages; ks++) {
                    if (!mbar_wait_warp(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    if (lane == 0u) {
                        mbar_arrive_expect_tx(&bars->full[slot], C::kBBytes);
                        tma_load_2d(smem_u32(smem) + C::kBRegion + slot * C::kBBytes, map, (int)(min(2u * ks, s.k_dim / 64u - 2u) * 64u), (int)cur.first,
                                    &bars->full[slot]);
                    }
                    if (++slot == C::kSlots) {
                        slot = 0u;
                        empty_parity ^= 1u;
                    }
                    if (ks == min(kAhead, s.stages) - 1u) look_ahead();
                }
            };
            auto run_scales = [&] {
                const uint32_t* row = (cur.phase == 0u ? p.stage[0].act_e8m0.words : p.stage[1].act_e8m0.words) + (size_t)(cur.first + lane) * s.stages;
                const uint32_t valid = cur.valid;
                uint32_t w[kAhead][kPer];
                auto fetch = [&](uint32_t ks, uint32_t (&into)[kPer]) {
#pragma unroll
                    for (uint32_t i = 0; i < kPer; i++)
                        into[i] = ks < s.stages && lane + 32u * i < valid ? __ldcg(row + (size_t)(32u * i) * s.stages + ks) : 0u;
                };
#pragma unroll
                for (uint32_t u = 0; u < kAhead; u++) fetch(u, w[u]);
                for (uint32_t ks0 = 0; ks0 < s.stages && alive; ks0 += kAhead) {
#pragma unroll
                    for (uint32_t u = 0; u < kAhead; u++) {
                        if (ks0 + u >= s.stages) break;
                        if (!mbar_wait_warp(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                            alive = false;
                            break;
                        }
                        uint32_t* block = reinterpret_cast<uint32_t*>(smem + C::kSfRegion + slot * C::kSfBytes + 2u * kScaleBlockBytes);
#pragma unroll
                        for (uint32_t i = 0; i < kPer; i++)
                            if (lane + 32u * i < N_TILE) block[lane * 4u + i] = w[u][i];
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0u) mbar_arrive(&bars->full[slot]);
                        fetch(ks0 + u + kAhead, w[u]);
                        if (++slot == C::kSlots) {
                            slot = 0u;
                            empty_parity ^= 1u;
                        }
                    }
                    if (ks0 == 0u && alive) look_ahead();
                }
            };
            if (rows) {
                run_rows();
            } else {
                run_scales();
            }
            if (nxt.tile == kUnboundSlot) break;
            if (nxt.phase != cur.phase) s = phase_of(nxt.phase);
            cur = nxt;
        }
    } else if (warp == 4u) {
        // ===== MMA issue (one elected lane) ======================================================
        if (elect_one()) {
            constexpr uint32_t kIdescCompact = idesc_mxf8f6f4(kFmtE2M1, kFmtE4M3, kBlockM, N_TILE);
            constexpr uint32_t kIdescBytes = idesc_mxf8f6f4(kFmtE4M3, kFmtE4M3, kBlockM, N_TILE);  // weights as E4M3 bytes
            const uint32_t base = smem_u32(smem);
            const uint64_t a_desc0 = desc_k_major_sw128(base);
            const uint64_t b_desc0 = desc_k_major_sw128(base + C::kBRegion);
            const uint64_t sf_desc0 = desc_scale_block(base + C::kSfRegion);
            const uint32_t tmem_scales = tmem_base + C::kScaleColumn0, sfb_tmem = tmem_scales + 8u;
            uint32_t acc_it = 0u, slot = 0u, full_parity = 0u;
            bool alive = true;
            for (uint32_t k = 0; alive; k++) {
                const uint32_t id = chunk_at(k);
                if (id >= 2u * G) break;
                const uint32_t phase = id >= G ? 1u : 0u;
                const LayerPhase s = phase_of(phase);
                const uint32_t tail_groups = (s.k_dim % kBlockK) / 32u;  // K steps of a trailing partial block, 0 = none
                for (uint32_t tile = id - phase * G; tile < s.tile_count && alive; tile += G, acc_it++) {
                    const uint32_t acc = acc_it & 1u;
                    if (!mbar_wait(&bars->acc_empty[acc], ((acc_it >> 1) & 1u) ^ 1u, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + acc * C::kAccColumns;
                    for (uint32_t ks = 0; ks < s.stages; ks++) {
                        if (!mbar_wait(&bars->full[slot], full_parity, abort_flag, wait_limit)) {
                            alive = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t idesc = *reinterpret_cast<volatile uint32_t*>(&bars->format[slot]) == 0u ? kIdescCompact : kIdescBytes;
                        // (a trailing half block lies in the second half of its operand tiles; a K step of 32 elements is two 16-byte
                        // units of the start address)
                        const uint32_t groups = ks + 1u == s.stages && tail_groups != 0u ? tail_groups : 4u;
                        const uint32_t first = 2u * (4u - groups);
                        const uint64_t sf_desc = sf_desc0 + (uint64_t)(slot * (C::kSfBytes >> 4));
                        const uint64_t a_desc = a_desc0 + (uint64_t)(slot * (C::kABytes >> 4) + first), b_desc = b_desc0 + (uint64_t)(slot * (C::kBBytes >> 4) + first);
                        tc_copy_scales(tmem_scales, sf_desc);
                        tc_copy_scales(tmem_scales + 4u, sf_desc + (kScaleBlockBytes >> 4));
                        tc_copy_scales(sfb_tmem, sf_desc + (2u * kScaleBlockBytes >> 4));
#pragma unroll
                        for (uint32_t j = 0; j < 4u; j++) {
                            if (j < groups) {
#pragma unroll
                                for (uint32_t mx = 0; mx < 2u; mx++)
                                    tc_mma_block_scaled(d_tmem + mx * N_TILE, a_desc + (mx * (kATileBytes >> 4) + 2u * j), b_desc + 2u * j,
                                                        idesc | (j << 4) | (j << 29), tmem_scales + 4u * mx, sfb_tmem, j == 0u ? (ks != 0u ? 1u : 0u) : 1u);
                            }
                        }
                        tc_commit(&bars->empty[slot]);  // the stage may be refilled once these MMAs retire
                        if (++slot == C::kSlots) {
                            slot = 0u;
                            full_parity ^= 1u;
                        }
                    }
                    if (alive) tc_commit(&bars->acc_full[acc]);
                }
            }
            // (nothing of this CTA may still be reading shared memory or using tensor memory when they are released)
            tc_commit(&bars->drain);
            mbar_wait_winddown(&bars->drain, 0u, kWinddownCycles);
        }
        __syncwarp();
    } else {
        // ===== epilogue: TMEM -> registers -> global =============================================
        const uint32_t quad = warp & 3u;  // the quadrant of tensor-memory lanes this warp may read
        const uint32_t group = warp < 4u ? 0u : warp / 4u - 1u;
        const bool whole_block = g.act_block == 128u;  // the scale block of the down operands is the tile's 128 rows
        uint32_t acc_it = 0u, set_it = 0u;
        bool alive = true;
        if (!maps_by_tile && (!maps_beside || warp == kLayerMapWarp)) {
            const uint32_t first = maps_beside ? lane : group * 128u + quad * 32u + lane, step = maps_beside ? 32u : 32u * kLayerEpilogueWarps;
#pragma unroll 1
            for (uint32_t m = first; m < experts; m += step) tensormap_acquire(p.stage[1].tmaps + (size_t)m * kWeightMaps * 128u + 256u);
            mbar_arrive(&bars->down_maps);
        }
        for (uint32_t k = 0; alive; k++) {
            if (warp == kLayerWatchWarp) {
                if (lane == 0u) *reinterpret_cast<volatile uint32_t*>(&bars->epilogue_chunk[k & 1u]) = chunk_at(k);
                __threadfence_block();
            }
            named_barrier(1u, 32u * kLayerEpilogueWarps);
            const uint32_t id = *reinterpret_cast<volatile uint32_t*>(&bars->epilogue_chunk[k & 1u]);
            if (id >= 2u * G) break;
            auto run = [&](auto tag) {
                constexpr uint32_t phase = decltype(tag)::value;
                const LayerPhase s = phase_of(phase);
                const ExpertLaunch& e = p.stage[phase];
                constexpr bool gate_up = phase == 0u;
                for (uint32_t tile = id - phase * G; tile < s.tile_count; tile += G, acc_it++) {
                    const uint32_t entry = __ldg(e.tile_list + tile / s.m_tiles), m_tile = tile % s.m_tiles, expert = entry >> 16;
                    const uint32_t first = __ldg(e.work.expert_offsets + expert) + (entry & 0xffffu) * N_TILE;
                    const uint32_t valid = min(N_TILE, __ldg(e.work.expert_offsets + expert + 1u) - first);
                    const uint32_t acc = acc_it & 1u;
                    // where token j of the tile goes (its row among the down operands, or its output row and weight): a chain of two
                    // loads, over before the accumulator is ready for narrow tiles, a lane per token
                    uint32_t my_row = kUnboundSlot;
                    float my_weight = 0.0f;
                    auto find = [&](uint32_t j, bool active) {
                        my_row = kUnboundSlot;
                        my_weight = 0.0f;
                        if (!active || j >= valid) return;
                        const uint32_t ri = __ldg(e.work.grouped_routes + first + j);
                        if (gate_up) {
                            my_row = __ldg(e.down_position + ri);
                        } else {
                            my_row = ri;
                            my_weight = nvmoe_bf16_to_f32(__ldg(e.routes + ri) >> 16);
                        }
                    };
                    constexpr bool kNarrow = N_TILE <= 32u;
                    if (kNarrow) find(lane, true);
                    // (one warp polls, the others sleep on a hardware barrier; every warp reaches it in every round)
                    if (warp == kLayerWatchWarp) {
                        const bool ready = mbar_wait_warp(&bars->acc_full[acc], (acc_it >> 1) & 1u, abort_flag, wait_limit);
                        if (lane == 0u) *reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc]) = ready ? 1u : 0u;
                        __threadfence_block();
                    }
                    named_barrier(1u, 32u * kLayerEpilogueWarps);
                    if (*reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc]) == 0u) {
                        alive = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t row = m_tile * (gate_up ? kBlockM : 2u * kBlockM) + quad * 32u + lane;
                    const bool row_ok = row < s.out_rows;
                    const uint32_t lane_addr = tmem_base + ((quad * 32u) << 16) + acc * C::kAccColumns;
                    // a narrow tile is shared out by sets of four tokens, a wide one by chunks of sixteen
                    for (uint32_t c0 = kNarrow ? 0u : 16u * group; c0 < valid; c0 += kNarrow ? 16u : 16u * kLayerGroups) {
                        if (kNarrow) {
                            bool mine = false;  // (uniform)
#pragma unroll
                            for (uint32_t g0 = 0; g0 < 16u; g0 += 4u) mine = mine || (c0 + g0 < valid && ((c0 + g0) / 4u) % kLayerGroups == group);
                            if (!mine) continue;
                        }
                        uint32_t d0[16], d1[16];
                        tmem_ld16(lane_addr + c0, d0);
                        tmem_ld16(lane_addr + N_TILE + c0, d1);  // up, or the second 128 rows
                        if (!kNarrow) find(c0 + lane, lane < 16u);
                        const uint32_t t0 = kNarrow ? c0 : 0u;  // the lane that knows token c0
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t g0 = 0; g0 < 16u; g0 += 4u) {
                            if (c0 + g0 >= valid) break;  // uniform
                            if (kNarrow && ((c0 + g0) / 4u) % kLayerGroups != group) continue;  // another group's
                            if constexpr (gate_up) {
                                // SwiGLU, then the activation quantisation of the down stage, as in experts_tc.cu (by one function for both,
                                // layers with scale blocks of 128 took up to 1.3 % longer)
                                uint32_t bits[4];
#pragma unroll
                                for (uint32_t t = 0; t < 4u; t++)
                                    bits[t] = swiglu_bf16_bits(__uint_as_float(d0[g0 + t]), __uint_as_float(d1[g0 + t]), g.swiglu_limit, g.swiglu_alpha, g.swiglu_up_offset);
                                float m[4];
#pragma unroll
                                for (uint32_t t = 0; t < 4u; t++) m[t] = row_ok ? fabsf(nvmoe_bf16_to_f32(bits[t])) : 0.0f;
#pragma unroll
                                for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                                    for (uint32_t t = 0; t < 4u; t++) m[t] = fmaxf(m[t], __shfl_xor_sync(0xffffffffu, m[t], o));
                                }
                                if (whole_block) {
                                    // (a set's maxima are overwritten two sets later, when every warp has passed the barrier of the set between)
                                    uint16_t(&quad_max)[4][4] = maxima[group][set_it++ & 1u];
                                    if (lane < 4u)
                                        quad_max[quad][lane] = (uint16_t)(__float_as_uint(lane == 0u ? m[0] : lane == 1u ? m[1] : lane == 2u ? m[2] : m[3]) >> 16);
                                    named_barrier(2u + group, 128u);
#pragma unroll
                                    for (uint32_t t = 0; t < 4u; t++)
                                        m[t] = fmaxf(fmaxf(fmaxf(0.0f, nvmoe_bf16_to_f32(quad_max[0][t])), nvmoe_bf16_to_f32(quad_max[1][t])),
                                                     fmaxf(nvmoe_bf16_to_f32(quad_max[2][t]), nvmoe_bf16_to_f32(quad_max[3][t])));
                                }
                                const uint32_t first_row = m_tile * kBlockM + quad * 32u;
                                const bool writes_scale = lane == 0u && first_row < s.out_rows;
#pragma unroll
                                for (uint32_t t = 0; t < 4u; t++) {
                                    const uint32_t dp = __shfl_sync(0xffffffffu, my_row, t0 + g0 + t);
                                    const float scale = nvmoe_rounded_fp8_scale(m[t]);
                                    const float inv = __uint_as_float(0x7f000000u - __float_as_uint(scale));  // 1 / scale, exact (a power of two)
                                    const uint8_t q = (uint8_t)__nv_cvt_float_to_fp8(nvmoe_bf16_to_f32(bits[t]) * inv, __NV_SATFINITE, __NV_E4M3);
                                    if (dp != kUnboundSlot) {  // (lanes past `valid` and routes the down stage skips)
                                        if (row_ok) e.q_out[(size_t)dp * I + row] = q;
                                        if (writes_scale) *e.q_e8m0.byte_at(dp, first_row / 32u) = (uint8_t)(nvmoe_f32_bits(scale) >> 23);
                                    }
                                }
                            } else {
#pragma unroll
                                for (uint32_t t = 0; t < 4u; t++) {
                                    const float weight = __shfl_sync(0xffffffffu, my_weight, t0 + g0 + t);
                                    uint16_t* out = e.outputs + (size_t)__shfl_sync(0xffffffffu, my_row, t0 + g0 + t) * H;
                                    if (c0 + g0 + t < valid && row_ok)
                                        out[row] = __bfloat16_as_ushort(__float2bfloat16_rn(__fmul_rn(__uint_as_float(d0[g0 + t]), weight)));
                                    if (c0 + g0 + t < valid && row + kBlockM < s.out_rows)
                                        out[row + kBlockM] = __bfloat16_as_ushort(__float2bfloat16_rn(__fmul_rn(__uint_as_float(d1[g0 + t]), weight)));
                                }
                            }
                        }
                    }
                    tc_fence_before();
                    mbar_arrive(&bars->acc_empty[acc]);
                    if (gate_up) {  // this warp's part of the tile is stored
                        fence_proxy_async_all();
                        __syncwarp();
                        if (lane == 0u) add_release(p.sync + 1u + expert, 1u);
                    }
                }
            };
            if (id < G) {
                run(PhaseTag<0u>{});
            } else {
                run(PhaseTag<1u>{});
            }
        }
    }

    // ---- teardown -------------------------------------------------------------------------------
    __syncthreads();
    if (warp == 4u) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::kTmemColumns);
    }
    if (threadIdx.x == 0u) {
        if (*abort_flag) {
            raise_status(p.stage[0].status, NVMOE_STATUS_WAIT_EXPIRED);
            winddown_pause();  // copies that no role waited for any more may still be landing
        }
    }
}

template <uint32_t N_TILE>
void launch_one(const LayerLaunch& p, int sms, cudaStream_t stream) {
    launch_chained(experts_layer_kernel<N_TILE>, dim3(sms), dim3(kLayerThreads), LayerConfig<N_TILE>::kSmemBytes, stream, p);
}
template <uint32_t N_TILE>
void configure_one() {
    cudaFuncSetAttribute(experts_layer_kernel<N_TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LayerConfig<N_TILE>::kSmemBytes);
}

}  // namespace

void layer_configure_kernels() {
    configure_one<16u>();
    configure_one<32u>();
    configure_one<64u>();
    configure_one<96u>();
}

// All maps ahead of the wait are acquired for nothing where the block would have waited anyway, but a block that starts late, on an SM that the kernel ahead still used,
// has 15 us of them before its first copy with 257 experts. Beside the first copies they hold up an epilogue warp as long, which short K can't hide. By tile the lane that
// issues the copies stands still for 0.4 us a tile, which costs bytes under way where K is long and a block has many tiles. Layers, us, ahead / beside / by tile: 17 tokens
// of 257 experts of 512 x 384 39.9 / 47.0 / 39.3, 579 of 1536 x 1152 167.9 / 174.6 / 164.0; 6 of 129 of 640 x 512 34.1 / 38.7 / 33.5; 165 of 3840 x 2432 396.0 / 392.3 / 401.1; 327 of 128 of
// 3072 x 2048 251.3 / 247.7 / 253.2; 64 tokens of 32 of 2880 x 2880 ahead. Of 420 drawn layers the rule takes the slower way by 0.15 % in the mean; beyond 64 experts it
// is 1.9 % faster than all ahead in the mean, at most 1.7 % slower.
static uint32_t layer_maps(const LayerLaunch& p, uint32_t sms) {
    const nvmoe_geometry& g = p.stage[0].g;
    const uint32_t experts = p.stage[0].work.num_experts;
    if (experts <= 64u) return kMapsAhead;
    const uint64_t routes = (uint64_t)p.stage[0].tokens * (g.routed_k + g.always_count), touched = routes < experts ? routes : experts;
    const uint64_t tiles = touched * ((g.intermediate_size + kBlockM - 1u) / kBlockM + (g.hidden_size + 2u * kBlockM - 1u) / (2u * kBlockM));
    return g.hidden_size > 2048u && tiles > 12u * (uint64_t)sms ? kMapsBeside : kMapsByTile;
}

void launch_experts_layer(const LayerLaunch& launch, int sms, cudaStream_t stream) {
    LayerLaunch p = launch;
    p.maps = layer_maps(p, (uint32_t)sms);
    switch (p.stage[0].token_rows) {
        case 16u: launch_one<16u>(p, sms, stream); break;
        case 32u: launch_one<32u>(p, sms, stream); break;
        case 64u: launch_one<64u>(p, sms, stream); break;
        default: launch_one<96u>(p, sms, stream); break;
    }
}

}  // namespace nvmoe
