// Grouped expert projections on the Blackwell tensor cores (tcgen05, sm_100a).
//
//   gate/up  runtime-rs/shaders/independent_sparse_moe_gate_up_batch1_mxfp4.comp.template:643-802
//   down     runtime-rs/shaders/independent_sparse_moe_down_batch1_mxfp4.comp.template:507-610
//
// Arithmetic.  The shaders multiply E4M3 activation codes by E2M1 weight codes, scale each group
// of products by (activation scale x E8M0 weight scale) and accumulate in f32.  That is exactly a
// block-scaled MMA of kind::mxf8f6f4: A = packaged E2M1 weight codes with their E8M0 scale per 32
// columns, B = E4M3 activation codes with a UE8M0 scale per 32 columns (the reference's
// power-of-two activation scale, repeated over the 32-column groups of its block), f32
// accumulators in tensor memory.  Products are exact; only the accumulation order differs.
//
// Shape.  The weights are the M side ("swap-AB"): D[128 weight rows x N tokens] = W . X^T, so the
// packaged row-major weight tensor is the K-major A operand as it lies in HBM, a decode batch with
// a handful of tokens per expert still fills an MMA (N = 16), and every weight byte is read once.
// One CTA per SM walks a list of (expert, token tile) x weight-row tiles.
//
// Roles: warps 0-3 epilogue (TMEM lane quadrant = warp); warp 4 allocates TMEM and one of its lanes
// issues the scale copies and MMAs; one lane of warp 5 issues TMA loads of whole 128 x 128 boxes of
// weight codes through a per-expert tensor map (the template map with the expert's address patched in
// on the device; the padded 4-bit tensor-map type spreads the codes into the 16-byte slots the f8f6f4
// kinds read and applies the 128-byte swizzle) and of the token rows; warp 6 stores the token scales.
// Shapes the tensor map cannot describe (K % 64 != 0) stage everything with cp.async by warps 6..,
// whose completion arrives on the stage's mbarrier without stalling the issuer: the codes in 8-byte
// pieces into the low half of the 16-byte slots.  Token rows are gathered
// through the expert-grouped route list (the permutation costs no pass of its own), and E8M0 scales
// come as ready 32x16-byte blocks (the layout tcgen05.cp expands into TMEM) from a derived copy of
// the packaged scale tensors that is rebuilt whenever a scale record's address or generation
// changes.  Stages are handed over with mbarriers; every wait is bounded (tcgen05.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <cstring>

#include "experts_device.cuh"
#include "experts_tc.cuh"
#include "quantize.cuh"
#include "tcgen05.cuh"

namespace nvmoe {
namespace {

using namespace tc;

constexpr uint32_t kFirstProducerThread = 192u;    // warps 0-3 epilogue, 4 MMA, 5 TMA, 6.. cp.async, then more epilogue warps
constexpr uint32_t kMaxStages = 8u;
constexpr uint32_t kRowPairRounds = 6u;  // rounds of the SMs, with every expert selected, from which down tiles of 32 tokens pair their rows
constexpr uint32_t kWatchWarp = 2u;     // the epilogue warp that polls for a finished accumulator (not on the MMA or TMA warp's scheduler)

// ROW_PAIR (down only): a tile covers two 128-row tiles of the one weight matrix, handled as the two
// "matrices" of a stage exactly as gate and up are: two accumulators alternate (one MMA cannot follow
// another into the same accumulator at full rate) and the token tile is fetched once for 256 rows. Used
// for the wide token tiles of large batches and for narrow ones when there are many (takes_row_pairs);
// small batches keep 128-row tiles, which spread better over the SMs.
template <bool GATE_UP, uint32_t N_TILE, bool USE_TMA, bool ROW_PAIR>
struct Config {
    static_assert(!(GATE_UP && ROW_PAIR), "gate/up already holds two matrices a stage");
    static constexpr uint32_t kMatrices = (GATE_UP || ROW_PAIR) ? 2u : 1u;
    static constexpr uint32_t kSources = GATE_UP ? 2u : 1u;        // weight tensors (and tensor maps) per expert
    static constexpr uint32_t kTileRows = kMatrices / kSources * kBlockM;  // weight rows a tile covers
    // matrix mx of a stage = weight tensor source_of(mx), rows shifted by row_shift(mx)
    static constexpr uint32_t source_of(uint32_t mx) { return GATE_UP ? mx : 0u; }
    static constexpr uint32_t row_shift(uint32_t mx) { return ROW_PAIR ? mx * kBlockM : 0u; }
    // Without tensor maps everything comes by cp.async: one warp sustains only about one copy instruction every 60-130
    // cycles, so the copies of a stage are spread over eight warps.
    // With TMA one warp is left with the token scales (a second idles, so that the ones after it keep warp % 4), and the warps
    // this frees become epilogue warps: the epilogue (activation, rounding, re-quantisation: a couple of hundred instructions
    // per value) is what large token tiles wait for, and a warp only issues one instruction at a time. Epilogue warps come in
    // groups of four, one per quadrant of tensor-memory lanes (a warp reads the quadrant warp_id % 4); the groups share out a
    // tile's columns.
    static constexpr uint32_t kProducerWarps = USE_TMA ? 2u : 8u;
    static constexpr uint32_t kProducerThreads = 32u * kProducerWarps;
    static constexpr uint32_t kRowsPerPass = kProducerThreads / 8u;  // eight threads cover the 128 bytes of one row
    static constexpr uint32_t kEpilogueGroups = USE_TMA ? 3u : 1u;
    static constexpr uint32_t kEpilogueThreads = 128u * kEpilogueGroups;
    static constexpr uint32_t kFirstExtraEpilogueWarp = 6u + kProducerWarps;  // a multiple of four
    static constexpr uint32_t kThreads = kFirstProducerThread + kProducerThreads + 128u * (kEpilogueGroups - 1u);
    static_assert(kFirstExtraEpilogueWarp % 4u == 0u || kEpilogueGroups == 1u, "extra epilogue warps keep warp % 4 = quadrant");
    static constexpr uint32_t kBTileBytes = N_TILE * 128u;
    // A stage holds kSub K blocks, each with its own operand tiles and scale blocks. Down moves one
    // matrix, so a stage of one block would carry half the bytes of a gate/up stage for the same
    // barrier traffic and issue overhead: it takes two blocks a stage.
    static constexpr uint32_t kSub = kMatrices == 2u ? 1u : 2u;
    // Shared memory is three regions, each an array over (slot, K block of the stage): the weight tiles, the token
    // tiles (both need 1024-byte alignment: the 128-byte swizzle is a function of the address) and the scale blocks.
    // Kept apart, nothing has to be padded to a 1024-byte boundary per K block, and the throughput of the pipeline is
    // the bytes its slots hold in flight: for the narrow down tiles the padding was the difference between five
    // slots and six.
    static constexpr uint32_t kScaleStride = kSources * kScaleBlockBytes;      // between K blocks of the derived weight scales
    static constexpr uint32_t kABytes = kMatrices * kATileBytes;               // weight tiles of one K block
    // weight scale blocks and the token scale block: 32 entries of 16 bytes, entry n % 32 holding token n's scales.
    // A tile of 16 tokens fills half of it; the copy into tensor memory still reads 512 bytes, the second half
    // being whatever follows in shared memory (the next block's scales, or the barriers): scales of token columns
    // that do not exist.
    static constexpr uint32_t kSfBytes = kMatrices * kScaleBlockBytes + (N_TILE <= 16u ? kScaleBlockBytes / 2u : kScaleBlockBytes);
    // offsets in the scale region: a slot's weight scale blocks (neighbouring K blocks come in one copy), then its token scales
    static constexpr uint32_t weight_scales(uint32_t slot, uint32_t sub, uint32_t mx) {
        return slot * kSub * kSfBytes + (sub * kMatrices + mx) * kScaleBlockBytes;
    }
    static constexpr uint32_t token_scales(uint32_t slot, uint32_t sub) {
        return slot * kSub * kSfBytes + kSub * kMatrices * kScaleBlockBytes + sub * (kSfBytes - kMatrices * kScaleBlockBytes);
    }
    static constexpr uint32_t kStageBytes = kSub * (kABytes + kBTileBytes + kSfBytes);
    static constexpr uint32_t kBarrierBytes = 256u + (GATE_UP ? 64u * kEpilogueGroups : 0u);  // barriers, then the block maxima
    // The arrays start at the first 1024-byte boundary of the dynamic shared memory. Room for that round-up is set
    // aside unless leaving it out buys another slot; the kernel then insists on a base that is aligned already
    // (it is when the kernel has no static shared memory) and does nothing, with NVMOE_STATUS_INTERNAL, otherwise.
    static constexpr uint32_t kSmemMax = 227u * 1024u;
    static constexpr uint32_t stages_for(uint32_t slack) {
        const uint32_t n = (kSmemMax - kBarrierBytes - slack) / kStageBytes;
        return n > kMaxStages ? kMaxStages : n;
    }
    static constexpr bool kNeedsAlignedBase = stages_for(0u) > stages_for(1024u);
    static constexpr uint32_t kStages = stages_for(kNeedsAlignedBase ? 0u : 1024u);
    static constexpr uint32_t kBlocks = kStages * kSub;                        // K blocks resident at once
    static constexpr uint32_t kBRegion = kBlocks * kABytes;                    // offset of the token tiles
    static constexpr uint32_t kSfRegion = kBRegion + kBlocks * kBTileBytes;    // offset of the scale blocks
    static constexpr uint32_t kAccColumns = kMatrices * N_TILE;
    static constexpr uint32_t kAccStages = 2u;
    static constexpr uint32_t kScaleColumns = 4u * (kMatrices + 1u);
    // Two accumulators of 128 tokens and two matrices (the widest tile of shapes without tensor maps; with them so many tokens
    // run by CTA pairs) would be all of tensor memory, with no columns left for the scales. They share 16 columns instead: the last tokens' second matrix of the first accumulator lies where the
    // second accumulator keeps the first tokens' first matrix. The epilogue reads that chunk before all others and
    // says so (acc_head), and the MMAs of the next tile wait for it: about a microsecond per tile, during which the
    // ring fills. Wider tiles fetch fewer weight bytes per token, and the MMA itself is bound by its operand reads
    // from shared memory below 128 columns (64.8 cycles at 96 columns, 68.5 at 128).
    static constexpr bool kOverlap = 2u * kAccColumns + kScaleColumns > 512u;
    static constexpr uint32_t kAccStride = kOverlap ? kAccColumns - 16u : kAccColumns;
    static constexpr uint32_t kScaleColumn0 = (kAccStages - 1u) * kAccStride + kAccColumns;
    static constexpr uint32_t kColumnsUsed = kScaleColumn0 + kScaleColumns;
    static_assert(kColumnsUsed <= 512u, "tensor memory");
    static constexpr uint32_t kTmemColumns = kColumnsUsed <= 32u ? 32u : kColumnsUsed <= 64u ? 64u : kColumnsUsed <= 128u ? 128u : kColumnsUsed <= 256u ? 256u : 512u;
    static constexpr uint32_t kSmemBytes = kStages * kStageBytes + (kNeedsAlignedBase ? 0u : 1024u) + kBarrierBytes;
    static_assert(N_TILE % 16u == 0u && N_TILE >= 16u && N_TILE <= 128u, "token tile");
    static_assert(kBTileBytes % 1024u == 0u && kABytes % 1024u == 0u, "operand tiles keep their 1024-byte alignment");
    static_assert(kStages >= 3u, "pipeline too shallow");
};

struct Barriers {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t acc_head[2];         // overlapping accumulators: the shared chunk of this one has been read
    uint64_t drain;
    uint32_t tmem_base;
    uint32_t abort;
    uint32_t format[kMaxStages];  // kFormat* of the weights staged in each slot (written before the slot's arrival)
    uint32_t acc_ready[2];        // the verdict of the epilogue warp that watches acc_full, for the others
};

// Block maxima of the fused quantisation with 128-row scale blocks: [set of four tokens, alternating][lane quadrant]
// [token] of each epilogue group, as the bf16 bits of the magnitude
using BlockMaxima = uint16_t[2][4][4];

// TRACE compiles the diagnostics in (cycle counters of CTA 0, per-CTA global-timer stamps): the
// instantiation that runs unless a plan's trace was armed has none of them in its loops.
template <bool GATE_UP, uint32_t N_TILE, bool USE_TMA, bool ROW_PAIR, bool TRACE>
__global__ void __launch_bounds__((Config<GATE_UP, N_TILE, USE_TMA, ROW_PAIR>::kThreads), 1)
    experts_tc_kernel(ExpertLaunch p, TileList list) {
    using C = Config<GATE_UP, N_TILE, USE_TMA, ROW_PAIR>;
    const long long wait_limit = p.wait_cycles;
    constexpr uint32_t kProducerThreads = C::kProducerThreads, kRowsPerPass = C::kRowsPerPass;
    extern __shared__ unsigned char smem_raw[];
    // operand tiles need 1024-byte alignment for the 128-byte swizzle
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023u));
    Barriers* bars = reinterpret_cast<Barriers*>(smem + C::kStages * C::kStageBytes);
    static_assert(sizeof(Barriers) <= 256u && sizeof(BlockMaxima) == 64u, "barrier block");
    BlockMaxima* maxima = reinterpret_cast<BlockMaxima*>(reinterpret_cast<unsigned char*>(bars) + 256u);
    volatile uint32_t* abort_flag = &bars->abort;
    if (C::kNeedsAlignedBase && smem != smem_raw) {  // (uniform) no room was set aside for the round-up
        grid_dependency_sync();
        if (threadIdx.x == 0u) raise_status(p.status, NVMOE_STATUS_INTERNAL);
        return;
    }

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t H = p.g.hidden_size, I = p.g.intermediate_size;
    const uint32_t K = p.g.routed_k + p.g.always_count;
    const uint32_t k_dim = GATE_UP ? H : I;
    const uint32_t out_rows = GATE_UP ? I : H;
    const uint32_t k_blocks = (k_dim + kBlockK - 1u) / kBlockK;
    // K blocks of a stage. By TMA a stage of two brings whole blocks only, both in one copy; a lone whole block and a trailing
    // half one are stages of their own.
    const uint32_t doubles = C::kSub == 2u ? (USE_TMA ? k_dim / kBlockK / 2u : k_blocks / 2u) : 0u;
    const uint32_t k_stages = k_blocks - doubles;
    auto first_block = [&](uint32_t ks) { return ks < doubles ? 2u * ks : doubles + ks; };
    const uint32_t m_tiles = (out_rows + C::kTileRows - 1u) / C::kTileRows;   // tiles along the weight rows
    const uint32_t row_tiles = (out_rows + kBlockM - 1u) / kBlockM;           // 128-row tiles (scale blocks are kept per these)
    // the derived scale blocks of matrix mx of tile m_tile (a second half past the last rows borrows the first's:
    // its weights arrive as zeros)
    auto scale_tile = [&](uint32_t m_tile, uint32_t mx) {
        const uint32_t t = ROW_PAIR ? 2u * m_tile + mx : m_tile;
        return t < row_tiles ? t : t - 1u;
    };
    // cycle counters of CTA 0, one writer per role (diagnostics; words 16.. of the tile-count block)
    uint64_t* trace = reinterpret_cast<uint64_t*>(const_cast<uint32_t*>(list.count) + 16) + (GATE_UP ? 0 : 12);
    if (TRACE && blockIdx.x == 0u && threadIdx.x == 0u) trace[8] = global_timer_ns();  // kernel entry of CTA 0

    // ---- one-time setup ---------------------------------------------------------------------
    if (threadIdx.x == 0u) {
        for (uint32_t s = 0; s < C::kStages; s++) {
            mbar_init(&bars->full[s], USE_TMA ? 2u : kProducerThreads);  // TMA: the announcement of the copies, the scale warp
            mbar_init(&bars->empty[s], 1u);
        }
        for (uint32_t a = 0; a < 2u; a++) {
            mbar_init(&bars->acc_full[a], 1u);
            mbar_init(&bars->acc_empty[a], C::kEpilogueThreads);
            mbar_init(&bars->acc_head[a], 128u);
        }
        mbar_init(&bars->drain, 1u);
        bars->abort = 0u;
        fence_mbar_init();
    }
    // (The padding halves of the 4-bit slots, the scale rows past the token tile and whatever else the
    // copies never write stay as they were found: the MMA does not read them. Checked by filling the
    // stages with 0xff first; rows and columns that are read but hold no data are written as zeros by the
    // copies themselves.)
    __syncthreads();
    if (warp == 4u) {
        tmem_alloc(&bars->tmem_base, C::kTmemColumns);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t tmem_scales = tmem_base + C::kScaleColumn0;
    auto acquire_maps = [&] {
        // The per-expert tensor maps were written to global memory by an earlier kernel. A thread block must
        // acquire such a map once before any of its threads hands it to the TMA unit; further uses by the
        // block need no fence. All threads share the maps out, so that the block pays one fence latency here
        // instead of one per map in the lane that issues the loads.
        for (uint32_t m = threadIdx.x; m < p.work.num_experts * C::kSources; m += blockDim.x) {
            const uint8_t* maps = p.tmaps + (size_t)m * kWeightMaps * 128u;
            tensormap_acquire(maps + (ROW_PAIR ? 256u : 0u));
            if (C::kSub == 2u) tensormap_acquire(maps + 128u);
        }
        if (threadIdx.x < C::kSub) tensormap_acquire(p.act_tmap + threadIdx.x * kTokenMaps * 128u);
        __syncthreads();
    };
    // Maps of earlier calls, or of this one with a launch between (which has completed by the time this kernel may start), are
    // acquired while the kernel ahead still runs.
    if (USE_TMA && !p.fresh_maps) acquire_maps();
    // everything above touched only this CTA's shared and tensor memory and maps that stand; what follows reads what the
    // kernels before this one wrote
    grid_dependency_sync();
    // (the first list entry is fetched with the count it may turn out to lie beyond, not after it)
    const uint32_t first_entry = USE_TMA && (warp == 5u || warp == 6u) ? __ldg(list.tiles + min(blockIdx.x / m_tiles, p.tile_capacity - 1u)) : 0u;
    const uint32_t pair_count = *list.count;
    const uint32_t tile_count = pair_count * m_tiles;
    if (USE_TMA && p.fresh_maps) acquire_maps();

    if (warp == 5u) {
        // ===== TMA issue (one lane): whole 128 x 128 boxes of weight codes, padded and swizzled by the unit =====
        if (USE_TMA && lane == 0u) {
            uint32_t slot = 0u, empty_parity = 1u;
            bool alive = true;
            long long trace_wait = 0;
            const long long trace_begin = TRACE ? clock64() : 0;
            // What the lane needs to know about a tile. The list entry of a tile is fetched two tiles ahead and
            // what hangs on it (the expert's offset, scale and tensor-map addresses) one tile ahead, so that the
            // chain of dependent loads is over by the time the tile starts: a lane that stalled on it at every
            // tile boundary would leave the memory pipe without new requests for about a microsecond per tile.
            // (The prefetch only loads: whatever is computed from a loaded value is computed when the tile
            // starts, because a thread stalls at the first instruction that needs a load's result.)
            struct Meta {
                uint32_t pair, m_tile, expert_begin, format;
                const uint8_t* ts[C::kSources];
            };
            auto entry_of = [&](uint32_t tile) {
                uint32_t pair = 0u;
                if (tile < tile_count) pair = __ldg(list.tiles + tile / m_tiles);
                return pair;
            };
            auto meta_of = [&](uint32_t tile, uint32_t pair, Meta& m) {
                m.pair = pair;
                m.m_tile = tile % m_tiles;
                const uint32_t expert = pair >> 16;
                m.expert_begin = __ldg(p.work.expert_offsets + expert);
                m.format = p.work.experts[expert].format;
#pragma unroll
                for (uint32_t src = 0; src < C::kSources; src++) m.ts[src] = p.work.experts[expert].ts[src];
            };
            Meta cur{}, nxt{};
            if (blockIdx.x < tile_count) meta_of(blockIdx.x, first_entry, cur);
            uint32_t pair_nxt = entry_of(blockIdx.x + gridDim.x);
            // (debug) leave out the very first arrival of CTA 0 or 1: its consumer's bounded wait must then give up
            bool withhold = blockIdx.x < 2u && ((p.debug_flags >> blockIdx.x) & 1u) != 0u;
            for (uint32_t tile = blockIdx.x; tile < tile_count && alive; tile += gridDim.x) {
                const uint32_t pair_nxt2 = entry_of(tile + 2u * gridDim.x);
                if (tile + gridDim.x < tile_count) meta_of(tile + gridDim.x, pair_nxt, nxt);
                const uint32_t m_tile = cur.m_tile;
                const int row0 = (int)(m_tile * C::kTileRows);
                const uint8_t* maps = p.tmaps + (size_t)(cur.pair >> 16) * C::kSources * kWeightMaps * 128u;
                // first operand row of this token tile in the expert-grouped activation matrix
                const int token0 = (int)(cur.expert_begin + (cur.pair & 0xffffu) * N_TILE);
                const uint8_t* scale_blocks[C::kMatrices];
#pragma unroll
                for (uint32_t mx = 0; mx < C::kMatrices; mx++)
                    scale_blocks[mx] = cur.ts[C::source_of(mx)] + (size_t)scale_tile(m_tile, mx) * k_blocks * C::kScaleStride;
                for (uint32_t ks = 0; ks < k_stages; ks++) {
                    const long long w0 = TRACE ? clock64() : 0;
                    if (!mbar_wait(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    if (TRACE) trace_wait += clock64() - w0;
                    const bool two = ks < doubles;
                    const uint32_t kb = first_block(ks), present = two ? 2u : 1u;
                    if (withhold) {
                        withhold = false;
                    } else {
                    // the K blocks' weight codes, token rows and weight scales: one copy each (gate and up: one each for the codes)
                    const uint32_t block = slot * C::kSub;  // index into the shared-memory arrays
                    const uint32_t smem_base = smem_u32(smem);
                    const uint32_t a = smem_base + block * C::kABytes, b = smem_base + C::kBRegion + block * C::kBTileBytes;
                    const uint32_t sf = smem_base + C::kSfRegion + C::weight_scales(slot, 0u, 0u);
                    // a box of one-byte elements brings twice the bytes of a box of packed 4-bit codes
                    const uint32_t box_bytes = cur.format == kFormatCompact ? kTmaBoxBytes : 2u * kTmaBoxBytes;
                    *reinterpret_cast<volatile uint32_t*>(&bars->format[slot]) = cur.format;
                    mbar_arrive_expect_tx(&bars->full[slot], present * (C::kMatrices * box_bytes + C::kBTileBytes + C::kMatrices * kScaleBlockBytes));
                    // (rows past the matrix arrive as zeros)
                    if (two) {
                        tma_load_3d(a, maps + 128u, 0, row0, (int)kb, &bars->full[slot]);
                        tma_load_3d(b, p.act_tmap + kTokenMaps * 128u, 0, token0, (int)kb, &bars->full[slot]);
                    } else {
                        // in units of 64 columns: a trailing half block comes as a whole one that ends with the row
                        const uint32_t k64 = min(2u * kb, k_dim / 64u - 2u);
                        if (ROW_PAIR) {
                            tma_load_3d(a, maps + 256u, 0, (int)k64, row0, &bars->full[slot]);
                        } else {
#pragma unroll
                            for (uint32_t src = 0; src < C::kSources; src++)
                                tma_load_3d(a + src * kATileBytes, maps + src * (kWeightMaps * 128u), 0, (int)k64, row0, &bars->full[slot]);
                        }
                        tma_load_2d(b, p.act_tmap, (int)(k64 * 64u), token0, &bars->full[slot]);
                    }
                    if (ROW_PAIR) {
#pragma unroll
                        for (uint32_t mx = 0; mx < C::kMatrices; mx++)
                            bulk_copy_g2s(sf + mx * kScaleBlockBytes, scale_blocks[mx] + (size_t)kb * C::kScaleStride, kScaleBlockBytes, &bars->full[slot]);
                    } else {
                        // the gate and the up block of this (row tile, K block) are neighbours in the derived copy, and so are two K blocks
                        bulk_copy_g2s(sf, scale_blocks[0] + (size_t)kb * C::kScaleStride, present * C::kMatrices * kScaleBlockBytes, &bars->full[slot]);
                    }
                    }
                    if (++slot == C::kStages) {
                        slot = 0u;
                        empty_parity ^= 1u;
                    }
                }
                cur = nxt;
                pair_nxt = pair_nxt2;
            }
            if (TRACE && blockIdx.x == 0u) {
                trace[0] = (uint64_t)trace_wait;                    // copy-issuing lane: cycles waiting for a free stage
                trace[1] = (uint64_t)(clock64() - trace_begin);     // copy-issuing lane: cycles in its loop
            }
        }
    } else if (USE_TMA && warp >= 6u && warp < 6u + C::kProducerWarps) {
        // ===== token scales (one warp): a lane per token, words fetched four stages ahead and stored to the stage's block =====
        // (As 4-byte asynchronous copies that arrived on the barrier by themselves, by 64 threads, with the trailing half block of
        // the weights, they were the last operands of many stages: layer of 64 tokens of 32 experts of 2880 x 2880 122.5 us, 114.7 this way.)
        if (warp == 6u) {
            constexpr uint32_t kAhead = 4u, kPer = (N_TILE + 31u) / 32u;
            struct Meta {
                uint32_t first, valid;
            };
            auto load_meta = [&](uint32_t pair, Meta& m) {
                const uint32_t expert = pair >> 16;
                m.first = __ldg(p.work.expert_offsets + expert) + (pair & 0xffffu) * N_TILE;
                m.valid = min(N_TILE, __ldg(p.work.expert_offsets + expert + 1u) - m.first);
            };
            uint32_t slot = 0u, empty_parity = 1u;
            bool alive = true;
            Meta cur{}, nxt{};
            if (blockIdx.x < tile_count) load_meta(first_entry, cur);
            for (uint32_t tile = blockIdx.x; tile < tile_count && alive; tile += gridDim.x) {
                const uint32_t* row = p.act_e8m0.words + (size_t)(cur.first + lane) * k_blocks;
                const uint32_t valid = cur.valid;
                uint32_t w[kAhead][C::kSub][kPer];
                auto fetch = [&](uint32_t ks, uint32_t (&into)[C::kSub][kPer]) {
#pragma unroll
                    for (uint32_t sub = 0; sub < C::kSub; sub++) {
#pragma unroll
                        for (uint32_t i = 0; i < kPer; i++) {
                            const bool ok = ks < k_stages && (sub == 0u || ks < doubles) && lane + 32u * i < valid;
                            into[sub][i] = ok ? __ldg(row + (size_t)(32u * i) * k_blocks + first_block(ks) + sub) : 0u;
                        }
                    }
                };
#pragma unroll
                for (uint32_t u = 0; u < kAhead; u++) fetch(u, w[u]);
                if (tile + gridDim.x < tile_count) load_meta(__ldg(list.tiles + (tile + gridDim.x) / m_tiles), nxt);
                for (uint32_t ks0 = 0; ks0 < k_stages && alive; ks0 += kAhead) {
#pragma unroll
                    for (uint32_t u = 0; u < kAhead; u++) {
                        if (ks0 + u >= k_stages) break;
                        if (!mbar_wait_warp(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                            alive = false;
                            break;
                        }
#pragma unroll
                        for (uint32_t sub = 0; sub < C::kSub; sub++) {
                            uint32_t* block = reinterpret_cast<uint32_t*>(smem + C::kSfRegion + C::token_scales(slot, sub));
#pragma unroll
                            for (uint32_t i = 0; i < kPer; i++)
                                if (lane + 32u * i < N_TILE) block[lane * 4u + i] = w[u][sub][i];
                        }
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0u) mbar_arrive(&bars->full[slot]);
                        fetch(ks0 + u + kAhead, w[u]);
                        if (++slot == C::kStages) {
                            slot = 0u;
                            empty_parity ^= 1u;
                        }
                    }
                }
                cur = nxt;
            }
        }
    } else if (!USE_TMA && warp >= 6u && warp < 6u + C::kProducerWarps) {
        // ===== operand producers: cp.async into the swizzled tiles, completion arrives on `full` =====
        const uint32_t pt = threadIdx.x - kFirstProducerThread;  // 0..kProducerThreads-1
        const uint32_t my_r = pt >> 3, my_c = pt & 7u;  // this thread's row (plus kRowsPerPass i) and 16-element chunk
        constexpr uint32_t kTokenPasses = (N_TILE + kRowsPerPass - 1u) / kRowsPerPass;
        const uint32_t row_bytes = k_dim / 2u;
        // What a thread needs to know about a tile; the next tile's copy is fetched while the current
        // tile streams, so that the dependent loads (tile list -> offsets -> routes) never stall the pipe.
        struct Meta {
            const uint8_t* w[C::kMatrices];
            const uint8_t* ts[C::kMatrices];
            uint32_t code_rows[kTokenPasses];  // activation row of token my_r + kRowsPerPass i
            uint32_t scale_row;                // activation row of token pt
            uint32_t valid, m_tile, first, format;
        };
        auto load_meta = [&](uint32_t tile, Meta& m) {
            const uint32_t pair = __ldg(list.tiles + tile / m_tiles);
            m.m_tile = tile % m_tiles;
            const uint32_t expert = pair >> 16, n_tile = pair & 0xffffu;
            const uint32_t e_begin = __ldg(p.work.expert_offsets + expert), e_end = __ldg(p.work.expert_offsets + expert + 1u);
            const uint32_t first = e_begin + n_tile * N_TILE;
            m.valid = min(N_TILE, e_end - first);
            m.first = first;
            const ExpertPtrs* ptrs = p.work.experts + expert;
            m.format = ptrs->format;
#pragma unroll
            for (uint32_t mx = 0; mx < C::kMatrices; mx++) {
                m.w[mx] = ptrs->w[C::source_of(mx)];
                m.ts[mx] = ptrs->ts[C::source_of(mx)];
            }
            // the operand matrices are expert-grouped: token n of the tile is row first + n
#pragma unroll
            for (uint32_t i = 0; i < kTokenPasses; i++) m.code_rows[i] = first + my_r + kRowsPerPass * i;
            // (the thread that copies token n's scales is kProducerThreads - 65 - n: see the copy below)
            m.scale_row = first + (kProducerThreads - 65u - pt);
        };
        uint32_t slot = 0u, empty_parity = 1u;  // a fresh barrier passes a wait on parity 1
        const uint32_t my_dst = swizzle128_offset(my_r, my_c);
        bool alive = true;
        Meta cur, nxt;
        if (blockIdx.x < tile_count) load_meta(blockIdx.x, cur);
        for (uint32_t tile = blockIdx.x; tile < tile_count && alive; tile += gridDim.x) {
            if (tile + gridDim.x < tile_count) load_meta(tile + gridDim.x, nxt);
            // this thread's first weight row of each matrix of the tile; its other rows are kRowsPerPass apart
            const uint8_t* wcol[C::kMatrices];
            uint32_t rows_here[C::kMatrices];
            // a matrix of one-byte elements (pre-expanded or native FP8) has rows, and pieces of 16 elements, twice as long
            const bool bytes_form = cur.format != kFormatCompact;
            const uint32_t form_row_bytes = bytes_form ? 2u * row_bytes : row_bytes;
#pragma unroll
            for (uint32_t mx = 0; mx < C::kMatrices; mx++) {
                const uint32_t row0 = cur.m_tile * C::kTileRows + C::row_shift(mx);
                rows_here[mx] = row0 < out_rows ? min(kBlockM, out_rows - row0) : 0u;
                wcol[mx] = cur.w[mx] + (size_t)(row0 + my_r) * form_row_bytes + my_c * (bytes_form ? 16u : 8u);
            }
            const size_t row_step = (size_t)kRowsPerPass * form_row_bytes;
            for (uint32_t ks = 0; ks < k_stages; ks++) {
                if (!mbar_wait_warp(&bars->empty[slot], empty_parity, abort_flag, wait_limit)) {
                    alive = false;
                    break;
                }
#pragma unroll
                for (uint32_t sub = 0; sub < C::kSub; sub++) {
                if (sub != 0u && ks >= doubles) break;  // the last stage of an odd count holds one block
                const uint32_t kb = first_block(ks) + sub;
                const uint32_t block = slot * C::kSub + sub;  // index into the shared-memory arrays
                unsigned char* a_tiles = smem + block * C::kABytes;
                const uint32_t k_left = k_dim - kb * kBlockK;  // elements of K from this block on
                const bool chunk_ok = my_c * 16u < k_left;
                // weights: 8-byte pieces of 16 codes into the low half of 16-byte slots
#pragma unroll
                for (uint32_t mx = 0; mx < C::kMatrices; mx++) {
                    const uint32_t a_dst = smem_u32(a_tiles + mx * kATileBytes) + my_dst;
                    const uint8_t* src = wcol[mx] + kb * (bytes_form ? 128u : 64u);
#pragma unroll
                    for (uint32_t i = 0; i < kBlockM / kRowsPerPass; i++) {
                        // rows my_r + kRowsPerPass i share (row & 7), so the swizzled offset only moves by whole rows
                        const bool ok = chunk_ok && (my_r + kRowsPerPass * i < rows_here[mx]);
                        if (bytes_form) {
                            cp_async_16(a_dst + i * (kRowsPerPass * 128u), ok ? src + i * row_step : cur.w[mx], ok ? 16u : 0u);
                        } else {
                            cp_async_8(a_dst + i * (kRowsPerPass * 128u), ok ? src + i * row_step : cur.w[mx], ok ? 8u : 0u);
                        }
                    }
                }
                // activations: 16-byte pieces of 16 E4M3 codes
                const uint32_t b_dst = smem_u32(smem + C::kBRegion + block * C::kBTileBytes) + my_dst;
#pragma unroll
                for (uint32_t i = 0; i < kTokenPasses; i++) {
                    const uint32_t n = my_r + kRowsPerPass * i;
                    if (n < N_TILE) {
                        const bool ok = chunk_ok && (n < cur.valid);
                        const uint8_t* src = ok ? p.act_q + (size_t)cur.code_rows[i] * k_dim + kb * kBlockK + my_c * 16u : p.act_q;
                        cp_async_16(b_dst + i * (kRowsPerPass * 128u), src, ok ? 16u : 0u);
                    }
                }
                // scales: the derived copy already has the 32x16-byte layout tcgen05.cp reads, one 512-byte
                // block per (row tile, K block); token scales are gathered four bytes (one K block) a row
                // (threads from the far end of the producer group, so that with few tokens a tile these are not
                // the threads that carry the token rows)
                const uint32_t st = kProducerThreads - 1u - pt;
                if (st < 32u * C::kMatrices) {
                    const uint32_t mx = st >> 5, l = st & 31u;
                    const uint8_t* src = cur.ts[mx] + ((size_t)scale_tile(cur.m_tile, mx) * k_blocks + kb) * C::kScaleStride + l * 16u;
                    cp_async_16(smem_u32(smem + C::kSfRegion + C::weight_scales(slot, sub, mx) + l * 16u), src, 16u);
                }
                if (st >= 64u && st < 64u + N_TILE) {
                    const uint32_t n = st - 64u;
                    const bool ok = n < cur.valid;
                    const uint32_t* src = ok ? p.act_e8m0.words + (size_t)cur.scale_row * k_blocks + kb : p.act_e8m0.words;
                    cp_async_4(smem_u32(smem + C::kSfRegion + C::token_scales(slot, sub) + (n & 31u) * 16u + (n >> 5) * 4u), src,
                               ok ? 4u : 0u);
                }
                }
                if (pt == 0u) *reinterpret_cast<volatile uint32_t*>(&bars->format[slot]) = cur.format;
                // the arrival fires when this thread's copies have landed; the thread moves on at once
                cp_async_arrive_noinc(&bars->full[slot]);
                if (++slot == C::kStages) {
                    slot = 0u;
                    empty_parity ^= 1u;
                }
            }
            cur = nxt;
        }
        cp_async_wait_all();  // nothing of this thread may still be landing when the CTA retires
    } else if (warp == 4u) {
        // ===== MMA issue (one elected lane) ======================================================
        if (elect_one()) {
            // One thread feeds the tensor pipe, and a lone thread retires an instruction every few
            // cycles at best: everything that does not depend on the stage is computed once, the four
            // K steps of a stage are unrolled with compile-time descriptors offsets and scale ids.
            constexpr uint32_t kIdescCompact = idesc_mxf8f6f4(kFmtE2M1, kFmtE4M3, kBlockM, N_TILE);
            constexpr uint32_t kIdescBytes = idesc_mxf8f6f4(kFmtE4M3, kFmtE4M3, kBlockM, N_TILE);  // weights as E4M3 bytes
            // descriptor start addresses count 16 bytes
            const uint32_t base = smem_u32(smem);
            const uint64_t a_desc0 = desc_k_major_sw128(base);
            const uint64_t b_desc0 = desc_k_major_sw128(base + C::kBRegion);
            const uint64_t sf_desc0 = desc_scale_block(base + C::kSfRegion);
            const uint32_t tail_groups = (k_dim % kBlockK) / 32u;  // K steps of a trailing partial block, 0 = none
            const uint32_t sfb_tmem = tmem_scales + 4u * C::kMatrices;
            uint32_t it = 0u, acc_it = 0u, slot = 0u, full_parity = 0u;
            bool alive = true;
            long long trace_full = 0, trace_acc = 0;
            const long long trace_begin = TRACE ? clock64() : 0;
            if (TRACE && blockIdx.x == 0u) trace[9] = global_timer_ns();  // MMA loop begins
            const uint64_t cta_begin = (TRACE && p.cta_trace) ? global_timer_ns() : 0u;
            for (uint32_t tile = blockIdx.x; tile < tile_count && alive; tile += gridDim.x, acc_it++) {
                const uint32_t acc = acc_it % C::kAccStages;
                const long long a0 = TRACE ? clock64() : 0;
                if (!mbar_wait(&bars->acc_empty[acc], ((acc_it / C::kAccStages) & 1u) ^ 1u, abort_flag, wait_limit)) break;
                if (C::kOverlap && acc_it != 0u &&
                    !mbar_wait(&bars->acc_head[acc ^ 1u], ((acc_it - 1u) / C::kAccStages) & 1u, abort_flag, wait_limit))
                    break;
                if (TRACE) trace_acc += clock64() - a0;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * C::kAccStride;
                for (uint32_t ks = 0; ks < k_stages; ks++, it++) {
                    const long long f0 = TRACE ? clock64() : 0;
                    if (!mbar_wait(&bars->full[slot], full_parity, abort_flag, wait_limit)) {
                        alive = false;
                        break;
                    }
                    if (TRACE) trace_full += clock64() - f0;
                    tc_fence_after();
                    const uint32_t kIdesc = *reinterpret_cast<volatile uint32_t*>(&bars->format[slot]) == kFormatCompact ? kIdescCompact
                                                                                                                 : kIdescBytes;
#pragma unroll
                    for (uint32_t sub = 0; sub < C::kSub; sub++) {
                    if (sub != 0u && ks >= doubles) break;
                    const uint32_t kb = first_block(ks) + sub;
                    const uint32_t block = slot * C::kSub + sub;  // index into the shared-memory arrays
                    const uint32_t groups = (kb + 1u == k_blocks && tail_groups != 0u) ? tail_groups : 4u;
                    // (by TMA a trailing half block lies in the second half of its operand tiles; a K step of 32 elements is 32 bytes:
                    // two 16-byte units of the start address)
                    const uint32_t first = USE_TMA ? 2u * (4u - groups) : 0u;
                    const uint64_t a_desc = a_desc0 + (uint64_t)(block * (C::kABytes >> 4) + first);
                    const uint64_t b_desc = b_desc0 + (uint64_t)(block * (C::kBTileBytes >> 4) + first);
#pragma unroll
                    for (uint32_t mx = 0; mx < C::kMatrices; mx++) tc_copy_scales(tmem_scales + 4u * mx, sf_desc0 + (C::weight_scales(slot, sub, mx) >> 4));
                    tc_copy_scales(sfb_tmem, sf_desc0 + (C::token_scales(slot, sub) >> 4));
#pragma unroll
                    for (uint32_t j = 0; j < 4u; j++) {
                        if (j < groups) {
#pragma unroll
                            for (uint32_t mx = 0; mx < C::kMatrices; mx++) {
                                tc_mma_block_scaled(d_tmem + mx * N_TILE, a_desc + (mx * (kATileBytes >> 4) + 2u * j),
                                                    b_desc + 2u * j, kIdesc | (j << 4) | (j << 29), tmem_scales + 4u * mx,
                                                    sfb_tmem, j == 0u ? (kb != 0u ? 1u : 0u) : 1u);
                            }
                        }
                    }
                    }
                    tc_commit(&bars->empty[slot]);  // the stage may be refilled once these MMAs retire
                    if (++slot == C::kStages) {
                        slot = 0u;
                        full_parity ^= 1u;
                    }
                }
                if (alive) tc_commit(&bars->acc_full[acc]);
            }
            // Nothing of this CTA may still be reading shared memory or using tensor memory when they are
            // released: the commit arrives once every MMA and scale copy issued above has retired. This wait has
            // its own limit and does not look at the abort flag, which is already set on the give-up path.
            tc_commit(&bars->drain);
            mbar_wait_winddown(&bars->drain, 0u, kWinddownCycles);
            if (TRACE && p.cta_trace) {  // per-CTA diagnostics: loop begin, loop end, stages, SM id
                uint32_t smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                uint64_t* mine = p.cta_trace + (size_t)((GATE_UP ? 0u : gridDim.x) + blockIdx.x) * 4u;
                mine[0] = cta_begin;
                mine[1] = global_timer_ns();
                mine[2] = it;
                mine[3] = smid;
            }
            if (TRACE && blockIdx.x == 0u) {
                trace[2] = (uint64_t)trace_full;                 // MMA thread: cycles waiting for operands
                trace[3] = (uint64_t)trace_acc;                  // MMA thread: cycles waiting for a free accumulator
                trace[4] = (uint64_t)(clock64() - trace_begin);  // MMA thread: cycles in its loop
                trace[5] = it;                                   // stages consumed
                trace[10] = global_timer_ns();                   // MMA loop ends
            }
        }
        __syncwarp();
    } else {
        // ===== epilogue: TMEM -> registers -> global =============================================
        const uint32_t quad = warp & 3u;  // the quadrant of tensor-memory lanes this warp may read
        const uint32_t epilogue_group = warp < 4u ? 0u : (warp - C::kFirstExtraEpilogueWarp) / 4u + 1u;
        const uint32_t frame_words = K * (I / 2u) + K;
        uint32_t acc_it = 0u, set_it = 0u;
        const bool whole_block = GATE_UP && p.g.act_block == 128u;  // the scale block of the fused quantisation is the tile's 128 rows
        long long trace_epi_wait = 0;
        const long long trace_begin = TRACE ? clock64() : 0;
        for (uint32_t tile = blockIdx.x; tile < tile_count; tile += gridDim.x, acc_it++) {
            const uint32_t pair = list.tiles[tile / m_tiles];
            const uint32_t m_tile = tile % m_tiles;
            const uint32_t expert = pair >> 16, n_tile = pair & 0xffffu;
            const uint32_t e_begin = p.work.expert_offsets[expert], e_end = p.work.expert_offsets[expert + 1u];
            const uint32_t first = e_begin + n_tile * N_TILE;
            const uint32_t valid = min(N_TILE, e_end - first);
            const uint32_t acc = acc_it % C::kAccStages;
            // where token j of the tile goes, and its route weight: a chain of two loads. With narrow tiles it is over before the
            // accumulator is ready, a lane per token; at the end of the kernel nothing else would hide it.
            uint64_t my_row = 0u;
            float my_weight = 0.0f;
            uint32_t my_route = kUnboundSlot;
            auto find = [&](uint32_t j, bool active) {
                my_row = 0u;
                my_weight = 0.0f;
                my_route = kUnboundSlot;
                if (!active || j >= valid) return;
                const uint32_t ri = __ldg(p.work.grouped_routes + first + j);
                // the row of the down stage's operand matrix that this route's activations go to
                my_route = (GATE_UP && p.q_out != nullptr) ? __ldg(p.down_position + ri) : kUnboundSlot;
                if (GATE_UP) {
                    if (p.intermediates != nullptr) my_row = reinterpret_cast<uint64_t>(reinterpret_cast<uint16_t*>(p.intermediates + (size_t)(ri / K) * frame_words) +
                                                        (size_t)(ri % K) * I);
                } else if (p.partial_outputs != nullptr) {
                    my_row = reinterpret_cast<uint64_t>(p.partial_outputs + (size_t)ri * H);
                } else {
                    my_row = reinterpret_cast<uint64_t>(p.outputs + (size_t)ri * H);
                    my_weight = nvmoe_bf16_to_f32(__ldg(p.routes + ri) >> 16);
                }
            };
            constexpr bool kNarrow = N_TILE <= 32u;
            if (kNarrow) find(lane, true);
            const long long e0 = TRACE ? clock64() : 0;
            // One warp watches the accumulator's barrier; the others sleep on a hardware barrier until it has a
            // verdict. A warp that polls takes issue slots from whatever shares its scheduler, and the epilogue warps
            // (three to a scheduler) wait through most of a tile beside the one thread that feeds the tensor pipe
            // and the one that issues the copies. Every epilogue warp reaches the hardware barrier in every round,
            // whatever the verdict, so none is left waiting there.
            if (warp == kWatchWarp) {
                const bool ready = mbar_wait_warp(&bars->acc_full[acc], (acc_it / C::kAccStages) & 1u, abort_flag, wait_limit);
                if (lane == 0u) *reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc_it & 1u]) = ready ? 1u : 0u;
                __threadfence_block();
            }
            named_barrier(1u, C::kEpilogueThreads);
            if (*reinterpret_cast<volatile uint32_t*>(&bars->acc_ready[acc_it & 1u]) == 0u) break;
            if (TRACE) trace_epi_wait += clock64() - e0;
            tc_fence_after();
            const uint32_t row = m_tile * C::kTileRows + quad * 32u + lane;  // (with row pairs: of the first half)
            const bool row_ok = row < out_rows;
            const uint32_t lane_addr = tmem_base + ((quad * 32u) << 16) + acc * C::kAccStride;
            // The epilogue groups share out a wide tile by 16-column chunks. A narrow tile (one or two chunks)
            // is shared out by sets of four tokens instead, every group reading the chunk: a tile of eight
            // tokens is then two groups' work side by side, not one group's in turn.
            constexpr bool kShareByFours = N_TILE <= 32u && C::kEpilogueGroups > 1u;
            for (uint32_t n0 = kShareByFours ? 0u : 16u * epilogue_group; n0 < N_TILE;
                 n0 += kShareByFours ? 16u : 16u * C::kEpilogueGroups) {
                // the chunk that overlapping accumulators share comes first: the last of the first one, the first of the second
                const uint32_t c0 = C::kOverlap && acc == 0u ? N_TILE - 16u - n0 : n0;
                const bool head = C::kOverlap && n0 == 0u;  // (group 0's)
                if (c0 >= valid) {  // uniform: no token of this tile lives in these columns
                    if (head) {
                        tc_fence_before();
                        mbar_arrive(&bars->acc_head[acc]);
                    }
                    continue;
                }
                if (kShareByFours) {
                    // does any of this chunk's sets of four fall to this group? (uniform)
                    bool mine = false;
#pragma unroll
                    for (uint32_t g0 = 0; g0 < 16u; g0 += 4u)
                        mine = mine || (c0 + g0 < valid && ((c0 + g0) / 4u) % C::kEpilogueGroups == epilogue_group);
                    if (!mine) continue;
                }
                uint32_t d0[16], d1[16];
                tmem_ld16(lane_addr + c0, d0);
                if (C::kMatrices == 2u) tmem_ld16(lane_addr + N_TILE + c0, d1);  // up, or the second 128 rows
                // lane j < 16 works out where token c0 + j of the tile goes (and its route weight) while the accumulators arrive; the
                // sixteen results are then handed round by shuffles. (A narrow tile has done so for all its tokens by now.)
                if (!kNarrow) find(c0 + lane, lane < 16u);
                const uint32_t t0 = kNarrow ? c0 : 0u;  // the lane that knows token c0
                tmem_ld_wait();
                if (head) {
                    tc_fence_before();
                    mbar_arrive(&bars->acc_head[acc]);
                }
                const bool quantise = GATE_UP && p.q_out != nullptr;  // host: only with scale blocks of 32 or 128 rows
                const bool store_rows = !GATE_UP || p.intermediates != nullptr;  // (uniform) a caller's rows; a layer only needs their codes
                // Four tokens at a time go through each step together, with no branch between them, so that
                // their instruction latencies overlap (the activation math is one long dependent chain per
                // value); columns past `valid` hold zeros and are only not stored.
#pragma unroll
                for (uint32_t g0 = 0; g0 < 16u; g0 += 4u) {
                    if (c0 + g0 >= valid) break;  // uniform
                    if (kShareByFours && ((c0 + g0) / 4u) % C::kEpilogueGroups != epilogue_group) continue;  // another group's
                    uint32_t bits[4];
#pragma unroll
                    for (uint32_t t = 0; t < 4u; t++) {
                        const uint32_t j = g0 + t;
                        if (GATE_UP) {
                            bits[t] = swiglu_bf16_bits(__uint_as_float(d0[j]), __uint_as_float(d1[j]), p.g.swiglu_limit,
                                                       p.g.swiglu_alpha, p.g.swiglu_up_offset);
                        } else {
                            const float weight = __shfl_sync(0xffffffffu, my_weight, t0 + j);
                            bits[t] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(__fmul_rn(__uint_as_float(d0[j]), weight)));
                        }
                    }
                    if (!GATE_UP && p.partial_outputs != nullptr) {
                        // tensor-parallel form: the raw f32 sums over this participant's columns, weighted and rounded
                        // only after the participants' planes have been added
#pragma unroll
                        for (uint32_t t = 0; t < 4u; t++) {
                            float* out = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, my_row, t0 + g0 + t));
                            if (c0 + g0 + t < valid && row_ok) out[row] = __uint_as_float(d0[g0 + t]);
                            if (ROW_PAIR && c0 + g0 + t < valid && row + kBlockM < out_rows) out[row + kBlockM] = __uint_as_float(d1[g0 + t]);
                        }
                        continue;
                    }
                    if (store_rows) {
#pragma unroll
                    for (uint32_t t = 0; t < 4u; t++) {
                        uint16_t* out = reinterpret_cast<uint16_t*>(__shfl_sync(0xffffffffu, my_row, t0 + g0 + t));
                        if (c0 + g0 + t < valid && row_ok) out[row] = (uint16_t)bits[t];
                        if (ROW_PAIR) {  // the second accumulator holds the next 128 output rows of the same tokens
                            const float weight = __shfl_sync(0xffffffffu, my_weight, t0 + g0 + t);
                            const uint32_t second = (uint32_t)__bfloat16_as_ushort(
                                __float2bfloat16_rn(__fmul_rn(__uint_as_float(d1[g0 + t]), weight)));
                            if (c0 + g0 + t < valid && row + kBlockM < out_rows) out[row + kBlockM] = (uint16_t)second;
                        }
                    }
                    }
                    if (quantise) {
                        // the activation quantisation of the down stage, on the values just rounded to bf16: one
                        // power-of-two scale per 32 rows, which is exactly this warp's share of the tile, or per 128
                        // rows, the share of the four warps of the group, which then hand their maxima round (a pass
                        // over the frames instead took 744 us for 147456 rows of 2048)
                        float m[4];
#pragma unroll
                        for (uint32_t t = 0; t < 4u; t++) m[t] = row_ok ? fabsf(nvmoe_bf16_to_f32(bits[t])) : 0.0f;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                            for (uint32_t t = 0; t < 4u; t++) m[t] = fmaxf(m[t], __shfl_xor_sync(0xffffffffu, m[t], o));
                        }
                        if (whole_block) {
                            // (the four warps of a group run through the same tokens; a set's maxima are overwritten two
                            // sets later, when every warp has passed the barrier of the set between)
                            uint16_t(&quad_max)[4][4] = maxima[epilogue_group][set_it++ & 1u];
                            if (lane < 4u)
                                quad_max[quad][lane] = (uint16_t)(__float_as_uint(lane == 0u ? m[0] : lane == 1u ? m[1] : lane == 2u ? m[2] : m[3]) >> 16);
                            named_barrier(2u + epilogue_group, 128u);
#pragma unroll
                            for (uint32_t t = 0; t < 4u; t++)
                                m[t] = fmaxf(fmaxf(fmaxf(0.0f, nvmoe_bf16_to_f32(quad_max[0][t])), nvmoe_bf16_to_f32(quad_max[1][t])),
                                             fmaxf(nvmoe_bf16_to_f32(quad_max[2][t]), nvmoe_bf16_to_f32(quad_max[3][t])));
                        }
                        const uint32_t first_row = m_tile * C::kTileRows + quad * 32u;
                        const bool writes_scale = lane == 0u && first_row < out_rows;
#pragma unroll
                        for (uint32_t t = 0; t < 4u; t++) {
                            const uint32_t dp = __shfl_sync(0xffffffffu, my_route, t0 + g0 + t);
                            const float scale = nvmoe_rounded_fp8_scale(m[t]);
                            // 1 / scale, exact: the scale is a power of two with a biased exponent in [107, 247]
                            const float inv = __uint_as_float(0x7f000000u - __float_as_uint(scale));
                            const uint8_t q =
                                (uint8_t)__nv_cvt_float_to_fp8(nvmoe_bf16_to_f32(bits[t]) * inv, __NV_SATFINITE, __NV_E4M3);
                            if (dp != kUnboundSlot) {  // (lanes past `valid` and routes the down stage skips)
                                if (row_ok) p.q_out[(size_t)dp * I + row] = q;
                                if (writes_scale)
                                    *p.q_e8m0.byte_at(dp, first_row / 32u) = (uint8_t)(nvmoe_f32_bits(scale) >> 23);
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&bars->acc_empty[acc]);
        }
        if (TRACE && blockIdx.x == 0u && threadIdx.x == 0u) {
            trace[6] = (uint64_t)trace_epi_wait;                 // epilogue: cycles waiting for an accumulator
            trace[7] = (uint64_t)(clock64() - trace_begin);      // epilogue: cycles in its loop
        }
    }

    // ---- teardown -------------------------------------------------------------------------------
    __syncthreads();
    if (warp == 4u) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::kTmemColumns);
    }
    if (threadIdx.x == 0u && *abort_flag) {
        raise_status(p.status, NVMOE_STATUS_WAIT_EXPIRED);
        winddown_pause();  // copies that no role waited for any more may still be landing
    }
    // latest exit over all CTAs (the timer only grows, so the last launch wins)
    if (TRACE && threadIdx.x == 0u) atomicMax(reinterpret_cast<unsigned long long*>(trace + 11), (unsigned long long)global_timer_ns());
}

// Re-tiles the packaged [rows][cols/32] scale bytes of one expert matrix into 512-byte blocks, one
// per (128-row tile, 128-column block): row r of the tile sits at (r % 32) * 16 + (r / 32) * 4 and
// holds the four scales of the block; positions past the matrix edge hold 127 (1.0) and are never
// multiplied with anything but zeros.  A block re-tiles only when the stamp differs.
__global__ void __launch_bounds__(128) derive_scales_kernel(const ExpertPtrs* experts, const uint64_t* stamps,
                                                           uint32_t matrices, uint32_t rows, uint32_t cols) {
    const uint32_t m_tiles = (rows + kBlockM - 1u) / kBlockM, k_blocks = (cols + kBlockK - 1u) / kBlockK;
    const uint32_t e = blockIdx.x / (matrices * m_tiles);
    const uint32_t mx = (blockIdx.x / m_tiles) % matrices, m_tile = blockIdx.x % m_tiles;
    const ExpertPtrs ptrs = experts[e];
    if (ptrs.w[0] == nullptr || ptrs.ts[mx] == nullptr) return;
    const uint64_t* stamp = stamps + ((size_t)e * matrices + mx) * 2u;
    if (stamp[0] == (uint64_t)(uintptr_t)ptrs.s[mx] && stamp[1] == ptrs.gen[mx]) return;
    const uint32_t r = threadIdx.x, row = m_tile * kBlockM + r, row_bytes = cols / 32u;
    // (the blocks of an expert's `matrices` tensors are interleaved: block (m_tile, kb) of tensor mx lies at
    // ((m_tile * k_blocks + kb) * matrices + mx) * 512, and ts[mx] already points at mx * 512)
    const size_t stride = (size_t)matrices * kScaleBlockBytes;
    uint8_t* out = const_cast<uint8_t*>(ptrs.ts[mx]) + (size_t)m_tile * k_blocks * stride + (r & 31u) * 16u + (r >> 5) * 4u;
    for (uint32_t kb = 0; kb < k_blocks; kb++) {
        uint32_t word = 0x7f7f7f7fu;
        if (row < rows && ptrs.format == kFormatNativeFp8) {
            // one exponent byte per 128 x 128 block, repeated over the block's four 32-column groups
            word = 0x01010101u * (uint32_t)ptrs.s[mx][(size_t)(row / 128u) * k_blocks + kb];
        } else if (row < rows) {
            word = 0u;
            for (uint32_t j = 0; j < 4u; j++) {
                const uint32_t c = kb * 4u + j;
                word |= (uint32_t)(c < row_bytes ? ptrs.s[mx][(size_t)row * row_bytes + c] : 127u) << (8u * j);
            }
        }
        *reinterpret_cast<uint32_t*>(out + (size_t)kb * stride) = word;
    }
}

__global__ void commit_stamps_kernel(const ExpertPtrs* experts, uint64_t* stamps, uint32_t matrices, uint32_t count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const ExpertPtrs ptrs = experts[i / matrices];
    const uint32_t mx = i % matrices;
    if (ptrs.w[0] == nullptr) return;
    stamps[(size_t)i * 2u] = (uint64_t)(uintptr_t)ptrs.s[mx];
    stamps[(size_t)i * 2u + 1u] = ptrs.gen[mx];
}

// (a whole warp) the template with an address patched in, as a map that the TMA unit may be given once it has been acquired
__device__ __forceinline__ void publish_map(uint8_t* map, const uint8_t* templ, unsigned char* smem_map, const uint8_t* address) {
    const uint32_t lane = threadIdx.x & 31u;
    reinterpret_cast<uint32_t*>(smem_map)[lane] = __ldg(reinterpret_cast<const uint32_t*>(templ) + lane);
    __syncwarp();
    if (lane == 0u) tensormap_replace_address(smem_map, address);
    __syncwarp();
    tensormap_publish(map, smem_map);
}

// One warp per map (an expert matrix's `per_matrix` of kWeightMaps): the template with the expert's weight address patched in;
// then one for the map of the set's derived scale copy. Bound by the latency of the copy's fence, once this way: tables that are
// resolved in every call add 35 us with 32 experts and 65 with 257 (38 and 69 with a warp that wrote three maps in turn).
__global__ void __launch_bounds__(32) build_tensormaps_kernel(const ExpertPtrs* experts, const uint8_t* templ, const uint8_t* derived,
                                                             uint8_t* maps, uint32_t matrices, uint32_t per_matrix) {
    __shared__ __align__(128) unsigned char sm[128];
    const uint32_t matrix = blockIdx.x / per_matrix, i = blockIdx.x % per_matrix;
    const uint32_t e = matrix / matrices, mx = matrix % matrices;
    const bool scales = derived != nullptr && blockIdx.x == gridDim.x - 1u;
    if (!scales && (experts[e].w[0] == nullptr || experts[e].w[mx] == nullptr)) return;
    // `templ` holds the maps of the compact form, those of the one-byte-per-element forms and that of the derived scales
    const uint8_t* mine = templ + ((scales ? 2u : experts[e].format == kFormatCompact ? 0u : 1u) * kWeightMaps + i) * 128u;
    publish_map(maps + ((size_t)matrix * kWeightMaps + i) * 128u, mine, sm, scales ? derived : experts[e].w[mx]);
}

// The same for the one matrix of a dense linear, whose addresses are the call's own: nothing about the matrix is kept
// between calls, so that scales rewritten in place by any means are what the next call reads. A block re-tiles 128 rows
// x 4 K blocks, a thread 4 rows of one K block and one 16-byte store. The last block writes the pointers and the tensor
// maps, a warp each. With scale blocks of 32 or 128 columns (LANES = block / 16; 0: none) further blocks quantise the input, a warp 512
// columns of one row, so that the launch takes little longer than that alone: bound by the latency of a load and a
// store; a warp takes a second piece, whose load is under way with the first's, where the pieces are more than a wave of blocks. Block of 777 x 7168 x 2048: 114.0 us
// with the quantisation in a launch of its own, 107 here; later 84.4 with one piece or two by blocks of 1.6 waves, 82.9 by one wave.
constexpr uint32_t kDenseKBlocks = 4u, kDenseThreads = 128u;
template <uint32_t LANES>
__global__ void __launch_bounds__(kDenseThreads) dense_prepare_kernel(DensePrepare p, uint32_t k_blocks, uint32_t retile_blocks) {
    __shared__ __align__(128) unsigned char sm[kWeightMaps * 128u];
    grid_dependency_sync();
    const uint32_t tile_total = p.tiles.list ? (p.tokens + p.tiles.n_tile - 1u) / p.tiles.n_tile : 0u;
    for (uint32_t i = blockIdx.x * kDenseThreads + threadIdx.x; p.lists && i < p.tokens; i += gridDim.x * kDenseThreads) {
        p.grouped[i] = i;
        if (i < tile_total) p.tiles.list[i] = i;  // (expert 0 << 16) | token tile
    }
    if (blockIdx.x < retile_blocks) {
        const uint32_t k_groups = (k_blocks + kDenseKBlocks - 1u) / kDenseKBlocks;
        const uint32_t m_tile = blockIdx.x / k_groups, row_bytes = p.cols / 32u;
        const uint32_t kb = blockIdx.x % k_groups * kDenseKBlocks + threadIdx.x % kDenseKBlocks, r = threadIdx.x / kDenseKBlocks;
        if (kb >= k_blocks) return;
        uint32_t word[4];
#pragma unroll
        for (uint32_t j = 0; j < 4u; j++) {
            const uint32_t row = m_tile * kBlockM + r + 32u * j;
            const uint8_t* in = p.scales + (size_t)row * row_bytes + kb * 4u;
            word[j] = 0x7f7f7f7fu;
            if (row < p.out_rows && row_bytes % 4u == 0u) {
                word[j] = __ldg(reinterpret_cast<const uint32_t*>(in));
            } else if (row < p.out_rows && row_bytes % 2u == 0u) {
                word[j] = __ldg(reinterpret_cast<const uint16_t*>(in)) |
                          (kb * 4u + 2u < row_bytes ? (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(in) + 1) : 0x7f7fu) << 16;
            } else if (row < p.out_rows) {
                word[j] = 0u;
#pragma unroll
                for (uint32_t b = 0; b < 4u; b++) word[j] |= (uint32_t)(kb * 4u + b < row_bytes ? __ldg(in + b) : 127u) << (8u * b);
            }
        }
        *reinterpret_cast<uint4*>(p.derived + ((size_t)m_tile * k_blocks + kb) * kScaleBlockBytes + r * 16u) =
            make_uint4(word[0], word[1], word[2], word[3]);
        return;
    }
    if (blockIdx.x != gridDim.x - 1u) {
        if (LANES == 0u) return;
        const uint32_t lane = threadIdx.x & 31u, chunks = (p.cols + 511u) / 512u, items = p.tokens * chunks;
        const uint32_t warps = (gridDim.x - 1u - retile_blocks) * (kDenseThreads / 32u);
        // two pieces at a time, whose loads are under way together
        for (uint32_t item = (blockIdx.x - retile_blocks) * (kDenseThreads / 32u) + (threadIdx.x >> 5); item < items; item += 2u * warps) {
            uint32_t out[2][4], word[2];
#pragma unroll
            for (uint32_t u = 0; u < 2u; u++) {
                const uint32_t at = item + u * warps, row = at / chunks, col = (at % chunks) * 512u + lane * 16u;
                // (columns come in whole blocks: the lanes of a block agree)
                quantize_sixteen<(LANES == 0u ? 1u : LANES)>(p.input + (size_t)row * p.cols + col, at < items && col < p.cols, lane, out[u], word[u]);
            }
#pragma unroll
            for (uint32_t u = 0; u < 2u; u++) {
                const uint32_t at = item + u * warps, row = at / chunks, col = (at % chunks) * 512u + lane * 16u;
                if (at >= items || col >= p.cols) continue;
                *reinterpret_cast<uint4*>(p.q + (size_t)row * p.cols + col) = make_uint4(out[u][0], out[u][1], out[u][2], out[u][3]);
                if ((lane & 7u) == 0u) *p.q_e8m0.at(row, col / 128u) = word[u];
            }
        }
        return;
    }
    if (!p.lists) return;
    if (threadIdx.x == 0u) {
        p.offsets[0] = 0u;
        p.offsets[1] = p.tokens;
        if (p.tiles.count) *p.tiles.count = tile_total;
        *p.ptrs = ExpertPtrs{{p.weights, nullptr}, {p.scales, nullptr}, {p.derived, nullptr}, {0u, 0u}, kFormatCompact, 0u};
    }
    const uint32_t i = threadIdx.x / 32u;
    if (p.map_template != nullptr && i < kWeightMaps) publish_map(p.map + i * 128u, p.map_template + i * 128u, sm + i * 128u, p.weights);
}

int g_sm_count[16] = {0};

int sm_count() {  // of the current device
    int dev = 0;
    cudaGetDevice(&dev);
    if (g_sm_count[dev & 15] == 0) cudaDeviceGetAttribute(&g_sm_count[dev & 15], cudaDevAttrMultiProcessorCount, dev);
    return g_sm_count[dev & 15];
}

template <bool GATE_UP, uint32_t N_TILE, bool USE_TMA, bool ROW_PAIR>
void launch_n(const ExpertLaunch& p, int sms, cudaStream_t stream) {
    using C = Config<GATE_UP, N_TILE, USE_TMA, ROW_PAIR>;
    // the traced instantiation only when a plan's trace was armed (and only for the TMA form)
    if (USE_TMA && p.cta_trace != nullptr) {
        launch_chained(experts_tc_kernel<GATE_UP, N_TILE, USE_TMA, ROW_PAIR, USE_TMA>, dim3(sms), dim3(C::kThreads), C::kSmemBytes, stream, p,
                       TileList{p.tile_list, p.tile_count});
    } else {
        launch_chained(experts_tc_kernel<GATE_UP, N_TILE, USE_TMA, ROW_PAIR, false>, dim3(sms), dim3(C::kThreads), C::kSmemBytes, stream, p,
                       TileList{p.tile_list, p.tile_count});
    }
}

// Whether a down launch takes two row tiles at a time: always with wide token tiles, and with narrow ones (TMA form)
// when that leaves the SMs enough tiles, counted as if every expert were selected (what routing, a partition
// or absent experts leave of them is not known here). A stage of a row pair is one K block: one box of 256 weight rows, one token
// box, two scale copies. One of a single row tile is two K blocks: a weight box, a token box and a scale copy, for the
// same weight bytes and twice the token rows. Single row tiles spread over the SMs in finer steps, which 32-token tiles gain
// from while there are few rounds, 16-token tiles only where pairs leave SMs without a tile. Layer of intermediate 1536, single rows /
// row pairs, us, by rounds: 32-token tiles 0.65 51.3 / 52.2, 1.3 62.9 / 67.4, 1.95 81.2 / 85.0, 2.6 100.4 / 101.4, 3.5 113.4 / 113.6, 3.9
// 124.6 / 126.0, 5.2 143.4 / 142.6, 6.05 167.8 / 165.9, 7.8 191.9 / 188.8, 10.4 234.1 / 228.7, 24 519 / 506; 16-token tiles 0.65 51.8 /
// 48.9, 1.3 60.7 / 58.3, 2.6 84.3 / 80.1, 5.2 129.9 / 126.5, 6.05 147.5 / 142.7, 10.4 212.2 / 207.1, 24 436 / 425; 16 experts of 2048 x 256 and x 512, 0.86
// 29.6 / 27.0, 32.3 / 29.3; 24 of 4096 x 256, 2.6 42.1 / 38.2.
bool takes_row_pairs(const ExpertLaunch& p, uint32_t n_tile, bool tma, int sms) {
    if (n_tile >= kRowPairTokens) return true;
    if (!tma) return false;
    const uint64_t routes = (uint64_t)p.tokens * (p.g.routed_k + p.g.always_count);
    const uint64_t lists = routes < p.work.num_experts ? routes : p.work.num_experts;
    const uint64_t tiles = lists * ((p.g.hidden_size + 2u * kBlockM - 1u) / (2u * kBlockM));
    return n_tile <= 16u ? 2u * tiles >= (uint64_t)sms : tiles >= (uint64_t)kRowPairRounds * (uint64_t)sms;
}

template <bool GATE_UP>
void launch(const ExpertLaunch& p, cudaStream_t stream) {
    const int sms = sm_count();
    const uint32_t n = p.token_rows;
    if (p.pairs) {
        launch_experts_pair(p, GATE_UP, sms, stream);
        return;
    }
    const bool tma = p.tmaps != nullptr;
    const bool pairs = !GATE_UP && takes_row_pairs(p, n, tma, sms);
    if (tma && pairs) {
        switch (n) {
            case 16u: launch_n<GATE_UP, 16u, true, !GATE_UP>(p, sms, stream); break;
            case 32u: launch_n<GATE_UP, 32u, true, !GATE_UP>(p, sms, stream); break;
            case 64u: launch_n<GATE_UP, 64u, true, !GATE_UP>(p, sms, stream); break;
            default: launch_n<GATE_UP, 96u, true, !GATE_UP>(p, sms, stream); break;
        }
    } else if (tma) {
        switch (n) {
            case 16u: launch_n<GATE_UP, 16u, true, false>(p, sms, stream); break;
            case 32u: launch_n<GATE_UP, 32u, true, false>(p, sms, stream); break;
            case 64u: launch_n<GATE_UP, 64u, true, !GATE_UP>(p, sms, stream); break;
            default: launch_n<GATE_UP, 96u, true, !GATE_UP>(p, sms, stream); break;
        }
    } else {
        switch (n) {
            case 16u: launch_n<GATE_UP, 16u, false, false>(p, sms, stream); break;
            case 32u: launch_n<GATE_UP, 32u, false, false>(p, sms, stream); break;
            case 64u: launch_n<GATE_UP, 64u, false, !GATE_UP>(p, sms, stream); break;
            case 96u: launch_n<GATE_UP, 96u, false, !GATE_UP>(p, sms, stream); break;
            default: launch_n<GATE_UP, 128u, false, !GATE_UP>(p, sms, stream); break;
        }
    }
}

template <bool GATE_UP, uint32_t N_TILE, bool USE_TMA, bool ROW_PAIR>
void configure_one() {
    constexpr int kBytes = (int)Config<GATE_UP, N_TILE, USE_TMA, ROW_PAIR>::kSmemBytes;
    cudaFuncSetAttribute(experts_tc_kernel<GATE_UP, N_TILE, USE_TMA, ROW_PAIR, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (USE_TMA)
        cudaFuncSetAttribute(experts_tc_kernel<GATE_UP, N_TILE, USE_TMA, ROW_PAIR, USE_TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
}

template <uint32_t N_TILE>
void configure_tile() {
    configure_one<true, N_TILE, false, false>();
    configure_one<false, N_TILE, false, (N_TILE >= 64u)>();
    if constexpr (N_TILE <= 96u) {
        configure_one<true, N_TILE, true, false>();
        configure_one<false, N_TILE, true, true>();
    }
    if constexpr (N_TILE < 64u) configure_one<false, N_TILE, true, false>();
}

}  // namespace

uint32_t device_sm_count() { return (uint32_t)sm_count(); }

bool tc_shape_supported(const nvmoe_geometry& g) {
    return g.hidden_size % 32u == 0u && g.intermediate_size % 32u == 0u && g.act_block % 32u == 0u;
}

bool tc_enabled_by_default() { return true; }

// The token tile of CTA pairs (the reasons stand with tc_token_tile_for).
static TokenTile pair_tile_for(uint32_t num_experts, uint32_t per_expert, uint32_t row_tiles) {
    const uint64_t sms = (uint64_t)sm_count();
    const uint32_t rows[4] = {kPairTokens, 192u, 128u, 64u};
    TokenTile best{kPairTokens, true};
    const uint64_t half_tiles = (uint64_t)num_experts * (2ull * per_expert + kPairTokens) / kPairTokens;
    if (num_experts > 1u && (half_tiles + 1u) / 2u * row_tiles > sms) return best;
    uint64_t best_cost = ~0ull;
    for (uint32_t i = 0; i < 4u; i++) {
        const uint64_t tiles = (uint64_t)num_experts * ((per_expert + rows[i] - 1u) / rows[i]) * row_tiles;
        const uint64_t cost = (tiles + sms / 2u - 1u) / (sms / 2u) * (256u + rows[i]);
        if (cost < best_cost) {
            best_cost = cost;
            best.rows = rows[i];
        }
    }
    return best;
}

// A dense linear has one matrix, whose row tiles leave most SMs idle, so that what a stage takes by itself counts: pairs from fewer tokens on than
// for a layer's experts, where K is long. One CTA a tile / pairs, us a call (quantisation included), 7168 columns to 2048 rows: 24 tokens 15.8 / 17.7,
// 32 23.9 / 17.6, 48 24.2 / 17.8, 64 26.3 / 17.9, 96 26.8 / 18.1; 2880 to 2880: 24 10.7 / 12.5, 32 14.6 / 12.7, 64 16.1 / 13.0; 2048 to 7168: 24 9.5 / 11.1, 32 12.2 /
// 11.3, 64 13.7 / 11.5; 1024 to 4096: 32 9.3 / 9.8, 48 9.6 / 9.9, 64 10.7 / 9.9; 512 to 1024: 24 7.0 / 8.8, 64 9.3 / 9.0. (Runs of a tile's stages by several
// pairs, whose sums the last one adds up: 2 us less for 7168 columns and up to 64 tokens, level or slower elsewhere. Token rows by linear copies from
// operands that lie as shared memory holds them, past the scale warp: 2 us more at 7168 columns.)
TokenTile tc_dense_tile_for(uint32_t tokens, uint32_t out_rows, uint32_t cols, bool tma) {
    const bool pairs = tma && tokens > (cols >= 2048u ? kTokenMapFrom[2] : kTokenMapFrom[3]) && tokens <= kPairsFrom;
    if (pairs) return pair_tile_for(1u, tokens, (out_rows + 2u * kBlockM - 1u) / (2u * kBlockM));
    return tc_token_tile_for(tokens, 1u, 1u, out_rows, false, tma);
}

TokenTile tc_token_tile_for(uint32_t tokens, uint32_t routes_per_token, uint32_t num_experts, uint32_t out_rows, bool gate_up, bool tma) {
    // tokens per expert if routing were uniform; skew only adds token tiles
    const uint32_t routes = tokens * routes_per_token;
    const uint32_t per_expert = (routes + num_experts - 1u) / num_experts;
    // the narrowest tile that holds an expert's tokens (with some room for skew: a second tile reads the weights again)
    if (per_expert <= kTokenMapFrom[1]) return {16u, false};
    if (per_expert <= kTokenMapFrom[2]) return {32u, false};
    if (per_expert <= kTokenMapFrom[3]) return {64u, false};
    if (per_expert <= kPairsFrom) return {96u, false};
    const uint32_t row_tiles = gate_up ? (out_rows + kBlockM - 1u) / kBlockM : (out_rows + 2u * kBlockM - 1u) / (2u * kBlockM);
    const uint64_t sms = (uint64_t)sm_count();
    // Beyond that CTA pairs. One CTA with tiles of 96 / pairs, us a layer, by tokens an expert: 32 experts of 2880 x 2880, 104
    // 205.7 / 183.8, 128 223.4 / 219.7, 192 290.4 / 264.7, 240 323.4 / 283.1; 128 of them, 104 731 / 711, 128 867 / 835, 192 1128 /
    // 1031. In layers that take one round of the SMs either way
    // the two are within a few percent: 16 experts of 768 x 512, 104 55.5 / 55.6, 128 54.0 / 55.3, 192 60.8 / 60.3, 240 61.9 / 66.0;
    // 8 of 1024 x 1024, 128 47.2 / 47.3, 192 60.3 / 61.2. (Dense linears have a lower line: tc_dense_tile_for.)
    // An expert takes several tiles. Where they are more than two rounds of the pairs, the widest: a stage takes 350 ns and 1.7 a
    // column (gate/up of 4096 tokens of 32 experts, all tiles of one width, ns a stage: 64 467, 128 581, 192 672, 240 761), a tile
    // with fewer tokens runs with fewer columns, and the loads of several experts differ, so that narrower tiles fit none of them
    // better: layers with the width that the count below chose / 240, 4096 tokens of 32 experts (192) 557.6 / 534.0 us, 8192 of 128
    // (128) 1439 / 1274, 16384 of 256 of 7168 x 2048 (192) 8606 / 8352. (An expert's last tile counts as half full.)
    // In fewer rounds, or with one expert, whose load is the call's, the fewest rounds x stage time wins, as 256 + columns, with
    // every expert at the mean load and its last tile at full width: dense block of 777 rows (128) 95.7 us, with 192 throughout
    // 110, with 240 139.
    if (tma) return pair_tile_for(num_experts, per_expert, row_tiles);
    // Shapes without tensor maps: the widest tile, by the same count of rounds. A stage of 128 columns takes 8/7 of the time
    // of one of 96 (0.527 and 0.461 us with whole rounds of either).
    const uint32_t widths[2] = {128u, 96u}, stage_time[2] = {8u, 7u};
    uint32_t best = 0u;
    uint64_t best_cost = ~0ull;
    for (uint32_t i = 0; i < 2u; i++) {
        const uint64_t tiles = (uint64_t)num_experts * ((per_expert + widths[i] - 1u) / widths[i]) * row_tiles;
        const uint64_t cost = (tiles + sms - 1u) / sms * stage_time[i];
        if (cost < best_cost) {
            best_cost = cost;
            best = widths[i];
        }
    }
    return {best, false};
}

size_t tc_derived_scale_bytes(uint32_t rows, uint32_t cols) {
    return (size_t)((rows + kBlockM - 1u) / kBlockM) * ((cols + kBlockK - 1u) / kBlockK) * kScaleBlockBytes;
}

void launch_derive_scales_tc(const ExpertLaunch& p, bool gate_up, cudaStream_t stream) {
    const uint32_t matrices = gate_up ? 2u : 1u;
    const uint32_t rows = gate_up ? p.g.intermediate_size : p.g.hidden_size;
    const uint32_t cols = gate_up ? p.g.hidden_size : p.g.intermediate_size;
    const uint32_t m_tiles = (rows + kBlockM - 1u) / kBlockM;
    derive_scales_kernel<<<p.work.num_experts * matrices * m_tiles, 128, 0, stream>>>(p.work.experts, p.scale_stamps,
                                                                                      matrices, rows, cols);
    const uint32_t count = p.work.num_experts * matrices;
    commit_stamps_kernel<<<(count + 127u) / 128u, 128, 0, stream>>>(p.work.experts, p.scale_stamps, matrices, count);
}

bool dense_prepare_quantises(const DensePrepare& p, uint32_t act_block) {
    return p.derived && (act_block == 32u || act_block == 128u) && (reinterpret_cast<uintptr_t>(p.input) & 15u) == 0u &&
           (uint64_t)p.tokens * ((p.cols + 511u) / 512u) <= 0x3fffffffull;
}

bool launch_dense_prepare(const DensePrepare& p, uint32_t act_block, cudaStream_t stream) {
    const uint32_t m_tiles = (p.out_rows + kBlockM - 1u) / kBlockM, k_blocks = (p.cols + kBlockK - 1u) / kBlockK;
    const uint32_t retile = p.derived ? m_tiles * ((k_blocks + kDenseKBlocks - 1u) / kDenseKBlocks) : 0u;
    const uint64_t warps = (uint64_t)p.tokens * ((p.cols + 511u) / 512u);
    const bool quantises = dense_prepare_quantises(p, act_block);
    // (without rows to quantise, as many blocks as the schedule's lists ask for)
    uint32_t others = quantises ? (uint32_t)((warps + 3u) / 4u) : (p.tokens + kDenseThreads - 1u) / kDenseThreads;
    // A warp takes further pieces of rows, two at a time, rather than that a second wave of blocks is needed (an SM holds 10): while that asks for two rounds
    // at most. Beyond, 16 blocks an SM, which even out the rounds. Block of 2048 rows of 7168 columns, us, 16 / 10 an SM: 501 tokens 75.6 / 73.8, 777 84.4 /
    // 82.9, 1200 (1.7 rounds) 99.8 / 99.4, 2048 (2.9) 139.4 / 140.9.
    const uint32_t sms = (uint32_t)sm_count();
    const uint32_t wave = sms * 10u > retile + 1u + sms ? sms * 10u - retile - 1u : sms;
    const uint32_t room = warps <= 16ull * wave ? wave : sms * 16u > retile + 1u + sms ? sms * 16u - retile - 1u : sms;
    if (quantises && others > room) others = room;
    const auto kernel = !quantises ? dense_prepare_kernel<0u> : act_block == 32u ? dense_prepare_kernel<2u> : dense_prepare_kernel<8u>;
    launch_chained(kernel, dim3(retile + others + 1u), dim3(kDenseThreads), 0, stream, p, k_blocks, retile);
    return quantises;
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's encoder, looked up through the runtime (no link-time dependency on libcuda)
static EncodeFn tensor_map_encoder() {
    static EncodeFn encode = nullptr;
    if (!encode) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return nullptr;
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    return encode;
}

bool tc_encode_bf16_map(void* map128, const void* base, uint32_t rows, uint32_t cols, uint32_t box_cols, uint32_t box_rows) {
    const EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {(cuuint64_t)cols * 2u};
    const cuuint32_t box[2] = {box_cols, box_rows}, step[2] = {1u, 1u};
    CUtensorMap map;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

bool tc_replace_map_address(void* map128, const void* device_address) {
    typedef CUresult (*ReplaceFn)(CUtensorMap*, void*);
    static const ReplaceFn replace = [] {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapReplaceAddress", &fn, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
        return reinterpret_cast<ReplaceFn>(ok ? fn : nullptr);
    }();
    CUtensorMap map;
    std::memcpy(&map, map128, 128);
    if (!replace || replace(&map, const_cast<void*>(device_address)) != CUDA_SUCCESS) return false;
    std::memcpy(map128, &map, 128);
    return true;
}

bool tc_encode_weight_map(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, uint32_t box_rows) {
    // The packaged [rows][cols/2] bytes seen as a 3-D tensor of 4-bit elements {128 elements, blocks, rows} whose blocks of
    // 128 columns start every 64: a box {128, 1, 128} is one operand tile, at block 2 kb that of K block kb, at the last
    // block the 128 columns that end with the row. (The padded 4-bit type wants 32-byte strides, so cols % 64 == 0, and
    // whole 128-element rows.)
    if (cols < kBlockK || cols % 64u != 0u) return false;
    EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[3] = {kBlockK, cols / 64u - 1u, rows};
    const cuuint64_t strides[2] = {32u, cols / 2u};
    const cuuint32_t box[3] = {kBlockK, 1u, box_rows};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    CUtensorMap map;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 3, any_device_address, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

bool tc_encode_weight_map_bytes(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, uint32_t box_rows) {
    // One E4M3 byte per element, seen like the compact form as {128 elements, blocks every 64 columns, rows}: the
    // same box coordinates fetch the same operand tile, now without padding.
    if (cols < kBlockK || cols % kBlockK != 0u) return false;
    EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[3] = {kBlockK, cols / 64u - 1u, rows};
    const cuuint64_t strides[2] = {64u, cols};
    const cuuint32_t box[3] = {kBlockK, 1u, box_rows};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    CUtensorMap map;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, any_device_address, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

// a 3-D map of one- or four-byte elements, rows of `dims[0]` elements
static bool encode_3d(void* map128, CUtensorMapDataType type, void* base, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2],
                      const cuuint32_t (&box)[3], CUtensorMapSwizzle swizzle) {
    EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    CUtensorMap map;
    if (encode(&map, type, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

bool tc_encode_pair_weight_map(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, bool bytes) {
    if (cols < kBlockK || cols % (bytes ? kBlockK : 64u) != 0u) return false;
    const uint32_t half = bytes ? 1u : 2u;  // elements to a byte
    return encode_3d(map128, bytes ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, any_device_address,
                     {kBlockK, rows, cols / kBlockK}, {cols / half, kBlockK / half}, {kBlockK, kBlockM, 2u}, CU_TENSOR_MAP_SWIZZLE_128B);
}

bool tc_encode_pair_token_map(void* map128, void* base, uint32_t rows, uint32_t cols, uint32_t box_rows) {
    if (cols < kBlockK || cols % 16u != 0u || rows == 0u) return false;
    return encode_3d(map128, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, {kBlockK, rows, cols / kBlockK}, {cols, kBlockK}, {kBlockK, box_rows, 2u},
                     CU_TENSOR_MAP_SWIZZLE_128B);
}

bool tc_encode_pair_scale_map(void* map128, void* any_device_address, uint32_t sources, uint32_t blocks) {
    return encode_3d(map128, CU_TENSOR_MAP_DATA_TYPE_UINT32, any_device_address, {kScaleBlockBytes / 4u, sources, blocks},
                     {kScaleBlockBytes, sources * kScaleBlockBytes}, {kScaleBlockBytes / 4u, 1u, 2u}, CU_TENSOR_MAP_SWIZZLE_NONE);
}

bool tc_encode_token_scale_map(void* map128, void* base, uint32_t words, uint32_t rows) {
    if (words % 4u != 0u || words == 0u || rows == 0u) return false;
    EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {words, rows};
    const cuuint64_t strides[1] = {4ull * words};
    const cuuint32_t box[2] = {kPairTokens + 4u, 2u};
    const cuuint32_t estr[2] = {1u, 1u};
    CUtensorMap map;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

bool tc_encode_activation_map(void* map128, void* base, uint32_t rows, uint32_t cols, uint32_t n_tile) {
    if (cols % 16u != 0u || rows == 0u) return false;
    EncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols};
    const cuuint32_t box[2] = {kBlockK, n_tile};
    const cuuint32_t estr[2] = {1u, 1u};
    CUtensorMap map;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(map128, &map, 128);
    return true;
}

void launch_build_tensormaps_tc(const ExpertLaunch& p, bool gate_up, const uint8_t* templ, cudaStream_t stream) {
    const uint32_t matrices = gate_up ? 2u : 1u, per_matrix = tc_weight_maps(gate_up, p.scale_base != nullptr);
    build_tensormaps_kernel<<<p.work.num_experts * matrices * per_matrix + (p.scale_base ? 1u : 0u), 32, 0, stream>>>(
        p.work.experts, templ, p.scale_base, const_cast<uint8_t*>(p.tmaps), matrices, per_matrix);
}

void tc_configure_kernels() {
    configure_tile<16u>();
    configure_tile<32u>();
    configure_tile<64u>();
    configure_tile<96u>();
    configure_tile<128u>();
    pair_configure_kernels();
    layer_configure_kernels();
}

// Both expert stages of a layer call in one launch, counted as if every expert were selected and had the mean load:
// - Gate/up is more than a round of the SMs. In less, the one kernel's longer set-up and its down tiles of 256 rows cost more than the second
//   launch: 16 gate/up tiles (tiny, 8 tokens) 22.0 us by two launches / 23.3, 32 (64 tokens) 25.2 / 28.0, 92 (one token of 32 experts of
//   2880 x 2880) 38.9 / 40.7.
// - Beyond 1.6 rounds, K of gate/up is long enough: 12 stages for tiles of 16 tokens, for wider ones 18 and one for every twenty tokens of an
//   expert. Short K loses by the one kernel, the more the more tokens a tile has, as if its epilogue took longer than that of the two and
//   the stages of the next tile alone hid it (announcements by a warp of their own made it no better). Layers, two / one, us: 16-token
//   tiles, 4 stages (512 x 4096, 32 experts) 49.7 / 63.7, 6 (768 x 3072, 64) 75.1 / 83.0, 12 (1536 x 2048, 128, 64 tokens) 120.6 / 114.3, 16 (2048 x 1536, 64)
//   86.3 / 78.8; 32 tokens, 12 stages (1536 x 2304, 32) 64.8 / 70.8, 23 (2880 x 2880, 32) 114.6 / 101.4; 64, 12 stages (1536 x 768, 128) 112.6 /
//   121.3, 23 128.3 / 120.9; 96, 12 stages 182.7 / 203.8, 16 (2048 x 1536, 64) 157.3 / 172.5, 23 180.2 / 172.5.
// - K of down is at least eight stages, or that of gate/up 32 with tiles of 64 tokens or more, and the down tiles of 256 rows fill the SMs:
//   4608 x 256, 128 experts, 32 tokens 65.2 / 70.7, 2048 x 2560, 16, eight tokens 44.0 / 46.6.
// Over 2000 layers drawn from 384 to 7168 columns, 256 to 4096 intermediate ones and 16 to 128 experts, two / one: the 932 beyond 1.6 rounds that
// these lines send here, medians 1.04 to 1.05 by width of the tile, 0.94 to 1.17; the 795 others there, medians 0.93 to 0.96, 0.70 to 1.10. In fewer
// rounds the two are level on the whole, whatever K is: medians 1.00 to 1.02, 0.84 to 1.37.
bool tc_layer_in_one_launch(uint32_t tokens, uint32_t routes_per_token, uint32_t num_experts, uint32_t hidden, uint32_t intermediate, uint32_t token_rows) {
    const uint64_t routes = (uint64_t)tokens * routes_per_token, lists = routes < num_experts ? routes : num_experts, sms = (uint64_t)sm_count();
    const uint64_t tiles = lists * ((intermediate + kBlockM - 1u) / kBlockM), down_tiles = lists * ((hidden + 2u * kBlockM - 1u) / (2u * kBlockM));
    if (tiles <= sms) return false;
    if (5u * tiles <= 8u * sms) return true;
    const uint64_t stages = (hidden + kBlockK - 1u) / kBlockK, per_expert = (routes + num_experts - 1u) / num_experts;
    const bool long_gate = token_rows <= 16u ? stages >= 12u : 20u * stages >= 360u + per_expert;
    const bool long_down = intermediate > 7u * kBlockK || (token_rows >= 64u && stages >= 32u);
    return long_gate && long_down && down_tiles >= sms;
}
void launch_layer_tc(const LayerLaunch& p, cudaStream_t stream) { launch_experts_layer(p, sm_count(), stream); }
void launch_gate_up_tc(const ExpertLaunch& p, cudaStream_t stream) { launch<true>(p, stream); }
void launch_down_tc(const ExpertLaunch& p, cudaStream_t stream) { launch<false>(p, stream); }

}  // namespace nvmoe
