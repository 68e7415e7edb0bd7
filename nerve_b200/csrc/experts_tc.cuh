// Interface of the tcgen05 grouped expert kernels (experts_tc.cu).
#pragma once
#include "common.cuh"

namespace nvmoe {

// Shapes the tensor-core path takes: columns in whole 32-blocks with a power-of-two activation
// scale per block (always true for the plan's own quantiser).
bool tc_shape_supported(const nvmoe_geometry& g);
// Whether "automatic" picks the tensor-core path.
bool tc_enabled_by_default();
void tc_configure_kernels();
// Encodes the template tensor map of a [rows][cols] weight matrix (any 32-byte aligned device address
// will do: it is replaced per expert). False when the shape cannot use TMA.
bool tc_encode_weight_map(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, uint32_t box_rows);
// The same for a matrix held as one E4M3 byte per element (pre-expanded or native FP8 resources).
bool tc_encode_weight_map_bytes(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, uint32_t box_rows);
// Tensor maps of a weight matrix: boxes of 128 rows x one K block, 128 rows x two, 256 rows x one; and how many of them a
// stage's kernels use (gate/up has tiles of 128 rows of either matrix, and two K blocks a copy in CTA pairs only).
constexpr uint32_t kWeightMaps = 3u;
constexpr uint32_t tc_weight_maps(bool gate_up, bool with_pairs) { return !gate_up ? 3u : with_pairs ? 2u : 1u; }
// Encodes the tensor map of an expert-grouped activation matrix [rows][cols] of E4M3 bytes with a box of
// n_tile rows x 128 bytes (the operand tile of one K block). False when tensor maps are unavailable.
bool tc_encode_activation_map(void* map128, void* base, uint32_t rows, uint32_t cols, uint32_t n_tile);
// The tensor maps whose boxes bring two K blocks at a time: a weight matrix in the compact or a one-byte form (128 rows),
// expert-grouped token rows, and for CTA pairs the derived scales of a set (blocks of 512 bytes, `sources` to a (row tile,
// K block)) and the token scales [rows = K blocks][words].
bool tc_encode_pair_weight_map(void* map128, void* any_device_address, uint32_t rows, uint32_t cols, bool bytes);
// Rows of bf16 numbers, in 128-byte swizzled boxes.
bool tc_encode_bf16_map(void* map128, const void* base, uint32_t rows, uint32_t cols, uint32_t box_cols, uint32_t box_rows);
// A map encoded above, for another address. False where the driver cannot.
bool tc_replace_map_address(void* map128, const void* device_address);
bool tc_encode_pair_token_map(void* map128, void* base, uint32_t rows, uint32_t cols, uint32_t box_rows);
bool tc_encode_pair_scale_map(void* map128, void* any_device_address, uint32_t sources, uint32_t blocks);
bool tc_encode_token_scale_map(void* map128, void* base, uint32_t words, uint32_t rows);
// per-expert tensor maps = template + the expert's weight address (p.tmaps must be set; tc_weight_maps of each matrix), and
// after them the map of the derived scales (p.scale_base: the plan's calls may run by CTA pairs)
void launch_build_tensormaps_tc(const ExpertLaunch& p, bool gate_up, const uint8_t* templ, cudaStream_t stream);
// What a dense linear needs before its expert kernel, in one launch: the schedule (every row a route of expert 0 in row
// order), what hangs on its matrix (the pointers and, for the tensor path (`derived` set), the re-tiled scales and the
// tensor map (map_template null: none); weights and scales are 32-byte aligned), and the quantised input rows. False when
// the input needs one of the general quantisations, which then follows: CUDA-core path, scale blocks other than 32 or 128
// columns, rows off the 16-byte grid.
struct DensePrepare {
    const uint8_t* weights;
    const uint8_t* scales;
    uint32_t out_rows, cols, tokens;
    uint32_t* grouped;
    uint32_t* offsets;
    TileOut tiles;
    ExpertPtrs* ptrs;
    uint8_t* derived;
    const uint8_t* map_template;
    uint8_t* map;
    bool lists;              // whether the lists, the pointers and the maps are asked for (CTA pairs need none of them)
    const uint16_t* input;
    uint8_t* q;
    ScaleWords q_e8m0;
};
bool dense_prepare_quantises(const DensePrepare& p, uint32_t act_block);  // whether it quantises the input too
bool launch_dense_prepare(const DensePrepare& p, uint32_t act_block, cudaStream_t stream);
// Token tile of a stage: rows of the operand matrix per entry of the (expert, token tile) list, by a CTA pair (experts_pair.cu)
// or by one CTA (then one of the kernel's tile widths).
struct TokenTile {
    uint32_t rows;
    bool pair;
};
// token tile of a stage for this many tokens and rows of its weight matrix (the (expert, token tile) list must be
// built with it); tma: the stage's shapes have tensor maps
TokenTile tc_token_tile_for(uint32_t tokens, uint32_t routes_per_token, uint32_t num_experts, uint32_t out_rows, bool gate_up, bool tma);
TokenTile tc_dense_tile_for(uint32_t tokens, uint32_t out_rows, uint32_t cols, bool tma);  // of a dense linear of a [out_rows][cols] matrix
constexpr uint32_t kPairTokens = 240u;    // the most tokens of a pair's tile
constexpr uint32_t kRowPairTokens = 64u;  // one CTA's down tiles of that many tokens and more always take two row tiles
void pair_configure_kernels();
void launch_experts_pair(const ExpertLaunch& p, bool gate_up, int sms, cudaStream_t stream);
// Tensor maps of a stage's operands: token rows in boxes of one K block, for one CTA's token tiles and, from the second on,
// for four of a pair's (half a tile); the same in boxes of two K blocks, kTokenMaps further on; the token scales.
constexpr uint32_t kTokenMaps = 5u, kTokenScaleMap = 2u * kTokenMaps, kActMaps = kTokenScaleMap + 1u;
constexpr uint32_t kTokenMapRows[kTokenMaps] = {16u, 32u, 64u, 96u, kPairTokens / 2u};
// tokens per expert above which a tile of those rows, or half a pair's tile, may be used (pairs above the last)
constexpr uint32_t kTokenMapFrom[kTokenMaps] = {0u, 12u, 24u, 48u, 96u}, kPairsFrom = kTokenMapFrom[kTokenMaps - 1u];
inline uint32_t tc_token_map_for(const TokenTile& t) {
    uint32_t i = 0u;
    while (i + 1u < kTokenMaps && kTokenMapRows[i] != t.rows) i++;
    return t.pair ? 1u : i;
}
// bytes of the derived (tiled) scale copy of one expert matrix with `rows` x `cols` elements
size_t tc_derived_scale_bytes(uint32_t rows, uint32_t cols);
// re-tiles the scales of every expert whose scale record changed since the last call
void launch_derive_scales_tc(const ExpertLaunch& p, bool gate_up, cudaStream_t stream);
// Both expert stages of a layer call in one launch (experts_layer.cu): one CTA a tile, the same token tile in both, tensor maps,
// the down operands made by gate/up.
struct LayerLaunch {
    ExpertLaunch stage[2];
    uint32_t* sync;    // experts + 1 words, cleared earlier in the call: chunks claimed, per expert the warps done with its gate/up tiles
    bool claim_late;   // the launch right before this one clears them
    uint32_t maps;     // who acquires the tensor maps of the weights (experts_layer.cu sets it)
};
constexpr uint32_t kLayerExperts = 1024u;  // at most
void layer_configure_kernels();
// whether a call gains by it
bool tc_layer_in_one_launch(uint32_t tokens, uint32_t routes_per_token, uint32_t num_experts, uint32_t hidden, uint32_t intermediate, uint32_t token_rows);
void launch_layer_tc(const LayerLaunch& p, cudaStream_t stream);
void launch_experts_layer(const LayerLaunch& p, int sms, cudaStream_t stream);
void launch_gate_up_tc(const ExpertLaunch& p, cudaStream_t stream);
void launch_down_tc(const ExpertLaunch& p, cudaStream_t stream);

}  // namespace nvmoe
