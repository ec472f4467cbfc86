// Building blocks of the tcgen05 "row-tile" kernels: a CTA owns tiles of 128 pair positions,
// loader warps normalise them into a bf16 A operand in shared memory (K-major, 128-byte swizzle:
// the layout TMA would produce), one thread issues tcgen05.mma against weight matrices kept in
// shared memory in the same layout, epilogue warps read the fp32 result from TMEM.
#pragma once

#include "pdl.cuh"
#include "sm100.cuh"
#include "tmap.cuh"

namespace b200pf {
namespace rtc {

constexpr int TM = 128;                     // positions per tile
constexpr int KC = 128;                     // channels
constexpr int A_KB_BYTES = TM * 128;        // one 64-channel k-block of the A tile
constexpr int A_TILE_BYTES = 2 * A_KB_BYTES;

// Byte offset of the 16-byte chunk `chunk` (8 channels) of row `row` inside one k-block.
__device__ __forceinline__ uint32_t sw128(int row, int chunk) {
    return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
}

// Fetch W[rows][128] (bf16, tensor map of weight_map) into shared memory as two k-blocks of [rows][128 bytes] with the
// 128-byte swizzle, counted on `bar`; issued by one thread.  The copy runs under the first tile's LayerNorm: done by all
// threads before anything else started (load, store, barrier), 128 KB of weights and the launch gap were 9 of the 22 us that
// a producer took at 45 tokens, where every CTA has one tile (22.5 -> 13.1 us; 1024 tokens 248 -> 240 us).
constexpr int W_BOX_ROWS = 128;
__device__ __forceinline__ void load_weights_tma(uint8_t* dst, const CUtensorMap* map, int rows, uint64_t* bar) {
    for (int kb = 0; kb < 2; ++kb)
        for (int r = 0; r < rows; r += W_BOX_ROWS)
            sm100::tma_load_4d(dst + kb * (rows * 128) + r * 128, map, bar, kb * 64, r, 0, 0);
}
static inline int weight_map(CUtensorMap* map, const void* w, int rows, const char* what) {
    cuuint64_t dims[4] = {(cuuint64_t)KC, (cuuint64_t)rows, 1, 1};
    cuuint64_t str[3] = {KC * 2, (cuuint64_t)rows * KC * 2, (cuuint64_t)rows * KC * 2};
    cuuint32_t box[4] = {64, W_BOX_ROWS, 1, 1};
    return tmap_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B, what);
}

}  // namespace rtc
}  // namespace b200pf
