// The packed int4 matrix as the tensor-core GEMMs load it (affine_b4_skinny.cu, affine_b4_gemm.cu, affine_b4_gemm_pair.cu): a chunk
// of 128 channels by 128 k is 8 blocks, KC blocks apart in memory, and arrives with ONE tiled copy.  With a 1-D bulk copy for each
// block the one lane that issued them was what bound these kernels: about 130 cycles a copy, 1050 a chunk, where the chunk's
// 9.2 KB take 400 from HBM and its MMAs 128 to 770.
#pragma once

#include "affine_b4.cuh"
#include "tc_common.cuh"

// [RB][KC][block] in 8-byte elements (a block is 144 or 160 of them; a box may hold 256 a side), box 1 chunk x 8 row-blocks.
static inline bool affine_w_map(CUtensorMap* map, tc_encode_tiled_fn enc, const uint8_t* packed, int RB, int KC, int gs) {
    const cuuint64_t block = (cuuint64_t)aff_block_bytes(gs);
    const cuuint64_t dims[3] = {block / 8, (cuuint64_t)KC, (cuuint64_t)RB};
    const cuuint64_t strides[2] = {block, (cuuint64_t)KC * block};
    const cuuint32_t box[3] = {(cuuint32_t)(block / 8), 1, 8};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, const_cast<uint8_t*>(packed), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Chunk `kc` of the row-blocks rb0 .. rb0 + 7 -> 8 blocks one after the other at `dst` (128-byte aligned).
__device__ __forceinline__ void affine_load_chunk(uint32_t dst, const CUtensorMap* map, int kc, int rb0, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(0), "r"(kc), "r"(rb0), "r"(bar) : "memory");
}
