// Tensor maps (TMA): host-side encoding and the rank-3 load.
#pragma once

#include <cuda.h>  // CUtensorMap and its enums; the encoder itself is looked up at run time

#include "common.cuh"

namespace reskv {

// FP16 tensor of `rank` dimensions (innermost first, strides[i] bytes between the elements of dimension i + 1) in boxes of
// box[]; elements beyond the ends read as zero.
int encode_tensor_map(CUtensorMap* map, const void* x, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                      CUtensorMapSwizzle swizzle, const char* who);

// One box of a rank-3 tensor map -> shared memory, completion counted on `bar`.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

}  // namespace reskv
