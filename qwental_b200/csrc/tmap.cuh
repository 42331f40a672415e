// 2-D tensor maps and their tiled loads.
#pragma once
#include "common.cuh"
#include <cuda.h>

namespace qw {

// rows x inner elements of a matrix whose rows are `pitch` bytes apart (base 16-byte aligned, pitch a multiple of 16), boxes of
// box_inner x box_rows; elements outside read as zero; `ahead` = what L2 fetches beyond a miss.  cuTensorMapEncodeTiled is a driver entry point, looked up through the runtime
// so that the library has no link dependency on libcuda (it must load, without running anything, on machines that have no driver).
inline bool tmap_2d(CUtensorMap *tm, CUtensorMapDataType type, const void *base, uint64_t inner, uint64_t rows, uint64_t pitch, uint32_t box_inner, uint32_t box_rows,
                    CUtensorMapSwizzle swizzle, CUtensorMapL2promotion ahead = CU_TENSOR_MAP_L2_PROMOTION_L2_256B) {
    typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const encode_fn fn = [] {
        void *q = nullptr;
        cudaDriverEntryPointQueryResult qr;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &qr) == cudaSuccess ? (encode_fn)q : (encode_fn) nullptr;
    }();
    if (!fn) return false;
    const cuuint64_t gdim[2] = {inner, rows}, gstride[1] = {pitch};
    const cuuint32_t box[2] = {box_inner, box_rows}, estr[2] = {1, 1};
    return fn(tm, type, 2, (void *)base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, ahead,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *tm, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(tm),
                 "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

}  // namespace qw
