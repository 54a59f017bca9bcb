// Tensor map of a row-major bf16 matrix for the GEMM kernels' TMA loads.
#pragma once
#include "common/log.h"
#include "core/device_api.h"
#include "kernels/fused/tc05.cuh"

namespace hcclb {
namespace tc05 {

// [rows, cols] from `base`, boxes of box_rows x BK elements, 128-byte swizzle.
inline HcclResult encode_2d(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint32_t box_rows)
{
    const DriverApi &d = driver_api();
    if (!d.ok || !d.TensorMapEncodeTiled) return HCCL_E_DRV;
    cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, box_rows}, estr[2] = {1, 1};
    CUresult r = d.TensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { HLOG_ERROR("cuTensorMapEncodeTiled failed: %s", cu_err(r)); return HCCL_E_DRV; }
    return HCCL_SUCCESS;
}

}  // namespace tc05
}  // namespace hcclb
