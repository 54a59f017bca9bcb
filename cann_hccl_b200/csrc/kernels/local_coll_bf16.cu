// Direct reduction kernels of one GPU for element type __nv_bfloat16 (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(__nv_bfloat16, bf16)
}  // namespace hcclb
