// Direct reduction kernels of one GPU for element type int32_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(int32_t, i32)
}  // namespace hcclb
