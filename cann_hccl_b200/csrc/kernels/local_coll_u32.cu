// Direct reduction kernels of one GPU for element type uint32_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(uint32_t, u32)
}  // namespace hcclb
