// Direct reduction kernels of one GPU for element type uint16_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(uint16_t, u16)
}  // namespace hcclb
