// Direct reduction kernels of one GPU for element type uint8_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(uint8_t, u8)
}  // namespace hcclb
