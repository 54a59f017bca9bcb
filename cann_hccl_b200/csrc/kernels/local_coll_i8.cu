// Direct reduction kernels of one GPU for element type int8_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(int8_t, i8)
}  // namespace hcclb
