// Direct reduction kernels of one GPU for element type int16_t (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(int16_t, i16)
}  // namespace hcclb
