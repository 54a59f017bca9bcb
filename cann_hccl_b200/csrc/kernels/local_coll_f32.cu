// Direct reduction kernels of one GPU for element type float (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(float, f32)
}  // namespace hcclb
