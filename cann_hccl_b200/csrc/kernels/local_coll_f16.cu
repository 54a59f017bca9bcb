// Direct reduction kernels of one GPU for element type __half (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(__half, f16)
}  // namespace hcclb
