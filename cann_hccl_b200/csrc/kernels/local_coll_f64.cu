// Direct reduction kernels of one GPU for element type double (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(double, f64)
}  // namespace hcclb
