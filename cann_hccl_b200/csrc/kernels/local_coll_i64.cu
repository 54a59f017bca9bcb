// Direct reduction kernels of one GPU for element type long long (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(long long, i64)
}  // namespace hcclb
