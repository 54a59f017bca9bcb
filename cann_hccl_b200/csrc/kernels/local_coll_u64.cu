// Direct reduction kernels of one GPU for element type unsigned long long (all four operators).
#include "kernels/local_coll.cuh"
namespace hcclb {
HCCLB_INSTANTIATE_LOCAL(unsigned long long, u64)
}  // namespace hcclb
