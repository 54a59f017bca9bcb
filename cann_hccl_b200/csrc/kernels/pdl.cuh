// Programmatic dependent launch: a kernel launched this way may take the SM slots that its predecessor in the stream leaves
// free and waits there (pdl_wait) until the predecessor has completed and its writes are visible; launch latency and block
// scheduling hide behind the predecessor's tail.  Nothing that the predecessor may touch is read or written before pdl_wait().
#pragma once
#include <cuda_runtime.h>
#include <cstring>
#include "common/log.h"

namespace hcclb {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches fn(*args) (one structure argument); cluster: CTAs of a cluster along x, 0 or 1 for none.
inline HcclResult launch_pdl(const void *fn, dim3 grid, unsigned threads, size_t smem, void *args, void *stream, const char *what, int cluster = 0)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = cluster > 1 ? 2 : 1;
    void *kargs[] = {args};
    cudaError_t e = cudaLaunchKernelExC(&cfg, fn, kargs);
    if (e != cudaSuccess) { HLOG_ERROR("%s launch failed (%u x %u CTAs): %s", what, grid.x, grid.y, cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

}  // namespace hcclb
