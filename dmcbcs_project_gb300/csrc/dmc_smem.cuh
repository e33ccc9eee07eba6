// Launch attributes of kernels whose dynamic shared memory depends on the system.
//
// The limit belongs to the function on the device, and contexts of any sizes
// launch it from their own host threads.  So it is only ever raised: set to
// each system's own size, a small system's call between a large one's set and
// its launch would have that launch refused.
#pragma once

#include <cuda_runtime.h>

#include "dmc_attr.h"

namespace dmc {

template <class... A>
cudaError_t allow_smem(AttrCache& cache, int kind, void (*kernel)(A...), size_t bytes)
{
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return (cudaError_t)cache.ensure(dev, kind, (int)bytes, [&](int v) {
        return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
    });
}

// the largest share of the SM's memory for shared memory, once per device
template <class... A>
cudaError_t max_carveout(AttrCache& cache, int kind, void (*kernel)(A...))
{
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return (cudaError_t)cache.ensure(dev, kind, 1, [&](int) {
        return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
    });
}

}  // namespace dmc
