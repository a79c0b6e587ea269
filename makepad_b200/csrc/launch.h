// A plain kernel launch that returns the status of this launch.  (cudaGetLastError after <<< >>> also returns an error that an
// earlier call of the program left behind.)
#pragma once
#include <cuda_runtime.h>

namespace mpq {

template <class... P, class... A>
cudaError_t launch(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace mpq
