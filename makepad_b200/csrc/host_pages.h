// Page-locked host memory of a context that kernels read and write in place: for rows that are too small for a copy engine to pay.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>

namespace mpq {

struct HostPages {
    static constexpr size_t MOST = (size_t)1 << 20;
    void *host = nullptr, *device = nullptr;       // the same bytes, as the host and as kernels address them
    size_t bytes = 0;

    // Room for `need` bytes; false where that is more than MOST or the system locks no more pages.  What was there is gone: no
    // launch may still be using it.
    bool reserve(size_t need)
    {
        if (need > MOST) return false;
        if (bytes >= need) return true;
        release();
        const size_t size = std::max(need, (size_t)1 << 16);
        if (cudaHostAlloc(&host, size, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            host = nullptr;
            return false;
        }
        if (cudaHostGetDevicePointer(&device, host, 0) != cudaSuccess) {
            cudaGetLastError();
            release();
            return false;
        }
        bytes = size;
        return true;
    }
    void release()
    {
        if (host) cudaFreeHost(host);
        host = device = nullptr;
        bytes = 0;
    }
};

}  // namespace mpq
