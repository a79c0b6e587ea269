// Page-locked host memory of a context that kernels read and write in place: for rows that are too small for a copy engine to pay.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace mpq {

struct HostPages {
    // The most that a context keeps per direction.  Activations pay for a copy by one host core that nothing overlaps: calls in us, by the
    // driver's copies / through pages, with bytes in + bytes out: 64 x 4096 x 4096 (1 + 1 MB) 185 / 204, 23 x 4096 x 11008 (1013 + 377 KB) 138 / 153, 40 x 4096 x
    // 4096 (655 + 655) 127 / 134, 32 x 4096 x 4096 (524 + 524) 112 / 103, 12 x 4096 x 11008 (528 + 197) 90 / 78.  Outputs are stored behind the arithmetic
    // and are worth it up to 1 MB (16 x 16384 x 4096, 262 KB + 1 MB, 143 / 135; one row of 262144 x 1024 116 / 99), behind activations that the driver
    // copies up to three quarters of that (outputs by copy / pages: 192 x 1024 x 1024, 786 KB, 143 / 139; 240 x 1000 x 2112, 960 KB, 234 / 245).
    static constexpr size_t MOST_IN = (size_t)1 << 19, MOST_OUT = (size_t)1 << 20, MOST_OUT_BEHIND_COPY = MOST_OUT / 4 * 3;
    void *host = nullptr, *device = nullptr;       // the same bytes, as the host and as kernels address them
    size_t bytes = 0;

    // Room for `need` bytes, in steps of a factor of two (rows that grow from call to call lock pages a few times, not every time); false
    // where that is more than `most` or the system locks no more pages.  What was there is gone: no launch may still be using it.
    bool reserve(size_t need, size_t most)
    {
        if (need > most) return false;
        if (bytes >= need) return true;
        release();
        size_t size = (size_t)1 << 16;
        while (size < need) size *= 2;
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
