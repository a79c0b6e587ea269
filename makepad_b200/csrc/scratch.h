// Device memory of a context that grows with the largest call seen.
//
// A captured graph holds the addresses that its launches were given, so a block that was replaced by a larger one must
// stay what it was: it is kept until the context is destroyed.  A new block is at least twice the one before, so that the
// blocks kept are together smaller than the one in use (where memory is too short for that, the new block is as large as needed).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>
#include <new>

namespace mpq {

class Scratch {
public:
    template <class T>
    T* as() const { return static_cast<T*>(mem_); }
    size_t bytes() const { return bytes_; }

    // At least `need` bytes.  On failure nothing changes, and the error is not left behind for the next cudaGetLastError.
    cudaError_t reserve(size_t need)
    {
        if (bytes_ >= need) return cudaSuccess;
        Old* old = nullptr;
        if (mem_ && !(old = new (std::nothrow) Old{mem_, old_})) return cudaErrorMemoryAllocation;
        size_t size = std::max(need, 2 * bytes_);
        void* mem = nullptr;
        cudaError_t e = cudaMalloc(&mem, size);
        if (e != cudaSuccess && size > need) {
            cudaGetLastError();
            e = cudaMalloc(&mem, size = need);
        }
        if (e != cudaSuccess) {
            cudaGetLastError();
            delete old;
            return e;
        }
        if (old) old_ = old;
        mem_ = mem;
        bytes_ = size;
        return cudaSuccess;
    }

    void release()
    {
        cudaFree(mem_);
        while (old_) {
            Old* next = old_->next;
            cudaFree(old_->mem);
            delete old_;
            old_ = next;
        }
        mem_ = nullptr;
        bytes_ = 0;
    }

private:
    struct Old { void* mem; Old* next; };
    void* mem_ = nullptr;
    size_t bytes_ = 0;
    Old* old_ = nullptr;
};

}  // namespace mpq
