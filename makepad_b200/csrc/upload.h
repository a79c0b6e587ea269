// Host memory or a file -> device memory through pinned slots.
//
// cudaMemcpy from pageable memory waits for each piece that it stages; a file adds a read into fresh pages before it.  Here
// the calling thread fills one pinned slot (memcpy or pread) while the slots filled before are on their way, so that the
// host's copy rate (16 GB/s: 1.8 ms for 28 MB) is what is left.  Two to eight filling threads were measured too: 20% faster on
// a quiet host (2.2 against 2.8 ms), but several times slower on a busy one.  The slots belong to a context: made by its
// first upload, 4 x 1 MiB, freed with it.
//
// Building a Q4 weight, median of 30 creations on three boxes, cudaMemcpy / slots (ms): from pageable arrays 1000 x 2112
// 1.0..1.1 / 0.50, 12288 x 4096 3.2..3.4 / 2.3..2.6, 28672 x 8192 13.7..14.8 / 12.4..14.3.  Page-locked arrays the copy engine
// reads by itself at the rate of PCIe (28672 x 8192: 4.5 against 11.5..15 through the slots; with the kept staging memory 3.4), so
// they are handed to it directly.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <mutex>

namespace mpq {

// memory that the driver can copy from by itself: page-locked, managed, or (given for host memory) device memory
inline bool driver_knows(const void* p)
{
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
}

class StagedUpload {
public:
    static constexpr int SLOTS = 4;
    static constexpr size_t PIECE = (size_t)1 << 20;
    enum Result { OK = 0, READ_FAILED, CUDA_FAILED };

    // One upload at a time per context (several host threads may build weights).  Returns when the bytes are in device
    // memory.  src: host memory, or null to read `bytes` at `offset` of the file `fd`.
    Result run(void* dst, const void* src, int fd, int64_t offset, size_t bytes, cudaStream_t stream, cudaError_t* err)
    {
        std::lock_guard<std::mutex> hold(lock_);
        Result result = OK;
        cudaError_t e = cudaSuccess;
        if (src) {
            const bool first = driver_knows(src), last = driver_knows(static_cast<const char*>(src) + (bytes - 1));
            if (first && last) {
                // By the legacy stream, as any cudaMemcpy: behind the copies that may still be filling the array.
                e = cudaStreamSynchronize(stream);
                if (e == cudaSuccess) e = cudaMemcpy(dst, src, bytes, cudaMemcpyDefault);
                if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
                *err = e;
                if (e == cudaSuccess) return OK;
                cudaGetLastError();                        // (parts in between may be unknown to the driver: through the slots then)
            }
            // (a core copies into the slots without waiting for anyone)
            e = first || last ? cudaDeviceSynchronize() : cudaSuccess;
        }
        for (size_t at = 0, k = 0; at < bytes && e == cudaSuccess && result == OK; at += PIECE, ++k) {
            Slot& slot = slots_[k % SLOTS];
            if (!slot.done) e = cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming);
            if (e == cudaSuccess && !slot.mem) e = slot.make();
            if (e == cudaSuccess) e = cudaEventSynchronize(slot.done);          // the slot's last piece has left it
            if (e != cudaSuccess) break;
            const size_t n = std::min(PIECE, bytes - at);
            if (src) memcpy(slot.mem, static_cast<const char*>(src) + at, n);
            else
                for (size_t got = 0; got < n && result == OK;) {
                    const ssize_t r = pread(fd, static_cast<char*>(slot.mem) + got, n - got, (off_t)(offset + (int64_t)(at + got)));
                    if (r <= 0) result = READ_FAILED;
                    else got += (size_t)r;
                }
            if (result == OK) e = cudaMemcpyAsync(static_cast<char*>(dst) + at, slot.mem, n, cudaMemcpyHostToDevice, stream);
            if (result == OK && e == cudaSuccess) e = cudaEventRecord(slot.done, stream);
        }
        const cudaError_t done = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) e = done;
        if (e != cudaSuccess) cudaGetLastError();
        *err = e;
        return result != OK ? result : e == cudaSuccess ? OK : CUDA_FAILED;
    }

    // Device memory for what an upload needs beside its destination, kept with the slots (a cudaMalloc and its cudaFree cost
    // 0.4 ms each): a buffer of at least `bytes`, at most STAGING_MOST.  Null when it cannot be had.
    static constexpr size_t STAGING_MOST = (size_t)32 << 20;
    uint8_t* staging(size_t bytes)
    {
        if (bytes > STAGING_MOST) return nullptr;
        if (staging_bytes_ < bytes) {
            cudaFree(staging_);
            staging_bytes_ = 0;
            if (cudaMalloc(&staging_, bytes) != cudaSuccess) {
                cudaGetLastError();
                staging_ = nullptr;
                return nullptr;
            }
            staging_bytes_ = bytes;
        }
        return staging_;
    }
    std::mutex& staging_lock() { return staging_lock_; }       // held from staging() until its use has been waited for

    void release()
    {
        cudaFree(staging_);
        staging_ = nullptr;
        staging_bytes_ = 0;
        for (Slot& s : slots_) {
            if (s.mem && s.locked) cudaFreeHost(s.mem);
            else free(s.mem);
            if (s.done) cudaEventDestroy(s.done);
            s = Slot();
        }
    }

private:
    struct Slot {
        void* mem = nullptr;
        bool locked = false;
        cudaEvent_t done = nullptr;
        // Where the system locks no more pages, ordinary memory: the driver then stages the copy, and is done with the slot
        // when cudaMemcpyAsync returns.
        cudaError_t make()
        {
            locked = cudaHostAlloc(&mem, PIECE, cudaHostAllocPortable) == cudaSuccess;
            if (locked) return cudaSuccess;
            cudaGetLastError();
            mem = malloc(PIECE);
            return mem ? cudaSuccess : cudaErrorMemoryAllocation;
        }
    };
    std::mutex lock_, staging_lock_;
    uint8_t* staging_ = nullptr;
    size_t staging_bytes_ = 0;
    Slot slots_[SLOTS];
};

}  // namespace mpq
