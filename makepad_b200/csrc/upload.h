// Host memory or a file -> device memory through pinned slots.
//
// cudaMemcpy from pageable memory is one thread's memcpy into the driver's staging (about 7 GB/s here); a file adds a
// read into fresh pages before it.  Several threads fill pinned slots (memcpy or pread) while the slots filled before
// are on their way.  The slots belong to a context: made by its first upload, at most 16 x 512 KiB, freed with it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <thread>

namespace mpq {

class StagedUpload {
public:
    static constexpr int THREADS = 8, SLOTS = 2;               // slots per thread: one is filled while the other travels
    static constexpr size_t PIECE = (size_t)1 << 19;
    enum Result { OK = 0, READ_FAILED, CUDA_FAILED };

    // One upload at a time per context (several host threads may build weights).  Returns when the bytes are in device
    // memory.  src: host memory, or null to read `bytes` at `offset` of the file `fd`.
    Result run(int device, void* dst, const void* src, int fd, int64_t offset, size_t bytes, cudaStream_t stream, cudaError_t* err)
    {
        std::lock_guard<std::mutex> hold(lock_);
        const size_t pieces = (bytes + PIECE - 1) / PIECE;
        const int want = (int)std::min<size_t>(THREADS, std::max<size_t>(1, pieces / SLOTS));
        std::atomic<size_t> next(0);
        std::atomic<int> result(OK), code(cudaSuccess);
        auto work = [&](int t) {
            cudaError_t e = cudaSetDevice(device);
            for (int k = 0; e == cudaSuccess && result.load() == OK; k = (k + 1) % SLOTS) {
                const size_t i = next.fetch_add(1);
                if (i >= pieces) break;
                Slot& slot = slots_[t * SLOTS + k];
                if (!slot.done) e = cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming);
                if (e == cudaSuccess && !slot.mem && cudaHostAlloc(&slot.mem, PIECE, cudaHostAllocPortable) != cudaSuccess) {
                    cudaGetLastError();
                    slot.mem = nullptr;
                    e = cudaErrorMemoryAllocation;
                }
                if (e == cudaSuccess) e = cudaEventSynchronize(slot.done);      // the slot's last piece has left it
                if (e != cudaSuccess) break;
                const size_t at = i * PIECE, n = std::min(PIECE, bytes - at);
                if (src) memcpy(slot.mem, static_cast<const char*>(src) + at, n);
                else
                    for (size_t got = 0; got < n;) {
                        const ssize_t r = pread(fd, static_cast<char*>(slot.mem) + got, n - got, (off_t)(offset + (int64_t)(at + got)));
                        if (r <= 0) { result.store(READ_FAILED); return; }
                        got += (size_t)r;
                    }
                e = cudaMemcpyAsync(static_cast<char*>(dst) + at, slot.mem, n, cudaMemcpyHostToDevice, stream);
                if (e == cudaSuccess) e = cudaEventRecord(slot.done, stream);
            }
            if (e != cudaSuccess) { code.store(e); result.store(CUDA_FAILED); }
        };
        std::thread threads[THREADS];
        int started = 0;
        try {
            for (; started < want - 1; ++started) threads[started] = std::thread(work, started + 1);
        } catch (...) {}                                       // no more threads to be had: those that run do the work
        work(0);
        for (int t = 0; t < started; ++t) threads[t].join();
        const cudaError_t e = cudaStreamSynchronize(stream);
        if (result.load() == OK && e != cudaSuccess) { code.store(e); result.store(CUDA_FAILED); }
        *err = (cudaError_t)code.load();
        return (Result)result.load();
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
            if (s.mem) cudaFreeHost(s.mem);
            if (s.done) cudaEventDestroy(s.done);
            s = Slot();
        }
    }

private:
    struct Slot { void* mem = nullptr; cudaEvent_t done = nullptr; };
    std::mutex lock_, staging_lock_;
    uint8_t* staging_ = nullptr;
    size_t staging_bytes_ = 0;
    Slot slots_[THREADS * SLOTS];
};

}  // namespace mpq
