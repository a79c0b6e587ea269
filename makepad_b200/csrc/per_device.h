// Bookkeeping for settings that CUDA keeps per DEVICE (cudaFuncSetAttribute, symbol addresses) while the
// code that applies them is shared by every context of the process: one flag per device index.
// Host-only, no CUDA dependency, so that it can be unit-tested without a GPU.
#pragma once
#include <mutex>

namespace mpq {

struct PerDeviceOnce {
    static constexpr int MAX_DEVICES = 64;
    bool done[MAX_DEVICES] = {};
    // true while the setting has not been applied on this device (always true for an index outside the
    // table: applying a per-device setting twice is harmless, skipping it is not)
    bool needs(int device) const { return device < 0 || device >= MAX_DEVICES || !done[device]; }
    void mark(int device)
    {
        if (device >= 0 && device < MAX_DEVICES) done[device] = true;
    }
};

// N numbers per device that a query finds, asked for once per device and by one thread at a time; asked for again where it failed.
template <int N>
struct PerDeviceNumbers {
    std::mutex lock;
    PerDeviceOnce known;
    int values[PerDeviceOnce::MAX_DEVICES][N] = {};
    // query(out) fills out and says whether that succeeded; zeros where it did not
    template <class Query>
    void get(int device, int (&out)[N], Query query)
    {
        std::lock_guard<std::mutex> hold(lock);
        if (!known.needs(device)) {
            for (int i = 0; i < N; ++i) out[i] = values[device][i];
            return;
        }
        for (int i = 0; i < N; ++i) out[i] = 0;
        if (!query(out)) {
            for (int i = 0; i < N; ++i) out[i] = 0;
            return;
        }
        if (device < 0 || device >= PerDeviceOnce::MAX_DEVICES) return;
        for (int i = 0; i < N; ++i) values[device][i] = out[i];
        known.mark(device);
    }
};

}  // namespace mpq
