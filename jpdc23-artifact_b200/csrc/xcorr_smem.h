// The dynamic shared memory a kernel instance may use beyond 48 KB is an attribute that has to be raised per
// device before a launch.  Kept apart from CUDA so that its threads can be tested with a stand-in for the call.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <mutex>

namespace xcorr {

// One per kernel instance (static).  After allow(device, bytes, ...) has succeeded, the attribute is at least `bytes`
// and is never lowered again, whatever other threads ask for meanwhile: the call and the note of what it granted
// happen under one lock and only upwards.  (Checked and set without one, a thread that asks for 130 KB can come
// between another's 200 KB and its launch, which then fails.)
struct SmemLimit {
    static constexpr int kDevices = 64;
    std::mutex mutex;
    std::atomic<size_t> granted[kDevices] = {};
    size_t beyond = 0;                       // devices the table has no place for: the largest size any of them was given

    // set(bytes) raises the attribute on the current device, which is `device`; 0 (cudaSuccess) means it did.
    template<typename Set>
    auto allow(int device, size_t bytes, Set set) -> decltype(set(bytes)) {
        using Status = decltype(set(bytes));
        if (bytes <= 48 * 1024) return Status{};
        const bool known = device >= 0 && device < kDevices;
        if (known && granted[device].load(std::memory_order_acquire) >= bytes) return Status{};
        std::lock_guard<std::mutex> lock(mutex);
        if (!known) {
            beyond = std::max(beyond, bytes);
            return set(beyond);
        }
        if (granted[device].load(std::memory_order_relaxed) >= bytes) return Status{};
        const Status s = set(bytes);
        if (s == Status{}) granted[device].store(bytes, std::memory_order_release);
        return s;
    }
};

}  // namespace xcorr
