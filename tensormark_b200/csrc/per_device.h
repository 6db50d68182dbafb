// per_device.h — what a process finds out or sets once on every device that it uses.
#pragma once

#include <atomic>
#include <mutex>

namespace tmc {

constexpr int kMaxDevices = 64;

// T as init(T&) leaves it, made by the first call on each device. Calls that arrive together wait for the one that makes it;
// where init returned false the next call tries again.
template <typename T> class PerDevice {
public:
    // nullptr: no such device, or init failed
    template <typename Init> const T* get(int device, Init init) {
        if (device < 0 || device >= kMaxDevices) return nullptr;
        Entry& e = entries_[device];
        if (!e.ready.load(std::memory_order_acquire)) {
            std::lock_guard<std::mutex> hold(making_);
            if (!e.ready.load(std::memory_order_relaxed)) {
                if (!init(e.value)) return nullptr;
                e.ready.store(true, std::memory_order_release);
            }
        }
        return &e.value;
    }

private:
    struct Entry {
        std::atomic<bool> ready{false};
        T value{};
    };
    Entry entries_[kMaxDevices];
    std::mutex making_;
};

}  // namespace tmc
