// A value per device, worked out by the first thread that asks for it and read by all others.
#pragma once
#include <atomic>
#include <mutex>

namespace bpdq {

template <class T>
class PerDevice {
public:
    // fill(T&) says whether it succeeded; null (and another attempt by the next call) where it did not.  A device beyond the table is
    // asked for every time.
    template <class Fill>
    const T* get(int device, Fill fill)
    {
        if (device < 0 || device >= kDevices) {
            thread_local T own;
            own = T();
            return fill(own) ? &own : nullptr;
        }
        Slot& s = slots_[device];
        if (!s.known.load(std::memory_order_acquire)) {
            std::lock_guard<std::mutex> lock(s.filling);
            if (!s.known.load(std::memory_order_relaxed)) {
                T value = T();
                if (!fill(value)) return nullptr;
                s.value = value;
                s.known.store(true, std::memory_order_release);
            }
        }
        return &s.value;
    }

private:
    static constexpr int kDevices = 64;
    struct Slot {
        std::mutex filling;
        std::atomic<bool> known{false};
        T value = T();
    };
    Slot slots_[kDevices];
};

}  // namespace bpdq
