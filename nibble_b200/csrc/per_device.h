// What a launcher learns once about each device (attributes it has set, SM counts), shared by all threads.
#pragma once

#include <atomic>
#include <mutex>

namespace w4a16 {

constexpr int kMaxDevices = 64;

// One State per device, set up by the first call there.  A set-up that fails is not kept: the next call tries again (with
// std::call_once, one passing error would have refused every later call on that device).
template <typename State>
class PerDevice {
public:
    // `learn(State&)` returns 0 or an error code, which is passed on; `*state` is valid after 0.
    template <typename Learn>
    int get(int device, Learn&& learn, const State** state) {
        Slot& slot = slots_[device];
        if (!slot.ready.load(std::memory_order_acquire)) {
            std::lock_guard<std::mutex> lock(slot.mutex);
            if (!slot.ready.load(std::memory_order_relaxed)) {
                State fresh{};
                const int status = learn(fresh);
                if (status != 0) return status;
                slot.state = fresh;
                slot.ready.store(true, std::memory_order_release);
            }
        }
        *state = &slot.state;
        return 0;
    }

private:
    struct Slot {
        std::mutex mutex;
        std::atomic<bool> ready{false};
        State state{};
    };
    Slot slots_[kMaxDevices];
};

}  // namespace w4a16
