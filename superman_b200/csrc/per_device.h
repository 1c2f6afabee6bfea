// Set-up that is due once on every device, such as a kernel's limit of dynamic
// shared memory: each device keeps its own outcome.
#pragma once

#include <mutex>

namespace spb {

template <class Status>
class OncePerDevice {
public:
    // Runs set_up the first time it is called for `device` and returns what that
    // run returned.
    template <class F>
    Status operator()(int device, F&& set_up)
    {
        Slot& s = slot_[device & 63];
        std::call_once(s.once, [&] { s.status = set_up(); });
        return s.status;
    }

private:
    struct Slot {
        std::once_flag once;
        Status status{};
    };
    Slot slot_[64];
};

}  // namespace spb
