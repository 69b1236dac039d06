// Facts that are asked, or settings that are made, once on every device: a kernel's shared-memory allowance, for one, belongs to
// the device that was current when it was raised.  Plain C++, safe with several threads.
#pragma once
#include <map>
#include <mutex>

namespace rb {

template <typename T>
class PerDevice {
public:
    // *out: the value of device number `device`.  The first call for a device has `ask(value)` fill it; an error it returns (not 0)
    // is passed on and nothing is kept, so that the next call asks again.
    template <typename Ask>
    int get(int device, const T** out, Ask ask) {
        std::lock_guard<std::mutex> hold(mu_);
        auto it = known_.find(device);
        if (it == known_.end()) {
            T value{};
            if (const int error = ask(value)) return error;
            it = known_.emplace(device, value).first;
        }
        *out = &it->second;          // a map's entries stay where they are
        return 0;
    }

private:
    std::mutex mu_;
    std::map<int, T> known_;
};

}  // namespace rb
