// Host state that belongs to a device: kernel attributes set on it, answers it
// gave.  A process may drive several devices from several threads, so none of
// it is kept once per process or per thread.
#pragma once

#include <map>
#include <mutex>

namespace rkdg {

template <class T>
class PerDevice {
public:
    // f(value of the device, default-constructed before its first use), one
    // thread at a time
    template <class F>
    auto use(int device, F&& f) {
        std::lock_guard<std::mutex> lock(mu_);
        return f(values_[device]);
    }

private:
    std::mutex mu_;
    std::map<int, T> values_;
};

}  // namespace rkdg
