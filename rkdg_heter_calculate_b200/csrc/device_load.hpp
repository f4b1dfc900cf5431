// What the calls in flight that step solves (contexts, packs, serving loops; of
// any thread) take of each device, in millionths: how many of the tiles it
// holds at once they have in flight.
#pragma once

#include <algorithm>
#include <cstdint>

#include "per_device.hpp"
#include "rkdg_internal.hpp"

namespace rkdg {

constexpr int64_t kWholeDevice = 1000000;
PerDevice<int64_t>& device_load();  // (capi.cpp)

// A call's share, for as long as the call lasts.
class LoadShare {
public:
    explicit LoadShare(int device) : device_(device) {}
    LoadShare(int device, int64_t share) : LoadShare(device) {
        take([&](int64_t) { return share; });
    }
    ~LoadShare() {
        if (share_ > 0) device_load().use(device_, [&](int64_t& load) { load -= share_; });
    }
    LoadShare(const LoadShare&) = delete;
    LoadShare& operator=(const LoadShare&) = delete;
    // once: f(the others' load) chooses the share
    template <class F>
    void take(F&& f) {
        device_load().use(device_, [&](int64_t& load) { load += share_ = f(load); });
    }

private:
    int device_;
    int64_t share_ = 0;
};

// Share of stage launches over n tiles, on a device that holds fit at once.
inline int64_t stage_share(int64_t n, int64_t fit) {
    return std::min(kWholeDevice, n * kWholeDevice / std::max<int64_t>(fit, 1));
}

}  // namespace rkdg
