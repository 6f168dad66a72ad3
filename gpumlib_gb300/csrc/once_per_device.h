// Runs something once on every device, as kernel attributes want it: they belong to the device that is
// current when they are set.  Host only, no CUDA types.
#pragma once

#include <mutex>

namespace gpunmf {

template <class Result>
class OncePerDevice {
    std::mutex mu_;
    bool done_[64] = {};
    Result result_[64] = {};

public:
    template <class F>
    Result run(int device, F &&f) {
        std::lock_guard<std::mutex> lock(mu_);
        const int k = device & 63;
        if (!done_[k]) {
            result_[k] = f();
            done_[k] = true;
        }
        return result_[k];
    }
};

}  // namespace gpunmf
