// A limit that only grows, set by the first caller that needs more and read by all others.  Plain C++, no CUDA.
#pragma once

#include <atomic>
#include <mutex>

namespace nmg {

class GrowingLimit {
    std::atomic<int> have_{0};
    std::mutex mu_;

  public:
    // set(v) sets the limit to v and returns 0, or an error that is handed on.  Two callers that both find too little come here one
    // after the other: set and recorded in any order, the smaller value could be the one in force and the larger the one recorded,
    // and nothing would set it again.
    template <typename Set> int ensure(int want, Set set) {
        if (have_.load(std::memory_order_acquire) >= want) return 0;
        std::lock_guard<std::mutex> lk(mu_);
        if (have_.load(std::memory_order_relaxed) >= want) return 0;
        const int rc = set(want);
        if (rc == 0) have_.store(want, std::memory_order_release);
        return rc;
    }
};

}  // namespace nmg
