// smem_limit.h -- the dynamic shared-memory limit of kernels whose launches
// take different amounts.  The limit is one per kernel and device, shared by
// the process's host threads: a thread that set it to its own launch's size
// could lower it between another thread's setting and launch, which then
// failed.  Here it only ever grows.  The setter is passed in, so the policy is
// plain host C++ and is tested on its own.
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace sp3mm {

template <class Set>
class SmemLimits {
public:
    explicit SmemLimits(Set set) : set_(set) {}

    // Make `device`'s limit of kernel `f` at least `bytes`; returns what the
    // setter returned.  The setter runs on every call (a device reset forgets
    // limits), under the lock, so that a larger one never goes in between.
    int need(int device, const void* f, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu_);
        size_t& most = most_[{device, f}];
        const size_t want = std::max(most, bytes);
        const int rc = set_(f, want);
        if (rc == 0) most = want;
        return rc;
    }

private:
    Set set_;
    std::mutex mu_;
    std::map<std::pair<int, const void*>, size_t> most_;   // guarded by mu_
};

}  // namespace sp3mm
