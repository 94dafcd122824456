// A setting that holds on one device (cudaFuncSetAttribute raises a kernel's
// shared-memory limit on the current device alone), made on first use there.
// Safe with several threads; a setting that failed is tried again.
#pragma once
#include <atomic>

namespace litho_b200 {

class PerDevice {
public:
    // Runs set() (0: success) unless it has succeeded on `dev` before; returns
    // its result.  Devices beyond 63 are set each time.
    template <typename Set>
    auto once(int dev, Set set) -> decltype(set()) {
        const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
        if (done_.load() & bit) return decltype(set())(0);
        const auto e = set();
        if (e == decltype(set())(0)) done_.fetch_or(bit);
        return e;
    }

private:
    std::atomic<unsigned long long> done_{0};
};

}  // namespace litho_b200
