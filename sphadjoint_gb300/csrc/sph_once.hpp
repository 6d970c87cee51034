// Work to be done once on each device of the process (a kernel's attributes belong to the
// device that was current when they were set), by whichever thread comes first; others wait
// until it is done. What throws is done again by the next caller.
#pragma once

#include <mutex>
#include <set>

namespace sphgb {

class OncePerDevice {
  public:
    template <typename F> void operator()(int device, F &&f)
    {
        std::lock_guard<std::mutex> g(mu_);
        if (done_.count(device)) return;
        f();
        done_.insert(device);
    }

  private:
    std::mutex mu_;
    std::set<int> done_;
};

} // namespace sphgb
