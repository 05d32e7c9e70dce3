// Shared objects for one call each, reused once nobody holds them any more.
#pragma once
#include <memory>
#include <vector>

namespace lpma {

// take() gives an object that nobody but the ring holds: one that was given
// out before and released by all its holders, else a new one from make()
// (null on failure, passed on).  The ring keeps as many objects as were ever
// held at the same time, and one more.  One thread takes; holders may release
// from any thread.
template <typename T>
class SpareRing {
    std::vector<std::shared_ptr<T>> all_;

  public:
    template <typename Make>
    std::shared_ptr<T> take(Make make) {
        for (const std::shared_ptr<T> &x : all_)
            if (x.use_count() == 1) return x;
        std::shared_ptr<T> x = make();
        if (x) all_.push_back(x);
        return x;
    }
    size_t size() const { return all_.size(); }
};

}  // namespace lpma
