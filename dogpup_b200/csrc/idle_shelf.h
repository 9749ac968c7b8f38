// Objects kept for reuse between calls, per device (host code only).
#pragma once

#include <cstddef>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

namespace dgp {

// Up to MAX idle objects of type T for each device's primary context, named by its id.  A device has one
// primary context at a time: when it shows another id, the one that the kept objects were made in has
// been reset, and their handles went with it (T::abandon: forget them, call nothing).  What does not
// fit is destroyed by the caller that returns it, whose context is the one that it belongs to.
template <class T> class IdleShelf {
 public:
  static constexpr size_t MAX = 4;

  std::unique_ptr<T> take(int dev, unsigned long long ctx) {
    std::lock_guard<std::mutex> lock(mutex_);
    auto &v = of(dev, ctx);
    if (v.empty()) return nullptr;
    std::unique_ptr<T> t = std::move(v.back());
    v.pop_back();
    return t;
  }

  void put(int dev, unsigned long long ctx, std::unique_ptr<T> t) {
    std::lock_guard<std::mutex> lock(mutex_);
    auto &v = of(dev, ctx);
    if (v.size() < MAX) v.push_back(std::move(t));
  }

 private:
  struct Device {
    unsigned long long ctx = 0;
    std::vector<std::unique_ptr<T>> idle;
  };
  std::vector<std::unique_ptr<T>> &of(int dev, unsigned long long ctx) {
    if ((size_t)dev >= devices_.size()) devices_.resize((size_t)dev + 1);
    Device &d = devices_[(size_t)dev];
    if (d.ctx != ctx) {
      for (auto &t : d.idle) t->abandon();
      d.idle.clear();
      d.idle.reserve(MAX);  // (put never allocates: it runs in destructors)
      d.ctx = ctx;
    }
    return d.idle;
  }
  std::mutex mutex_;
  std::vector<Device> devices_;
};

}  // namespace dgp
