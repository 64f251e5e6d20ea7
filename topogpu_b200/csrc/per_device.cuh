// per_device.cuh - host-side tables with one entry per CUDA device.
#pragma once

#include <cstddef>
#include <deque>
#include <mutex>

namespace topo {

// An entry stays where it is while the table grows: a thread keeps using its
// device's entry outside the lock while another thread meets a new device.
template <typename T>
class PerDevice {
 public:
  T& at(int dev) {
    std::lock_guard<std::mutex> lk(mu_);
    while (d_.size() <= (std::size_t)dev) d_.emplace_back();
    return d_[(std::size_t)dev];
  }

 private:
  std::mutex mu_;
  std::deque<T> d_;
};

}  // namespace topo
