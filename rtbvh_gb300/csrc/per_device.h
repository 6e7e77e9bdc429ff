// A value that belongs to a CUDA device (kernel attributes that are set on it,
// what it can launch), found on the first use there.
#pragma once

#include <mutex>
#include <vector>

namespace rtbvh {

template <class T>
class PerDevice {
 public:
  // The value of `device` into *out. find(T*) runs on the first call for that
  // device and returns an error (0: none); after an error nothing is kept and
  // the next call tries again.
  template <class Find>
  auto get(int device, T* out, Find&& find) -> decltype(find(out)) {
    std::lock_guard<std::mutex> lock(mu_);
    for (const Known& k : known_) {
      if (k.device == device) {
        *out = k.value;
        return {};
      }
    }
    T value{};
    const auto e = find(&value);
    if (e) return e;
    known_.push_back({device, value});
    *out = value;
    return e;
  }

 private:
  struct Known {
    int device;
    T value;
  };
  std::mutex mu_;
  std::vector<Known> known_;
};

}  // namespace rtbvh
