// What holds for a device and is found out or set up once: kernel attributes,
// whether a launch shape can be scheduled.
#pragma once
#include <atomic>
#include <mutex>

namespace rsg {

class PerDevice {
 public:
  // f's answer for this device, asked for once (again if f threw).
  template <class F>
  bool ask(int device, F&& f) {
    if (device < 0 || device >= DEVICES) return f();
    std::atomic<int>& a = answer_[device];
    if (int v = a.load(std::memory_order_acquire)) return v > 0;
    std::lock_guard<std::mutex> lk(mu_);
    if (!a.load(std::memory_order_relaxed)) a.store(f() ? 1 : -1, std::memory_order_release);
    return a.load(std::memory_order_relaxed) > 0;
  }

 private:
  static constexpr int DEVICES = 64;  // further ones are asked each time
  std::mutex mu_;
  std::atomic<int> answer_[DEVICES] = {};  // 0 not asked, 1 yes, -1 no
};

}  // namespace rsg
