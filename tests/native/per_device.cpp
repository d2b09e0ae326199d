// rsg::PerDevice: asked once for each device, by however many threads; no
// answer is kept of a question that threw, nor for devices beyond its range.
#include "../../ressim_gb300/csrc/perdevice.hpp"

#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

int main() {
  rsg::PerDevice p;
  int asked[2] = {0, 0};
  std::vector<std::thread> pool;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    pool.emplace_back([&] {
      for (int k = 0; k < 1000; ++k)
        for (int d = 0; d < 2; ++d)
          if (p.ask(d, [&] { return ++asked[d], d == 0; }) != (d == 0)) ++wrong;
    });
  for (auto& t : pool) t.join();
  if (wrong || asked[0] != 1 || asked[1] != 1) return std::puts("once per device"), 1;
  int thrown = 0;
  try {
    p.ask(2, []() -> bool { throw std::runtime_error("no"); });
  } catch (const std::runtime_error&) {
    ++thrown;
  }
  if (!thrown || !p.ask(2, [] { return true; }) || !p.ask(2, [] { return false; })) return std::puts("after a throw"), 1;
  int far = 0;
  for (int k = 0; k < 3; ++k) p.ask(1000, [&] { return ++far, true; });
  return far == 3 ? 0 : (std::puts("far devices"), 1);
}
