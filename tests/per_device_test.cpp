// PerDevice from several threads on several devices: one make() per device, its value for everybody.
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#include "per_device.h"

int main() {
  static thc::PerDevice value;
  std::atomic<int> made[4] = {};
  std::atomic<int> wrong{0};
  try { value.get(2, []() -> int { throw std::runtime_error("no"); }); return 1; } catch (const std::runtime_error &) {}
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 1000; i++) {
        const int device = (i + t) % 4;
        if (value.get(device, [&] { made[device]++; return 10 + device; }) != 10 + device) wrong++;
      }
    });
  for (auto &t : ts) t.join();
  for (int d = 0; d < 4; d++) if (made[d] != 1) { std::printf("device %d: made %d times\n", d, made[d].load()); return 1; }
  return wrong ? 1 : 0;
}
