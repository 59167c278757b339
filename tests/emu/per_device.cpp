// per_device.cpp - csrc/per_device.h on the CPU, for tests/test_per_device_cpu.py.
#include <thread>
#include <vector>

#include "per_device.h"

using arbor::PerDevice;

// Calls of `find` when `rounds` rounds ask for each of `devices` devices.
extern "C" int finds(int devices, int rounds) {
  PerDevice p;
  int n = 0;
  for (int r = 0; r < rounds; r++)
    for (int d = 0; d < devices; d++)
      if (p.get(d, [&] { return n++, 100 + d; }) != 100 + d) return -1;
  return n;
}
// Calls when the first `failures` fail (0).
extern "C" int finds_after_failures(int failures, int asks) {
  PerDevice p;
  int n = 0;
  for (int k = 0; k < asks; k++)
    if ((p.get(3, [&] { return n++ < failures ? 0 : 7; }) == 7) != (k >= failures)) return -1;
  return n;
}
// Threads asking for `devices` devices at once: wrong answers.
extern "C" int wrong_answers(int threads, int devices) {
  PerDevice p;
  std::vector<std::thread> t;
  std::atomic<int> wrong{0};
  for (int k = 0; k < threads; k++)
    t.emplace_back([&, k] {
      for (int r = 0; r < 1000; r++) {
        const int d = (r + k) % devices;
        if (p.get(d, [&] { return 100 + d; }) != 100 + d) wrong++;
      }
    });
  for (auto& x : t) x.join();
  return wrong;
}
