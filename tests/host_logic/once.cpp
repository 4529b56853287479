// OncePerDevice (pwm_gb300/csrc/device_once.hpp) on fake devices: prints "ok",
// or what went wrong.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "../../pwm_gb300/csrc/device_once.hpp"

using namespace pwmgpu;

static int wrong(const char* what) {
  printf("%s\n", what);
  return 1;
}

int main() {
  {  // one thread a device and device after device: every device gets the setting, none twice
    static OncePerDevice once;
    for (int round = 0; round < 3; ++round)
      for (int dev = 0; dev < 64; ++dev) {
        int calls = 0;
        if (once.run(dev, [&]() { ++calls; return 0; }) != 0) return wrong("an error from nowhere");
        if (calls != (round == 0)) return wrong("not once a device");
      }
    int calls = 0;
    for (int k = 0; k < 2; ++k)
      for (int dev : {-1, 64, 1000}) once.run(dev, [&]() { ++calls; return 0; });
    if (calls != 6) return wrong("a device without a bit is set every time");
  }
  {  // a failure is reported and tried again
    static OncePerDevice once;
    if (once.run(5, []() { return 7; }) != 7) return wrong("the error is lost");
    int calls = 0;
    if (once.run(5, [&]() { ++calls; return 0; }) != 0 || calls != 1) return wrong("a failure counted as done");
    if (once.run(5, []() { return 7; }) != 0) return wrong("a success was forgotten");
  }
  for (int trial = 0; trial < 50; ++trial) {  // threads of many devices: set before run returns
    OncePerDevice once;
    std::atomic<int> set[8] = {};
    std::atomic<bool> early{false};
    std::vector<std::thread> pool;
    for (int t = 0; t < 16; ++t)
      pool.emplace_back([&, t]() {
        const int dev = t % 8;
        for (int k = 0; k < 100; ++k) {
          once.run(dev, [&]() { set[dev].store(1); return 0; });
          if (!set[dev].load()) early = true;
        }
      });
    for (auto& t : pool) t.join();
    if (early) return wrong("run returned before the setting was made");
  }
  printf("ok\n");
  return 0;
}
