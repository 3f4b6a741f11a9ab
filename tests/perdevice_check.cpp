// Checks of lace_gb300/csrc/perdevice.h against a stand-in for the current
// device: an action runs once on each device, again where it failed, from many
// threads on the device each of them has chosen.  Prints "ok" and exits 0 when
// all hold.
#include <cstdio>
#include <thread>
#include <vector>

#include "perdevice.h"

static thread_local int t_device = 0;
cudaError_t cudaGetDevice(int *d) {
  if (t_device < 0) return 1;
  *d = t_device;
  return cudaSuccess;
}

int main() {
  std::vector<int> set(130, 0);
  lace::PerDevice once;
  auto act = [&] {
    ++set[t_device];
    return true;
  };
  for (int rep = 0; rep < 3; ++rep)
    for (int d : {0, 1, 0, 7, 63}) {
      t_device = d;
      if (!once.done(act)) return printf("device %d\n", d), 1;
    }
  for (int d : {0, 1, 7, 63})
    if (set[d] != 1) return printf("device %d: %d times\n", d, set[d]), 1;
  t_device = 100;  // past the devices it remembers: every time
  if (!once.done(act) || !once.done(act) || set[100] != 2) return printf("device 100\n"), 1;
  // a failure is not remembered, and none of another device's
  lace::PerDevice other;
  t_device = 2;
  if (other.done([] { return false; }) || !other.done(act) || set[2] != 1) return printf("failure\n"), 1;
  t_device = -1;
  if (other.done(act)) return printf("no device\n"), 1;
  // threads on devices of their own
  lace::PerDevice shared;
  std::vector<std::atomic<int>> hits(8);
  std::vector<std::thread> th;
  for (int d = 0; d < 8; ++d)
    th.emplace_back([&, d] {
      t_device = d;
      for (int k = 0; k < 1000; ++k)
        shared.done([&] {
          ++hits[t_device];
          return true;
        });
    });
  for (auto &x : th) x.join();
  for (int d = 0; d < 8; ++d)
    if (hits[d] != 1) return printf("thread of device %d: %d times\n", d, (int)hits[d]), 1;
  printf("ok\n");
  return 0;
}
