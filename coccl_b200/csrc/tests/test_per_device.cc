// Values that kernels' launchers keep per device (kernels/per_device.h).
#include <thread>
#include <vector>

#include "host_test.h"
#include "kernels/per_device.h"

using coccl::PerDevice;

TEST(per_device_every_device_is_initialised_once) {
  PerDevice<int> p;
  int calls = 0;
  for (int round = 0; round < 3; ++round) {
    for (int dev : {0, 3, 1}) {
      const int* v = nullptr;
      EXPECT(p.get(dev, &v, [&](int& x) { x = 10 + dev; ++calls; return 0; }) == 0);
      EXPECT(v != nullptr && *v == 10 + dev);
    }
  }
  EXPECT(calls == 3);
}

TEST(per_device_a_failure_is_returned_and_tried_again) {
  PerDevice<int> p;
  const int* v = nullptr;
  EXPECT(p.get(2, &v, [](int&) { return 7; }) == 7);
  EXPECT(v == nullptr);
  EXPECT(p.get(2, &v, [](int& x) { x = 5; return 0; }) == 0 && *v == 5);
}

TEST(per_device_devices_beyond_the_table_are_initialised_at_every_use) {
  PerDevice<int> p;
  int calls = 0;
  for (int dev : {PerDevice<int>::kDevices, -1, PerDevice<int>::kDevices}) {
    const int* v = nullptr;
    EXPECT(p.get(dev, &v, [&](int& x) { x += 3; ++calls; return 0; }) == 0);
    EXPECT(v != nullptr && *v == 3);
  }
  EXPECT(calls == 3);
}

TEST(per_device_threads_share_one_initialisation) {
  PerDevice<int> p;
  std::atomic<int> calls{0}, wrong{0};
  std::vector<std::thread> ts;
  for (int i = 0; i < 8; ++i)
    ts.emplace_back([&] {
      for (int dev = 0; dev < 8; ++dev) {
        const int* v = nullptr;
        if (p.get(dev, &v, [&](int& x) { x = dev + 1; ++calls; return 0; }) != 0 || *v != dev + 1) ++wrong;
      }
    });
  for (auto& t : ts) t.join();
  EXPECT(calls == 8 && wrong == 0);
}
