// Values made once per device (csrc/psv_device.hpp), by several threads at once.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "psv_device.hpp"

int main()
{
    psv::PerDevice<int> v;
    std::atomic<int> made[4] = {}, wrong{0};
    std::vector<std::thread> th;
    for (int t = 0; t < 8; t++)
        th.emplace_back([&, t] {
            for (int k = 0; k < 4000; k++) {
                const int dev = (t + k) % 4;
                if (v.get(dev, [&] { return made[dev]++, 100 + dev; }) != 100 + dev) wrong++;
            }
        });
    for (auto &t : th) t.join();
    for (int d = 0; d < 4; d++)
        if (made[d] != 1) return printf("device %d: made %d times\n", d, (int)made[d]), 1;
    if (wrong) return printf("%d wrong values\n", (int)wrong), 1;
    printf("ok %d devices\n", 4);
    return 0;
}
