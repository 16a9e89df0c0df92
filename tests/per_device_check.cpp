// csrc/per_device.h by itself (test_per_device.py): each device is asked once, a failure again, devices beyond the table every time.
#include "per_device.h"

#include <cstdio>
#include <thread>
#include <vector>

#define CHECK(c) do { if (!(c)) { std::printf("failed: %s\n", #c); return 1; } } while (0)

int main() {
    static ib::PerDevice once;
    int made[3] = {0, 0, 0};
    for (int pass = 0; pass < 3; pass++)
        for (int d = 0; d < 3; d++) CHECK(once.get(d, [&] { made[d]++; return 10 + d; }) == 10 + d);
    for (int d = 0; d < 3; d++) CHECK(made[d] == 1);
    int tries = 0;
    CHECK(once.get(5, [&] { tries++; return 0; }) == 0);
    CHECK(once.get(5, [&] { tries++; return 7; }) == 7);
    CHECK(once.get(5, [&] { tries++; return 8; }) == 7 && tries == 2);
    for (int d : {-1, 64, 1000}) CHECK(once.get(d, [&] { return 3; }) == 3 && once.get(d, [&] { return 4; }) == 4);
    static ib::PerDevice shared;
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; t++)
        threads.emplace_back([&] {
            for (int i = 0; i < 10000; i++)
                if (shared.get(i % 8, [&] { return 100 + i % 8; }) != 100 + i % 8) wrong++;
        });
    for (auto& t : threads) t.join();
    CHECK(wrong == 0);
    return 0;
}
