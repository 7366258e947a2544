// Answers are kept by device and key, what is no answer is not kept, and threads may ask at once.
#include "device_table.h"

#include <cstdio>
#include <thread>
#include <vector>

static int fails = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++fails; } } while (0)

int main() {
    static DeviceTable<6> table;
    int asked = 0;
    auto says = [&](int n) { return [&asked, n] { ++asked; return n; }; };
    CHECK(table.get(0, 1, says(73)) == 73 && asked == 1);
    CHECK(table.get(0, 1, says(9)) == 73 && asked == 1);            // kept
    CHECK(table.get(1, 1, says(66)) == 66 && asked == 2);           // another device's
    CHECK(table.get(0, 2, says(48)) == 48 && asked == 3);           // another key's
    CHECK(table.get(0, 1, says(9)) == 73 && table.get(1, 1, says(9)) == 66 && asked == 3);
    CHECK(table.get(2, 0, says(0)) == 0 && table.get(2, 0, says(-3)) == -3 && table.get(2, 0, says(5)) == 5 && asked == 6);
    for (int device : {-1, 64, 1000}) CHECK(table.get(device, 0, says(7)) == 7 && table.get(device, 0, says(8)) == 8);
    CHECK(table.get(0, 6, says(1)) == 1 && table.get(0, 6, says(2)) == 2 && table.get(1, 0, says(3)) == 3);
    static DeviceTable<4> shared;
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            for (int i = 0; i < 4000; ++i) {
                const int device = i % 64, key = (i / 64) % 4, want = 1 + 4 * device + key;
                if (shared.get(device, key, [&] { return want; }) != want) ++wrong;
            }
        });
    for (auto &t : threads) t.join();
    CHECK(wrong == 0);
    if (!fails) std::printf("OK\n");
    return fails ? 1 : 0;
}
