// Values found once a device: found again for another device, not for one seen before, by several threads too.
#include <cassert>
#include <thread>
#include <vector>

#include "perdevice.hpp"

int main() {
    avbdg::PerDevice values;
    int found = 0;
    const auto value = [&](int device) { return values.get(device, [&] { return ++found, 10 + device; }); };
    for (int turn = 0; turn < 3; turn++)
        for (int device = 0; device < 64; device++)
            assert(value(device) == 10 + device);
    assert(found == 64);
    assert(value(64) == 74 && value(64) == 74 && value(-1) == 9 && found == 67); // not kept
    avbdg::PerDevice shared;
    int runs = 0;
    std::vector<std::thread> threads;
    for (int k = 0; k < 8; k++)
        threads.emplace_back([&] {
            for (int n = 0; n < 1000; n++)
                assert(shared.get(n & 3, [&] { return ++runs, 1 + (n & 3); }) == 1 + (n & 3));
        });
    for (std::thread &t : threads)
        t.join();
    assert(runs == 4);
    return 0;
}
