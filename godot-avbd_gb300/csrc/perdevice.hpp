// A value found once for each device of the process.
#pragma once

#include <mutex>

namespace avbdg {

// What a kernel may use (clusters beyond eight CTAs, shared memory beyond 48 KB) is allowed device by device, and
// how much of it a device holds is its own: `find` runs at the first `get` for a device, with that device current,
// and its value (> 0) is kept. Safe with several threads.
class PerDevice {
public:
    template <typename F>
    int get(int device, F find) {
        std::lock_guard<std::mutex> lock(mutex);
        if (device < 0 || device >= kMost)
            return find();
        if (values[device] <= 0)
            values[device] = find();
        return values[device];
    }

private:
    static constexpr int kMost = 64; // (beyond: found each time)
    std::mutex mutex;
    int values[kMost] = {};
};

} // namespace avbdg
