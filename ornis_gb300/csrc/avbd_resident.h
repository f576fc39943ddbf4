// Blocks of one kernel that a device holds at once, asked for once per device.
// Worlds are stepped from any host thread, so an entry is an atomic: two
// threads may both ask, and store the same number.
#pragma once
#include <atomic>

namespace avbd {

class Resident {
    static constexpr int DEVICES = 64;
    std::atomic<int> blocks[DEVICES] = {};

  public:
    // ask(): sets what the kernel needs on the current device `dev` and
    // returns its resident blocks; beyond DEVICES it is asked every time.
    template <class Ask>
    int on(int dev, Ask ask) {
        if (dev < 0 || dev >= DEVICES) return ask();
        int n = blocks[dev].load(std::memory_order_acquire);
        if (n == 0) {
            n = ask();
            blocks[dev].store(n, std::memory_order_release);
        }
        return n;
    }
};

}  // namespace avbd
