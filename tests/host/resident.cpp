// The per-device cache of resident block counts: every device asks for
// itself, once (a device beyond the table each time), and threads that step
// worlds of one device at once agree.  Built with the thread sanitiser where
// there is one: a data race ends the program with its status.
#include <cstdio>
#include <thread>
#include <vector>

#include "../../ornis_gb300/csrc/avbd_resident.h"

int main() {
    static avbd::Resident r;
    int bad = 0;
    for (int dev = 0; dev < 80; dev++)
        for (int k = 0; k < 2; k++) {
            int asked = 0;
            const int n = r.on(dev, [&] { asked++; return 100 + dev; });
            if (n != 100 + dev || asked != (k == 0 || dev >= 64 ? 1 : 0)) {
                std::printf("device %d, call %d: %d blocks, asked %d times\n", dev, k, n, asked);
                bad++;
            }
        }
    static avbd::Resident shared;
    int got[8] = {};
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; t++)
        ts.emplace_back([&, t] {
            for (int k = 0; k < 1000; k++) got[t] = shared.on(t & 1, [&] { return 456 + (t & 1); });
        });
    for (auto& t : ts) t.join();
    for (int t = 0; t < 8; t++) bad += got[t] != 456 + (t & 1);
    std::printf("bad %d\n", bad);
    return bad != 0;
}
