// each_item (vbd_internal.h): an exception of the work reaches the caller from any worker, after every worker has ended.
#include <atomic>
#include <cstdio>
#include <new>
#include <set>
#include <stdexcept>

#include "vbd_internal.h"

int main() {
    for (bool large : {false, true})
        for (int bad : {0, 5, 199}) {
            std::atomic<int> running{0};
            bool caught = false;
            try {
                vbd::each_item(200, large, [&](int, int i) {
                    ++running;
                    std::this_thread::sleep_for(std::chrono::microseconds(200));
                    --running;
                    if (i == bad) throw std::bad_alloc();
                });
            } catch (const std::bad_alloc&) {
                caught = running == 0;
            }
            if (!caught) return std::printf("large %d, item %d: not passed on\n", large, bad), 1;
        }
    // several at once: one of them
    try {
        vbd::each_range(1000000, true, [](int, long long, long long) { throw std::runtime_error("x"); });
        return 1;
    } catch (const std::runtime_error&) {
    }
    // every item once, workers in range
    for (int items : {0, 1, 3, 1000}) {
        std::vector<std::atomic<int>> n(items);
        std::atomic<bool> in_range{true};
        vbd::each_item(items, true, [&](int w, int i) {
            ++n[i];
            if (w < 0 || w >= vbd::kMaxWorkers) in_range = false;
        });
        for (auto& k : n)
            if (k != 1) return 1;
        if (!in_range) return 1;
    }
    return 0;
}
