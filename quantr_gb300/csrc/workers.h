// workers.h — host threads that share the circuits of a batch.
#pragma once

#include <system_error>
#include <thread>
#include <vector>

namespace qgpu {

// Runs work() on `count` threads at most, the calling one among them, and waits for all of them. A new
// thread starts without the caller's per-thread state (the CUDA runtime's current device is device 0
// there), so each calls enter() first and leaves at once where that returns false. Where the system
// gives no further thread the ones there are do the work.
template <class Enter, class Work>
void run_workers(int count, Enter enter, Work work) {
    auto body = [&]() {
        if (enter()) work();
    };
    std::vector<std::thread> pool;
    pool.reserve(count > 1 ? (size_t)count - 1 : 0);
    try {
        for (int w = 1; w < count; ++w) pool.emplace_back(body);
    } catch (const std::system_error&) {
    }
    body();
    for (auto& t : pool) t.join();
}

}  // namespace qgpu
