// workers_host.cpp — run_workers (quantr_gb300/csrc/workers.h): every thread enters once, before its work and
// with the caller's setting; a thread that may not enter does no work; all items are taken once.
// Prints "fails <n>"; exit code 0 when there are none.
#include <atomic>
#include <cstdio>
#include <mutex>
#include <set>
#include <thread>

#include "../../quantr_gb300/csrc/workers.h"

static thread_local int current = 0;  // stands for the CUDA runtime's current device

int main() {
    int fails = 0;
    for (int count : {0, 1, 2, 4, 16}) {
        current = 3;
        const int caller = current;
        std::atomic<int> next{0}, entered{0}, wrong{0};
        std::mutex mu;
        std::multiset<int> items;
        std::set<std::thread::id> threads;
        qgpu::run_workers(
            count,
            [&]() {
                current = caller;
                ++entered;
                return true;
            },
            [&]() {
                for (int i; (i = next.fetch_add(1)) < 1000;) {
                    if (current != caller) ++wrong;
                    std::lock_guard<std::mutex> lk(mu);
                    items.insert(i);
                    threads.insert(std::this_thread::get_id());
                }
            });
        fails += wrong != 0;
        fails += entered != (count > 1 ? count : 1);
        fails += items.size() != 1000 || std::set<int>(items.begin(), items.end()).size() != 1000;
        // only the caller may enter: the others take nothing
        const std::thread::id me = std::this_thread::get_id();
        std::atomic<int> others{0}, taken{0};
        qgpu::run_workers(
            count, [&]() { return std::this_thread::get_id() == me; },
            [&]() {
                ++taken;
                if (std::this_thread::get_id() != me) ++others;
            });
        fails += others != 0 || taken != 1;
    }
    std::printf("fails %d\n", fails);
    return fails != 0;
}
