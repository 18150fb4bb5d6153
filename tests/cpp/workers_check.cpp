// Exercises tgbm::WorkerPool with threads that cannot be started.  Prints "<name> <sum of the tasks run> <threads started>".
#include <atomic>
#include <cstdio>
#include <memory>
#include <system_error>
#include <vector>

#include "../../thundergbm_b200/csrc/tgbm_workers.h"

struct Worker { int tasks = 0; };

static void scenario(const char *name, int most, int startable, int callers, int n) {
    auto started = std::make_shared<std::atomic<int>>(0);
    auto *pool = new tgbm::WorkerPool<Worker>(most, [=](std::function<void()> f) {   // (its threads wait on it until the process ends)
        if (*started >= startable) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        ++*started;
        std::thread(std::move(f)).detach();
    });
    std::atomic<int> sum{0};
    std::vector<std::thread> t;
    for (int c = 0; c < callers; ++c)
        t.emplace_back([&] {
            for (int round = 0; round < 50; ++round)   // a later call finds what an earlier one left
                pool->run(n, [&](Worker &w, int k) { ++w.tasks; sum += k + 1; });
        });
    for (auto &x : t) x.join();
    printf("%s %d %d\n", name, sum.load(), started->load());
}

int main() {
    scenario("all", 4, 4, 1, 8);
    scenario("some", 4, 2, 3, 8);
    scenario("one", 4, 1, 3, 8);
    scenario("none", 4, 0, 3, 8);
    scenario("empty", 4, 4, 1, 0);
    return 0;
}
