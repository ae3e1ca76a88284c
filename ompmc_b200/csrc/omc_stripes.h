// Host threads for work that falls into a few equal stripes.
#pragma once
#include <exception>
#include <thread>
#include <vector>

namespace omc {

// work(0) .. work(n - 1), each once: work(0) here, the others on threads of
// their own, or here too where no more threads (or memory for them) are to be
// had.  `work` does not throw, and neither does this.
template <typename F>
void run_stripes(int n, const F &work) {
    std::vector<std::thread> pool;
    int rest = 1;
    try {
        pool.reserve(n - 1);
        for (; rest < n; rest++) pool.emplace_back(work, rest);
    } catch (const std::exception &) {
    }
    work(0);
    for (; rest < n; rest++) work(rest);
    for (auto &t : pool) t.join();
}

}  // namespace omc
