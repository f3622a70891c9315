// gbh_parallel.h -- host work spread over threads.
#pragma once
#include <cstddef>
#include <exception>
#include <thread>
#include <vector>

namespace gbh {

// f(i) for every i below n that `want` names, each on a thread of its own; the
// rest runs here where no more threads are to be had (a thread object
// destroyed while it runs would end the process).
template <class Thread = std::thread, class Want, class F> void in_threads(size_t n, Want want, F f)
{
    std::vector<Thread> th;
    size_t i = 0;
    try {
        th.reserve(n);
        for (; i < n; ++i)
            if (want(i)) th.emplace_back(f, i);
    } catch (const std::exception &) {
    }
    for (; i < n; ++i)
        if (want(i)) f(i);
    for (Thread &t : th) t.join();
}

}  // namespace gbh
