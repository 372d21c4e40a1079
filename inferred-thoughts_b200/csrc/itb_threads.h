// Host work in shares, a thread each.
#pragma once
#include <exception>
#include <thread>
#include <vector>

// fn(0) .. fn(n - 1), each on a thread of its own; the shares whose thread the system refuses run on the caller's, one after the other.
// Returns when all are done. fn must not throw.
template <class F>
static void on_threads(unsigned n, F&& fn) {
    std::vector<std::thread> th;
    unsigned t = 0;
    try {
        th.reserve(n);
        for (; t < n; ++t) th.emplace_back([&fn, t] { fn(t); });
    } catch (const std::exception&) {}
    for (; t < n; ++t) fn(t);
    for (auto& x : th) x.join();
}
