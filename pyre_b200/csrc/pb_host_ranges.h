// Host memory that a kernel may be given: the page-locked allocations of this library, by address (pb_host_alloc / pb_host_free).  Memory that a
// caller page-locked itself is not in here: its attributes can be asked for one address only, not for a range, and it may be read-only for the GPU.
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <map>
#include <mutex>

class PbHostRanges {
    std::mutex mu;
    std::map<uintptr_t, size_t> at;   // first byte -> bytes
public:
    // (without memory for the entry the range stays unknown: the copy engine moves it)
    void add(const void* p, size_t n) {
        std::lock_guard<std::mutex> lock(mu);
        try { at[(uintptr_t)p] = n; } catch (...) {}
    }
    void drop(const void* p) {
        std::lock_guard<std::mutex> lock(mu);
        at.erase((uintptr_t)p);
    }
    // whether all of [p, p + n) lies in one of them
    bool inside(const void* p, size_t n) {
        std::lock_guard<std::mutex> lock(mu);
        const uintptr_t a = (uintptr_t)p;
        auto it = at.upper_bound(a);
        if (it == at.begin()) return false;
        --it;
        const size_t o = a - it->first;
        return o <= it->second && n <= it->second - o;
    }
};
