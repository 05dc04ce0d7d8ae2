// A driver's entry point that is looked up once and kept. Host code, without CUDA.
#pragma once
#include <atomic>

// find() gives the address or null. An address is kept for every later call; a
// failure is not, so that the next call looks again. Safe with several threads: they
// find the same address.
struct GamEntry {
    std::atomic<void*> at{nullptr};
    template <class F> void* get(F&& find) {
        void* p = at.load(std::memory_order_acquire);
        if (!p && (p = find())) at.store(p, std::memory_order_release);
        return p;
    }
};
