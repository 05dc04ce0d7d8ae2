// Shared allocations for the small arrays of a handle. Host code, without CUDA: the
// allocator is the caller's.
#pragma once
#include <stddef.h>

// Arrays below a quarter of SLAB share allocations of that size, one after the other
// on 512-byte boundaries; larger ones get allocations of their own, unless the rest of
// the last one holds them.
struct GamSlab {
    static constexpr size_t SLAB = 16u << 20;
    char* at = nullptr;  // what is left of the last shared allocation
    size_t left = 0;
    // bytes of memory, or null with err set: alloc(&p, n) gives n bytes at p or returns
    // an error code. An err that is set already stays, and nothing is given out then, so
    // that one look at it after several calls finds the first failure.
    template <class E, class F> void* take(size_t bytes, E& err, F&& alloc) {
        if (err != E()) return nullptr;
        bytes = (bytes + 511) / 512 * 512;
        void* p = nullptr;
        if (bytes <= left) {
            p = at;
            at += bytes;
            left -= bytes;
            return p;
        }
        const size_t n = bytes < SLAB / 4 ? SLAB : bytes;
        err = alloc(&p, n);
        if (err != E()) return nullptr;
        if (n > bytes) {  // the rest serves the arrays that follow
            at = (char*)p + bytes;
            left = n - bytes;
        }
        return p;
    }
};
