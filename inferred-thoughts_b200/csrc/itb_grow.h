// Device scratch that grows with what a call needs.
#pragma once
#include <cuda_runtime.h>

#include <initializer_list>

struct Scratch {
    void** p;
    size_t bytes;
};
// Replaces buffers that share one capacity by larger ones. All or none: after a failure the pointers are null and the capacity 0, so that a
// later, smaller call makes them again and meets no buffer that is gone. The stream's work on the old ones must be done or be waited
// for by cudaFree.
inline bool grow_scratch(size_t* cap, size_t need, std::initializer_list<Scratch> bufs) {
    if (*cap >= need) return true;
    *cap = 0;
    for (const Scratch& b : bufs) { cudaFree(*b.p); *b.p = nullptr; }
    bool ok = true;
    for (const Scratch& b : bufs)
        if (ok && cudaMalloc(b.p, b.bytes) != cudaSuccess) { *b.p = nullptr; ok = false; }
    if (!ok) {
        for (const Scratch& b : bufs) { cudaFree(*b.p); *b.p = nullptr; }
        cudaGetLastError();
        return false;
    }
    *cap = need;
    return true;
}
