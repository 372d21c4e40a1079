// Work beside a pass's main stream.
#pragma once
#include <cuda_runtime.h>

// beside(f) runs f with `cur` set to the second stream, between an event on the main one and an event behind it; what f's kernels write
// may be read, and what they read may be written, behind meet(). A pass that ends early, on an error, meets on its way out: the next pass's
// kernels would otherwise write rows that the second stream still reads. Where an event or a wait is refused, f runs on the main stream,
// or the host waits.
struct SideStream {
    cudaStream_t main, side;                // side null: everything on the main stream
    cudaEvent_t fork, join;
    cudaStream_t cur;
    bool open = false;
    SideStream(cudaStream_t main, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) : main(main), side(side), fork(fork), join(join), cur(main) {}
    SideStream(const SideStream&) = delete;
    SideStream& operator=(const SideStream&) = delete;
    template <class F>
    void beside(F f) {
        meet();
        if (!side || cudaEventRecord(fork, main) != cudaSuccess || cudaStreamWaitEvent(side, fork, 0) != cudaSuccess) { f(); return; }
        cur = side; open = true;
        f();
        cur = main;
        if (cudaEventRecord(join, side) != cudaSuccess) { cudaStreamSynchronize(side); open = false; }
    }
    void meet() {
        if (!open) return;
        open = false; cur = main;
        if (cudaStreamWaitEvent(main, join, 0) != cudaSuccess) cudaStreamSynchronize(side);
    }
    ~SideStream() { meet(); }
};
