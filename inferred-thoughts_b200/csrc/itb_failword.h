// One context's word for kernels that give up a bounded wait.
#pragma once
#include <cuda_runtime.h>

// Host memory, so that a look costs nothing; where four pinned bytes are refused, device memory, and a look is a copy of four bytes. A look
// belongs behind a wait for the stream. It takes the word: the kernels of the next call start from zero.
struct FailWord {
    int* word = nullptr;                       // where kernels store: 0, or what was waited for (3 operands, 4 issue, 5 accumulators)
    bool on_device = false;
    cudaError_t open() {
        if (cudaHostAlloc((void**)&word, 4, cudaHostAllocMapped) == cudaSuccess) { *(volatile int*)word = 0; return cudaSuccess; }
        cudaGetLastError();
        word = nullptr; on_device = true;
        cudaError_t e = cudaMalloc((void**)&word, 4);
        if (e != cudaSuccess) word = nullptr;
        else if ((e = cudaMemset(word, 0, 4)) != cudaSuccess) close();
        return e;
    }
    void set(int v) { if (on_device) cudaMemcpy(word, &v, 4, cudaMemcpyHostToDevice); else *(volatile int*)word = v; }
    int take() {
        int v = 0;
        if (!word) return 0;
        if (!on_device) v = *(volatile int*)word; else if (cudaMemcpy(&v, word, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return 0;      // a device error, which the caller's own wait reports
        if (v) set(0);
        return v;
    }
    void close() {
        if (on_device) cudaFree(word); else cudaFreeHost(word);
        word = nullptr;
    }
};
