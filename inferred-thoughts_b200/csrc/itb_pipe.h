// Host transfers of one context: pinned staging buffers and the threads that copy into and out of them.
#pragma once
#include <cuda_runtime.h>
#include <semaphore.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <exception>
#include <thread>
#include <vector>

// A copy from or to pageable memory goes through a staging buffer somewhere: the driver's does it on one thread and asks for a stream
// synchronise to be sure of it. Here: a small copy is one memcpy into a pinned ring and an asynchronous copy behind it (no
// synchronise); a large one runs in chunks, the chunk in flight on the bus while the next is copied by up to eight threads. The threads start
// with the first large copy and end with the context. Nothing here throws, and a refused thread, event or pinned buffer costs only time:
// the caller copies alone, waits for the stream where an event would have told it, or takes the driver's own copy.
// Chunks up are small: the bus idles while the first is copied and the threads while the last is sent, and a chunk that waits for a thread
// to wake holds up less. (4.1 MB up, mean: 2 MB chunks and four threads 437 us, 1 MB and eight 264, 0.5 MB and four 186, six 163, eight 155;
// 16.8 MB: 895, 883, 712, 633, 588.) Down, large ones want few waits for events: 16.8 MB in 2 MB chunks 491 us, in 0.5 MB ones 611; 4.1 MB 199
// in three, 157 in 0.5 MB ones. Eight pinned chunks up, three down: 11 MB a context that makes such copies.
struct HostPipe {
    static constexpr size_t RING = 1 << 20, SMALL = 128 << 10, CHUNK = 2 << 20, UP_CHUNK = 512 << 10;
    static constexpr int N_CHUNK = 3, N_UP = 8, MAX_THREAD = 7;
    uint8_t* ring = nullptr; size_t ring_at = 0; int ring_half = 0; cudaEvent_t half_ev[2] = {nullptr, nullptr}; bool half_used[2] = {false, false};
    uint8_t* chunk[N_CHUNK] = {nullptr, nullptr, nullptr}; cudaEvent_t chunk_ev[N_CHUNK] = {nullptr, nullptr, nullptr}; bool chunk_used[N_CHUNK] = {false, false, false};
    uint8_t* up_mem = nullptr; cudaEvent_t up_ev[N_UP] = {}; bool up_used[N_UP] = {};
    // Copy threads. A copy is cut into PARTS; whoever is free takes the next one, the caller included, so a thread that wakes late costs
    // nothing but its help. turn = (copy number << 8) | next part: a part is taken by raising it from the value under which the
    // copy's arguments were read, and the arguments change only after every part of the copy before is done.
    static constexpr uint64_t PARTS = 16;
    std::vector<std::thread> threads; sem_t wake; std::atomic<bool> quit{false}; std::atomic<int> asleep{0};
    std::atomic<uint64_t> turn{PARTS}, done{0};
    std::atomic<uint8_t*> jd{nullptr}; std::atomic<const uint8_t*> js{nullptr}; std::atomic<size_t> jn{0};
    void take_parts() {
        for (;;) {
            uint64_t t = turn.load(std::memory_order_acquire);
            if ((t & 255) >= PARTS) return;
            uint8_t* d = jd.load(std::memory_order_relaxed); const uint8_t* s = js.load(std::memory_order_relaxed); const size_t n = jn.load(std::memory_order_relaxed);
            if (!turn.compare_exchange_strong(t, t + 1, std::memory_order_acq_rel)) continue;
            const size_t per = ((n + PARTS - 1) / PARTS + 4095) & ~(size_t)4095, a = std::min(n, per * (t & 255)), z = std::min(n, a + per);
            if (z > a) memcpy(d + a, s + a, z - a);
            done.fetch_add(1, std::memory_order_release);
        }
    }
    bool work_left() const { return (turn.load() & 255) < PARTS; }
    // The caller pays for one wake at most, and for none while the pieces of a transfer follow each other: a thread that wakes wakes two more
    // while there is work for them, and one that finds no part looks for the next piece for LOOK_NS before it sleeps again. (The copies alone, up,
    // on eight CPUs, with seven threads each woken for each piece / three so / one memcpy, us: 4.2 MB 490 / 156 / 327, 16.8 MB 1,880 / 493 / 1,340.
    // On sixteen, seven threads either way: 16.8 MB up and down around 2,048 rows of kernels 1,650 -> 1,520; 500 rows 730 as before, and 740 when a thread
    // woke one more and not two.)
    static constexpr long long LOOK_NS = 50000;
    void help() {
        for (;;) {
            take_parts();
            const auto since = std::chrono::steady_clock::now();
            while (!work_left() && !quit.load(std::memory_order_acquire)) {
                for (int i = 0; i < 16; ++i) cpu_relax();
                if (std::chrono::steady_clock::now() - since > std::chrono::nanoseconds(LOOK_NS)) {
                    asleep.fetch_add(1);
                    if (!work_left() && !quit.load()) while (sem_wait(&wake) != 0) {}
                    asleep.fetch_sub(1);
                    for (int i = 0; i < 2; ++i) if (work_left() && asleep.load() > i) sem_post(&wake);
                    break;
                }
            }
            if (quit.load(std::memory_order_acquire)) return;
        }
    }
    static void cpu_relax() {
#if defined(__x86_64__) || defined(__i386__)
        __builtin_ia32_pause();
#endif
    }
    bool threads_tried = false;
    // Half of the CPUs, the caller's own among them, and eight at most: as many as the system grants, possibly none.
    bool start_threads() {
        if (!threads_tried) {
            threads_tried = true;
            const int n = std::min((int)MAX_THREAD, (int)std::thread::hardware_concurrency() / 2 - 1);
            try {
                if (n > 0) threads.reserve(n);
                for (int i = 0; i < n; ++i) threads.emplace_back([this] { help(); });
            } catch (const std::exception&) {}
        }
        return !threads.empty();
    }
    // Below `alone` bytes waking the threads costs more than they save: 384 KB on the way up (0.26 MB: 29 us alone, 46 with them), 512 KB down,
    // where they have slept while the device worked (1 MB of logits in three steps: a decode step of 2.49 ms took 2.54 with them).
    void copy(void* d, const void* s, size_t n, size_t alone) {
        if (n < alone || !start_threads()) { memcpy(d, s, n); return; }
        jd.store((uint8_t*)d, std::memory_order_relaxed); js.store((const uint8_t*)s, std::memory_order_relaxed); jn.store(n, std::memory_order_relaxed);
        done.store(0, std::memory_order_relaxed);
        turn.store(((turn.load(std::memory_order_relaxed) >> 8) + 1) << 8);
        if (asleep.load() > 0) sem_post(&wake);
        take_parts();
        while (done.load(std::memory_order_acquire) < PARTS) std::this_thread::yield();
    }
    HostPipe() { sem_init(&wake, 0, 0); }
    // Pinned memory with its events, all or nothing.
    template <int N>
    static bool ready(uint8_t** mem, size_t bytes, cudaEvent_t (&ev)[N]) {
        if (*mem) return true;
        bool ok = cudaMallocHost(mem, bytes) == cudaSuccess;
        if (!ok) *mem = nullptr;
        for (int i = 0; i < N && ok; ++i) ok = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming) == cudaSuccess || (ev[i] = nullptr, false);
        if (ok) return true;
        for (auto& e : ev) if (e) { cudaEventDestroy(e); e = nullptr; }
        if (*mem) { cudaFreeHost(*mem); *mem = nullptr; }
        cudaGetLastError();
        return false;
    }
    bool ready_small() { return ready(&ring, RING, half_ev); }
    bool ready_large() {
        if (!ready(&chunk[0], CHUNK * N_CHUNK, chunk_ev)) return false;
        for (int i = 1; i < N_CHUNK; ++i) chunk[i] = chunk[0] + i * CHUNK;
        return true;
    }
    bool ready_up() { return ready(&up_mem, UP_CHUNK * N_UP, up_ev); }
    // After the copies out of (or into) a staging buffer have been queued: `used` until they have run.
    static cudaError_t queued(cudaStream_t st, cudaEvent_t ev, bool& used) {
        used = true;
        if (cudaEventRecord(ev, st) == cudaSuccess) return cudaSuccess;
        cudaGetLastError();
        const cudaError_t e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) used = false;
        return e;
    }
    // Before it is touched again.
    static cudaError_t settle(cudaStream_t st, cudaEvent_t ev, bool& used) {
        if (!used) return cudaSuccess;
        cudaError_t e = cudaEventSynchronize(ev);
        if (e != cudaSuccess) { cudaGetLastError(); e = cudaStreamSynchronize(st); }
        if (e == cudaSuccess) used = false;
        return e;
    }
    ~HostPipe() {
        quit.store(true);
        for (size_t i = 0; i < threads.size(); ++i) sem_post(&wake);
        for (auto& t : threads) t.join();
        sem_destroy(&wake);
        for (auto& e : half_ev) if (e) cudaEventDestroy(e);
        for (auto& e : chunk_ev) if (e) cudaEventDestroy(e);
        for (auto& e : up_ev) if (e) cudaEventDestroy(e);
        cudaFreeHost(ring); cudaFreeHost(chunk[0]); cudaFreeHost(up_mem);
    }
    cudaError_t up(cudaStream_t st, void* dev, const void* host, size_t bytes) {
        cudaError_t e = cudaSuccess;
        if (bytes <= SMALL && ready_small()) {
            // the ring's halves alternate: a half is written again only after the copies out of it have run
            const size_t need = (bytes + 255) & ~(size_t)255, half = RING / 2;
            if (ring_at + need > half) {
                e = queued(st, half_ev[ring_half], half_used[ring_half]);
                if (e != cudaSuccess) return e;
                e = settle(st, half_ev[ring_half ^ 1], half_used[ring_half ^ 1]);
                if (e != cudaSuccess) return e;
                ring_half ^= 1; ring_at = 0;
            }
            const size_t at = half * ring_half + ring_at;
            memcpy(ring + at, host, bytes);
            ring_at += need;
            return cudaMemcpyAsync(dev, ring + at, bytes, cudaMemcpyHostToDevice, st);
        }
        if (!ready_up()) return plain(st, dev, host, bytes, cudaMemcpyHostToDevice);
        int i = 0;
        for (size_t at = 0; at < bytes; at += UP_CHUNK, i = (i + 1) % N_UP) {
            const size_t n = std::min(UP_CHUNK, bytes - at);
            if ((e = settle(st, up_ev[i], up_used[i])) != cudaSuccess) return e;
            copy(up_mem + i * UP_CHUNK, (const uint8_t*)host + at, n, 384 << 10);
            if ((e = cudaMemcpyAsync((uint8_t*)dev + at, up_mem + i * UP_CHUNK, n, cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
            if ((e = queued(st, up_ev[i], up_used[i])) != cudaSuccess) return e;
        }
        return e;
    }
    cudaError_t down(cudaStream_t st, void* host, const void* dev, size_t bytes) {
        if (bytes <= (64 << 10) || !ready_large()) return plain(st, host, dev, bytes, cudaMemcpyDeviceToHost);
        cudaError_t e = cudaSuccess;
        const size_t step = bytes >= 4 * CHUNK ? CHUNK : std::min(UP_CHUNK, (bytes / 3 + 65535) & ~(size_t)65535), n_step = (bytes + step - 1) / step;
        auto issue = [&](size_t s) {
            const int i = (int)(s % N_CHUNK);
            e = settle(st, chunk_ev[i], chunk_used[i]);
            if (e == cudaSuccess) e = cudaMemcpyAsync(chunk[i], (const uint8_t*)dev + s * step, std::min(step, bytes - s * step), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = queued(st, chunk_ev[i], chunk_used[i]);
        };
        for (size_t s = 0; s < n_step && s < (size_t)N_CHUNK && e == cudaSuccess; ++s) issue(s);
        for (size_t s = 0; s < n_step && e == cudaSuccess; ++s) {
            const int i = (int)(s % N_CHUNK);
            if ((e = settle(st, chunk_ev[i], chunk_used[i])) != cudaSuccess) break;
            copy((uint8_t*)host + s * step, chunk[i], std::min(step, bytes - s * step), 512 << 10);
            if (s + N_CHUNK < n_step) issue(s + N_CHUNK);
        }
        return e;
    }
    static cudaError_t plain(cudaStream_t st, void* to, const void* from, size_t bytes, cudaMemcpyKind kind) {
        const cudaError_t e = cudaMemcpyAsync(to, from, bytes, kind, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
};
