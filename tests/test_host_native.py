"""Host-side native code that the CUDA runtime surrounds, compiled for the CPU: the headers under test are included into a small
program in which the runtime's calls are stand-ins that count, fail or run late as a case asks."""
import os
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "inferred-thoughts_b200" / "csrc"
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def run(tmp_path, source):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-g", "-Wall", f"-I{CSRC}", f"-I{CUDA}/include", str(src), "-o", str(exe), "-pthread", "-ldl"], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, f"exit {r.returncode}\n{r.stdout}{r.stderr}"


CHECK = """
#include <stdio.h>
#include <stdlib.h>
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\\n", __LINE__, #x); exit(1); } } while (0)
"""


def test_shared_memory_limits_are_kept_by_device_and_only_raised(tmp_path):
    run(tmp_path, CHECK + r"""
#include <map>
#include <thread>
#include <utility>
#include <vector>
#include "itb_smem.h"
static std::map<std::pair<int, const void*>, size_t> limit;     // the driver's own state: what the last set left
static int calls = 0, refuse = 0;
static SmemLimits table;
static int raise(int dev, const void* fn, size_t bytes) {
    return table.raise(dev, fn, bytes, [&] { ++calls; if (refuse) return 1; limit[{dev, fn}] = bytes; return 0; });
}
int main() {
    int a, b;
    CHECK(raise(0, &a, 100) == 0 && calls == 1 && (limit[{0, &a}] == 100));
    CHECK(raise(0, &a, 100) == 0 && raise(0, &a, 60) == 0 && calls == 1 && (limit[{0, &a}] == 100));     // seen there: nothing to do, and never lowered
    CHECK(raise(1, &a, 60) == 0 && calls == 2 && (limit[{1, &a}] == 60));                                // the same kernel on another device
    CHECK(raise(0, &b, 60) == 0 && calls == 3 && raise(0, &a, 120) == 0 && calls == 4 && (limit[{0, &a}] == 120));
    refuse = 1;
    CHECK(raise(1, &a, 300) == 1 && raise(1, &a, 300) == 1 && calls == 6);                               // an error is handed back each time
    refuse = 0;
    CHECK(raise(1, &a, 60) == 0 && calls == 6 && raise(1, &a, 200) == 0 && calls == 7);
    CHECK(raise(-1, &a, 10) == 0 && raise(1000, &a, 10) == 0 && raise(1000, &a, 10) == 0 && calls == 10); // beyond the table: set each time
    std::vector<std::thread> th;                                                                          // threads that need different amounts
    for (int t = 0; t < 8; ++t) th.emplace_back([t, &b] { for (int i = 0; i < 2000; ++i) raise(2, &b, 1 + (i * 7 + t * 13) % 997); });
    for (auto& t : th) t.join();
    CHECK((limit[{2, &b}] == 997));
    return 0;
}
""")


def test_every_kernel_limit_goes_through_that_table():
    """No launch keeps a "set once" of its own: those were per process or thread, and a second device never got its limit."""
    hits = [f"{p.name}:{i + 1}" for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh", ".h")
            for i, line in enumerate(p.read_text().splitlines()) if "cudaFuncAttributeMaxDynamicSharedMemorySize" in line]
    assert len(hits) == 1 and hits[0].startswith("itb_ctx.cu"), hits
    for p in CSRC.iterdir():
        if p.suffix in (".cu", ".cuh"):
            assert not re.search(r"static (thread_local )?bool attr", p.read_text()), p.name


# The runtime calls that itb_pipe.h makes, with a stream whose copies run only when something waits for them -- so a staging buffer that is
# written again too early is seen in the data -- and switches that make one kind of call fail.
FAKE_RUNTIME = CHECK + r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <deque>
#include <vector>
#include "itb_pipe.h"
struct CUevent_st { size_t at = 0; };
struct Copy { void* d; const void* s; size_t n; };
static std::deque<Copy> queue;
static size_t issued = 0, ran = 0;
static int events = 0;                       // alive
static bool no_pinned = false, no_event = false, no_record = false, no_wait = false, no_thread = false;
static int event_after = 1 << 30;            // with no_event: that many are still made
static void run_to(size_t at) { for (; ran < at; ++ran) { memcpy(queue.front().d, queue.front().s, queue.front().n); queue.pop_front(); } }
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { if (no_pinned) return cudaErrorMemoryAllocation; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { if (no_event && event_after-- <= 0) return cudaErrorMemoryAllocation; *e = new CUevent_st; ++events; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --events; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { if (!e || no_record) return cudaErrorInvalidResourceHandle; e->at = issued; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { if (!e || no_wait) return cudaErrorInvalidResourceHandle; run_to(e->at); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { run_to(issued); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { queue.push_back({d, s, n}); ++issued; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    if (no_thread) return EAGAIN;
    return ((int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
}
static void transfers() {
    {
        HostPipe p;
        unsigned seed = 1;
        std::vector<std::vector<uint8_t>> dev, want;
        for (int round = 0; round < 3; ++round)
            for (size_t n : {(size_t)1, (size_t)4096, (size_t)131072, (size_t)131072, (size_t)131072, (size_t)131072, (size_t)131072, (size_t)131073, (size_t)3000001, (size_t)9000000, (size_t)524288}) {
                std::vector<uint8_t> h(n);
                for (auto& b : h) b = (uint8_t)((seed = seed * 1664525u + 1013904223u) >> 24);
                dev.emplace_back(n); want.push_back(h);
                CHECK(p.up(nullptr, dev.back().data(), h.data(), n) == cudaSuccess);
                memset(h.data(), 0, n);                    // the caller may change its bytes once the call is back
            }
        run_to(issued);
        for (size_t i = 0; i < dev.size(); ++i) CHECK(dev[i] == want[i]);
        for (size_t i = 0; i < dev.size(); ++i) {
            std::vector<uint8_t> h(dev[i].size());
            CHECK(p.down(nullptr, h.data(), dev[i].data(), h.size()) == cudaSuccess);
            CHECK(h == want[i]);
        }
    }
    CHECK(events == 0);
}
"""


def test_transfers_come_through(tmp_path):
    run(tmp_path, FAKE_RUNTIME + "int main() { transfers(); return 0; }")


def test_transfers_without_copy_threads(tmp_path):
    """The system refuses a thread: the caller copies alone, and nothing is thrown out of the C interface."""
    run(tmp_path, FAKE_RUNTIME + "int main() { no_thread = true; transfers(); return 0; }")


def test_transfers_without_pinned_memory_or_events(tmp_path):
    run(tmp_path, FAKE_RUNTIME + """int main() {
        no_pinned = true; transfers(); no_pinned = false;
        for (int made = 0; made < 6; ++made) { no_event = true; event_after = made; transfers(); }
        return 0;
    }""")


def test_transfers_whose_events_cannot_be_recorded_or_waited_for(tmp_path):
    """A staging buffer is not written again while a copy may still read it, whichever call fails."""
    run(tmp_path, FAKE_RUNTIME + "int main() { no_record = true; transfers(); no_record = false; no_wait = true; transfers(); return 0; }")


def test_copy_threads_are_counted_by_the_cpus_and_woken_once(tmp_path):
    """Half of the CPUs copy, the caller's own among them, and the caller pays for one wake a piece at most (for none of the pieces that
    find the threads still looking): threads by the dozen, each woken for each piece, made a copy on eight CPUs slower than one memcpy."""
    run(tmp_path, FAKE_RUNTIME + r"""
#include <unistd.h>
static int cpus = 1, wakes = 0;
static pthread_t caller;
extern "C" {
int get_nprocs() noexcept { return cpus; }
int sem_post(sem_t* s) noexcept { wakes += pthread_equal(pthread_self(), caller) != 0; return ((int (*)(sem_t*))dlsym(RTLD_NEXT, "sem_post"))(s); }
}
int main() {
    caller = pthread_self();
    const int want[][2] = {{1, 0}, {2, 0}, {4, 1}, {8, 3}, {16, 7}, {128, 7}};
    std::vector<uint8_t> h((size_t)16 << 20), d(h.size()), back(h.size());
    for (size_t i = 0; i < h.size(); ++i) h[i] = (uint8_t)(i * 2654435761u >> 13);
    for (auto& w : want) {
        HostPipe p;
        cpus = w[0]; wakes = 0;
        memset(d.data(), 0, d.size()); memset(back.data(), 0, back.size());
        CHECK(p.up(nullptr, d.data(), h.data(), h.size()) == cudaSuccess);
        run_to(issued);
        CHECK((int)p.threads.size() == w[1]);
        CHECK(wakes <= (int)(h.size() / HostPipe::UP_CHUNK));
        usleep(2000);                                          // they sleep again, and are woken for the way down
        wakes = 0;
        CHECK(p.down(nullptr, back.data(), d.data(), h.size()) == cudaSuccess);
        CHECK(wakes <= (int)(h.size() / HostPipe::CHUNK));
        CHECK(d == h && back == h);
    }
    return 0;
}
""")


def test_shares_whose_thread_is_refused_run_on_the_caller(tmp_path):
    """The correction table of log is built on all host threads inside a C entry point: a refused thread must not end the program."""
    run(tmp_path, FAKE_RUNTIME + r"""
#include "itb_threads.h"
int main() {
    for (int refused : {0, 1}) {
        no_thread = refused;
        for (unsigned n : {1u, 2u, 33u}) {
            std::vector<int> seen(n, 0);
            on_threads(n, [&](unsigned t) { seen[t]++; });
            for (int s : seen) CHECK(s == 1);
        }
    }
    return 0;
}
""")


def test_scratch_that_cannot_grow_leaves_no_stale_pointer(tmp_path):
    """One of two buffers cannot be had: both are gone and the capacity says so; a later call that needs less makes them again."""
    run(tmp_path, CHECK + r"""
#include <set>
#include "itb_grow.h"
static std::set<void*> alive;
static int made = 0, fail_at = -1;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { if (made++ == fail_at) return cudaErrorMemoryAllocation; *p = malloc(n); alive.insert(*p); return cudaSuccess; }
cudaError_t cudaFree(void* p) { if (p) { CHECK(alive.erase(p) == 1); free(p); } return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
int main() {
    for (int f : {-1, 2, 3}) {
        made = 0; fail_at = f;
        void *a = nullptr, *b = nullptr; size_t cap = 0;
        CHECK(grow_scratch(&cap, 100, {{&a, 100}, {&b, 400}}) && cap == 100 && alive.count(a) && alive.count(b) && alive.size() == 2);
        CHECK(grow_scratch(&cap, 60, {{&a, 60}, {&b, 240}}) && cap == 100 && made == 2);
        const bool ok = grow_scratch(&cap, 1000, {{&a, 1000}, {&b, 4000}});
        CHECK(ok == (f < 0));
        if (!ok) CHECK(!a && !b && cap == 0 && alive.empty());
        CHECK(grow_scratch(&cap, 50, {{&a, 50}, {&b, 200}}) && alive.count(a) && alive.count(b) && alive.size() == 2);
        cudaFree(a); cudaFree(b);
    }
    return 0;
}
""")


def test_work_beside_the_main_stream_is_met_on_every_way_out(tmp_path):
    """A pass that ends early between beside and meet leaves the main stream waiting for the second one, whatever call was refused."""
    run(tmp_path, CHECK + r"""
#include <stdexcept>
#include "itb_side.h"
struct CUstream_st { int seen[2] = {0, 0}, done = 0; };      // per stream: work queued; of each stream's work, how much is ordered before what comes next
struct CUevent_st { int at[2] = {0, 0}; };
static CUstream_st S[2];
static int refuse = 0, calls = 0;
static bool no() { return ++calls == refuse; }
extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { if (no()) return cudaErrorInvalidResourceHandle; const int i = (int)(s - S); for (int k = 0; k < 2; ++k) e->at[k] = k == i ? s->done : s->seen[k]; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { if (no()) return cudaErrorInvalidResourceHandle; for (int k = 0; k < 2; ++k) if (s->seen[k] < e->at[k]) s->seen[k] = e->at[k]; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { const int i = (int)(s - S); S[1 - i].seen[i] = s->done; return cudaSuccess; }
}
static bool pass(bool two, int leave) {
    CUevent_st fork, join;
    SideStream x(&S[0], two ? &S[1] : nullptr, &fork, &join);
    for (int layer = 0; layer < 3; ++layer) {
        CHECK(S[0].seen[1] == S[1].done);                    // this layer's main chain comes behind all of the last one's side work
        S[0].done++;
        x.beside([&] { if (x.cur == &S[1]) CHECK(S[1].seen[0] == S[0].done); x.cur->done++; });
        CHECK(x.cur == &S[0]);
        S[0].done++;
        if (layer == leave) return false;
        if (layer == leave - 10) throw std::runtime_error("out");
        x.meet();
    }
    return true;
}
int main() {
    for (bool two : {false, true})
        for (int r = 0; r < 12; ++r)
            for (int leave : {-1, 0, 1, 2, 10, 11, 12}) {
                S[0] = S[1] = CUstream_st(); refuse = r; calls = 0;
                try { pass(two, leave); } catch (const std::exception&) {}
                CHECK(S[0].seen[1] == S[1].done);            // the next pass too
            }
    return 0;
}
""")


def test_word_of_a_wait_that_ran_out_where_pinned_memory_is_refused(tmp_path):
    """Host memory or, without it, device memory: the word reads as stored, once, and a context needs both refused to fail."""
    run(tmp_path, CHECK + r"""
#include <string.h>
#include "itb_failword.h"
static bool no_pinned = false, no_device = false; static int alive = 0, device_reads = 0;
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { if (no_pinned) return cudaErrorMemoryAllocation; ++alive; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { if (p) { --alive; free(p); } return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { if (no_device) return cudaErrorMemoryAllocation; ++alive; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { if (p) { --alive; free(p); } return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { ++device_reads; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
int main() {
    for (bool refused : {false, true}) {
        no_pinned = refused;
        FailWord f;
        CHECK(f.take() == 0 && f.open() == cudaSuccess && f.on_device == refused && f.take() == 0);
        for (int v : {3, 4, 5}) { *f.word = v; CHECK(f.take() == v && f.take() == 0); }
        CHECK(refused == (device_reads > 0));
        f.close();
        CHECK(alive == 0 && !f.word);
    }
    no_device = true;
    FailWord f;
    CHECK(f.open() == cudaErrorMemoryAllocation && !f.word && f.take() == 0 && alive == 0);
    return 0;
}
""")
