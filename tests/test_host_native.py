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
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-g", "-Wall", f"-I{CSRC}", f"-I{CUDA}/include", str(src), "-o", str(exe), "-pthread"], check=True, timeout=120)
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
