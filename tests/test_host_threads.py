"""Host threads of the engine build (cospdnn_b200/csrc/host_threads.h): with no
memory to be had, even for a message, a failure is an error code and every
thread is joined."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdlib>
#include <cstring>
#include <string>
#include "host_threads.h"

static std::atomic<long> left{-1};  // allocations that still succeed (-1: all)
void *operator new(size_t n) {
    for (long v = left.load(); v >= 0;) {
        if (v == 0) throw std::bad_alloc();
        if (left.compare_exchange_weak(v, v - 1)) break;
    }
    if (void *p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

using namespace cospdnn;
int main() {
    // from none to enough allocations for threads and work
    for (long allowed = 0; allowed < 200; ++allowed) {
        std::atomic<int> next{0}, done{0};
        FirstError err;
        left = allowed;
        on_threads(8, 3, err, [&] {
            while (err.code.load() == 0 && next++ < 32) {
                std::vector<std::string> v;
                v.emplace_back(100, 'x');
                ++done;
            }
        });
        left = -1;
        if (err.code.load() == 0 ? done.load() != 32 : err.code.load() != 3 || std::strcmp(err.message, "build: out of host memory"))
            return 1;
        if (allowed == 0 && err.code.load() != 3) return 2;
        if (allowed == 199 && err.code.load() != 0) return 3;
    }
    FirstError other;
    on_threads(4, 3, other, [&] { throw 7; });
    if (other.code.load() != 3) return 4;
    FirstError first;
    first.set(5, "five");
    first.set(6, "six");
    return first.code.load() == 5 && !std::strcmp(first.message, "five") ? 0 : 5;
}
"""


def test_failures_are_codes(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-pthread", "-I", os.path.join(ROOT, "cospdnn_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    for _ in range(5):
        assert subprocess.run([str(exe)], timeout=60).returncode == 0
