"""run_threads (csrc/host_threads.hpp): every part runs exactly once and no exception, of a part or of starting a
thread, leaves while a thread runs (which would end the process)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multem_b200" / "csrc"

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>
#include "host_threads.hpp"
static std::atomic<int> left{-1};  // allocations until one fails (-1: none does)
void* operator new(size_t n) {
    if (left >= 0 && left-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
int main() {
    constexpr int N = 6;
    int refused = 0;
    for (int k = -1; k < 20; k++) {
        std::atomic<int> ran[N] = {};
        left = k;
        try {
            mtb::run_threads(N, [&](int i) { ran[i]++; });
            left = -1;
            for (auto& r : ran)
                if (r != 1) return 1;
        } catch (const std::bad_alloc&) {  // before the first part
            left = -1;
            refused++;
            for (auto& r : ran)
                if (r != 0) return 2;
        }
    }
    if (refused == 0) return 3;
    std::atomic<int> ran{0};
    try {
        mtb::run_threads(N, [&](int i) {
            ran++;
            if (i == 1 || i == 4) throw std::runtime_error(i == 1 ? "one" : "four");
        });
        return 4;
    } catch (const std::runtime_error& e) {
        if (ran != N || std::string(e.what()) != "one") return 5;
    }
    mtb::run_threads(0, [](int) { std::abort(); });
    return 0;
}
"""


def test_parts_run_once_whatever_fails(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text("#include <string>\n" + PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", "-o", tmp_path / "t", tmp_path / "t.cpp"], check=True)
    assert subprocess.run([tmp_path / "t"], timeout=60).returncode == 0


def test_threads_are_started_nowhere_else():
    """A std::thread of its own would end the process where an exception passes it by."""
    for f in CSRC.glob("*.c*"):
        assert "std::thread>" not in f.read_text() and "std::thread " not in f.read_text(), f.name
