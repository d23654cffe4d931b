"""The threads a large copy is shared out over (csrc/parts.cuh, plain C++, built with the host compiler): every
part is done once, also where no memory or no thread is to be had for some of them."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "physics-engine_b200", "csrc")

MAIN = r"""
#include <atomic>
#include <cstdlib>
#include <new>
#include "parts.cuh"
static std::atomic<int> left{1 << 30};  // allocations that still succeed
void* operator new(std::size_t n) {
    if (left.fetch_sub(1) <= 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main(int argc, char** argv) {
    const int parts = std::atoi(argv[1]);
    std::atomic<int> done[8] = {};
    auto run = [&](int t) noexcept { done[t] += 1; };
    left = std::atoi(argv[2]);
    pe::run_parts<8>(parts, run);
    left = 1 << 30;
    for (int t = 0; t < 8; ++t)
        if (done[t] != (t < parts ? 1 : 0)) return 1;
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("parts")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("parts", [1, 2, 5, 8])
@pytest.mark.parametrize("allocations", [0, 1, 3, 1000])
def test_every_part_is_done_once(program, parts, allocations):
    assert subprocess.run([program, str(parts), str(allocations)]).returncode == 0
