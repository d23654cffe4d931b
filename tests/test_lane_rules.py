"""The lanes a world's pair passes take, and the slots their threads work on, from the counts alone
(csrc/lane_rules.cuh is plain C++; built here with the host compiler)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "physics-engine_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include "lane_rules.cuh"
using namespace pe;
template <int G>
int slots(uint64_t n, uint32_t threads) {  // the first and the last blocks of a launch over n slots
    const uint64_t blocks = (n * G + threads - 1) / threads;
    for (uint64_t b = 0; b < blocks; b += (b == 2 && blocks > 6) ? blocks - 5 : 1)
        for (uint32_t t = 0; t < threads; ++t)
            if (lane_slot<G>((uint32_t)b, threads, t) != (b * threads + t) / G) return 1;
    return 0;
}
int main(int argc, char** argv) {
    if (!std::strcmp(argv[1], "slots")) {
        int bad = 0;
        for (uint64_t n : {1ull, 1000ull, 134217727ull, 134217729ull, 268435457ull, 536870911ull})
            for (uint32_t threads : {64u, 128u, 256u})
                bad += slots<1>(n, threads) + slots<4>(n, threads) + slots<8>(n, threads) + slots<16>(n, threads) +
                       slots<32>(n, threads);
        return bad;
    }
    const uint64_t fluid = std::strtoull(argv[2], nullptr, 10), slots = std::strtoull(argv[3], nullptr, 10);
    const PassLanes a = pass_lanes(std::atoi(argv[1]), fluid, slots), b = pass_lanes_f32(std::atoi(argv[1]), fluid, slots);
    std::printf("%u %u %u %u %u %u %u %u %u %u\n", a.density, a.forces, a.xsph, a.boundary, b.density, b.forces, b.xsph,
                pbf_lanes(fluid, slots), dfsph_lanes(fluid, slots), dfsph_boundary_lanes(fluid, slots));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


def _lanes(program, dim, fluid, boundary):
    out = subprocess.run([program, str(dim), str(fluid), str(fluid + boundary)], check=True, capture_output=True, text=True)
    names = ("density", "forces", "xsph", "boundary", "density32", "forces32", "xsph32", "pbf", "dfsph", "dfsph_boundary")
    return dict(zip(names, map(int, out.stdout.split())))


def test_every_thread_has_its_slot(program):
    """Up to the largest world (2^29 - 1 slots), where the thread's number in the launch passes 2^32."""
    assert subprocess.run([program, "slots"]).returncode == 0


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("fluid,boundary", [(10_000_000, 0), (1_000_000, 4008), (4_096_000, 46_082), (500_000_000, 1000)])
def test_a_world_of_fluid_gives_its_boundary_pass_one_lane(program, dim, fluid, boundary):
    got = _lanes(program, dim, fluid, boundary)
    assert got["boundary"] == 1
    assert set(got.values()) <= {1, 8}
    if boundary == 0:
        assert got["dfsph_boundary"] == 1


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("fluid", [1, 256, 2197, 15_625, 60_000])
@pytest.mark.parametrize("boundary", [0, 700, 100_000, 540_002, 5_000_000, 500_000_000])
def test_the_threads_of_idle_slots_stay_bounded(program, dim, fluid, boundary):
    """Beyond 13 million threads a pass takes one lane a slot."""
    for k, lanes in _lanes(program, dim, fluid, boundary).items():
        assert lanes in (1, 4, 8, 16, 32)
        assert lanes == 1 or lanes * (fluid + boundary) <= 13_000_000, k


def test_the_measured_worlds_take_their_fastest_lanes(program):
    tiny, mid, large = (_lanes(program, 3, f, b) for f, b in ((256, 674), (32_768, 24_802), (1_000_000, 396_802)))
    assert [tiny[k] for k in ("density", "forces", "xsph", "boundary", "dfsph")] == [32] * 5
    assert [mid[k] for k in ("density", "forces", "xsph", "boundary", "pbf", "dfsph")] == [8, 8, 8, 16, 8, 8]
    assert set(large.values()) - {large["dfsph_boundary"]} == {1}
    few = _lanes(program, 3, 2197, 540_002)
    assert [few[k] for k in ("density", "forces", "xsph", "boundary", "density32", "pbf", "dfsph")] == [8, 8, 8, 4, 8, 1, 8]
