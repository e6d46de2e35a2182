"""The path state carved out of the fixed scratch of pe_device_render_tile_noalloc (carveWave, pe_wave.h):
every column that the trace, binning and shading kernels take for granted is there, inside the
scratch, aligned, and apart from the others.  Host arithmetic only: no GPU."""
import importlib
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "pe_wave.h"
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace pe;

struct Range {
    const char* name;
    size_t at, bytes;
};

int main(int, char** argv) {
    const size_t slots = static_cast<size_t>(std::atoll(argv[1]));
    unsigned char* const base = reinterpret_cast<unsigned char*>(size_t(1) << 20); // arithmetic only, never read
    const Paths P = carveWave(base, slots);
    std::vector<Range> r;
#define COLUMN(c, n) r.push_back({#c, reinterpret_cast<size_t>(P.c), (n) * sizeof(*P.c)})
    COLUMN(rayO, slots); COLUMN(rayD, slots); COLUMN(thr, slots); COLUMN(L, slots); COLUMN(lastN, slots); COLUMN(lastP, slots);
    COLUMN(pickP, slots); COLUMN(pickN, slots); COLUMN(hit, slots); COLUMN(med, slots); COLUMN(key, slots);
    COLUMN(queueA, slots); COLUMN(queueB, slots); COLUMN(sortQ, slots * kShadeKeys);
    COLUMN(shadowQ, slots); COLUMN(shO, slots); COLUMN(shD, slots); COLUMN(shC, slots); COLUMN(shT, slots);
    COLUMN(blocks, kCounters);
    std::sort(r.begin(), r.end(), [](const Range& a, const Range& b) { return a.at < b.at; });
    size_t end = reinterpret_cast<size_t>(base);
    for (const Range& c : r) {
        if (c.at < end || c.at % 256 != 0) {
            std::printf("%s at %zu, the scratch is taken to %zu\n", c.name, c.at, end);
            return 1;
        }
        end = c.at + c.bytes;
    }
    if (end > reinterpret_cast<size_t>(base) + waveBytes(slots) || P.capacity != slots) {
        std::printf("%zu bytes past the scratch, capacity %u\n", end - reinterpret_cast<size_t>(base) - waveBytes(slots), P.capacity);
        return 1;
    }
    if (P.now != P.blocks || P.next != P.blocks + kBounceBlock || P.counters != P.blocks + 2 * kBounceBlock) {
        std::printf("counters\n");
        return 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("wave_columns")
    (d / "t.cpp").write_text(PROGRAM)
    csrc = ROOT / "photon-engine_b200" / "csrc"
    nvcc = pathlib.Path(importlib.import_module("photon_engine_b200.build")._nvcc())
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{csrc}", f"-I{nvcc.resolve().parent.parent / 'include'}", "-o", str(d / "t"),
                    str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("slots", [256, 512, 1 << 15])
def test_carved_columns_are_whole_and_apart(program, slots):
    r = subprocess.run([program, str(slots)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
