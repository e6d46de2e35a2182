"""Which paths of a wave train the learned proposal (trainOrder, pe_wave.h): counted sample by sample and
row by row, one in guideStride, whatever order the paths themselves are in.  Host arithmetic, no GPU."""
import importlib
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "pe_wave.h"
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace pe;

int main(int, char** argv) {
    WaveSeg A{};
    A.width = 3000;
    A.height = 2000;
    A.tileX = 17;
    A.tileY = 5;
    A.tileW = std::atoi(argv[1]);
    A.tileH = std::atoi(argv[2]);
    A.nSamples = std::atoi(argv[3]);
    A.slotFirst = std::atoi(argv[4]);
    const int kind = std::atoi(argv[5]); // 0 the whole rectangle, 1 its last two thirds, 2 a pixel list
    const int all = A.tileW * A.tileH;
    A.nPix = all;
    std::vector<int32_t> list;
    if (kind == 1) {
        A.pixelFirst = all / 3;
        A.nPix = all - A.pixelFirst;
    } else if (kind == 2) {
        for (int i = 0; i < all; ++i) list.push_back((i * 7919) % (A.width * A.height));
        A.pixList = list.data();
    }
    std::vector<char> seen(static_cast<size_t>(A.nPix) * A.nSamples, 0);
    for (int p = 0; p < A.nPix; ++p)
        for (int s = 0; s < A.nSamples; ++s) {
            const int path = pathOfSample(A, p, s);
            int x, y;
            tilePixel(A, A.pixelFirst + p, x, y);
            const int r = kind == 0 ? (y - A.tileY) * A.tileW + x - A.tileX : p;
            const int order = trainOrder(A, path);
            if (order != A.slotFirst + s * A.nPix + r || pathOfTrainOrder(A, order) != path || seen[order - A.slotFirst]++) {
                std::printf("pixel %d sample %d: path %d order %d back %d\n", p, s, path, order, pathOfTrainOrder(A, order));
                return 1;
            }
        }
    // the paths of a stride: every sample, and of the whole rectangle every row (a stride no wider than a row)
    for (int stride = 1; stride <= 16; stride *= 2) {
        std::vector<char> samples(static_cast<size_t>(A.nSamples), 0), rows(static_cast<size_t>(A.tileH), 0);
        for (int o = 0; o < A.nPix * A.nSamples; ++o) {
            if ((A.slotFirst + o) % stride != 0) continue;
            const int path = pathOfTrainOrder(A, A.slotFirst + o);
            samples[static_cast<size_t>(sampleOfPath(A, path))] = 1;
            int x, y;
            tilePixel(A, A.pixelFirst + (path - A.slotFirst) / A.nSamples, x, y);
            if (kind == 0) rows[static_cast<size_t>(y - A.tileY)] = 1;
        }
        for (char c : samples)
            if (!c && A.nPix >= stride) return 2;
        for (char c : rows)
            if (kind == 0 && !c && A.tileW >= stride) return 3;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("train_order")
    (d / "t.cpp").write_text(PROGRAM)
    csrc = ROOT / "photon-engine_b200" / "csrc"
    nvcc = pathlib.Path(importlib.import_module("photon_engine_b200.build")._nvcc())
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{csrc}", f"-I{nvcc.resolve().parent.parent / 'include'}", "-o", str(d / "t"),
                    str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("w,h,spp,first", [(320, 180, 16, 0), (64, 36, 4, 0), (33, 7, 5, 0), (16, 1, 16, 0), (1, 1, 1, 0), (97, 41, 3, 1000)])
def test_one_path_in_a_stride_trains(program, w, h, spp, first):
    for kind in range(3):
        if kind == 1 and w * h < 3:
            continue
        r = subprocess.run([program, str(w), str(h), str(spp), str(first), str(kind)], capture_output=True, text=True)
        assert r.returncode == 0, (kind, r.returncode, r.stdout + r.stderr)
