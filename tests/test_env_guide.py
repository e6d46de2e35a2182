"""The bucket guide of an environment's sampling CDFs (cdfFind, pe_light.h) finds the entry that the
search of the whole CDF finds, for every number in [0, 1) and for those outside it: bucket ends,
CDF values and their neighbours, runs of equal values, rows without light, odd sizes."""
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "pe_light.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
using namespace pe;

int main(int, char** argv) {
    const int n = std::atoi(argv[1]), kind = std::atoi(argv[2]);
    std::mt19937 rng(static_cast<unsigned>(n * 7 + kind));
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    std::vector<float> cdf(static_cast<size_t>(n) + 1, 0.0f);
    for (int i = 0; i < n; ++i) {
        float f = U(rng);
        if (kind == 1) f = U(rng) < 0.8f ? 0.0f : f;       // runs of equal values
        if (kind == 2) f = i == n / 2 ? 1.0f : 0.0f;       // one lit texel
        if (kind == 3) f = 0.0f;                           // a row without light
        if (kind == 4) f = std::exp(12.0f * U(rng));       // a bright sky
        cdf[static_cast<size_t>(i) + 1] = cdf[static_cast<size_t>(i)] + f;
    }
    const float total = cdf[static_cast<size_t>(n)];
    for (float& c : cdf) c = total > 0.0f ? c / total : 0.0f;
    int buckets = 1;
    while (2 * buckets <= n && buckets < 2048) buckets *= 2;
    std::vector<uint16_t> guide;
    for (int k = 0; k <= buckets; ++k)
        guide.push_back(static_cast<uint16_t>(cdfUpper(cdf.data(), 0, n + 1, static_cast<float>(k) / static_cast<float>(buckets))));
    std::vector<float> us = {0.0f, 0.99999994f, 1.0f, 1.5f, -0.25f, NAN};
    auto around = [&](float u) {
        for (float v : {u, std::nextafterf(u, -1.0f), std::nextafterf(u, 2.0f)}) us.push_back(v);
    };
    for (int k = 0; k <= buckets; ++k) around(static_cast<float>(k) / static_cast<float>(buckets));
    for (float c : cdf) around(c);
    for (int i = 0; i < 20000; ++i) us.push_back(U(rng));
    for (float u : us)
        if (cdfFind(cdf.data(), n, u, guide.data(), buckets) != cdfFind(cdf.data(), n, u, nullptr, 0)) {
            std::printf("n %d kind %d u %.9g\n", n, kind, u);
            return 1;
        }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("env_guide")
    (d / "t.cpp").write_text(PROGRAM)
    csrc = ROOT / "photon-engine_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{csrc}", f"-I{ROOT / 'include'}", "-o", str(d / "t"),
                    str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("n", [1, 2, 3, 31, 64, 65, 1023, 2048, 4097, 60001])
def test_guided_search_equals_the_whole_search(program, n):
    for kind in range(5):
        r = subprocess.run([program, str(n), str(kind)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
