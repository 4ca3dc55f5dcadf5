"""The tuner's choice from measured times, without a GPU: a small program linked
against the library makes it for tables of times."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dcu-winograd-conv2d_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "wg_plan.h"
// stdin: fallback, direct us (-1: none), direct GFLOP, candidates, then "algo bn us" each
int main() {
    int fallback, n;
    double direct_us, gflop;
    while (std::scanf("%d %lf %lf %d", &fallback, &direct_us, &gflop, &n) == 4) {
        std::vector<wg::TunedTime> t(n);
        for (auto& x : t) {
            double us;
            if (std::scanf("%d %d %lf", &x.algo, &x.bn, &us) != 3) return 2;
            x.ms = static_cast<float>(us * 1e-3);
        }
        wg::TunedTime best;
        bool direct;
        wg::pick_tuned(t.data(), n, fallback, static_cast<float>(direct_us * 1e-3), gflop * 1e9, &best, &direct);
        std::printf("%d %d %d\n", best.algo, best.bn, direct ? 1 : 0);
    }
}
"""

F4, F2, FUSED, ROW = 0, 1, 2, 4


@pytest.fixture(scope="module")
def pick(wg, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    d = tmp_path_factory.mktemp("tuner")
    src, exe = d / "pick.cpp", d / "pick"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda, str(src), "-o", str(exe), wg.LIB_PATH,
                    "-Wl,-rpath," + os.path.dirname(wg.LIB_PATH)], check=True, capture_output=True, text=True)

    def run(fallback, direct, times, gflop=0.0):
        text = f"{fallback} {direct} {gflop} {len(times)}\n" + "".join("%d %d %f\n" % t for t in times)
        r = subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True)
        algo, bn, d = (int(v) for v in r.stdout.split())
        return algo, bn, bool(d)

    return run


@pytest.mark.parametrize("f4,direct,runs", [(14.2, 15.5, True), (14.2, 16.0, True), (14.2, 16.1, False), (40.0, 43.8, True),
                                            (40.0, 44.0, False)])
def test_direct_in_a_near_tie(pick, f4, direct, runs):
    assert pick(F4, direct, [(F4, 256, f4), (F2, 256, 1.5 * f4), (ROW, 0, 3 * f4)])[2] == runs


@pytest.mark.parametrize("f2,f4,algo", [(12.1, 12.1, F2), (12.8, 12.1, F2), (12.1, 12.8, F2), (13.7, 12.1, F2), (13.9, 12.1, F4)])
def test_more_accurate_of_two_alike(pick, f2, f4, algo):
    # whichever of the two the reference rule names
    for fallback in (F4, F2):
        got = pick(fallback, -1, [(F4, 128, f4), (F2, 256, f2)])
        if fallback == F4 or algo == F2:
            assert got == (algo, 256 if algo == F2 else 128, False)


def test_clear_winners(pick):
    assert pick(F2, 100.0, [(FUSED, 0, 300.0), (ROW, 0, 90.0), (F2, 128, 70.0), (F2, 256, 65.0), (F4, 256, 40.0), (F4, 128, 45.0)]) == (F4, 256, False)
    assert pick(F4, 30.0, [(F2, 128, 70.0), (F4, 256, 40.0)]) == (F4, 256, True)
    # by its products at the rate of the power cap the direct kernel is slower (80 us)
    assert pick(F4, 70.5, [(F4, 256, 65.5), (F2, 256, 93.0)], gflop=118.5) == (F4, 256, False)
    # the reference rule's pick unless another is more than 3% faster
    assert pick(FUSED, -1, [(FUSED, 0, 102.0), (F2, 128, 100.0)]) == (FUSED, 0, False)
    assert pick(FUSED, -1, [(FUSED, 0, 104.0), (F2, 128, 100.0)]) == (F2, 128, False)
    assert pick(ROW, -1, [(ROW, 0, 100.0), (F4, 256, 94.0)]) == (ROW, 0, False)
    # nothing could be planned
    assert pick(F4, -1, []) == (F4, 0, False)
