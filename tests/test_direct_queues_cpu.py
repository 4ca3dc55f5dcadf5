"""Host logic of the direct kernel's queues of many problems, without a GPU: a
small program linked against the library plans sets of problems (sizes only)
and prints the queues, which are checked here."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dcu-winograd-conv2d_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "wg_kernels.h"
using namespace wg;
// stdin: sets of problems, "count" then "n c h w k" each; stdout: a JSON list per set
int main() {
    int count;
    while (std::scanf("%d", &count) == 1) {
        std::vector<DirectProblem> p;
        for (int i = 0; i < count; ++i) {
            int n, c, h, w, k;
            if (std::scanf("%d %d %d %d %d", &n, &c, &h, &w, &k) != 5) return 2;
            const Geom g = make_geom(n, c, h, w, k, 1, 1, 2);
            if (!direct_supported(g, false)) return 3;
            p.push_back({g, reinterpret_cast<const void*>(256), reinterpret_cast<void*>(256 + i), nullptr});
        }
        std::vector<DirectDesc> d(p.size());
        std::vector<DirectQueue> q;
        const cudaError_t e = make_direct_queues(p.data(), count, 76, d.data(), q);
        std::printf("{\"status\": %d, \"queues\": [", static_cast<int>(e));
        for (size_t i = 0; i < q.size(); ++i) {
            std::printf("%s{\"first\": %d, \"items\": %d, \"na\": %d, \"nb\": %d, \"a\": %d, \"b\": %d, \"smem\": %d, \"problems\": [",
                        i ? ", " : "", q[i].first, q[i].items, q[i].ring.na, q[i].ring.nb, q[i].ring.a_bytes,
                        q[i].ring.b_bytes, q[i].ring.smem_bytes);
            for (int j = 0; j < q[i].n; ++j) {
                const DirectDesc& x = d[q[i].first + j];
                std::printf("%s{\"i\": %d, \"begin\": %d, \"items\": %d, \"win\": %d, \"gran\": %d, \"bn\": %d, \"mb\": %d}",
                            j ? ", " : "", static_cast<int>(reinterpret_cast<size_t>(x.y)) - 256, x.item_begin, x.items, x.win,
                            x.gran, x.bn, x.mb);
            }
            std::printf("]}");
        }
        std::printf("]}\n");
    }
}
"""


@pytest.fixture(scope="module")
def planner(wg, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    d = tmp_path_factory.mktemp("queues")
    src, exe = d / "queues.cpp", d / "queues"
    src.write_text(PROGRAM)
    libdir = os.path.dirname(wg.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda, str(src), "-o", str(exe), wg.LIB_PATH,
                    "-Wl,-rpath," + libdir], check=True, capture_output=True, text=True)

    def plan(sets):
        text = "".join("%d\n" % len(s) + "".join("%d %d %d %d %d\n" % p for p in s) for s in sets)
        r = subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True)
        return [json.loads(line) for line in r.stdout.splitlines()]

    return plan


def own_stages(a, b):
    """Window and filter stages of a ring for these sizes: as many of the
    filter as of both, the rest to the windows, three of those and two at least."""
    room = 227 * 1024 - 1536
    for nb in range(min(12, room // (a + b)), 1, -1):
        na = min(12, (room - nb * b) // a)
        if na >= 3:
            return na, nb
    raise AssertionError((a, b))


def check(shapes, got):
    assert got["status"] == 0, shapes
    seen, first = [], 0
    for q in got["queues"]:
        assert q["first"] == first
        first += len(q["problems"])
        # the rings: fewest stages, all of shared memory at most (barriers and alignment 1,536 bytes)
        assert q["na"] >= 3 and q["nb"] >= 2 and q["smem"] <= 227 * 1024
        assert q["na"] * q["a"] + q["nb"] * q["b"] + 1536 <= q["smem"]
        if len(q["problems"]) > 1:
            # as deep as a problem alone would have it, or three of each
            for p in q["problems"]:
                own = own_stages((2 * p["gran"] + 127) // 128 * 128 + 32, 9 * 16 * p["bn"])
                assert q["na"] >= min(3, own[0]) and q["nb"] >= min(3, own[1])
        begin = 0
        for p in q["problems"]:
            n, c, h, w, k = shapes[p["i"]]
            assert p["begin"] == begin
            positions = (n - 1) * (h + 1) * (w + 1) + (h - 1) * (w + 1) + w
            assert p["items"] == -(-positions // (256 * p["mb"])) * -(-k // p["bn"])
            begin += p["items"]
            assert p["win"] == 128 * p["mb"] + 2 * (w + 1) + 2
            assert 16 * p["win"] <= p["gran"] and 2 * p["gran"] <= q["a"] and 9 * 16 * p["bn"] <= q["b"]
            assert p["bn"] * p["mb"] <= 256
            seen.append(p["i"])
        assert q["items"] == begin
    assert sorted(seen) == list(range(len(shapes)))


def test_wide_rows_beside_many_channels(planner):
    """Every width that the kernel takes beside every filter tile, both ways
    round, and several of each: all are planned, the narrow ones together."""
    sets = []
    for w in (222, 300, 500, 640, 750, 751, 847, 943, 1000, 1079, 1080):
        for k in (8, 64, 96, 128, 192, 256, 512):
            wide, many = (1, 64, 200, w, 64), (8, 256, 14, 14, k)
            sets += [[wide, many], [many, wide], [many, (3, 8, 9, w, 300), (32, 256, 28, 28, k), wide, (1, 3, 1, 1, 1)]]
    for shapes, got in zip(sets, planner(sets)):
        check(shapes, got)
        narrow = {i for i, s in enumerate(shapes) if s[3] <= 220}
        assert narrow == set(p["i"] for p in got["queues"][0]["problems"]) & narrow
    split = [[(1, 64, 800, 800, 64), (8, 256, 14, 14, 256)]]
    got = planner(split)[0]
    assert [[p["i"] for p in q["problems"]] for q in got["queues"]] == [[1], [0]]


def test_ordinary_sets_share_one_queue(planner):
    sets = [[(2, 16, 7, 7, 40), (20, 32, 40, 40, 256), (3, 17, 13, 9, 33), (1, 20, 5, 300, 8)],
            [(16, 512, 56, 56, 512), (1, 64, 112, 112, 256), (128, 64, 14, 14, 64)], [(1, 80, 4, 1080, 40)]]
    for shapes, got in zip(sets, planner(sets)):
        check(shapes, got)
        assert len(got["queues"]) == 1
        one = got["queues"][0]["problems"]
        assert len(one) == len(shapes)
