"""The cached shared-memory limit of a kernel under concurrent launches, without
a GPU: a small program stands in for the runtime and makes two threads raise
one kernel's limit, by unlike sizes, in the order that loses the larger one."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dcu-winograd-conv2d_gb300", "csrc")

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <cuda_runtime.h>
static std::atomic<int> limit{0}, sets{0};
static void pause_ms(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }
extern "C" cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
    limit = bytes;
    ++sets;
    // the larger size's thread is held up here until the smaller one's has been and gone
    if (bytes == 200000) {
        for (int i = 0; i < 30 && sets < 2; ++i) pause_ms(10);
        pause_ms(100);
    }
    return cudaSuccess;
}
// as the runtime's own header has it for nvcc
template <class T> cudaError_t cudaFuncSetAttribute(T* f, cudaFuncAttribute a, int v) {
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(f), a, v);
}
#include "wg_launch.h"
void kernel(int) {}
void other(int) {}
int main() {
    std::thread large([] { wg::allow_smem<kernel>(200000); });
    while (sets == 0) std::this_thread::yield();
    std::thread small([] { wg::allow_smem<kernel>(100000); });
    large.join();
    small.join();
    // a launch of any size up to those asked for finds its limit in force
    for (int bytes : {100000, 150000, 200000}) {
        wg::allow_smem<kernel>(bytes);
        if (limit < bytes) return std::printf("%d allowed, %d in force\n", bytes, limit.load()), 1;
    }
    // a larger one raises it, a smaller one leaves it; another kernel has its own
    wg::allow_smem<kernel>(220000);
    if (limit != 220000) return 2;
    const int n = sets;
    wg::allow_smem<kernel>(1000);
    if (sets != n) return 3;
    wg::allow_smem<other>(1000);
    return sets == n + 1 && limit == 1000 ? 0 : 4;
}
"""


def test_two_threads_raise_one_limit(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", cuda, str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout)
