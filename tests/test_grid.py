"""The persistent kernels' grids: each instantiation of a kernel template has
its own occupancy, whichever was asked first, also from several threads.  The
header is compiled for the host with stand-ins for the two functions that it
calls."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wavefrontpathtracing_gb300", "csrc")
INCLUDE = next((p for p in ("/usr/local/cuda/include",) if os.path.exists(os.path.join(p, "cuda_runtime.h"))), None)

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "wf_grid.h"

template <int LAY> void kernel(int*) {}   // one type, several kernels
static std::atomic<int> asked{0};

extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* k, int block, size_t) {
    asked++;
    *n = k == (const void*)kernel<0> ? 9 : k == (const void*)kernel<1> ? 8 : k == (const void*)kernel<2> ? block / 32 : 0;
    return cudaSuccess;
}
namespace wf { int sm_count() { return 10; } }

int main() {
    std::vector<std::thread> t;
    for (int i = 0; i < 8; ++i) t.emplace_back([] { wf::persistent_grid<kernel<1>, 128>(); });
    for (auto& x : t) x.join();
    std::printf("%u %u %u %u %u ", wf::persistent_grid<kernel<1>, 128>(), wf::persistent_grid<kernel<0>, 128>(),
                wf::persistent_grid<kernel<2>, 128>(), wf::persistent_grid<kernel<2>, 256>(),
                wf::persistent_grid<kernel<3>, 128>());
    std::printf("%d\n", asked.load());
}
"""


@pytest.mark.skipif(INCLUDE is None or shutil.which("g++") is None, reason="needs g++ and the CUDA headers")
def test_each_kernel_has_its_own_grid(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", INCLUDE, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    # kernels <1>, <0>, <2> by block size, and one whose query says nothing; one query per kernel and block
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == \
        ["80", "90", "40", "80", "10", "5"]
