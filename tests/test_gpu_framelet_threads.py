"""Framelet analyses of volumes that want different shared memory, from two threads of
a C++ host (Python's lock would keep their calls apart)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HOST = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <cuda_runtime.h>
#include "framelab_gb300.h"
// analyses of one volume for two seconds; 0, or the first status that is not
static void work(int nx, int ny, int nz, int *status)
{
    fl_framelet *w = nullptr;
    cudaStream_t s;
    float *u, *c;
    *status = fl_framelet_create(nx, ny, nz, 1, FL_FRAMELET_LINEAR, &w);
    if (*status) return;
    const size_t n = (size_t)nx * ny * nz * sizeof(float);
    if (cudaStreamCreate(&s) || cudaMalloc(&u, n) || cudaMalloc(&c, fl_framelet_ncoef(w) * sizeof(float)) ||
        cudaMemsetAsync(u, 0, n, s)) { *status = -1000; return; }
    const auto end = std::chrono::steady_clock::now() + std::chrono::seconds(2);
    for (int k = 0; !*status && std::chrono::steady_clock::now() < end; k++) {
        *status = fl_framelet_analysis(w, u, c, s);
        if (n > 1 << 20 || k % 64 == 0) cudaStreamSynchronize(s);     // neither queue fills
    }
    cudaStreamSynchronize(s);
    cudaFree(u); cudaFree(c);
    fl_framelet_destroy(w);
}
int main()
{
    int a = 0, b = 0;                        // coefficients above and below 400 MB
    std::thread ta(work, 161, 160, 160, &a), tb(work, 34, 10, 12, &b);
    ta.join(); tb.join();
    std::printf("%d %d\n", a, b);
    return a || b;
}
"""


def test_two_threads_of_unlike_rows(tmp_path):
    """Rows off the memory sector hold shared memory by their volume's size, under a
    limit that is the kernel's and not the call's: no launch may fail over another
    thread's."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = os.path.join(root, "framelab_gb300")
    src, exe = tmp_path / "host.cpp", tmp_path / "host"
    src.write_text(HOST)
    subprocess.run([nvcc, "-std=c++17", "-O1", str(src), "-I" + os.path.join(root, "include"), "-L" + lib,
                    "-l:libframelab_gb300.so", "-Xlinker", "-rpath=" + lib, "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
