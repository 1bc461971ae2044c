"""CPU test of the once-per-device set-up of the kernels' launchers, against a
stand-in for the CUDA runtime: a second device in the process is set up too, a
failed set-up is tried again, and devices beyond the mask are set up each time."""
import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "phase-field-project-3d_b200", "csrc")

MAIN = r"""
#include "pf3d_once.h"
#include <cstdio>
static int dev = 0;
cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
int main()
{
    static pf3d::DeviceOnce once;
    int calls = 0;
    cudaError_t next = cudaSuccess;
    auto on = [&](int d) { dev = d; return (int)once([&] { ++calls; return next; }); };
    next = cudaErrorInvalidValue;
    int e = on(0);
    next = cudaSuccess;
    e = e * 10 + on(0) + on(0) + on(1) + on(0) + on(1) + on(63) + on(63);
    std::printf("%d %d", e, calls);
    on(64); on(64);
    std::printf(" %d\n", calls);
}
"""


def test_once_per_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(
        "#pragma once\nenum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };\ncudaError_t cudaGetDevice(int*);\n")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "once")
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["10", "4", "6"]
