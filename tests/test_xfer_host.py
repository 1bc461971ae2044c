"""CPU test of the staged field transfers' host side (pf3d_xfer.cu), built by the
host compiler against a stand-in for the CUDA runtime: the copies are memcpy,
events and streams belong to devices, and a call can be made to fail.  Every
transfer must deliver its bytes whatever the runtime refuses on the way."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "phase-field-project-3d_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstring>
#include <cstdlib>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2,
                   cudaErrorInvalidResourceHandle = 400 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
enum cudaStreamCaptureMode { cudaStreamCaptureModeGlobal, cudaStreamCaptureModeThreadLocal, cudaStreamCaptureModeRelaxed };
struct FakeStream { int device; };
struct FakeEvent { int device; };
typedef FakeStream* cudaStream_t;
typedef FakeEvent* cudaEvent_t;
struct cudaPointerAttributes { cudaMemoryType type; int device; };
constexpr unsigned cudaEventDisableTiming = 2, cudaHostAllocPortable = 1;
cudaError_t cudaSetDevice(int);
cudaError_t cudaGetDevice(int*);
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned);
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t);
cudaError_t cudaEventSynchronize(cudaEvent_t);
cudaError_t cudaEventDestroy(cudaEvent_t);
cudaError_t cudaStreamSynchronize(cudaStream_t);
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t);
cudaError_t cudaHostAlloc(void**, size_t, unsigned);
cudaError_t cudaFreeHost(void*);
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*);
cudaError_t cudaGetLastError();
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*);
"""

HARNESS = r"""
#include "pf3d_xfer.h"
#include <atomic>
#include <cstdio>
#include <vector>

static thread_local int t_dev = 0;
static thread_local cudaError_t t_err = cudaSuccess;
static thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;
static std::atomic<int> n_alloc{0}, live{0}, unsafe{0};
static int allocs_allowed = 1 << 30;
static const char *dev_lo, *dev_hi;
static const int kDevice = 1;                       // where the field and its stream live
static cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) t_err = e; return e; }

cudaError_t cudaSetDevice(int d) { t_dev = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = t_dev; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new FakeEvent{t_dev}; ++live; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    return ret(e->device == s->device ? cudaSuccess : cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --live; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t)
{
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    if (t_mode != cudaStreamCaptureModeRelaxed) ++unsafe;   // fails while another thread captures
    if (n_alloc >= allocs_allowed) return ret(cudaErrorMemoryAllocation);
    ++n_alloc;
    ++live;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); --live; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    const char* c = (const char*)p;
    if (c >= dev_lo && c < dev_hi) *a = {cudaMemoryTypeDevice, kDevice};
    else *a = {cudaMemoryTypeUnregistered, -2};
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { cudaError_t e = t_err; t_err = cudaSuccess; return e; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) { std::swap(*m, t_mode); return cudaSuccess; }

// argv: element size, nx, rows, allocations allowed, the caller's device
int main(int argc, char** argv)
{
    const int es = std::atoi(argv[1]), nx = std::atoi(argv[2]);
    const long long rows = std::atoll(argv[3]), px = (nx + 31) / 32 * 32;
    allocs_allowed = std::atoi(argv[4]);
    cudaSetDevice(std::atoi(argv[5]));
    FakeStream st{kDevice};
    std::vector<char> dev((size_t)px * rows * es, 77);
    std::vector<double> a((size_t)nx * rows), b(a.size(), -1.0);
    dev_lo = dev.data();
    dev_hi = dev_lo + dev.size();
    for (size_t i = 0; i < a.size(); ++i) a[i] = (double)(i * 2654435761u % 1000003) / 997.0 - 300.0;
    pf3d::xfer_ref();
    const cudaError_t up = pf3d::xfer_to_device(dev.data(), es, nx, px, rows, a.data(), &st);
    const cudaError_t down = pf3d::xfer_to_host(dev.data(), es, nx, px, rows, b.data(), &st);
    int cur = -1;
    cudaGetDevice(&cur);
    size_t bad = 0;
    for (size_t i = 0; i < a.size(); ++i) bad += b[i] != (es == 8 ? a[i] : (double)(float)a[i]);
    const int left = (int)cudaGetLastError();
    pf3d::xfer_unref();
    std::printf("up %d down %d bad %zu error left %d device %d live %d allocations %d unsafe %d\n", (int)up, (int)down,
                bad, left, cur, (int)live, (int)n_alloc, (int)unsafe);
    return 0;
}
"""


@pytest.fixture(scope="session")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("xfer")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text("#include <utility>\n" + HARNESS)
    exe = str(d / "xfer")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(d), "-I", CSRC, str(d / "main.cpp"), "-x", "c++",
                    os.path.join(CSRC, "pf3d_xfer.cu"), "-o", exe], check=True)

    def run(*args):
        return subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True, timeout=60).stdout

    return run


def result(out):
    w = out.split()
    return dict(up=int(w[1]), down=int(w[3]), bad=int(w[5]), left=int(w[8]), device=int(w[10]), live=int(w[12]),
                allocations=int(w[14]), unsafe=int(w[16]))


SIZES = [(4, 1), (33, 7000), (200, 9000), (131, 20011), (140000, 9)]


@pytest.mark.parametrize("es", [8, 4])
@pytest.mark.parametrize("nx,rows", SIZES)
@pytest.mark.parametrize("allowed", [0, 1, 100])
def test_delivers_without_pinned_chunks(harness, es, nx, rows, allowed):
    """The staging chunks cannot be allocated, or only some of them: the copy is
    made all the same, and no error is left behind."""
    r = result(harness(es, nx, rows, allowed, 1))
    assert (r["up"], r["down"], r["bad"], r["left"], r["live"]) == (0, 0, 0, 0, 0), r


@pytest.mark.parametrize("es", [8, 4])
@pytest.mark.parametrize("nx,rows", SIZES)
def test_field_of_another_device(harness, es, nx, rows):
    """The calling thread's current device is not the field's (a thread that
    only reads fields back): the transfer runs on the field's device, and the
    thread keeps its own."""
    r = result(harness(es, nx, rows, 100, 0))
    assert (r["up"], r["down"], r["bad"], r["left"], r["live"], r["device"]) == (0, 0, 0, 0, 0, 0), r


def test_allocates_beside_a_capture(harness):
    """Another thread may be capturing a graph, during which an allocation in the
    default capture mode fails (and can end the capture): the chunks are
    allocated in the relaxed mode."""
    r = result(harness(8, 200, 9000, 100, 1))
    assert r["allocations"] > 0 and r["unsafe"] == 0, r
