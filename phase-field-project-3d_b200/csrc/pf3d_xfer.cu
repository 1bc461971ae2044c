// pf3d_xfer.cu -- transfers between device fields and pageable host arrays.
//
// A copy engine reaches pinned memory only, so a plain copy to a pageable
// array goes through the driver's staging on one host thread, page faults of
// a fresh array included (measured: 4.6 GB/s for a 64 MB field; FP32 fields
// were converted on one thread besides, 2 GB/s of doubles).  Here a few host
// threads each own a pinned chunk and take the field's chunks in turn: the
// copy of one thread's chunk runs while the others move (and convert) theirs.
// FP32 fields cross the link as floats.  Measured,
// into fresh arrays: 200^3 FP64 13.2 -> 3.8 ms, 256^3 FP32 53.7 -> 10.0 ms,
// 340x340x200 FP64 43 -> 12 ms, twelve FP32 fields of 33 .. 128 cells across
// 44 -> 17 ms.
//
// The chunks belong to the process, one transfer at a time uses them (a
// caller first waits for its own stream, so it never holds them while it
// waits for kernels), and the last object frees them.
#include "pf3d_xfer.h"
#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace pf3d {
namespace {

constexpr int kXferThreads = 6;
constexpr size_t kChunk = 1u << 20;   // allocating pinned memory costs about 1 ms a MB, once
// doubles (bytes) below which the threads cost more than they save: a 2.8 MB
// FP64 field takes 0.18 ms through the driver and 0.67 ms through the chunks
constexpr size_t kSmall64 = 8u << 20, kSmall32 = 4u << 20;

std::mutex g_mu;      // the staging buffers and their use
int g_refs = 0;       // under g_mu
void* g_buf[kXferThreads] = {};

void free_buffers()
{
    for (void*& b : g_buf) {
        if (b) cudaFreeHost(b);
        b = nullptr;
    }
}

struct Job {
    char* dev;
    int es, nx;
    long long px, n_rows, rows_per;
    double* host;
    bool to_host;
    cudaStream_t stream;
    int device;
};

cudaError_t run_thread(const Job& j, int t, int nt)
{
    cudaError_t e = cudaSetDevice(j.device);
    cudaEvent_t ev = nullptr;
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    const size_t row = (size_t)j.nx * j.es;
    for (long long r0 = (long long)t * j.rows_per; e == cudaSuccess && r0 < j.n_rows; r0 += (long long)nt * j.rows_per) {
        const long long nr = std::min(j.rows_per, j.n_rows - r0);
        const size_t n = (size_t)nr * j.nx;
        char* dev = j.dev + (size_t)r0 * j.px * j.es;
        double* host = j.host + (size_t)r0 * j.nx;
        float* f = (float*)g_buf[t];
        if (j.to_host) {
            e = cudaMemcpy2DAsync(g_buf[t], row, dev, (size_t)j.px * j.es, row, (size_t)nr, cudaMemcpyDeviceToHost,
                                  j.stream);
        } else {
            if (j.es == 8) std::memcpy(g_buf[t], host, n * 8);
            else for (size_t q = 0; q < n; ++q) f[q] = (float)host[q];
            e = cudaMemcpy2DAsync(dev, (size_t)j.px * j.es, g_buf[t], row, row, (size_t)nr, cudaMemcpyHostToDevice,
                                  j.stream);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ev, j.stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev);
        if (e == cudaSuccess && j.to_host) {
            if (j.es == 8) std::memcpy(host, g_buf[t], n * 8);
            else for (size_t q = 0; q < n; ++q) host[q] = (double)f[q];
        }
    }
    if (ev) cudaEventDestroy(ev);
    return e;
}

// without the chunks: the driver's copy, FP32 through one conversion
cudaError_t direct(const Job& j)
{
    const size_t row = (size_t)j.nx * j.es;
    std::vector<float> f;
    void* buf = j.host;
    if (j.es == 4) {
        try {
            f.resize((size_t)j.nx * j.n_rows);
        } catch (...) {
            return cudaErrorMemoryAllocation;
        }
        buf = f.data();
        if (!j.to_host)
            for (size_t q = 0; q < f.size(); ++q) f[q] = (float)j.host[q];
    }
    cudaError_t e = j.to_host ? cudaMemcpy2DAsync(buf, row, j.dev, (size_t)j.px * j.es, row, (size_t)j.n_rows,
                                                  cudaMemcpyDeviceToHost, j.stream)
                              : cudaMemcpy2DAsync(j.dev, (size_t)j.px * j.es, buf, row, row, (size_t)j.n_rows,
                                                  cudaMemcpyHostToDevice, j.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(j.stream);
    if (e == cudaSuccess && j.to_host)
        for (size_t q = 0; q < f.size(); ++q) j.host[q] = (double)f[q];
    return e;
}

// chunk t is there, or could be allocated (in the relaxed capture mode: while
// another thread captures a graph, an allocation is refused in the default one)
bool have_chunk(int t)
{
    if (g_buf[t]) return true;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(&g_buf[t], kChunk, cudaHostAllocPortable) != cudaSuccess) {
        g_buf[t] = nullptr;
        cudaGetLastError();
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return g_buf[t] != nullptr;
}

cudaError_t transfer(Job j)
{
    cudaError_t e = cudaStreamSynchronize(j.stream);
    if (e != cudaSuccess) return e;
    const size_t row = (size_t)j.nx * j.es;
    const size_t bytes = row * (size_t)j.n_rows;
    const bool small = (size_t)j.nx * j.n_rows * 8 < (j.es == 8 ? kSmall64 : kSmall32);
    if (small || row > kChunk) return direct(j);
    // the field's device, which need not be the calling thread's
    cudaPointerAttributes at;
    e = cudaPointerGetAttributes(&at, j.dev);
    if (e != cudaSuccess) return e;
    j.device = at.device;
    // equal chunks, at least one a thread where the field is large enough
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency() / 2);
    int nt = (int)std::min<size_t>(std::min(kXferThreads, hw), (bytes + (1u << 20) - 1) >> 20);
    long long n_chunks = (long long)((bytes + kChunk - 1) / kChunk);
    n_chunks = (n_chunks + nt - 1) / nt * nt;
    j.rows_per = std::max<long long>(1, (j.n_rows + n_chunks - 1) / n_chunks);
    j.rows_per = std::min<long long>(j.rows_per, (long long)(kChunk / row));
    std::unique_lock<std::mutex> lk(g_mu);
    int have = 0;
    while (have < nt && have_chunk(have)) ++have;
    if (have == 0) {   // no pinned memory to be had
        lk.unlock();
        return direct(j);
    }
    nt = have;
    cudaError_t rc[kXferThreads] = {};
    std::thread thr[kXferThreads];
    int started = 1;
    try {
        for (; started < nt; ++started) {
            const int t = started;
            thr[t] = std::thread([&j, &rc, t, nt] { rc[t] = run_thread(j, t, nt); });
        }
    } catch (...) {   // no more threads: this one takes the shares that are left
    }
    int own = j.device;
    cudaGetDevice(&own);
    for (int t = started; t < nt; ++t) rc[t] = run_thread(j, t, nt);
    rc[0] = run_thread(j, 0, nt);
    if (own != j.device) cudaSetDevice(own);
    for (int t = 1; t < started; ++t) thr[t].join();
    for (int t = 0; t < nt; ++t)
        if (rc[t] != cudaSuccess) e = rc[t];
    if (e != cudaSuccess) cudaStreamSynchronize(j.stream);   // no copy into a chunk is left in flight
    return e;
}

}  // namespace

void xfer_ref()
{
    std::lock_guard<std::mutex> lk(g_mu);
    ++g_refs;
}

void xfer_unref()
{
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_refs <= 0) {
        g_refs = 0;
        free_buffers();
    }
}

bool xfer_pinned(const void* host)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

cudaError_t xfer_to_host(const void* dev, int es, int nx, long long px, long long n_rows, double* host,
                         cudaStream_t stream)
{
    return transfer(Job{(char*)const_cast<void*>(dev), es, nx, px, n_rows, 1, host, true, stream, 0});
}

cudaError_t xfer_to_device(void* dev, int es, int nx, long long px, long long n_rows, const double* host,
                           cudaStream_t stream)
{
    return transfer(Job{(char*)dev, es, nx, px, n_rows, 1, const_cast<double*>(host), false, stream, 0});
}

}  // namespace pf3d
