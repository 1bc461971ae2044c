// pf3d_xfer.h -- whole fields between the device and the caller's pageable
// host arrays (pinned arrays are copied by the callers without staging).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace pf3d {

// Every object that transfers fields holds a reference; the staging buffers
// (kXferThreads pinned chunks, allocated by the first large transfer) are
// freed with the last one.
void xfer_ref();
void xfer_unref();

// whether host is pinned or managed memory the device's copy engines reach directly
bool xfer_pinned(const void* host);

// The field at `dev` (rows of nx elements of es bytes, pitch px elements, n_rows
// rows) to or from the doubles at `host`, complete on return: device ordering
// through `stream`.  es 4 converts on the way, rounding to nearest.
cudaError_t xfer_to_host(const void* dev, int es, int nx, long long px, long long n_rows, double* host,
                         cudaStream_t stream);
cudaError_t xfer_to_device(void* dev, int es, int nx, long long px, long long n_rows, const double* host,
                           cudaStream_t stream);

}  // namespace pf3d
