// pf3d_simple.cuh -- kernels without a stencil window: the heat equation and
// the interior copy of concentracao_soluto (one thread per cell, reference
// form), the diagnostics and the staging conversions.
#pragma once
#include <cfloat>
#include "pf3d_launch.h"

namespace pf3d {

__device__ __forceinline__ long long cell_off(const DomainDesc& d, int x, int y, int z)
{
    return (long long)x + (long long)y * d.px + (long long)z * d.plane;
}

// Both kernels below stream whole fields, so HBM (or L2, for small domains)
// bounds them: a thread takes the same column of kPlanes planes with their
// loads in flight together, and the loop constants come by value
// (temperatura on 128x128x256 FP64: 29.9 -> 19.3 us).
constexpr int kPlanes = 4;

// ---- temperatura.f90 (TNEW = TOLD; temp_body.inc on 2..N-1) ----
template <typename T>
__global__ void __launch_bounds__(256) k_heat(DomainDesc d, const KC<T> c, const T* __restrict__ Told,
                                              const T* __restrict__ phi, const T* __restrict__ dpp,
                                              T* __restrict__ Tnew)
{
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z0 = blockIdx.z * kPlanes;
    if (x >= d.nx || y >= d.ny) return;
    const bool xy = x >= 1 && x <= d.nx - 2 && y >= 1 && y <= d.ny - 2;
    const long long id0 = cell_off(d, x, y, z0);
    T a[kPlanes], b[kPlanes];
#pragma unroll
    for (int k = 0; k < kPlanes; ++k) {
        const int z = z0 + k;
        const long long id = id0 + k * d.plane;
        if (z >= d.nz) continue;
        if (xy && z >= 1 && z <= d.nz - 2) {
            a[k] = phi[id];
            b[k] = dpp[id];
        } else {
            a[k] = Told[id];
        }
    }
#pragma unroll
    for (int k = 0; k < kPlanes; ++k) {
        const int z = z0 + k;
        const long long id = id0 + k * d.plane;
        if (z >= d.nz) continue;
        T v = a[k];
        if (xy && z >= 1 && z <= d.nz - 2) {
            T TE = 0, TW = 0, TN = 0, TS = 0, TT = 0, TB = 0;
            if (c.lap) {
                TE = Told[id + 1]; TW = Told[id - 1]; TN = Told[id + d.px]; TS = Told[id - d.px];
                TT = Told[id + d.plane]; TB = Told[id - d.plane];
            }
            v = heat_new<T>(a[k], b[k], TE, TW, TN, TS, TT, TB, c);
        }
        Tnew[id] = v;
    }
}

// conc_soluto_old = conc_soluto_new on 2..N-1 (the wall cells of
// conc_soluto_old keep their values; concentracao_soluto.f90:116)
template <typename T>
__global__ void __launch_bounds__(256) k_copy_inner(DomainDesc d, const T* __restrict__ src, T* __restrict__ dst)
{
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z0 = blockIdx.z * kPlanes;
    if (x < 1 || x > d.nx - 2 || y < 1 || y > d.ny - 2) return;
    const long long id0 = cell_off(d, x, y, z0);
    T v[kPlanes];
#pragma unroll
    for (int k = 0; k < kPlanes; ++k)
        if (z0 + k >= 1 && z0 + k <= d.nz - 2) v[k] = src[id0 + k * d.plane];
#pragma unroll
    for (int k = 0; k < kPlanes; ++k)
        if (z0 + k >= 1 && z0 + k <= d.nz - 2) dst[id0 + k * d.plane] = v[k];
}

// ---- diagnosticos.f90 + diag_body.inc ----
// FP64 accumulation with Neumaier compensation; max/min exact and NaN-
// propagating (fmax/fmin would drop a NaN and report finite extremes for a
// blown-up field); plus the watchdog: the count of cells where phi, c, or
// (when given) T or DPP is not finite.  The clamp of the phase update maps a
// NaN or infinite update to 1, so a blow-up can leave phi finite and show
// only in DPP and T.  Partials: kDiagRow doubles per block (pf3d_launch.h).

// max / min that return NaN when either argument is NaN
__device__ __forceinline__ double nan_max(double a, double b) { return (a > b || a != a) ? a : b; }
__device__ __forceinline__ double nan_min(double a, double b) { return (a < b || a != a) ? a : b; }
struct KSum {
    double s, c;
    __device__ __forceinline__ void add(double v)
    {
        double t = s + v;
        if (fabs(s) >= fabs(v)) c += (s - t) + v;
        else c += (v - t) + s;
        s = t;
    }
    __device__ __forceinline__ void merge(double os, double oc)
    {
        add(os);
        c += oc;
    }
};

// whether a value is NaN or infinite, from its bits
__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }

// The grid walks 32 x 8-column tiles, each marched along z over a chunk of zlen
// planes (a persistent grid: block b takes tiles b, b + gridDim.x, ...; the
// per-thread sums carry across its tiles, so the reduction order is fixed by
// the launch shape).  The march goes in groups of kDiagG planes: a thread
// first issues the reads of the whole group -- phi of the next kDiagG planes
// and c, T, DPP of the group's planes, each cell read once from HBM, all in
// flight together -- then shares the group's phase planes through shared
// memory (one barrier a group) and evaluates its cells, with the phase field
// of the planes above and below in registers (indexed at compile time, so no
// register is moved before its load lands).
//
// FP64 arithmetic bounds the pass where memory does not (FP32 fields, small
// domains), so a cell contributes bare squares -- phi^2, the three squared
// central differences and (phi (1-phi))^2, eleven operations -- and the
// factors of diag_body.inc (0.5 E0^2, (0.5/dx)^2, W0, dx dy dz) multiply the
// column's sums once.  T and DPP, which only the watchdog reads, are tested
// on their bits and never converted.  A column's at most kDiagZ terms are
// summed in plain FP64 (every term is nonnegative: phi^2, c and the energy's
// parts, so the relative error stays below kDiagZ ulps) and the column sums go
// into compensated (Neumaier) totals.
//
// The last block to finish merges the blocks' partials (block order, fixed), so
// the whole reduction is one launch.  pf_diagnosticos, call to answer, before and
// after: 340x340x700 FP64 768 -> 488 us (5.3 TB/s, 0.81 of the measured HBM
// rate), 256x256x512 FP32 576 -> 172 us, 64x64x128 FP64 84 -> 34 us.
constexpr int kDiagZ = 64;
constexpr int kDiagG = 4;   // planes a group
constexpr int kDiagBlocks = 592;

// the block's nine values reduced over its threads into v on thread 0 (fixed
// order): l2, its compensation, max, min, sol, comp., fe, comp., bad cells
__device__ __forceinline__ void diag_merge(double* v, const double* o)
{
    KSum a{v[0], v[1]}; a.merge(o[0], o[1]); v[0] = a.s; v[1] = a.c;
    v[2] = nan_max(v[2], o[2]); v[3] = nan_min(v[3], o[3]);
    KSum b{v[4], v[5]}; b.merge(o[4], o[5]); v[4] = b.s; v[5] = b.c;
    KSum e{v[6], v[7]}; e.merge(o[6], o[7]); v[6] = e.s; v[7] = e.c;
    v[8] += o[8];
}
__device__ __forceinline__ void diag_block_reduce(double* v, double (*sh)[9])
{
    for (int off = 16; off > 0; off >>= 1) {
        double o[9];
        for (int q = 0; q < 9; ++q) o[q] = __shfl_down_sync(0xffffffffu, v[q], off);
        diag_merge(v, o);
    }
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 9; ++q) sh[w][q] = v[q];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int ww = 1; ww < (int)(blockDim.x >> 5); ++ww) diag_merge(v, sh[ww]);
}

template <typename T>
__global__ void __launch_bounds__(256, 4) k_diag(DomainDesc d, const T* __restrict__ pn, const T* __restrict__ cn,
                                                 const T* __restrict__ tw, const T* __restrict__ dw, int zlen,
                                                 double* __restrict__ part, double* __restrict__ out)
{
    KSum l2{0, 0}, sol{0, 0}, fe{0, 0};
    double mx = -DBL_MAX, mn = DBL_MAX;
    int bad = 0;
    bool nan_phi = false;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const long long px = d.px, pl = d.plane;
    const double hE2 = 0.5 * d.E0 * d.E0, vol = d.dx * d.dy * d.dz;
    const double kx = hE2 * d.hx * d.hx, ky = hE2 * d.hy * d.hy, kz = hE2 * d.hz * d.hz;
    constexpr int W = 34, H = 10;
    __shared__ double sp[2][kDiagG][H * W];   // the group's phase planes and their ring, double-buffered by group parity
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int ntx = (nx + 31) >> 5, nty = (ny + 7) >> 3, ntz = (nz + zlen - 1) / zlen;
    const long long ntiles = (long long)ntx * nty * ntz;
    const int me = (ty + 1) * W + tx + 1;
    // the first 80 threads fetch the tile's ring (its corners are not read)
    const int h = threadIdx.x;
    const bool ringer = h < 80;
    const int hx = h < 64 ? (h & 31) : (h < 72 ? -1 : 32), hy = h < 32 ? -1 : h < 64 ? 8 : (h & 7);
    const int hs = (hy + 1) * W + hx + 1;
    int g = 0;   // group parity across the whole walk
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int bx = (int)(t % ntx);
        const long long r = t / ntx;
        const int by = (int)(r % nty), bz = (int)(r / nty);
        const int x = bx * 32 + tx, y = by * 8 + ty;
        const bool own = x < nx && y < ny;
        const bool xy_in = x > 0 && x < nx - 1 && y > 0 && y < ny - 1;
        const int z0 = bz * zlen, z1 = min(z0 + zlen, nz);
        // threads outside the domain repeat its last column: their loads and
        // extremes are harmless, their sums are dropped
        const uint32_t col = (uint32_t)min(x, nx - 1) + (uint32_t)min(y, ny - 1) * (uint32_t)px;
        const uint32_t hcol = (uint32_t)max(min(bx * 32 + hx, nx - 1), 0) +
                              (uint32_t)max(min(by * 8 + hy, ny - 1), 0) * (uint32_t)px;
        // phase field of this column at planes z-1 (pprev) and z (pcur) of the group's first plane z
        double pprev = (double)(pn + (long long)max(z0 - 1, 0) * pl)[col];
        double pcur = (double)(pn + (long long)z0 * pl)[col];
        double s_l2 = 0.0, s_sol = 0.0, s_x = 0.0, s_y = 0.0, s_z = 0.0, s_w = 0.0;   // this column's sums
        int s_bad = 0;
        for (int zb = z0; zb < z1; zb += kDiagG, g ^= 1) {
            const int ng = min(kDiagG, z1 - zb);          // planes in this group (uniform)
            // phi of plane zb+k+1; c, T, DPP and the ring of zb+k.  Planes are
            // clamped to the domain and no load stands under a condition: a
            // conditional load is waited for inside its branch when a
            // conversion follows it
            T pnx[kDiagG], cv[kDiagG], tv[kDiagG], dv[kDiagG], rv[kDiagG];
#pragma unroll
            for (int k = 0; k < kDiagG; ++k) {
                const long long zo = (long long)min(zb + k, nz - 1) * pl;
                pnx[k] = (pn + (long long)min(zb + k + 1, nz - 1) * pl)[col];
                cv[k] = (cn + zo)[col];
                tv[k] = (tw + zo)[col];
                dv[k] = (dw + zo)[col];
                rv[k] = (pn + zo)[hcol];
            }
            double p[kDiagG + 2];   // phi of planes zb-1 .. zb+kDiagG
            p[0] = pprev;
            p[1] = pcur;
#pragma unroll
            for (int k = 0; k < kDiagG; ++k) p[k + 2] = (double)pnx[k];
#pragma unroll
            for (int k = 0; k < kDiagG; ++k) {
                sp[g][k][me] = p[k + 1];
                if (ringer) sp[g][k][hs] = (double)rv[k];
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kDiagG; ++k) {
                if (k >= ng) continue;
                const int z = zb + k;
                const double phi = p[k + 1];
                s_l2 = __fma_rn(phi, phi, s_l2);
                mx = phi > mx ? phi : mx;
                mn = phi < mn ? phi : mn;
                s_sol += (double)cv[k];
                if (not_finite(phi) || not_finite(cv[k]) || not_finite(tv[k]) || not_finite(dv[k])) {
                    ++s_bad;
                    nan_phi = nan_phi || phi != phi;
                }
                const double w = phi * (1.0 - phi);
                s_w = __fma_rn(w, w, s_w);
                if (z > 0 && z < nz - 1) {
                    const double* const q = &sp[g][k][me];
                    const double gx = q[1] - q[-1], gy = q[W] - q[-W], gz = p[k + 2] - p[k];
                    s_x = __fma_rn(gx, gx, s_x);
                    s_y = __fma_rn(gy, gy, s_y);
                    s_z = __fma_rn(gz, gz, s_z);
                }
            }
            pprev = p[kDiagG];   // the next group's planes z-1 and z (a short group ends the chunk)
            pcur = p[kDiagG + 1];
        }
        if (own) {
            const double e = xy_in ? __fma_rn(kx, s_x, __fma_rn(ky, s_y, kz * s_z)) : 0.0;
            l2.add(s_l2);
            sol.add(s_sol);
            fe.add(vol * __fma_rn(d.W0, s_w, e));
            bad += s_bad;
        }
    }
    if (nan_phi) mx = mn = __longlong_as_double(0x7ff8000000000000ll);
    __shared__ double sh[8][9];
    __shared__ bool last;
    double v[9] = {l2.s, l2.c, mx, mn, sol.s, sol.c, fe.s, fe.c, (double)bad};
    diag_block_reduce(v, sh);
    unsigned* const done = (unsigned*)(out + 7);   // blocks that have written their partials; 0 between launches
    if (threadIdx.x == 0) {
        for (int q = 0; q < 9; ++q) part[(long long)blockIdx.x * kDiagRow + q] = v[q];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int q = 0; q < 9; ++q) v[q] = 0.0;
    v[2] = -DBL_MAX;
    v[3] = DBL_MAX;
    for (int b = (int)threadIdx.x; b < (int)gridDim.x; b += (int)blockDim.x) {
        double o[9];
        for (int q = 0; q < 9; ++q) o[q] = __ldcg(part + (long long)b * kDiagRow + q);
        diag_merge(v, o);
    }
    diag_block_reduce(v, sh);
    if (threadIdx.x == 0) {
        out[0] = sqrt(v[0] + v[1]);
        out[1] = v[2];
        out[2] = v[3];
        out[3] = v[4] + v[5];
        out[4] = v[6] + v[7];
        out[5] = v[8];   // cells with a non-finite phi, c, T or DPP (the watchdog)
        *done = 0u;
    }
}

// ---- host conversion staging (FP32 contexts) ----
template <typename T>
__global__ void k_convert_in(DomainDesc d, const double* __restrict__ stage, T* __restrict__ dst, long long z0, long long nzc)
{
    long long n = (long long)d.nx * d.ny * nzc;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        int x = (int)(q % d.nx);
        long long r = q / d.nx;
        int y = (int)(r % d.ny);
        long long z = z0 + r / d.ny;
        dst[x + (long long)y * d.px + z * d.plane] = (T)stage[q];
    }
}

template <typename T>
__global__ void k_convert_out(DomainDesc d, const T* __restrict__ src, double* __restrict__ stage, long long z0, long long nzc)
{
    long long n = (long long)d.nx * d.ny * nzc;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        int x = (int)(q % d.nx);
        long long r = q / d.nx;
        int y = (int)(r % d.ny);
        long long z = z0 + r / d.ny;
        stage[q] = (double)src[x + (long long)y * d.px + z * d.plane];
    }
}

// ---- launchers ----
inline dim3 cell_grid(const DomainDesc& d)
{
    return dim3((d.nx + 31) / 32, (d.ny + 7) / 8, (d.nz + kPlanes - 1) / kPlanes);
}

template <typename T>
cudaError_t launch_heat(const DomainDesc& d, const StepArgs& s, const Fields& f, cudaStream_t st)
{
    KC<T> c;
    c.load(d, s);
    k_heat<T><<<cell_grid(d), dim3(32, 8), 0, st>>>(d, c, (const T*)f.T_old, (const T*)f.phi_old, (const T*)f.dpp,
                                                    (T*)f.T_new);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_copy_inner(const DomainDesc& d, const void* src, void* dst, cudaStream_t st)
{
    k_copy_inner<T><<<cell_grid(d), dim3(32, 8), 0, st>>>(d, (const T*)src, (T*)dst);
    return cudaGetLastError();
}

// part: kDiagBlocks rows; out: 8 doubles, the last one zero before the first call
template <typename T>
cudaError_t launch_diag(const DomainDesc& d, const void* phi, const void* c, const void* Tw, const void* dppw,
                        double* part, double* out, cudaStream_t st)
{
    // chunks of whole groups, short enough for a small domain's tiles to fill
    // the grid, at most kDiagZ planes
    const long long cols = (long long)((d.nx + 31) / 32) * ((d.ny + 7) / 8);
    const long long want = (kDiagBlocks + cols - 1) / cols;   // chunks a column
    long long zlen = ((d.nz + want - 1) / want + kDiagG - 1) / kDiagG * kDiagG;
    zlen = zlen < kDiagZ ? zlen : kDiagZ;
    const long long tiles = cols * ((d.nz + zlen - 1) / zlen);
    const int nblk = (int)(tiles < kDiagBlocks ? tiles : kDiagBlocks);
    // a field the watchdog does not look at is replaced by c, which it does
    k_diag<T><<<nblk, 256, 0, st>>>(d, (const T*)phi, (const T*)c, (const T*)(Tw ? Tw : c),
                                    (const T*)(dppw ? dppw : c), (int)zlen, part, out);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_convert_in(const DomainDesc& d, const double* stage, void* dst, long long z0, long long nzc,
                              cudaStream_t st)
{
    k_convert_in<T><<<592, 256, 0, st>>>(d, stage, (T*)dst, z0, nzc);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_convert_out(const DomainDesc& d, const void* src, double* stage, long long z0, long long nzc,
                               cudaStream_t st)
{
    k_convert_out<T><<<592, 256, 0, st>>>(d, (const T*)src, stage, z0, nzc);
    return cudaGetLastError();
}

}  // namespace pf3d
