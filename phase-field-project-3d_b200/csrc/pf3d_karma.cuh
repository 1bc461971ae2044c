// pf3d_karma.cuh -- the quantitative Karma model of the reference
// (karma/karma3d.f90: Karma PRL 87 115701 2001; Echebarria, Folch, Karma &
// Plapp PRE 70 061604 2004) on the z-marching tile scheme of the main model.
//
// State: phi in [-1, 1] and the dimensionless supersaturation U, interior
// cells only, Fortran order with a padded row pitch.  The reference keeps a
// ghost layer refreshed by mirror copies on every face (espelho,
// karma3d.f90:318-339); a mirror ghost equals the interior value at the
// clamped index, so the kernels clamp their neighbour indices instead.
//
// One step = two passes (the U equation needs dphi/dt at the face
// neighbours, karma3d.f90:209):
//   pass A (karma3d.f90:166-207): dphi from phi (19-point stencil: centre,
//           6 faces, 12 edges) and U at the centre;
//   pass B (karma3d.f90:212-287): U_new from phi, U and dphi (anti-trapping
//           current through the 6 faces) and phi_new = clamp(phi + dt dphi).
// Each CTA owns a 32 x TY column tile and marches a z-chunk.  Planes (tile +
// 1-cell ring) come by TMA, one tiled load a field and plane issued by one
// thread two planes ahead into 4-slot windows; the mirror ghosts of tiles on
// the domain's faces, which the load fills with zeros, are copied from the
// neighbouring cells in shared memory, and a z ghost is the clamped plane.
// Where the phase field is exactly +1 or -1 on a warp's 34 x 3 x 3
// neighbourhood -- the crystal's interior and the melt beyond the interface's
// tanh tails, most of a domain -- every gradient is zero, so both passes
// reduce to what is left of the same expressions (no phase flux, no
// anti-trapping current, dphi = 0): the same values with a tenth of the work.
// A warp finds that out with one vote a plane on the bits it has just loaded.
// Measured against element-wise cp.async planes and the full arithmetic
// everywhere (crystals a third of the domain's extent): 200^3 FP64 with noise
// 512 -> 328 us a step, 256^3 FP32 612 -> 365 us, 72x60x80 FP64 49 -> 44 us;
// the seeded 512^3 FP64 domain 7.0 -> 2.6 ms.
// Every operation is the reference's, in its order, with IEEE division and
// square root and no contraction: the FP64 result is the reference's
// arithmetic bit for bit (checked against the C oracle).
#pragma once
#include <cstdint>
#include "pf3d_launch.h"
#include "pf3d_tma.cuh"

namespace pf3d {

struct KarmaDesc {
    int nx, ny, nz;
    long long px, plane;    // row pitch and plane stride (elements)
    int it;                 // step being computed (noise)
};

// loop constants, each computed on the host exactly as the reference's
// expression computes it (same operations, same rounding)
template <typename T>
struct KarmaK {
    T idx;        // 1/dx
    T q;          // 0.25*idx
    T h;          // 0.5*idx
    T om3;        // 1 - 3 eps4
    T e4;         // 4 eps4
    T e16;        // 16 eps4
    T lambda, dt, Fnoise, sqdt;   // sqdt = sqrt(dt)
    T omk;        // 1 - k
    T Ahalf1;     // 0.5*(1+k)
    T Ahalf2;     // 0.5*(1-k)
    T D;          // a2*lambda
    T at;         // 1/(2 sqrt 2)
    T z0;         // dphi without the term in U where phi is +1 or -1 all around: 0, or NaN where a parameter makes it so
};

template <typename T>
__device__ __forceinline__ T k_fluxn(T g1, T g2, T g3, const KarmaK<T>& c)
{
    const T g2s = g1 * g1 + g2 * g2 + g3 * g3;
    if (g2s < (T)1.e-20) return (c.om3 * c.om3) * g1;
    const T a = g1 * g1, b = g2 * g2, d = g3 * g3;
    const T s4 = a * a + b * b + d * d;
    const T as = c.om3 + c.e4 * s4 / (g2s * g2s);
    return as * (as * g1 + c.e16 * ((g1 * g1) * g1 - g1 * s4 / g2s) / g2s);
}

// karma3d.f90:52-67 in [-1, 1)
__device__ __forceinline__ double k_ruido(int i, int j, int k, int it)
{
    uint64_t h = (uint64_t)(int64_t)i * 2654435761ull + (uint64_t)(int64_t)j * 2246822519ull +
                 (uint64_t)(int64_t)k * 3266489917ull + (uint64_t)(int64_t)it * 668265263ull + 1ull;
    h ^= h >> 33;
    h *= 0xff51afd7ed558ccdull;
    h ^= h >> 33;
    h *= 0xc4ceb9fe1a85ec53ull;
    h ^= h >> 33;
    const double m = (double)(long long)(h & 0x7fffffffffffffffull);
    return __dsub_rn(__dmul_rn(m, 0x1p-62), 1.0);   // 2 m / 2^63: both scalings are exact
}

__device__ __forceinline__ int kclamp(int v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// One plane of a tile in shared memory: the tile plus a 1-cell ring, widened
// in x so that the TMA box starts on a 16-byte boundary.
template <typename T, int TY>
struct KarmaTile {
    static constexpr int XOFF = (sizeof(T) == 8) ? 2 : 4;
    static constexpr int W = 32 + 2 * XOFF, H = TY + 2;
    static constexpr int BYTES = W * H * (int)sizeof(T);
    static constexpr int STRIDE = (BYTES + 127) / 128 * 128 / (int)sizeof(T);   // elements a slot
};
inline int karma_box_x(int es) { return es == 8 ? 36 : 40; }

// The planes of NF fields of a tile, marched along z: plane z0 - 1 + q lives in
// slot q % 4.  `lead` issues; `pend` (lead only) are the slots in flight.
template <typename T, int TY, int NF>
struct KarmaWindow {
    using KT = KarmaTile<T, TY>;
    T* buf;
    const CUtensorMap* const* tm;   // NF maps
    uint32_t bar0;
    int x0, y0, zfirst, nz;
    uint32_t pend;
    __device__ __forceinline__ const T* plane(int f, int q) const { return buf + (f * 4 + (q & 3)) * KT::STRIDE; }
    __device__ __forceinline__ void issue(int q)
    {
        const int s = q & 3;
        const uint32_t bar = bar0 + 8 * s;
        mbar_arrive_expect_tx(bar, NF * KT::BYTES);
        const int zc = kclamp(zfirst + q, nz);
#pragma unroll
        for (int f = 0; f < NF; ++f)
            tma_load_3d(smem_u32(buf + (f * 4 + s) * KT::STRIDE), tm[f], x0 - KT::XOFF, y0 - 1, zc, bar);
        pend |= 1u << s;
    }
    __device__ __forceinline__ bool wait(int q)
    {
        const int s = q & 3;
        const bool ok = mbar_wait(bar0 + 8 * s, (q >> 2) & 1);
        if (ok) pend &= ~(1u << s);
        return ok;
    }
    // after a failed wait: the loads still in flight land (bounded wait) before
    // the CTA leaves its shared memory; q is the last plane waited for, and
    // at most q-2 .. q+1 (the prologue's planes among them) are in flight
    __device__ __forceinline__ void drain(int q)
    {
        for (int k = q - 2; k < q + 2; ++k)
            if ((pend >> (k & 3)) & 1u) mbar_wait(bar0 + 8 * (k & 3), (k >> 2) & 1);
    }
    // mirror ghosts of a tile on the domain's faces (espelho,
    // karma3d.f90:318-339): each is the landed cell at the clamped index
    __device__ __forceinline__ void ghosts(int q, int nx, int ny, int tid)
    {
        const int cr = min(33, nx - x0 + 1), rt = min(TY + 1, ny - y0 + 1);   // ring positions in 0..33, 0..TY+1
        const bool left = x0 == 0, right = nx - x0 <= 32, low = y0 == 0, top = ny - y0 <= TY;
        for (int i = tid; i < 2 * KT::H + 2 * 34; i += 32 * TY) {
            int c, r;
            if (i < KT::H) { if (!left) continue; c = 0; r = i; }
            else if (i < 2 * KT::H) { if (!right) continue; c = cr; r = i - KT::H; }
            else if (i < 2 * KT::H + 34) { if (!low) continue; r = 0; c = i - 2 * KT::H; }
            else { if (!top) continue; r = rt; c = i - 2 * KT::H - 34; }
            if (c > cr || r > rt) continue;
            const int cc = kclamp(x0 + c - 1, nx) - x0 + 1, rr = kclamp(y0 + r - 1, ny) - y0 + 1;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                T* p = buf + (f * 4 + (q & 3)) * KT::STRIDE + KT::XOFF - 1;
                p[r * KT::W + c] = p[rr * KT::W + cc];
            }
        }
        fence_proxy_async_smem();   // before the barrier that lets a later load overwrite these cells
    }
};

__device__ __forceinline__ uint32_t k_bits_diff(double a, double s)
{
    return (uint32_t)(__double2hiint(a) ^ __double2hiint(s)) | (uint32_t)(__double2loint(a) ^ __double2loint(s));
}
__device__ __forceinline__ uint32_t k_bits_diff(float a, float s)
{
    return __float_as_uint(a) ^ __float_as_uint(s);
}

// +1 or -1 when the three rows around the warp's own row hold exactly that
// value in the warp's columns and the two beside them, else 0 (warp-uniform).
// o: the lane's cell; oe: the edge column of the lane's half warp, same row.
template <typename T, int W>
__device__ __forceinline__ int k_uniform3(const T* p, int o, int oe, int o0, bool own)
{
    const T s = p[o0];
    uint32_t d = (uint32_t)0;
    if (own) d = k_bits_diff(p[o - W], s) | k_bits_diff(p[o], s) | k_bits_diff(p[o + W], s);
    d |= k_bits_diff(p[oe - W], s) | k_bits_diff(p[oe], s) | k_bits_diff(p[oe + W], s);
    const bool one = s == (T)1 || s == (T)-1;
    return __all_sync(0xffffffffu, d == 0 && one) ? (s > (T)0 ? 1 : -1) : 0;
}

// resident CTAs the register budget is sized for
template <typename T> struct KarmaOcc { static constexpr int v = sizeof(T) == 8 ? 3 : 5; };

// pass A: dphi of karma3d.f90:166-207
template <typename T, int TY>
__global__ void __launch_bounds__(32 * TY, (KarmaOcc<T>::v))
    k_karma_phase(const __grid_constant__ CUtensorMap tm_phi, KarmaDesc d, const KarmaK<T> c, const T* __restrict__ U,
                  T* __restrict__ dphi, int zchunk, int* __restrict__ err)
{
    using KT = KarmaTile<T, TY>;
    __shared__ __align__(128) T sbuf[4 * KT::STRIDE];
    __shared__ __align__(8) uint64_t sbar[4];
    constexpr int W = KT::W;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * TY;
    const int zb = blockIdx.z * zchunk, ze = min(zb + zchunk, d.nz);
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + 32 * ty;
    const int x = x0 + tx, y = y0 + ty;
    const bool own = x < d.nx && y < d.ny, lead = tid == 0;
    const bool edge = x0 == 0 || x0 + 32 >= d.nx || y0 == 0 || y0 + TY >= d.ny;
    const CUtensorMap* tms[1] = {&tm_phi};
    KarmaWindow<T, TY, 1> w{sbuf, tms, smem_u32(sbar), x0, y0, zb - 1, d.nz, 0u};
    if (lead) {
        for (int s = 0; s < 4; ++s) mbar_init(w.bar0 + 8 * s, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (lead)
        for (int q = 0; q < 4 && zb - 1 + q <= ze; ++q) w.issue(q);
    const int o = (ty + 1) * W + tx + KT::XOFF;                       // own cell
    const int o0 = (ty + 1) * W + KT::XOFF - 1;                       // left ring column
    const int oe = tx < 16 ? o0 : o0 + min(33, d.nx - x0 + 1);        // ring column of the lane's half warp
    long long id = (long long)x + (long long)y * d.px + (long long)zb * d.plane;
    T u_next = own ? U[id] : (T)0;
    bool bad = false;
    int ub = 0, up = 0;   // phase field uniform around the own row in planes z-1, z
    for (int q = 0; q < 2; ++q) {
        bad |= !w.wait(q);
        if (edge) w.ghosts(q, d.nx, d.ny, tid);
    }
    if (edge) __syncthreads();
    ub = k_uniform3<T, W>(w.plane(0, 0), o, oe, o0, own);
    up = k_uniform3<T, W>(w.plane(0, 1), o, oe, o0, own);
    for (int z = zb, q = 0; z < ze; ++z, ++q) {   // plane z is sequence q + 1
        const T uc = u_next;
        if (own && z + 1 < ze) u_next = U[id + d.plane];
        bad |= !w.wait(q + 2);
        if (edge) {
            w.ghosts(q + 2, d.nx, d.ny, tid);
            __syncthreads();
        }
        const T* const P = w.plane(0, q + 1) + o;
        const T* const Tp = w.plane(0, q + 2) + o;
        const int ut = k_uniform3<T, W>(w.plane(0, q + 2), o, oe, o0, own);
        if (up != 0 && ub == up && ut == up) {
            // every gradient and 1 - phi^2 are zero: dphi = 0 (0 times U keeps a non-finite U visible)
            if (own) dphi[id] = c.z0 * uc + c.z0;
        } else if (own) {
            const T* const B = w.plane(0, q) + o;
            const T pp = P[0];
            const T qq = c.q, idx = c.idx;
            const T Jxp = k_fluxn<T>((P[1] - pp) * idx, qq * (P[W] + P[W + 1] - P[-W] - P[-W + 1]),
                                     qq * (Tp[0] + Tp[1] - B[0] - B[1]), c);
            const T Jxm = k_fluxn<T>((pp - P[-1]) * idx, qq * (P[W] + P[W - 1] - P[-W] - P[-W - 1]),
                                     qq * (Tp[0] + Tp[-1] - B[0] - B[-1]), c);
            const T Jyp = k_fluxn<T>((P[W] - pp) * idx, qq * (P[1] + P[W + 1] - P[-1] - P[W - 1]),
                                     qq * (Tp[0] + Tp[W] - B[0] - B[W]), c);
            const T Jym = k_fluxn<T>((pp - P[-W]) * idx, qq * (P[1] + P[-W + 1] - P[-1] - P[-W - 1]),
                                     qq * (Tp[0] + Tp[-W] - B[0] - B[-W]), c);
            const T Jzp = k_fluxn<T>((Tp[0] - pp) * idx, qq * (P[1] + Tp[1] - P[-1] - Tp[-1]),
                                     qq * (P[W] + Tp[W] - P[-W] - Tp[-W]), c);
            const T Jzm = k_fluxn<T>((pp - B[0]) * idx, qq * (P[1] + B[1] - P[-1] - B[-1]),
                                     qq * (P[W] + B[W] - P[-W] - B[-W]), c);
            const T divJ = (Jxp - Jxm + Jyp - Jym + Jzp - Jzm) * idx;
            const T g1 = c.h * (P[1] - P[-1]);
            const T g2 = c.h * (P[W] - P[-W]);
            const T g3 = c.h * (Tp[0] - B[0]);
            const T gm = g1 * g1 + g2 * g2 + g3 * g3;
            T as2;
            if (gm > (T)1.e-20) {
                const T a = g1 * g1, b = g2 * g2, e = g3 * g3;
                const T s4 = (a * a + b * b + e * e) / (gm * gm);
                const T t = c.om3 + c.e4 * s4;
                as2 = t * t;
            } else {
                as2 = c.om3 * c.om3;
            }
            const T om = (T)1 - pp * pp;
            T v = (divJ + pp - (pp * pp) * pp - c.lambda * (om * om) * uc) / as2;
            if (c.Fnoise != (T)0) {   // without noise the reference adds a zero
                const T r = (T)k_ruido(x + 1, y + 1, z + 1, d.it);
                v = v + c.Fnoise * r * ((T)1 - pp * pp) / c.sqdt;
            }
            dphi[id] = v;
        }
        id += d.plane;
        ub = up;
        up = ut;
        if (__syncthreads_or(bad)) {   // everyone learns of a failed load; the slot of plane z-1 is free
            if (lead) {
                w.drain(q + 2);
                atomicExch(err, kErrTmaTimeout);
            }
            return;
        }
        if (lead && z + 3 <= ze) w.issue(q + 4);   // into a slot only read since its last barrier
    }
}

// flux of U through one face of the own cell (karma3d.f90:219-264): g = the
// face gradient (gn its normal component), nb = phi across the face, du =
// the U difference in the face's orientation, un / dn = U and dphi across
template <typename T>
__device__ __forceinline__ T k_uflux(T g1, T g2, T g3, T gn, T pp, T nb, T du, T cl, T un, T dn, const KarmaK<T>& c)
{
    const T gm = sqrt(g1 * g1 + g2 * g2 + g3 * g3);
    const T qf = (T)0.25 * ((T)2 - pp - nb);
    const T cf = (T)0.5 * (cl + ((T)1 + c.omk * un) * dn);
    T F = c.D * qf * du * c.idx;
    if (gm > (T)1.e-10) F = F + c.at * cf * gn / gm;
    return F;
}

// pass B: U_new and phi_new of karma3d.f90:212-287
template <typename T, int TY>
__global__ void __launch_bounds__(32 * TY, (KarmaOcc<T>::v))
    k_karma_solute(const __grid_constant__ CUtensorMap tm_phi, const __grid_constant__ CUtensorMap tm_u,
                   const __grid_constant__ CUtensorMap tm_dphi, KarmaDesc d, const KarmaK<T> c,
                   T* __restrict__ phi_out, T* __restrict__ U_out, int zchunk, int* __restrict__ err)
{
    using KT = KarmaTile<T, TY>;
    __shared__ __align__(128) T sbuf[12 * KT::STRIDE];
    __shared__ __align__(8) uint64_t sbar[4];
    constexpr int W = KT::W;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * TY;
    const int zb = blockIdx.z * zchunk, ze = min(zb + zchunk, d.nz);
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + 32 * ty;
    const int x = x0 + tx, y = y0 + ty;
    const bool own = x < d.nx && y < d.ny, lead = tid == 0;
    const bool edge = x0 == 0 || x0 + 32 >= d.nx || y0 == 0 || y0 + TY >= d.ny;
    const CUtensorMap* tms[3] = {&tm_phi, &tm_u, &tm_dphi};
    KarmaWindow<T, TY, 3> w{sbuf, tms, smem_u32(sbar), x0, y0, zb - 1, d.nz, 0u};
    if (lead) {
        for (int s = 0; s < 4; ++s) mbar_init(w.bar0 + 8 * s, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (lead)
        for (int q = 0; q < 4 && zb - 1 + q <= ze; ++q) w.issue(q);
    const int o = (ty + 1) * W + tx + KT::XOFF;
    const int o0 = (ty + 1) * W + KT::XOFF - 1;
    const int oe = tx < 16 ? o0 : o0 + min(33, d.nx - x0 + 1);
    long long id = (long long)x + (long long)y * d.px + (long long)zb * d.plane;
    bool bad = false;
    int ub = 0, up = 0;
    for (int q = 0; q < 2; ++q) {
        bad |= !w.wait(q);
        if (edge) w.ghosts(q, d.nx, d.ny, tid);
    }
    if (edge) __syncthreads();
    ub = k_uniform3<T, W>(w.plane(0, 0), o, oe, o0, own);
    up = k_uniform3<T, W>(w.plane(0, 1), o, oe, o0, own);
    for (int z = zb, s = 0; z < ze; ++z, ++s) {   // plane z is sequence s + 1
        bad |= !w.wait(s + 2);
        if (edge) {
            w.ghosts(s + 2, d.nx, d.ny, tid);
            __syncthreads();
        }
        const T* const P = w.plane(0, s + 1) + o;
        const T* const UB = w.plane(1, s) + o;
        const T* const UP = w.plane(1, s + 1) + o;
        const T* const UT = w.plane(1, s + 2) + o;
        const T* const DP = w.plane(2, s + 1) + o;
        const int ut = k_uniform3<T, W>(w.plane(0, s + 2), o, oe, o0, own);
        if (own) {
            const T pp = P[0], uc = UP[0], dc = DP[0];
            const T q = c.q, idx = c.idx;
            T Fxp, Fxm, Fyp, Fym, Fzp, Fzm;
            if (up != 0 && ub == up && ut == up) {
                // no phase gradient at any face: the diffusive flux alone
                const T Dq = c.D * ((T)0.25 * ((T)2 - pp - pp));
                Fxp = Dq * (UP[1] - uc) * idx;
                Fxm = Dq * (uc - UP[-1]) * idx;
                Fyp = Dq * (UP[W] - uc) * idx;
                Fym = Dq * (uc - UP[-W]) * idx;
                Fzp = Dq * (UT[0] - uc) * idx;
                Fzm = Dq * (uc - UB[0]) * idx;
            } else {
                const T* const B = w.plane(0, s) + o;
                const T* const Tp = w.plane(0, s + 2) + o;
                const T* const DB = w.plane(2, s) + o;
                const T* const DT = w.plane(2, s + 2) + o;
                const T cl = ((T)1 + c.omk * uc) * dc;   // the own cell's term of cf
                T g1, g2, g3;
                g1 = (P[1] - pp) * idx;
                g2 = q * (P[W] + P[W + 1] - P[-W] - P[-W + 1]);
                g3 = q * (Tp[0] + Tp[1] - B[0] - B[1]);
                Fxp = k_uflux<T>(g1, g2, g3, g1, pp, P[1], UP[1] - uc, cl, UP[1], DP[1], c);
                g1 = (pp - P[-1]) * idx;
                g2 = q * (P[W] + P[W - 1] - P[-W] - P[-W - 1]);
                g3 = q * (Tp[0] + Tp[-1] - B[0] - B[-1]);
                Fxm = k_uflux<T>(g1, g2, g3, g1, pp, P[-1], uc - UP[-1], cl, UP[-1], DP[-1], c);
                g2 = (P[W] - pp) * idx;
                g1 = q * (P[1] + P[W + 1] - P[-1] - P[W - 1]);
                g3 = q * (Tp[0] + Tp[W] - B[0] - B[W]);
                Fyp = k_uflux<T>(g1, g2, g3, g2, pp, P[W], UP[W] - uc, cl, UP[W], DP[W], c);
                g2 = (pp - P[-W]) * idx;
                g1 = q * (P[1] + P[-W + 1] - P[-1] - P[-W - 1]);
                g3 = q * (Tp[0] + Tp[-W] - B[0] - B[-W]);
                Fym = k_uflux<T>(g1, g2, g3, g2, pp, P[-W], uc - UP[-W], cl, UP[-W], DP[-W], c);
                g3 = (Tp[0] - pp) * idx;
                g1 = q * (P[1] + Tp[1] - P[-1] - Tp[-1]);
                g2 = q * (P[W] + Tp[W] - P[-W] - Tp[-W]);
                Fzp = k_uflux<T>(g1, g2, g3, g3, pp, Tp[0], UT[0] - uc, cl, UT[0], DT[0], c);
                g3 = (pp - B[0]) * idx;
                g1 = q * (P[1] + B[1] - P[-1] - B[-1]);
                g2 = q * (P[W] + B[W] - P[-W] - B[-W]);
                Fzm = k_uflux<T>(g1, g2, g3, g3, pp, B[0], uc - UB[0], cl, UB[0], DB[0], c);
            }
            const T Au = c.Ahalf1 - c.Ahalf2 * pp;
            const T rhsU = (Fxp - Fxm + Fyp - Fym + Fzp - Fzm) * idx + (T)0.5 * ((T)1 + c.omk * uc) * dc;
            U_out[id] = uc + c.dt * rhsU / Au;
            const T pn = pp + c.dt * dc;
            phi_out[id] = fmax((T)-1, fmin((T)1, pn));
        }
        id += d.plane;
        ub = up;
        up = ut;
        if (__syncthreads_or(bad)) {
            if (lead) {
                w.drain(s + 2);
                atomicExch(err, kErrTmaTimeout);
            }
            return;
        }
        if (lead && z + 3 <= ze) w.issue(s + 4);   // into a slot only read since its last barrier
    }
}

// karma3d.f90:290-296 on the device: largest 1-based i with phi(i,1,1) > 0
// and with phi(i,i,i) > 0 (i up to the smallest extent); out[2] ints
template <typename T>
__global__ void k_karma_tip(KarmaDesc d, const T* __restrict__ phi, int* __restrict__ out)
{
    const int nd = min(d.nx, min(d.ny, d.nz));
    int tx = 0, td = 0;
    for (int i = threadIdx.x; i < d.nx; i += blockDim.x)
        if (phi[i] > (T)0) tx = max(tx, i + 1);
    for (int i = threadIdx.x; i < nd; i += blockDim.x)
        if (phi[(long long)i + (long long)i * d.px + (long long)i * d.plane] > (T)0) td = max(td, i + 1);
    for (int o = 16; o > 0; o >>= 1) {
        tx = max(tx, __shfl_xor_sync(0xffffffffu, tx, o));
        td = max(td, __shfl_xor_sync(0xffffffffu, td, o));
    }
    __shared__ int s[2][32];
    const int w = threadIdx.x / 32, l = threadIdx.x % 32;
    if (l == 0) {
        s[0][w] = tx;
        s[1][w] = td;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0, b = 0;
        for (int q = 0; q < (int)(blockDim.x / 32); ++q) {
            a = max(a, s[0][q]);
            b = max(b, s[1][q]);
        }
        out[0] = a;
        out[1] = b;
    }
}

}  // namespace pf3d
