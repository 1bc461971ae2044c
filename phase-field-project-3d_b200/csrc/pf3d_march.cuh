// pf3d_march.cuh -- the z-marching passes of the coupled step, TMA-staged.
//
// A CTA owns a 32 x TY column tile and a z-chunk and marches along z, like
// the passes of pf3d_fused.cuh, with the same per-cell arithmetic (the fast
// form of pf3d_device.cuh), so every output has the bits of those passes.
// What differs is how data moves and how the boundary is treated:
//
//  * Plane staging.  Each plane of the input phase field (tile + 2-cell halo)
//    is one TMA tiled load (cp.async.bulk.tensor.3d, no multicast) issued by
//    one thread into a 6-slot window and completed on that slot's mbarrier;
//    the loads run two planes ahead of the stencil.  Cells outside the domain
//    read as zero.  Every wait is bounded: a load that does not arrive sets
//    the context's status word and the CTA stops (pf3d_tma.cuh).
//  * Node windows.  The anisotropy quantities (eps^2, exy, eyz, ezx) of every
//    node of the tile and its 1-cell ring, and the solute point quantities
//    (Gamma bracket, mu), are computed once per plane into 3-plane windows,
//    one barrier a plane (MarchLayout).
//  * Uniform arithmetic, fan-out stores.  Every cell of every tile -- also
//    the tiles on the domain boundary -- goes through the same arithmetic
//    (two cells per thread as lane pairs when L = 2, packed f32x2 in FP32),
//    in copies of the body that differ in their checks only; in deep domains
//    the cells of a uniform plane keep their value instead (FLAT).
//    The boundary decoration of the reference (plane copies after the sweep,
//    equacao_campo_fase.f90:151-167, concentracao_soluto.f90:116-124) is a
//    per-cell store fan-out: a cell writes its value to every cell whose
//    copy source it is (one store in the interior, up to 27 at a corner).
//    Only the stores diverge; small domains, whose tiles are all boundary
//    tiles, run the paired arithmetic at the interior's cost.
//
// Template switches: HEAT (temperatura), DPPW (write DPP: last sweep), SOL
// (concentracao_soluto from the same input phase field), SMOOTH (the deck
// may draw the smooth noise).  The first pass of a multi-sweep step stores
// the step's REAL(4) noise in the DPP buffer and the last pass reads it back
// (both sweeps use the same it, so the same noise: principal.f90:127-151).
#pragma once
#include <type_traits>
#include "pf3d_launch.h"
#include "pf3d_once.h"
#include "pf3d_pair.cuh"
#include "pf3d_tma.cuh"

namespace pf3d {

// L lanes (cells) per thread: the arithmetic type and its packing
template <typename S, int L> struct Lanes;
template <typename S> struct Lanes<S, 1> {
    using V = S;
    static __device__ __forceinline__ V make(const S* a) { return a[0]; }
    static __device__ __forceinline__ S get(const V& v, int) { return v; }
};
template <typename S> struct Lanes<S, 2> {
    using V = typename PairOf<S>::type;
    static __device__ __forceinline__ V make(const S* a) { return V(a[0], a[1]); }
    static __device__ __forceinline__ S get(const V& v, int l) { return l ? v.y() : v.x(); }
};

// Shared-memory layout of one tile (bytes from a 128-byte aligned base): six
// phase planes (z-1 .. z+4), their barriers, and the node / solute-point
// windows of three planes, a plane's node and point arrays in one slot.
//
// Three planes suffice with one barrier a plane: the cells of plane z read
// plane z's nodes and points at their neighbours' positions, written by other
// threads before the previous plane's barrier, and those of planes z-1 and
// z+1 only at their own position, written by the same thread; so when the
// nodes of plane z+1 overwrite plane z-2's slot, the last cross-thread reader
// of that slot (the cells of plane z-2) is behind the previous plane's
// barrier.
template <typename S, int TY, bool SOL, bool PHASE = true, bool FAST = true>
struct MarchLayout {
    static constexpr int TX = 32;
    static constexpr int ES = (int)sizeof(S);
    // the TMA box starts XOFF cells left of the tile: x * sizeof(S) must be a
    // multiple of 16 bytes (tile origins are multiples of 32 cells)
    static constexpr int XOFF = (sizeof(S) == 8) ? 2 : 4;
    static constexpr int TW = TX + 2 * XOFF;       // phase tile width (box x)
    static constexpr int PH = TY + 4;              // phase tile height (box y)
    static constexpr int NW = TX + 2, NH = TY + 2; // node / point tile (ring 1)
    static constexpr int NB = NW * NH * ES;        // bytes of one node or point array
    static constexpr int NPHI = 6;
    static constexpr int PHI_BYTES = TW * PH * ES;
    static_assert(PHI_BYTES % 128 == 0, "TMA destinations are 128-byte aligned");
    static constexpr int BAR_OFF = NPHI * PHI_BYTES;
    static constexpr int BAD_OFF = BAR_OFF + NPHI * 8;   // set by a thread whose plane load did not arrive
    static constexpr int NODE_OFF = (BAD_OFF + 4 + 127) / 128 * 128;
    // arrays of a slot: eps^2, exy, eyz, ezx; Gamma bracket, mu (reference
    // form 1/GAMMA, mu, 1/GAMMA of the solid)
    static constexpr int Q_SOL = PHASE ? 4 : 0;
    static constexpr int SLOT = (Q_SOL + (SOL ? (FAST ? 2 : 3) : 0)) * NB;
    static constexpr int BYTES = NODE_OFF + 3 * SLOT;
    static constexpr int ALLOC = BYTES + 128;      // slack to align the dynamic base
};

// shared memory by 32-bit address (base + an offset the compiler folds into
// the instruction)
__device__ __forceinline__ void lds(uint32_t a, double& v) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); }
__device__ __forceinline__ void lds(uint32_t a, float& v) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void sts(uint32_t a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v)); }
__device__ __forceinline__ void sts(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v)); }

// temperatura at one own cell (temp_body.inc:31-41): the neighbours of TOLD
// are read only when the deck has heat diffusion (D != 0)
template <typename S, int HQ>
__device__ __forceinline__ S heat_at(const S* __restrict__ T_old, long long id, long long px, long long pl, S PP,
                                     S dppv, const KC<S>& c)
{
    S TE = 0, TW = 0, TN = 0, TS = 0, TT = 0, TB = 0;
    if (c.lap) {
        TE = T_old[id + 1]; TW = T_old[id - 1]; TN = T_old[id + px]; TS = T_old[id - px];
        TT = T_old[id + pl]; TB = T_old[id - pl];
    }
    return heat_new<S, true, HQ>(PP, dppv, TE, TW, TN, TS, TT, TB, c);
}

// the dynamic shared-memory base rounded up to 128 bytes.  The offset is
// added to the shared array itself (not computed through an integer cast of
// its address), so the compiler still knows every pointer derived from it
// is a shared-memory pointer and emits shared loads and stores, not generic
// ones with 64-bit address arithmetic.
__device__ __forceinline__ unsigned char* align128(unsigned char* p)
{
    return p + ((128u - (smem_u32(p) & 127u)) & 127u);
}

// Initialises the six plane barriers of a tile's window (one thread), made
// visible to the TMA unit and to every thread of the CTA.
template <typename LY>
__device__ __forceinline__ void march_init_barriers(unsigned char* smem)
{
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        const uint32_t b0 = smem_u32(smem + LY::BAR_OFF);
        for (int s = 0; s < LY::NPHI; ++s) mbar_init(b0 + 8 * s, 1);
        *reinterpret_cast<int*>(smem + LY::BAD_OFF) = 0;
        fence_mbar_init();
    }
    __syncthreads();
}

// One 32 x TY x zchunk tile (tile coordinates bx, by, bz) of one domain, read
// from the phase field the tensor map `tm` describes.  `par` carries the
// parity of each plane barrier across the tiles a CTA processes (every load
// issued is waited for).  Returns false if a plane load did not arrive in
// time; the CTA must then stop.  SPLIT: a second copy of the plane body for
// the interior planes, without their z checks (FP64 single domains).  INT: every
// column and row of the tile lies in [3, N-4], so no cell needs a check or a
// second store (FP64).
// PHASE = false leaves the phase sweep out (the solute subroutine alone);
// FAST = false is the reference form of the per-subroutine entry points (FP64,
// one lane).  FLAT: planes on which the tile and its 2-cell halo hold nothing but
// 0 or nothing but 1 (melt beyond the interface's tail, the crystal's interior)
// leave out what is exactly zero there (two-sweep steps, below).
//
// The arithmetic is a third to a half of what a plane executes: the rest is
// addresses, conditions and moves, and every thread repeats it in every
// plane.  So shared memory is reached by 32-bit addresses kept per plane of
// the windows and rotated with them (all neighbours are immediate offsets,
// ring items one added delta), global memory by a plane pointer that is the
// same for the CTA plus a 32-bit offset, and the conditions that only tiles on
// the domain's faces need exist in their copy of the body alone.  FP64
// 340x340x200, pass 1 / pass 2: 602 + 815 -> 553 + 744 us (563 / 758 -> 490 /
// 685 instructions a cell on 256x256x128); FP32 256^3: 292 + 351 -> 262 + 305
// us.  Also tried: one loop over own cells and ring items (half the node and
// point code; 2 % slower for the run-time addresses), the prologue as two
// planes of the march without cells (small domains 3 to 18 % slower for the
// barriers), the logarithm's coefficients in the constant bank (pass 2 10 %
// slower), 2 CTAs an SM with 128 registers (4 % slower).
template <typename S, int L, int TY, bool HEAT, bool DPPW, bool SOL, bool SMOOTH, bool SPLIT, bool PHASE, bool FAST,
          int HQ, bool FLAT, bool INT>
__device__ __forceinline__ bool march_tile(const DomainDesc& d, const KC<S>& c, const KC<typename Lanes<S, L>::V>& cv,
                                           const CUtensorMap* tm, const S* __restrict__ c_in,
                                           S* __restrict__ phi_out, S* __restrict__ dpp, S* __restrict__ c_out,
                                           const S* __restrict__ T_old, S* __restrict__ T_new, int zchunk, int bx,
                                           int by, int bz, unsigned char* smem, uint32_t& par)
{
    using LN = Lanes<S, L>;
    using V = typename LN::V;
    using LY = MarchLayout<S, TY, SOL, PHASE, FAST>;
    constexpr int ES = LY::ES, TX = 32, NW = LY::NW, NH = LY::NH, NB = LY::NB, XOFF = LY::XOFF;
    constexpr int TR = TY / L;                                   // thread rows; lane l owns row ty + l*TR
    constexpr int PR = LY::TW * ES, NR = NW * ES;                // bytes of a phase / node row
    constexpr int LP = TR * PR, LNB = TR * NR;                   // from a thread's lane to its next
    constexpr int ran_mode = (HEAT && !DPPW) ? 1 : ((!HEAT && DPPW && SOL) ? 2 : 0);
    constexpr int NRING = (L == 1) ? 2 * NW + 2 * TY : NW + TY;  // ring items (pairs when L = 2)
    constexpr int NT = 32 * TY / L;
    static_assert(TY % L == 0, "tile height must be a multiple of the lanes");
    constexpr int NOUT = FLAT ? (2 * TX + 2 * TY) / L : 0;       // second halo's items (FLAT)
    static_assert(2 * NRING + NOUT <= NT, "the threads of the two rings and of the second halo are disjoint");

    const uint32_t sb = smem_u32(smem);
    const uint32_t bar0 = sb + LY::BAR_OFF;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const long long px = d.px, pl = d.plane;
    const int x0 = bx * TX, y0 = by * TY;
    const int zb = bz * zchunk;
    const int ze = min(zb + zchunk, nz);
    const int zlast = min(nz - 1, ze + 1);   // the last plane any computation of this tile reads
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = tx + TX * ty;
    const bool lead = tid == 0;
    const bool tile_int = INT || (x0 >= 3 && x0 + TX + 3 <= nx && y0 >= 3 && y0 + TY + 3 <= ny);

    // ---- the cells of this thread, and its ring items.  The first NRING
    // threads compute the ring's node quantities, the last NRING its solute
    // points (solute passes), so that no warp carries both ring parts of a
    // plane while the others wait for it at the plane's barrier ----
    const uint32_t own_phi = (uint32_t)((ty + 2) * PR + (tx + XOFF) * ES);   // lane 0, in a phase slot
    const uint32_t own_node = (uint32_t)((ty + 1) * NR + (tx + 1) * ES);     // lane 0, in a node array
    const bool ring = tid < NRING;                      // ring nodes
    const bool outer = FLAT && tid >= NRING && tid < NRING + NOUT;   // second halo's phase values
    const bool ring_s = SOL && tid >= NT - NRING;       // ring solute points
    uint32_t col[L], rcol[L];      // element offsets in the plane: own cells, ring points
    uint32_t rphi[L], rnode[L];    // bytes from the thread's own position (lane 0) to its ring (or second halo) items
    bool own[L], xyin[L], rin[L], rdom[L];
    {
        int r = ring ? tid : (ring_s ? tid - (NT - NRING) : 0), rx[L], ry[L];
        if (outer) {   // what the ring's nodes read beyond the ring, without corners
            r = tid - NRING;
            if (L == 1) {
                const bool lo = r < TX + TY;
                if (!lo) r -= TX + TY;
                rx[0] = r < TX ? 1 + r : (lo ? -1 : NW);
                ry[0] = r < TX ? (lo ? -1 : NH) : 1 + (r - TX);
            } else {
                rx[0] = r < TX ? 1 + r : -1;
                ry[0] = r < TX ? -1 : 1 + (r - TX);
                rx[L - 1] = r < TX ? 1 + r : NW;
                ry[L - 1] = r < TX ? NH : 1 + (r - TX);
            }
        } else if (L == 1) {
            if (r < NW) { rx[0] = r; ry[0] = 0; }
            else if ((r -= NW) < NW) { rx[0] = r; ry[0] = NH - 1; }
            else if ((r -= NW) < TY) { rx[0] = 0; ry[0] = 1 + r; }
            else { r -= TY; rx[0] = NW - 1; ry[0] = 1 + r; }
        } else if (r < NW) {
            rx[0] = rx[L - 1] = r;
            ry[0] = 0;
            ry[L - 1] = NH - 1;
        } else {
            rx[0] = 0;
            rx[L - 1] = NW - 1;
            ry[0] = ry[L - 1] = 1 + (r - NW);
        }
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int x = x0 + tx, y = y0 + ty + l * TR, gx = x0 - 1 + rx[l], gy = y0 - 1 + ry[l];
            own[l] = INT || (x < nx && y < ny);
            xyin[l] = INT || (x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2);
            rdom[l] = (ring || outer) && (INT || (gx >= 0 && gx < nx && gy >= 0 && gy < ny));    // its phase value counts
            rin[l] = ring_s && (INT || (gx >= 0 && gx < nx && gy >= 0 && gy < ny));   // its concentration is read
            col[l] = (uint32_t)x + (uint32_t)y * (uint32_t)px;
            rcol[l] = (uint32_t)gx + (uint32_t)gy * (uint32_t)px;
            rphi[l] = (uint32_t)((ry[l] + 1) * PR + (rx[l] - 1 + XOFF) * ES) - own_phi;
            rnode[l] = (uint32_t)(ry[l] * NR + rx[l] * ES) - own_node;
        }
    }

    // ---- plane loads ----
    uint32_t pend = 0;          // slots with a load issued and not yet seen complete (lead thread)
    auto issue = [&](int p, int s) {   // one thread: plane p into its slot s = p mod 6
        const uint32_t bar = bar0 + 8 * s;
        mbar_arrive_expect_tx(bar, (uint32_t)LY::PHI_BYTES);
        tma_load_3d(sb + s * LY::PHI_BYTES, tm, x0 - XOFF, y0 - 2, p, bar);
        pend |= 1u << s;
    };
    auto wait_plane = [&](int s) -> bool {   // the load into slot s has landed
        const bool ok = mbar_wait(bar0 + 8 * s, (par >> s) & 1u);
        if (ok) {
            par ^= 1u << s;
            pend &= ~(1u << s);
        }
        return ok;
    };
    // after a failed wait: the lead thread waits (bounded) for the loads
    // still in flight, so that no TMA write lands in shared memory the CTA
    // has left
    auto drain = [&]() {
        if (!lead) return;
        for (int s = 0; s < 6; ++s)
            if ((pend >> s) & 1u) mbar_wait(bar0 + 8 * s, (par >> s) & 1u);
    };
    auto phi_at = [&](int s) { return sb + (uint32_t)(s * LY::PHI_BYTES) + own_phi; };        // own cell, slot s
    auto node_at = [&](int s) { return sb + (uint32_t)(LY::NODE_OFF + s * LY::SLOT) + own_node; };

    // own lanes (ring = false) or ring items of a plane: the address of lane l
    auto pa = [&](uint32_t a, int l, bool rg) { return rg ? a + rphi[l] : a + (uint32_t)(l * LP); };
    auto na = [&](uint32_t a, int l, bool rg) { return rg ? a + rnode[l] : a + (uint32_t)(l * LNB); };
    // the difference of two neighbours, lane by lane
    auto ldv = [&](uint32_t a, int off, bool rg) -> V {
        S t[L];
#pragma unroll
        for (int l = 0; l < L; ++l) lds(pa(a, l, rg) + (uint32_t)off, t[l]);
        return LN::make(t);
    };
    auto ldn = [&](uint32_t a, int off) -> V {   // own lanes' neighbour in a node / point array
        S t[L];
#pragma unroll
        for (int l = 0; l < L; ++l) lds(a + (uint32_t)(l * LNB + off), t[l]);
        return LN::make(t);
    };
    auto stn = [&](uint32_t a, int q, V v, bool rg) {
#pragma unroll
        for (int l = 0; l < L; ++l) sts(na(a, l, rg) + (uint32_t)(q * NB), LN::get(v, l));
    };
    // node quantities of a plane into its slot `dst`, from the phase planes
    // below, at and above it (own addresses)
    auto node_one = [&](uint32_t dst, uint32_t m, uint32_t p0, uint32_t pp, bool rg) {
        const V gx = grad<V, FAST>(ldv(p0, ES, rg), ldv(p0, -ES, rg), cv.dx, cv.hx);
        const V gy = grad<V, FAST>(ldv(p0, PR, rg), ldv(p0, -PR, rg), cv.dy, cv.hy);
        const V gz = grad<V, FAST>(ldv(pp, 0, rg), ldv(m, 0, rg), cv.dz, cv.hz);
        const Node<V> q = aniso_node<V, FAST>(gx, gy, gz, cv);
        stn(dst, 0, q.eps * q.eps, rg);   // the stencil reads eps only squared
        stn(dst, 1, q.exy, rg);
        stn(dst, 2, q.eyz, rg);
        stn(dst, 3, q.ezx, rg);
    };
    // own_flat / ring_flat: the warp's gradients there are all zero
    auto node_plane = [&](uint32_t dst, uint32_t m, uint32_t p0, uint32_t pp, bool own_flat, bool ring_flat) {
        auto zero = [&](bool rg) {
            const Node<S> q = aniso_flat<S>(c);
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const uint32_t o = na(dst, l, rg);
                sts(o, q.eps * q.eps);
                sts(o + NB, (S)0);
                sts(o + 2 * NB, (S)0);
                sts(o + 3 * NB, (S)0);
            }
        };
        if (FLAT && own_flat) zero(false);
        else node_one(dst, m, p0, pp, false);
        if (ring) {
            if (FLAT && ring_flat) zero(true);
            else node_one(dst, m, p0, pp, true);
        }
    };
    // solute point quantities of a plane into its slot, from its phase plane
    // and the concentration at the own (co) and ring (cr) points
    auto sol_one = [&](uint32_t dst, uint32_t p0, const S* cc, bool rg) {
        const SolNode<V> q = sol_node<V, FAST, HQ>(ldv(p0, 0, rg), LN::make(cc), cv);
        stn(dst, LY::Q_SOL, FAST ? q.br : q.il, rg);
        stn(dst, LY::Q_SOL + 1, q.mu, rg);
        if constexpr (!FAST) stn(dst, LY::Q_SOL + 2, q.is, rg);
    };
    auto sol_plane = [&](uint32_t dst, uint32_t p0, const S* co, const S* cr) {
        sol_one(dst, p0, co, false);
        if (ring_s) sol_one(dst, p0, cr, true);
    };
    // concentration of plane s at the own and ring points (a benign value
    // outside the domain, so that no logarithm there leaves the normal range)
    auto load_c = [&](int s, const S* cz, S* co, S* cr, bool zin) {
#pragma unroll
        for (int l = 0; l < L; ++l) {
            co[l] = (zin && own[l]) ? cz[col[l]] : (S)0.02;
            if (SOL) cr[l] = (zin && rin[l]) ? cz[rcol[l]] : (S)0.02;
        }
    };

    // ---- prologue: planes zb-2 .. zb+3 in flight, nodes zb-1, zb ----
    if (lead) {
        for (int p = zb - 2; p <= zb + 3; ++p)
            if (p >= 0 && p <= zlast) issue(p, (p + 6) % 6);
    }
    S co[L], c1[L], c2[L];      // concentration at the own points of planes z, z+1, z+2
    S cr1[L], cr2[L];           // ... at the ring points of planes z+1, z+2
    S nd[L], nt[L];             // centre values of the next plane: DPP (or the noise), TOLD
#pragma unroll
    for (int l = 0; l < L; ++l) nd[l] = nt[l] = c1[l] = c2[l] = cr1[l] = cr2[l] = 0;
    // DPP / noise and TOLD of the own cells of plane z.  TOLD is read only
    // where the heat equation keeps it (outside 2..N-1): inside, TNEW is TP
    // plus the latent term (and the Laplacian reads its own neighbours)
    auto load_centre = [&](int z, long long zo, bool zi) {
        if (!(HEAT || ran_mode == 2)) return;
        const S* const dz = dpp + zo;
#pragma unroll
        for (int l = 0; l < L; ++l) {
            if (!own[l]) continue;
            nd[l] = dz[col[l]];
            if (HEAT && !(zi && xyin[l])) nt[l] = (T_old + zo)[col[l]];
        }
    };
    auto zin = [&](int z) { return z >= 1 && z <= nz - 2; };
    auto zdom = [&](int z) { return z >= 0 && z < nz; };
    bool bad = false;
    const long long zo0 = (long long)zb * pl;
    auto wait_first = [&]() {
        for (int p = zb - 2; p <= zb + 1; ++p)
            if (p >= 0 && p <= zlast) bad |= !wait_plane((p + 6) % 6);
    };
    uint32_t n0 = node_at(0), np = node_at(1), nm = node_at(2);   // slots of planes z, z+1, z-1
    if (SOL) {
        S ca[L], cra[L];
        load_c(zb - 1, c_in + zo0 - pl, ca, cra, zdom(zb - 1));
        load_c(zb, c_in + zo0, co, cr2, true);
        load_c(zb + 1, c_in + zo0 + pl, c1, cr1, zdom(zb + 1));
        wait_first();
        if (zb - 1 >= 0) sol_plane(nm, phi_at((zb + 5) % 6), ca, cra);
        sol_plane(n0, phi_at(zb % 6), co, cr2);
    } else {
        load_c(zb, c_in + zo0, co, cr2, true);
        wait_first();
    }
    load_centre(zb, zo0, zin(zb));
    if (PHASE && zin(zb - 1)) node_plane(nm, phi_at((zb + 4) % 6), phi_at((zb + 5) % 6), phi_at(zb % 6), false, false);
    if (PHASE && zin(zb)) node_plane(n0, phi_at((zb + 5) % 6), phi_at(zb % 6), phi_at((zb + 1) % 6), false, false);

    // the smooth noise's lattice layers below and above the plane, blended at the
    // own columns: they change every six planes, and the upper one becomes the
    // lower, so a cell costs a blend of two numbers and two thirds of a hash
    // where it took eight hashes (97x131x201 FP64, one
    // sweep: 211 -> 177 us a step)
    double slo[L], shi[L];
    const bool smooth = SMOOTH && c.rt == 2;
    auto smooth_layer = [&](int l, int k0) { return ruido_layer64(x0 + tx + 1, y0 + ty + l * TR + 1, k0, c.it); };
#pragma unroll
    for (int l = 0; l < L; ++l) {
        slo[l] = smooth ? smooth_layer(l, (zb + 1) / 6) : 0.0;
        shi[l] = smooth ? smooth_layer(l, (zb + 1) / 6 + 1) : 0.0;
    }
    uint64_t hin[L];   // noise hash input of the own cells, carried along z (k = z + 1)
#pragma unroll
    for (int l = 0; l < L; ++l)
        hin[l] = hash_base(x0 + tx + 1, y0 + ty + l * TR + 1, c.it, 1) + (uint64_t)(zb + 1) * kHashK;
    uint32_t am = phi_at((zb + 5) % 6), a0 = phi_at(zb % 6), ap = phi_at((zb + 1) % 6);   // planes z-1, z, z+1
    int sq = (zb + 2) % 6;       // phase slot of plane z+2
    long long zoff = zo0;
    // what planes z-2 .. z+1 hold all over the tile and its 2-cell halo (inside
    // the domain), two bits a plane, z+1 in the lowest: 1 exactly 0, 2 exactly 1,
    // 0 anything else or not known yet
    int uh = 0;

    // One plane of the march.  IN: every z-dependent condition of the plane
    // is known true (z in [3, N-4], the planes it reads and the load it
    // issues all inside the domain and the chunk), so that copy of the body
    // carries none of the checks; the other copy serves the first and last
    // planes.  Returns false when a plane load did not arrive.  Always
    // inlined: an outlined copy would pass every captured value through the
    // stack (measured: 5x slower).
    auto plane = [&](int z, auto in_tag) __attribute__((always_inline)) -> bool {
        constexpr bool IN = decltype(in_tag)::value;
        const uint32_t aq = phi_at(sq);
        S dcur[L], tcur[L];
#pragma unroll
        for (int l = 0; l < L; ++l) { dcur[l] = nd[l]; tcur[l] = nt[l]; }
        if (IN || z + 1 < ze) load_centre(z + 1, zoff + pl, IN || zin(z + 1));
        if (SOL) load_c(z + 2, c_in + zoff + 2 * pl, c2, cr2, IN || zdom(z + 2));
        else load_c(z + 1, c_in + zoff + pl, c1, cr1, IN || zdom(z + 1));

        if (!IN && z == ze - 1) pdl_release();   // the last plane is never an IN one
        // A: plane z+2 has landed
        if (IN || z + 2 <= zlast) bad |= !wait_plane(sq);
        // whether plane z+2 holds one of the two values all over, and the
        // concentrations of plane z keep the driving force's logarithm finite
        // (KC::cflat); and whether the warp's nodes of plane z+1 are flat
        bool mixed = false, own_flat = false, ring_flat = false;
        int u2 = uh & 3;
        if constexpr (FLAT) {
            if (IN || z + 2 <= zlast) {
                S v;
                lds(sb + (uint32_t)(sq * LY::PHI_BYTES + 2 * PR + XOFF * ES), v);   // the tile's first cell
                u2 = is_bits0(v) ? 1 : is_bits1(v) ? 2 : 0;
                bool od = false, rd = false;   // own cells, ring and second halo items that differ from it
#pragma unroll
                for (int l = 0; l < L; ++l) {
                    S a, b;
                    lds(pa(aq, l, false), a);
                    lds(pa(aq, l, true), b);
                    od = od || (own[l] && a != v);
                    rd = rd || (rdom[l] && b != v);
                }
                mixed = u2 == 0 || od || rd;
                if (u2 != 0 && (uh & 15) == 5 * u2) {   // planes z and z+1 hold it too (CTA-uniform)
                    own_flat = !__any_sync(0xffffffffu, od);
                    ring_flat = !__any_sync(0xffffffffu, rd);
                }
            }
#pragma unroll
            for (int l = 0; l < L; ++l) mixed = mixed || (own[l] && !(co[l] > (S)0 && co[l] < c.cflat));
        }
        // B, C: nodes and solute points of plane z+1
        if (PHASE && (IN || zin(z + 1))) node_plane(np, a0, ap, aq, own_flat, ring_flat);
        if (SOL && (IN || z + 1 <= nz - 1)) sol_plane(np, ap, c1, cr1);
        // D: one barrier orders the plane; everyone learns of a failed load, and
        // whether the plane is mixed
        if constexpr (FLAT) {
            int* const flag = reinterpret_cast<int*>(smem + LY::BAD_OFF);
            if (bad) *flag = 1;
            if (__syncthreads_or(bad || mixed)) {
                if (*(volatile int*)flag) {
                    drain();
                    return false;
                }
                u2 = 0;
            }
        } else {
            if (__syncthreads_or(bad)) {
                drain();
                return false;
            }
        }
        // E: the load of plane z+4 into the slot plane z-2 has left (read
        // only, by threads that are behind the barrier)
        if (lead && (IN || z + 4 <= zlast)) issue(z + 4, sq + 2 >= 6 ? sq - 4 : sq + 2);

        // F: the cells of plane z.  Where all that their sweep reads -- planes
        // z-2 .. z+2 of the tile and its 2-cell halo -- holds nothing but 0 or
        // nothing but 1, every difference, g', h' and the noise's
        // phi^2 (1-phi)^2 are zero and the sweep changes nothing: the cells
        // keep their value and DPP is zero, the bits the arithmetic gives as
        // long as its logarithm is finite.  (The noise is not drawn either:
        // the second sweep multiplies it by the same zero.)  All that is read
        // counts, not only what the zeros multiply: a node beside a NaN makes
        // NaN of a zero difference.
        if constexpr (FLAT) uh = ((uh << 2) | u2) & 0x3ff;
        const bool flat = FLAT && u2 != 0 && uh == 0x155 * u2;
        const bool zi = IN || zin(z);                     // T interior / phase source / solute interior
        const bool zph = IN || (z >= 2 && z <= nz - 3);   // phase interior
        const V PP = ldv(a0, 0, false);
        const V CPP = LN::make(co);

        // the REAL(4) noise of the own cells, exact in S
        S ran[L];
#pragma unroll
        for (int l = 0; l < L; ++l) {
            if (!PHASE || flat) {
                ran[l] = (S)0;
            } else if (ran_mode == 2) {
                ran[l] = dcur[l];
            } else if constexpr (SMOOTH) {
                if (smooth) {
                    if ((z + 1) % 6 == 0 && z > zb) {
                        slo[l] = shi[l];
                        shi[l] = smooth_layer(l, (z + 1) / 6 + 1);
                    }
                    ran[l] = (S)__double2float_rn(ruido_blend64(slo[l], shi[l], z + 1));
                } else {
                    ran[l] = (S)__double2float_rn(ran64(hash63_mix(hin[l])));
                }
            } else {
                ran[l] = (S)__double2float_rn(ran64(hash63_mix(hin[l])));
            }
            hin[l] += kHashK;
        }

        V ppn = PP;
        if (PHASE && zph && !flat) {
            Nbr<V> nb;
            nb.PP = PP;
            nb.PN = ldv(a0, PR, false); nb.PS = ldv(a0, -PR, false);
            nb.PE = ldv(a0, ES, false); nb.PW = ldv(a0, -ES, false);
            nb.PT = ldv(ap, 0, false); nb.PB = ldv(am, 0, false);
            nb.PNT = ldv(ap, PR, false); nb.PNB = ldv(am, PR, false);
            nb.PST = ldv(ap, -PR, false); nb.PSB = ldv(am, -PR, false);
            nb.PET = ldv(ap, ES, false); nb.PEB = ldv(am, ES, false);
            nb.PWT = ldv(ap, -ES, false); nb.PWB = ldv(am, -ES, false);
            nb.PNE = ldv(a0, PR + ES, false); nb.PSE = ldv(a0, -PR + ES, false);
            nb.PNW = ldv(a0, PR - ES, false); nb.PSW = ldv(a0, -PR - ES, false);
            Node<V> E, W, N, So, Tt, B;
            E.eps = ldn(n0, ES); E.exy = ldn(n0, ES + NB); E.ezx = ldn(n0, ES + 3 * NB);
            W.eps = ldn(n0, -ES); W.exy = ldn(n0, -ES + NB); W.ezx = ldn(n0, -ES + 3 * NB);
            N.eps = ldn(n0, NR); N.exy = ldn(n0, NR + NB); N.eyz = ldn(n0, NR + 2 * NB);
            So.eps = ldn(n0, -NR); So.exy = ldn(n0, -NR + NB); So.eyz = ldn(n0, -NR + 2 * NB);
            Tt.eps = ldn(np, 0); Tt.eyz = ldn(np, 2 * NB); Tt.ezx = ldn(np, 3 * NB);
            B.eps = ldn(nm, 0); B.eyz = ldn(nm, 2 * NB); B.ezx = ldn(nm, 3 * NB);
            E.eyz = W.eyz = N.ezx = So.ezx = Tt.exy = B.exy = V((S)0);   // unused by the body
            ppn = phase_ppnew<V, FAST, true, HQ>(nb, E, W, N, So, Tt, B, CPP, LN::make(ran), cv);
        }
        V cn = CPP;
        if (SOL && zi) {
            constexpr int Q = LY::Q_SOL * NB;
            auto sol_at = [&](uint32_t a, int off) {
                SolNode<V> q;
                q.br = q.il = ldn(a, off + Q);
                q.mu = ldn(a, off + Q + NB);
                if constexpr (!FAST) q.is = ldn(a, off + Q + 2 * NB);
                return q;
            };
            cn = conc_new<V, FAST>(PP, CPP, sol_at(n0, 0), sol_at(n0, ES), sol_at(n0, -ES), sol_at(n0, NR),
                                   sol_at(n0, -NR), sol_at(np, 0), sol_at(nm, 0), cv);
        }
        const V U = clamp01(ppn);
        const V DP = ppn - PP;

        if (tile_int && (IN || (z >= 3 && z <= nz - 4))) {
            // every cell of the tile plane is interior and its own only
            // preimage (CTA-uniform branch)
#pragma unroll
            for (int l = 0; l < L; ++l) {
                const uint32_t id = col[l];
                if (HEAT) (T_new + zoff)[id] = heat_at<S, HQ>(T_old, zoff + id, px, pl, LN::get(PP, l), dcur[l], c);
                if (ran_mode == 1) (dpp + zoff)[id] = ran[l];
                if (DPPW) (dpp + zoff)[id] = LN::get(DP, l);
                if (PHASE) (phi_out + zoff)[id] = LN::get(U, l);
                if (SOL) (c_out + zoff)[id] = LN::get(cn, l);
            }
        } else {
#pragma unroll
            for (int l = 0; l < L; ++l) {
                if (!own[l]) continue;
                const int x = x0 + tx, y = y0 + ty + l * TR;
                const long long id = zoff + col[l];
                const bool xin = x >= 1 && x <= nx - 2;          // T interior, phase source, solute interior
                const bool src = xyin[l] && zi;                  // T interior; phase copy source
                if (HEAT) {
                    S tn = tcur[l];
                    if (src) tn = heat_at<S, HQ>(T_old, id, px, pl, LN::get(PP, l), dcur[l], c);
                    T_new[id] = tn;
                }
                if (PHASE && src) {
                    const bool inner = x >= 2 && x <= nx - 3 && y >= 2 && y <= ny - 3 && zph;
                    S u = LN::get(PP, l);
                    if (inner) {
                        if (ran_mode == 1) dpp[id] = ran[l];
                        if (DPPW) dpp[id] = LN::get(DP, l);
                        u = LN::get(U, l);
                    }
                    if (x >= 3 && x <= nx - 4 && y >= 3 && y <= ny - 4 && z >= 3 && z <= nz - 4) {
                        phi_out[id] = u;   // its own only preimage
                    } else {
                        int xl, xh, yl, yh, zl, zh;
                        fpre_range(x, nx, &xl, &xh);
                        fpre_range(y, ny, &yl, &yh);
                        fpre_range(z, nz, &zl, &zh);
                        for (int zz = zl; zz <= zh; ++zz)
                            for (int yy = yl; yy <= yh; ++yy)
                                for (int xx = xl; xx <= xh; ++xx)
                                    phi_out[(long long)xx + (long long)yy * px + (long long)zz * pl] = u;
                    }
                }
                if (SOL) {
                    // concentracao_soluto.f90:116-124 as a fan-out: the point
                    // writes its value to the face cells copied from it
                    const S uc = src ? LN::get(cn, l) : co[l];
                    if (src) c_out[id] = uc;
                    if (z == 1) c_out[id - pl] = uc;
                    if (z == nz - 2) c_out[id + pl] = uc;
                    if (zi && x == 1) c_out[id - 1] = uc;
                    if (zi && x == nx - 2) c_out[id + 1] = uc;
                    if (zi && xin && y == 1) c_out[id - px] = uc;
                    if (zi && xin && y == ny - 2) c_out[id + px] = uc;
                }
            }
        }

        // the next plane's view of the windows and the carried concentrations
#pragma unroll
        for (int l = 0; l < L; ++l) {
            co[l] = c1[l];
            if (SOL) {
                c1[l] = c2[l];
                cr1[l] = cr2[l];
            }
        }
        am = a0;
        a0 = ap;
        ap = aq;
        sq = sq == 5 ? 0 : sq + 1;
        const uint32_t t = nm;
        nm = n0;
        n0 = np;
        np = t;
        zoff += pl;
        return true;
    };
    if constexpr (SPLIT) {
        // interior planes [zi0, zi1): z >= 3, z <= nz - 4 and z + 4 <= zlast
        const int zi0 = max(zb, 3), zi1 = min(min(ze, nz - 3), zlast - 3);
        int z = zb;
        for (; z < ze && z < zi0; ++z)
            if (!plane(z, std::false_type{})) return false;
        for (; z < zi1; ++z)
            if (!plane(z, std::true_type{})) return false;
        for (; z < ze; ++z)
            if (!plane(z, std::false_type{})) return false;
    } else {
        for (int z = zb; z < ze; ++z)
            if (!plane(z, std::false_type{})) return false;
    }
    return true;
}

// Whether a chunk of the tile looks uniform: four cells of its middle column
// hold 0, or all 1 (the same answer in every thread).  A guess: the copy of
// the body it selects is right for any plane.
template <typename S>
__device__ __forceinline__ bool looks_flat(const DomainDesc& d, const S* phi, int x0, int y0, int zb, int ze)
{
    const S* const p = phi + min(x0 + 16, d.nx - 1) + (long long)min(y0 + 4, d.ny - 1) * d.px;
    const int n = ze - 1 - zb;
    S v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = p[(long long)(zb + i * n / 3) * d.plane];
    bool zero = true, one = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        zero = zero && is_bits0(v[i]);
        one = one && is_bits1(v[i]);
    }
    return zero || one;
}

// The tile in the copy of the body that its position in the domain needs.  The
// FP32 passes, with twice the CTAs in flight and half the instructions a cell,
// are short of instruction cache and run the one copy with all its checks
// (256^3: 668 us a step with interior copies of tiles and planes, 561 without;
// FP64 340x340x200: 1290 us with, 1405 without).
// FLAT: FP64 chunks that look uniform take the copy that leaves out what is zero
// on uniform planes; its checks cost a mixed plane 5 %, so the others take the
// plain one.  FP32 runs the one copy with those checks, for the same reason as
// above (with both, 256x256x512 took 1.23 ms a step, against 1.06).
template <typename S, int L, int TY, bool HEAT, bool DPPW, bool SOL, bool SMOOTH, bool SPLIT, bool PHASE, bool FAST,
          int HQ, bool FLAT>
__device__ __forceinline__ bool march_any(const DomainDesc& d, const KC<S>& c, const KC<typename Lanes<S, L>::V>& cv,
                                          const CUtensorMap* tm, const S* phi_in, const S* c_in, S* phi_out, S* dpp,
                                          S* c_out, const S* T_old, S* T_new, int zchunk, int bx, int by, int bz,
                                          unsigned char* smem, uint32_t& par)
{
    const int x0 = bx * 32, y0 = by * TY;
    constexpr bool copies = sizeof(S) == 8;
    const bool inside = copies && x0 >= 3 && x0 + 32 + 3 <= d.nx && y0 >= 3 && y0 + TY + 3 <= d.ny;
    if constexpr (FLAT && copies) {
        if (inside && looks_flat<S>(d, phi_in, x0, y0, bz * zchunk, min(bz * zchunk + zchunk, d.nz)))
            return march_tile<S, L, TY, HEAT, DPPW, SOL, SMOOTH, SPLIT, PHASE, FAST, HQ, true, true>(
                d, c, cv, tm, c_in, phi_out, dpp, c_out, T_old, T_new, zchunk, bx, by, bz, smem, par);
    }
    if (inside)
        return march_tile<S, L, TY, HEAT, DPPW, SOL, SMOOTH, SPLIT, PHASE, FAST, HQ, false, true>(
            d, c, cv, tm, c_in, phi_out, dpp, c_out, T_old, T_new, zchunk, bx, by, bz, smem, par);
    return march_tile<S, L, TY, HEAT, DPPW, SOL, SMOOTH, SPLIT, PHASE, FAST, HQ, FLAT && !copies, false>(
        d, c, cv, tm, c_in, phi_out, dpp, c_out, T_old, T_new, zchunk, bx, by, bz, smem, par);
}

// resident CTAs per SM the register budget is sized for (shared memory
// allows no more): FP64 3 (80 registers a thread), or 2 for the reference form
// of the sweep and for the whole step of one sweep in one pass (300x300x200:
// 755 us a step with 3 and its spills, 683 with 2); FP32 pairs 6, FP32 single
// cells 3
template <typename S, int L, bool PHASE = true, bool FAST = true, bool ONE = false>
struct MarchOcc {
    static constexpr int v = (sizeof(S) == 8) ? (((PHASE && !FAST) || ONE) ? 2 : 3) : (L == 2 ? 6 : 3);
};

// single domain: one CTA per tile; the phase field comes through `tm`
template <typename S, int L, int TY, bool HEAT, bool DPPW, bool SOL, bool SMOOTH, bool PHASE, bool FAST, int HQ,
          bool FLAT>
__global__ void __launch_bounds__(32 * TY / L, (MarchOcc<S, L, PHASE, FAST, HEAT && SOL>::v))
    k_march(const __grid_constant__ CUtensorMap tm, DomainDesc d, const KC<S> c,
            const KC<typename Lanes<S, L>::V> cv, const S* __restrict__ phi_in, const S* __restrict__ c_in,
            S* __restrict__ phi_out,
            S* __restrict__ dpp, S* __restrict__ c_out, const S* __restrict__ T_old, S* __restrict__ T_new,
            int zchunk, int* __restrict__ err)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = align128(smem_raw);
    if (threadIdx.x == 0 && threadIdx.y == 0) prefetch_tensormap(&tm);
    march_init_barriers<MarchLayout<S, TY, SOL, PHASE, FAST>>(smem);
    pdl_wait();
    uint32_t par = 0;
    if (!march_any<S, L, TY, HEAT, DPPW, SOL, SMOOTH, sizeof(S) == 8, PHASE, FAST, HQ, FLAT>(
            d, c, cv, &tm, phi_in, c_in, phi_out, dpp, c_out, T_old, T_new, zchunk, blockIdx.x, blockIdx.y, blockIdx.z, smem,
            par)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) atomicExch(err, kErrTmaTimeout);
    }
}

// many domains: a persistent grid walks the work list (head[0] items, chunks
// of head[1] planes).  PASS 0 is the first
// pass of a step (temperatura + sweep 1, or the whole step with one sweep),
// PASS 1 the last (sweep 2 + solute).  tmaps[2 d + b] describes buffer b of
// domain d's phase field.  Items are handed out dynamically: each CTA starts
// with item blockIdx.x and then takes the next unclaimed item from the
// counter *ctr (zero before the launch), so CTAs that drew short items (thin
// z-chunks, small domains at the end of the largest-first list) keep
// working while others finish long ones.
template <typename S, int L, int TY, int PASS, bool ONE_SWEEP, bool SMOOTH>
__global__ void __launch_bounds__(32 * TY / L, (MarchOcc<S, L, true, true, ONE_SWEEP>::v))
    k_march_batch(const BatchDomain* __restrict__ doms, const CUtensorMap* __restrict__ tmaps,
                  const BatchStep* __restrict__ steps, const BatchItem* __restrict__ items,
                  const int* __restrict__ head, int* __restrict__ ctr, int* __restrict__ err)
{
    using V = typename Lanes<S, L>::V;
    constexpr bool SOL = PASS == 1 || ONE_SWEEP;
    __shared__ int s_next;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(16) KC<S> skc;   // the loop constants of the current item
    __shared__ __align__(16) KC<V> skv;   // the same, broadcast to the lanes (L = 2)
    constexpr int nf = (int)(offsetof(KC<S>, hq) / sizeof(S));
    constexpr int NT = 32 * TY / L;
    unsigned char* smem = align128(smem_raw);
    march_init_barriers<MarchLayout<S, TY, SOL>>(smem);
    uint32_t par = 0;
    const int n = head[0], zchunk = head[1];
    const int tid = threadIdx.x + 32 * threadIdx.y;
    for (int w = blockIdx.x; w < n;) {
        const BatchItem it = items[w];
        const BatchStep& st = steps[it.dom];
        // the next item, claimed now so the atomic's latency hides behind this one
        __syncthreads();            // every thread has read the previous claim
        if (tid == 0) s_next = (int)gridDim.x + atomicAdd(ctr, 1);
        if (!st.active) {           // uniform across the CTA
            __syncthreads();
            w = s_next;
            continue;
        }
        const BatchDomain& D = doms[it.dom];
        const int q = st.q_phi, qc = st.q_c, qt = st.q_T;
        __syncthreads();            // the previous item is done with the constants and the windows
        static_assert(sizeof(KC<S>) % 4 == 0, "KC is copied as words");
        for (int i = tid; i < (int)(sizeof(KC<S>) / 4); i += NT)
            reinterpret_cast<int*>(&skc)[i] = reinterpret_cast<const int*>(st.kc)[i];
        if (L == 2) {
            __syncthreads();
            for (int i = tid; i < nf; i += NT)
                reinterpret_cast<V*>(&skv)[i] = V(reinterpret_cast<const S*>(&skc)[i]);
            if (tid == 0) {
                skv.hq = skc.hq;
                skv.rt = skc.rt;
                skv.it = skc.it;
                skv.lap = skc.lap;
            }
        }
        __syncthreads();
        const KC<V>& kv = (L == 2) ? skv : *reinterpret_cast<const KC<V>*>(&skc);
        bool ok;
        if (PASS == 0) {
            const CUtensorMap* tm = tmaps + 2 * it.dom + q;
            if (ONE_SWEEP)
                ok = march_any<S, L, TY, true, true, true, SMOOTH, false, true, true, 2, false>(
                    D.d, skc, kv, tm, nullptr, (const S*)D.c[qc], (S*)D.phi[1 - q], (S*)D.dpp, (S*)D.c[1 - qc],
                    (const S*)D.T[qt], (S*)D.T[1 - qt], zchunk, it.bx, it.by, it.bz, smem, par);
            else
                ok = march_any<S, L, TY, true, false, false, SMOOTH, false, true, true, 2, false>(
                    D.d, skc, kv, tm, nullptr, (const S*)D.c[qc], (S*)D.phi[1 - q], (S*)D.dpp, nullptr, (const S*)D.T[qt],
                    (S*)D.T[1 - qt], zchunk, it.bx, it.by, it.bz, smem, par);
        } else {
            const CUtensorMap* tm = tmaps + 2 * it.dom + (1 - q);
            ok = march_any<S, L, TY, false, true, true, false, false, true, true, 2, false>(
                D.d, skc, kv, tm, nullptr, (const S*)D.c[qc], (S*)D.phi[q], (S*)D.dpp, (S*)D.c[1 - qc], nullptr, nullptr,
                zchunk, it.bx, it.by, it.bz, smem, par);
        }
        if (!ok) {
            if (tid == 0) atomicExch(err, kErrTmaTimeout);
            return;
        }
        __syncthreads();            // the claim is visible (and the tile is done)
        w = s_next;
    }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------

// KC with every scalar constant broadcast to the lanes (host side)
template <typename S, int L>
KC<typename Lanes<S, L>::V> kc_lanes(const KC<S>& k)
{
    using V = typename Lanes<S, L>::V;
    if constexpr (L == 1) {
        return k;
    } else {
        KC<V> r;
        constexpr int n = (int)(offsetof(KC<S>, hq) / sizeof(S));
        static_assert(offsetof(KC<V>, hq) == n * sizeof(V), "KC layout");
        const S* src = reinterpret_cast<const S*>(&k);
        V* dst = reinterpret_cast<V*>(&r);
        for (int i = 0; i < n; ++i) dst[i] = V::splat(src[i]);
        r.hq = k.hq;
        r.rt = k.rt;
        r.it = k.it;
        r.lap = k.lap;
        return r;
    }
}

template <typename S, int L, int TY, bool HEAT, bool DPPW, bool SOL, bool SMOOTH, bool PHASE, bool FAST, int HQ,
          bool FLAT = false>
cudaError_t launch_march_t(const CUtensorMap& tm, const DomainDesc& d, const StepArgs& s, const void* phi_in,
                           const void* c_in,
                           void* phi_out, void* dpp, void* c_out, const void* T_old, void* T_new, int zchunk,
                           int* err, cudaStream_t st)
{
    using LY = MarchLayout<S, TY, SOL, PHASE, FAST>;
    auto kern = k_march<S, L, TY, HEAT, DPPW, SOL, SMOOTH, PHASE, FAST, HQ, FLAT>;
    static DeviceOnce once;   // one attribute call per instantiation and device
    const cudaError_t e = once(
        [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::ALLOC); });
    if (e != cudaSuccess) return e;
    if (zchunk <= 0) zchunk = d.nz;
    KC<S> kc;
    kc.load(d, s);
    const auto kv = kc_lanes<S, L>(kc);
    dim3 grid((d.nx + 31) / 32, (d.ny + TY - 1) / TY, (d.nz + zchunk - 1) / zchunk);
    return launch_pdl(kern, grid, dim3(32, TY / L), LY::ALLOC, st, tm, d, kc, kv, (const S*)phi_in, (const S*)c_in, (S*)phi_out,
                      (S*)dpp, (S*)c_out, (const S*)T_old, (S*)T_new, zchunk, err);
}

// the passes of a step (32 x 8 tiles).  lanes: cells per thread (1 or 2); the
// smooth noise runs one cell per thread.  h(phi) is known at compile time.
//
// flat: with what serves uniform planes.  How much of a domain is uniform grows
// with its depth around the interface (in a run under way the FP64 phase is
// exactly 1 some 37 cells inside the crystal, the FP32 phase also exactly 0 some
// 105 cells into the melt; a young run's melt is exactly 0 altogether), and a
// chunk learns of its first planes' uniformity four planes late.  So it serves
// domains of kFlatDepth planes and chunks of kFlatChunk and more, of steps with
// two sweeps (with more, a middle sweep may need the noise of a cell the first
// one left alone).  The depth stands in for the state, which the host does not
// know; the line lies where a grown crystal begins to gain.  Microseconds a step,
// without / with.  Crystal a third grown: FP64 340x340 x 200 1294 / 1326, x 330
// 2069 / 2103, x 448 2847 / 2895, x 700 4236 / 4150; FP32 192x192 x 256 380 / 387,
// x 384 572 / 581, x 448 663 / 667, 256x256 x 512 1096 / 1040, x 700 1533 / 1447.
// Seeded start: FP64 192x192 x 200 470 / 481, x 384 880 / 902, 256x256x512
// 1864 / 1629, 512x512x1024 12648 / 8959; FP32 192x192 x 200 302 / 267, x 384
// 571 / 476, 256x256x512 1096 / 870, 1024^3 27723 / 18911.
template <typename S>
cudaError_t launch_march_first(const CUtensorMap& tm, const DomainDesc& d, const StepArgs& s, const Fields& f,
                               bool with_solute, int lanes, bool flat, int zchunk, int* err, cudaStream_t st)
{
#define PF3D_MF(L, SO, SM, HQ, FL)                                                                              \
    launch_march_t<S, L, 8, true, SO, SO, SM, true, true, HQ, FL>(tm, d, s, f.phi_old, f.c_old, f.phi_mid, f.dpp, \
                                                                  SO ? f.c_new : nullptr, f.T_old, f.T_new,     \
                                                                  zchunk, err, st)
#define PF3D_MQ(L, SO, SM, FL) (d.hq ? PF3D_MF(L, SO, SM, 1, FL) : PF3D_MF(L, SO, SM, 0, FL))
    constexpr int L0 = sizeof(S) == 4 ? 2 : 1;   // the default lanes, which the flat copies have
    if (d.rt == 2) return with_solute ? PF3D_MQ(1, true, true, false) : PF3D_MQ(1, false, true, false);
    if (with_solute) return lanes == 2 ? PF3D_MQ(2, true, false, false) : PF3D_MQ(1, true, false, false);
    if (flat && lanes == L0) return PF3D_MQ(L0, false, false, true);
    return lanes == 2 ? PF3D_MQ(2, false, false, false) : PF3D_MQ(1, false, false, false);
#undef PF3D_MQ
#undef PF3D_MF
}

template <typename S>
cudaError_t launch_march_last(const CUtensorMap& tm, const DomainDesc& d, const StepArgs& s, const Fields& f,
                              int lanes, bool flat, int zchunk, int* err, cudaStream_t st)
{
#define PF3D_ML(L, HQ, FL)                                                                                      \
    launch_march_t<S, L, 8, false, true, true, false, true, true, HQ, FL>(tm, d, s, f.phi_mid, f.c_old, f.phi_new, f.dpp, \
                                                                          f.c_new, nullptr, nullptr, zchunk,   \
                                                                          err, st)
#define PF3D_MQ(L, FL) (d.hq ? PF3D_ML(L, 1, FL) : PF3D_ML(L, 0, FL))
    constexpr int L0 = sizeof(S) == 4 ? 2 : 1;
    if (flat && lanes == L0) return PF3D_MQ(L0, true);
    return lanes == 2 ? PF3D_MQ(2, false) : PF3D_MQ(1, false);
#undef PF3D_MQ
#undef PF3D_ML
}

// One subroutine alone, for the per-subroutine entry points and the middle
// sweeps of a step with more than two: equacao_campo_fase (dpp null: DPP is
// not written) and concentracao_soluto without its copy to conc_soluto_old.
// FP64 runs the reference form, FP32 the fast form; every node's and point's
// quantities are computed once and shared, where one thread per cell computed
// six nodes and seven points a cell.  128x128x256 FP64: a whole step of
// subroutine calls 1146 -> 453 us (a sweep 440 -> 149 us, the solute step with
// its copy 237 -> 115 us; with the general divisions the sweep took 336 us).
template <typename S>
cudaError_t launch_march_sweep(const CUtensorMap& tm, const DomainDesc& d, const StepArgs& s, const void* c_in,
                               void* phi_out, void* dpp, int zchunk, int* err, cudaStream_t st)
{
    constexpr bool FAST = sizeof(S) == 4;
    const bool smooth = d.rt == 2;
#define PF3D_MS(DW, SM)                                                                                          \
    launch_march_t<S, 1, 8, false, DW, false, SM, true, FAST, 2>(tm, d, s, nullptr, c_in, phi_out, dpp, nullptr, nullptr, \
                                                                 nullptr, zchunk, err, st)
    if (dpp) return smooth ? PF3D_MS(true, true) : PF3D_MS(true, false);
    return smooth ? PF3D_MS(false, true) : PF3D_MS(false, false);
#undef PF3D_MS
}

template <typename S>
cudaError_t launch_march_solute(const CUtensorMap& tm, const DomainDesc& d, const StepArgs& s, const void* c_in,
                                void* c_out, int zchunk, int* err, cudaStream_t st)
{
    return launch_march_t<S, 1, 8, false, false, true, false, false, sizeof(S) == 4, 2>(
        tm, d, s, nullptr, c_in, nullptr, nullptr, c_out, nullptr, nullptr, zchunk, err, st);
}

// The persistent grid is the SM count times the CTAs of this kernel that are
// resident on one SM.
template <typename S, int L, int PASS, bool ONE_SWEEP, bool SMOOTH>
cudaError_t launch_march_batch_t(const BatchDomain* doms, const CUtensorMap* tmaps, const BatchStep* steps,
                                 const BatchItem* items, const int* head, int n_sm, int* ctr, int* err,
                                 cudaStream_t st)
{
    constexpr bool SOL = PASS == 1 || ONE_SWEEP;
    using LY = MarchLayout<S, 8, SOL>;
    auto kern = k_march_batch<S, L, 8, PASS, ONE_SWEEP, SMOOTH>;
    static int per_sm = 0;   // one attribute and occupancy query per instantiation
    if (per_sm == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::ALLOC);
        if (e != cudaSuccess) return e;
        int nb = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 32 * 8 / L, LY::ALLOC);
        if (e != cudaSuccess) return e;
        per_sm = nb > 0 ? nb : 1;
    }
    kern<<<n_sm * per_sm, dim3(32, 8 / L), LY::ALLOC, st>>>(doms, tmaps, steps, items, head, ctr, err);
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_march_batch(const BatchDomain* doms, const CUtensorMap* tmaps, const BatchStep* steps,
                               const BatchItem* items, const int* head, int pass, bool one_sweep, bool smooth,
                               int lanes, int n_sm, int* ctr, int* err, cudaStream_t st)
{
#define PF3D_MB(L, P, ONE, SM) \
    launch_march_batch_t<S, L, P, ONE, SM>(doms, tmaps, steps, items, head, n_sm, ctr, err, st)
    if (pass == 0) {
        if (smooth) return one_sweep ? PF3D_MB(1, 0, true, true) : PF3D_MB(1, 0, false, true);
        if (lanes == 2) return one_sweep ? PF3D_MB(2, 0, true, false) : PF3D_MB(2, 0, false, false);
        return one_sweep ? PF3D_MB(1, 0, true, false) : PF3D_MB(1, 0, false, false);
    }
    return lanes == 2 ? PF3D_MB(2, 1, false, false) : PF3D_MB(1, 1, false, false);
#undef PF3D_MB
}

}  // namespace pf3d
