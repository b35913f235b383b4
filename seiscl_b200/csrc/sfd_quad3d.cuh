// sfd_quad3d.cuh -- 4-cell vectorised 3D kernels (forward and adjoint) and
// their launchers, templates on the kind of rows R (sfd_kernels.h).  The
// instantiations live in sfd_quad3d_*.cu, one translation unit per half
// width and direction.
#pragma once

#include <type_traits>

#include "sfd_device.cuh"
#include "sfd_internal.h"
#include "sfd_kernels.h"
#include "sfd_launch.cuh"

namespace sfd {

// ------------------------------------------------- 4-cell vectorised 3D kernels
// One thread updates four consecutive z cells with 128-bit loads and stores:
// the per-cell streams cost one load per four cells, a z derivative one
// 12-value window (three loads) for four cells, and an x or y derivative one
// load per tap for four cells -- about a fifth of the load instructions of
// the one-cell kernels, which are bound by load issue and latency, not by
// DRAM bytes.  Every row's first physical cell must lie on a 16-byte boundary
// and rows must be whole quads: Grid::zpad fills rows of 4 n + 2 cells up with
// dummy cells (zero parameters, so their fields stay zero), Grid::zshift
// moves the fields' base for F = 2 and L > 0.  Same operation order per cell as k_v3d.
struct Q4 {
    float v[4];
};
__device__ __forceinline__ Q4 ldq(const float *p)
{
    float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    return Q4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ Q4 ldq_rw(const float *p)
{
    float4 t = *reinterpret_cast<const float4 *>(p);
    return Q4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void stq(float *p, const Q4 &q)
{
    *reinterpret_cast<float4 *>(p) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
// FP16 storage: four halves move as one 64-bit access
__device__ __forceinline__ Q4 q4_of(uint2 u)
{
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return Q4{{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ Q4 ldq(const __half *p) { return q4_of(__ldg(reinterpret_cast<const uint2 *>(p))); }
__device__ __forceinline__ Q4 ldq_rw(const __half *p) { return q4_of(*reinterpret_cast<const uint2 *>(p)); }
__device__ __forceinline__ void stq(__half *p, const Q4 &q)
{
    const __half2 a = __floats2half2_rn(q.v[0], q.v[1]), b = __floats2half2_rn(q.v[2], q.v[3]);
    uint2 u;
    u.x = *reinterpret_cast<const unsigned *>(&a);
    u.y = *reinterpret_cast<const unsigned *>(&b);
    *reinterpret_cast<uint2 *>(p) = u;
}
// Load policy of the stencil reads (template parameter LP): 0 the read-only
// path (__ldg; arrays no thread writes during the launch), 2 L2 only (__ldcg:
// values other CTAs wrote earlier in the same launch, which a stale L1 line
// must not hide).
template <int LP>
__device__ __forceinline__ Q4 ldq_p(const float *p)
{
    float4 t;
    if constexpr (LP == 0) t = __ldg(reinterpret_cast<const float4 *>(p));
    else t = __ldcg(reinterpret_cast<const float4 *>(p));
    return Q4{{t.x, t.y, t.z, t.w}};
}
template <int LP>
__device__ __forceinline__ Q4 ldq_p(const __half *p)
{
    static_assert(LP == 0, "FP16 fields are read through the read-only path");
    return ldq(p);
}

// add a quad to its FP64 sums
__device__ __forceinline__ void grad_add4(double *g, i64 ip, const float (&d)[4])
{
    double2 *p = reinterpret_cast<double2 *>(g + ip);
    double2 a = p[0], b = p[1];
    a.x += (double)d[0]; a.y += (double)d[1]; b.x += (double)d[2]; b.y += (double)d[3];
    p[0] = a;
    p[1] = b;
}

// the stored forward field of a checkpointed adjoint, four cells (the segment
// store has the fields' alignment)
template <class T>
__device__ __forceinline__ Q4 fwd_quad(const Grid &g, const AdjFields &a, int w, i64 iv)
{
    const T *p = (const T *)a.fwd[w] + iv;
    Q4 q;
    if constexpr (std::is_same<T, float>::value) {
        q = ldq(p);
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
        const T *h = reinterpret_cast<const T *>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) q.v[j] = to_f<T>(h[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) q.v[j] *= g.bsci[w];
    return q;
}

// memory variables of four cells in storage type TR: with TR FP16 under
// FP32 wave fields (Grid::rhalf) they are stored times g.rsc
template <class T, class TR>
__device__ __forceinline__ Q4 ldr_q(const Grid &g, const TR *p)
{
    Q4 r = ldq_rw(p);
    if constexpr (!std::is_same<T, TR>::value) {
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] *= g.rsci;
    }
    return r;
}
template <class T, class TR>
__device__ __forceinline__ void str_q(const Grid &g, TR *p, const Q4 &q)
{
    if constexpr (!std::is_same<T, TR>::value) {
        Q4 r;
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] = q.v[j] * g.rsc;
        stq(p, r);
    } else {
        stq(p, q);
    }
}

// forward / backward differences of four cells along a stride (x or y)
template <int F, class T, int LP = 0>
__device__ __forceinline__ Q4 dfw_q(const T *__restrict__ v, i64 i, i64 st, const float *hc)
{
    Q4 a = ldq_p<LP>(v + i + st), b = ldq_p<LP>(v + i), r;
#pragma unroll
    for (int j = 0; j < 4; j++) r.v[j] = __fmul_rn(hc[0], a.v[j] - b.v[j]);
#pragma unroll
    for (int m = 2; m <= F; m++) {
        a = ldq_p<LP>(v + i + m * st);
        b = ldq_p<LP>(v + i - (m - 1) * st);
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
    }
    return r;
}
template <int F, class T, int LP = 0>
__device__ __forceinline__ Q4 dbw_q(const T *__restrict__ v, i64 i, i64 st, const float *hc)
{
    Q4 a = ldq_p<LP>(v + i), b = ldq_p<LP>(v + i - st), r;
#pragma unroll
    for (int j = 0; j < 4; j++) r.v[j] = __fmul_rn(hc[0], a.v[j] - b.v[j]);
#pragma unroll
    for (int m = 2; m <= F; m++) {
        a = ldq_p<LP>(v + i + (m - 1) * st);
        b = ldq_p<LP>(v + i - m * st);
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
    }
    return r;
}
// the 12 values z0-4 .. z0+7 around four cells starting at z0 (a multiple of 4)
struct W12 {
    float w[12];
};
template <class T, int LP = 0>
__device__ __forceinline__ W12 ldw(const T *__restrict__ v, i64 i)
{
    W12 r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const Q4 t = ldq_p<LP>(v + i - 4 + 4 * k);
        r.w[4 * k] = t.v[0]; r.w[4 * k + 1] = t.v[1]; r.w[4 * k + 2] = t.v[2]; r.w[4 * k + 3] = t.v[3];
    }
    return r;
}
template <int F>
__device__ __forceinline__ Q4 dfw_z(const W12 &w, const float *hc)
{
    Q4 r;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float acc = __fmul_rn(hc[0], w.w[5 + j] - w.w[4 + j]);
#pragma unroll
        for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], w.w[4 + j + m] - w.w[4 + j - (m - 1)], acc);
        r.v[j] = acc;
    }
    return r;
}
template <int F>
__device__ __forceinline__ Q4 dbw_z(const W12 &w, const float *hc)
{
    Q4 r;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float acc = __fmul_rn(hc[0], w.w[4 + j] - w.w[3 + j]);
#pragma unroll
        for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], w.w[4 + j + m - 1] - w.w[4 + j - m], acc);
        r.v[j] = acc;
    }
    return r;
}

// CPML recursion on four consecutive z cells sharing one profile index
// (y and x slabs: the psi arrays are z-fastest and 16-byte aligned there).
// DIV: cpml()'s recursion with its division by K, so that grids that reach
// these kernels by dummy rows or a shifted base, and 2D ones, have the bits of
// the one-cell kernels.  Otherwise (whole rows at order 8) d is multiplied by
// 1/K (Fields::kinv, rounded to FP32 on the host): within one rounding of the
// quotient per cell, and cheaper -- the FP32 divisions had cost the velocity
// update at 256^3 with 20-cell slabs 0.031 ms of its 0.306.  A run keeps one
// of the two: where shells are saved under a free surface, the adjoint's
// surface amplifies a difference of one rounding a thousandfold and more.
template <bool DIV> struct KVal;   // 1/K of one node
template <> struct KVal<true> {
    double k;
    __device__ __forceinline__ KVal(const KTab &t, int ci) : k(__ldg(t.kq + ci)) {}
    __device__ __forceinline__ float operator()(float d, float psi) const { return cpml_quot(d, k, psi); }
};
template <> struct KVal<false> {
    float k;
    __device__ __forceinline__ KVal(const KTab &t, int ci) : k(__ldg(t.kinv + ci)) {}
    __device__ __forceinline__ float operator()(float d, float psi) const { return __fmaf_rn(d, k, psi); }
};
template <bool DIV>
__device__ __forceinline__ void cpml_q(float *psi, i64 q, KTab t, const float *a, const float *b, int ci,
                                       Q4 &d)
{
    const KVal<DIV> k(t, ci);
    const float aa = __ldg(a + ci), bb = __ldg(b + ci);
    Q4 p = ldq_rw(psi + q);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float ps = cpml_psi(p.v[j], aa, bb, d.v[j]);
        p.v[j] = ps;
        d.v[j] = k(d.v[j], ps);
    }
    stq(psi + q, p);
}

// z-slab CPML on a quad that lies entirely inside the slab: the psi cells
// are consecutive (z-type psi is [nx][ny][2 nab], k fastest), the profile
// index differs per cell (ci0 + step * j)
template <bool DIV>
__device__ __forceinline__ void cpml_zq(float *psi, i64 q, KTab t, const float *a, const float *b, int ci0,
                                        int step, Q4 &d)
{
    Q4 p = ldq_rw(psi + q);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int ci = ci0 + step * j;
        const float ps = cpml_psi(p.v[j], __ldg(a + ci), __ldg(b + ci), d.v[j]);
        p.v[j] = ps;
        d.v[j] = KVal<DIV>(t, ci)(d.v[j], ps);
    }
    stq(psi + q, p);
}

// Grids whose absorbing slabs cannot overlap (every axis at least 2 nab
// cells, the z axis 2 nab + 4) with nab % 4 == 0: a cell lies in at most one
// slab per axis and a z quad lies wholly inside or outside a z slab, so each
// axis takes one path, its side picked by selects.  The general forms below
// follow the reference's branch structure, which small grids need.
__device__ __forceinline__ bool cpml_slabs_apart(const Grid &g)
{
    return g.nab % 4 == 0 && g.nz - g.zpad >= 2 * g.nab + 4 && g.ny >= 2 * g.nab && g.nx >= 2 * g.nab;
}
// z slabs made of whole quads (the bottom one only without dummy rows), apart.
// zpad stays a run-time value in the corrections below, whatever the rows: the
// instances of whole rows compiled without it were slower, 256^3, L = 2, 946
// against 931 us a step, 72 x 64 x 80 28.5 against 26.9.
__device__ __forceinline__ bool z_quads(const Grid &g) { return g.nab % 4 == 0 && g.nz - g.zpad >= 2 * g.nab + 4; }

// The CPML corrections of cpml_v3d for a quad of z cells: z slabs per cell
// (a quad may straddle a z-slab edge), y and x slabs per quad.
template <bool DIV>
__device__ __forceinline__ void cpml_v3d_q4(const Grid &g, const Fields &f, int gz0, int gy, int gx, Q4 &sxx_x,
                                            Q4 &syy_y, Q4 &szz_z, Q4 &sxy_y, Q4 &sxy_x, Q4 &syz_y, Q4 &syz_z,
                                            Q4 &sxz_x, Q4 &sxz_z)
{
    const int F = g.F, NAB = g.nab, NZ = g.NZl, NY = g.NY, NX = g.NX;
    const i64 nz = g.nz, ny = g.ny;
    // side-merged forms where the slabs are apart: far-side profile indices are
    // 2 nab - k (integer grid) and 2 nab - 1 - k (half grid) of the slab-local
    // index k.  zq: a quad lies wholly inside or outside a z slab
    const bool apart = cpml_slabs_apart(g), zq = DIV ? z_quads(g) : NAB % 4 == 0;
    const int zpad = g.zpad;
    const i64 k0 = gz0 - F;
    if (apart && !zpad) {
        const bool zhi = gz0 > NZ - NAB - F - 1, zlo = !g.freesurf && gz0 - F < NAB;
        if (zhi || zlo) {
            const int k = zhi ? gz0 - NZ + 2 * NAB + F : gz0 - F;
            const int st = zhi ? -1 : 1, cf = zhi ? 2 * NAB - k : k, ch = zhi ? 2 * NAB - 1 - k : k;
            const i64 q = ((i64)(gx - F) * ny + (gy - F)) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], cf, st, sxz_z);
            cpml_zq<DIV>(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], cf, st, syz_z);
            cpml_zq<DIV>(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ch, st, szz_z);
        }
    } else {
        if (zq && !zpad && gz0 > NZ - NAB - F - 1) {
            i64 i = gx - F, jj = gy - F, k = gz0 - NZ + NAB + F + NAB;
            int ind = 2 * NAB - 1 - (int)k;
            i64 q = (i * ny + jj) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, -1, sxz_z);
            cpml_zq<DIV>(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, -1, syz_z);
            cpml_zq<DIV>(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, -1, szz_z);
        } else if (zq && !g.freesurf && gz0 - F < NAB) {
            i64 i = gx - F, jj = gy - F, k = gz0 - F;
            i64 q = (i * ny + jj) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, 1, sxz_z);
            cpml_zq<DIV>(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, 1, syz_z);
            cpml_zq<DIV>(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, 1, szz_z);
        } else if (gz0 + 3 > NZ - NAB - F - 1 || (!zq && !g.freesurf && gz0 - F < NAB)) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int gz = gz0 + j;
                if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
                    i64 i = gx - F, jj = gy - F, k = gz - NZ + NAB + F + NAB;
                    int ind = 2 * NAB - 1 - (int)k;
                    i64 q = (i * ny + jj) * (2 * NAB) + k;
                    cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, sxz_z.v[j]);
                    cpml(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, syz_z.v[j]);
                    cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, szz_z.v[j]);
                } else if (!g.freesurf && gz - F < NAB) {
                    i64 i = gx - F, jj = gy - F, k = gz - F;
                    i64 q = (i * ny + jj) * (2 * NAB) + k;
                    cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, sxz_z.v[j]);
                    cpml(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, syz_z.v[j]);
                    cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, szz_z.v[j]);
                }
            }
        }
    }
    if (apart) {
        const bool ylo = gy - F < NAB, yhi = gy > NY - NAB - F - 1;
        if (ylo || yhi) {
            const int j = ylo ? gy - F : gy - NY + 2 * NAB + F;
            const int cf = ylo ? j : 2 * NAB - j, ch = ylo ? j : 2 * NAB - 1 - j;
            const i64 q = ((i64)(gx - F) * (2 * NAB) + j) * nz + k0;
            cpml_q<DIV>(f.psi[PSXY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], cf, sxy_y);
            cpml_q<DIV>(f.psi[PSYY_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ch, syy_y);
            cpml_q<DIV>(f.psi[PSYZ_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], cf, syz_y);
        }
        const bool xlo = gx - F < NAB, xhi = gx > NX - NAB - F - 1;
        if (xlo || xhi) {
            const int i = xlo ? gx - F : gx - NX + 2 * NAB + F;
            const int cf = xlo ? i : 2 * NAB - i, ch = xlo ? i : 2 * NAB - 1 - i;
            const i64 q = ((i64)i * ny + (gy - F)) * nz + k0;
            cpml_q<DIV>(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ch, sxx_x);
            cpml_q<DIV>(f.psi[PSXY_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], cf, sxy_x);
            cpml_q<DIV>(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], cf, sxz_x);
        }
        return;
    }
    if (gy - F < NAB) {
        i64 i = gx - F, j = gy - F;
        i64 q = (i * (2 * NAB) + j) * nz + k0;
        cpml_q<DIV>(f.psi[PSXY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, sxy_y);
        cpml_q<DIV>(f.psi[PSYY_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, syy_y);
        cpml_q<DIV>(f.psi[PSYZ_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, syz_y);
    } else if (gy > NY - NAB - F - 1) {
        i64 i = gx - F, j = gy - NY + NAB + F + NAB;
        int ind = 2 * NAB - 1 - (int)j;
        i64 q = (i * (2 * NAB) + j) * nz + k0;
        cpml_q<DIV>(f.psi[PSXY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, sxy_y);
        cpml_q<DIV>(f.psi[PSYY_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, syy_y);
        cpml_q<DIV>(f.psi[PSYZ_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, syz_y);
    }
    if (gx - F < NAB) {
        i64 i = gx - F, j = gy - F;
        i64 q = (i * ny + j) * nz + k0;
        cpml_q<DIV>(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, sxx_x);
        cpml_q<DIV>(f.psi[PSXY_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, sxy_x);
        cpml_q<DIV>(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, sxz_x);
    }
    if (gx > NX - NAB - F - 1) {
        i64 i = gx - NX + NAB + F + NAB, j = gy - F;
        int ind = 2 * NAB - 1 - (int)i;
        i64 q = (i * ny + j) * nz + k0;
        cpml_q<DIV>(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, sxx_x);
        cpml_q<DIV>(f.psi[PSXY_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, sxy_x);
        cpml_q<DIV>(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, sxz_x);
    }
}

// MB (a template parameter of the kernel): the launch covers several shots
#define CELL3D_Q4                                                                      \
    int shot = 0, xb_ = blockIdx.z;                                                    \
    if (MB) {                                                                          \
        const int nxb_ = gridDim.z / g.nb;                                             \
        shot = blockIdx.z / nxb_;                                                      \
        xb_ = blockIdx.z - shot * nxb_;                                                \
    }                                                                                  \
    const int gz0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4 + F;                   \
    const int gy = blockIdx.y * blockDim.y + threadIdx.y + F;                          \
    const int gx = xb_ * blockDim.z + threadIdx.z + F;                                 \
    if (gz0 > g.NZ - F - 1 || gy > g.NY - F - 1 || gx > g.NX - F - 1) return;          \
    if (MB) shot_fields(g, f, shot);                                                   \
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;                                        \
    const i64 iv = gx * sx + (i64)gy * sy + gz0;                                       \
    const i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz0 - F);

// velocity update of the quad (gz0..gz0+3, gy, gx); LP: load policy of the
// stress reads
template <int R, class T, int LP = 0>
__device__ __forceinline__ void v3d_q4_at(const Grid &g, const Fields &f, int gz0, int gy, int gx, i64 iv, i64 ip)
{
    constexpr int F = half_width(R);
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    const float *hc = g.hc;
    T *wvx = fld<T>(f.w[VX]), *wvy = fld<T>(f.w[VY]), *wvz = fld<T>(f.w[VZ]);
    const T *Sxx = fld<T>(f.w[SXX]), *Syy = fld<T>(f.w[SYY]), *Szz = fld<T>(f.w[SZZ]);
    const T *Sxy = fld<T>(f.w[SXY]), *Syz = fld<T>(f.w[SYZ]), *Sxz = fld<T>(f.w[SXZ]);
    Q4 vx = ldq_rw(wvx + iv), vy = ldq_rw(wvy + iv), vz = ldq_rw(wvz + iv);
    const Q4 rip = ldq(f.p[PRIP] + ip), rjp = ldq(f.p[PRJP] + ip), rkp = ldq(f.p[PRKP] + ip);
    const W12 wzz = ldw<T, LP>(Szz, iv), wxz = ldw<T, LP>(Sxz, iv), wyz = ldw<T, LP>(Syz, iv);
    Q4 szz_z = dfw_z<F>(wzz, hc);
    Q4 sxx_x = dfw_q<F, T, LP>(Sxx, iv, sx, hc);
    Q4 sxz_x = dbw_q<F, T, LP>(Sxz, iv, sx, hc);
    Q4 sxz_z = dbw_z<F>(wxz, hc);
    Q4 syz_y = dbw_q<F, T, LP>(Syz, iv, sy, hc);
    Q4 syz_z = dbw_z<F>(wyz, hc);
    Q4 syy_y = dfw_q<F, T, LP>(Syy, iv, sy, hc);
    Q4 sxy_x = dbw_q<F, T, LP>(Sxy, iv, sx, hc);
    Q4 sxy_y = dbw_q<F, T, LP>(Sxy, iv, sy, hc);
    if (g.abs_type == 1)
        cpml_v3d_q4<!whole_rows(R)>(g, f, gz0, gy, gx, sxx_x, syy_y, szz_z, sxy_y, sxy_x, syz_y, syz_z, sxz_x, sxz_z);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float v3[3] = {__fmaf_rn(__fadd_rn(__fadd_rn(sxx_x.v[j], sxy_y.v[j]), sxz_z.v[j]), rip.v[j], vx.v[j]),
                       __fmaf_rn(__fadd_rn(__fadd_rn(syy_y.v[j], sxy_x.v[j]), syz_z.v[j]), rjp.v[j], vy.v[j]),
                       __fmaf_rn(__fadd_rn(__fadd_rn(szz_z.v[j], sxz_x.v[j]), syz_y.v[j]), rkp.v[j], vz.v[j])};
        if (g.abs_type == 2) taper_regs<3>(g, f.taper, gz0 + j, gy, gx, v3);
        vx.v[j] = v3[0]; vy.v[j] = v3[1]; vz.v[j] = v3[2];
    }
    stq(wvx + iv, vx);
    stq(wvy + iv, vy);
    stq(wvz + iv, vz);
}

template <int R, class T, bool MB>
__device__ __forceinline__ void v3d_q4(const Grid &g, Fields f)
{
    constexpr int F = half_width(R);
    CELL3D_Q4
    v3d_q4_at<R, T, 0>(g, f, gz0, gy, gx, iv, ip);
}

template <int R, class T, bool MB = false>
__global__ void __launch_bounds__(128) k_v3d_q4(Grid g, Fields f)
{
    constexpr int F = half_width(R);
    v3d_q4<R, T, MB>(g, f);
}

// The single-shot FP32 launch asks for NB resident CTAs per SM: 4, or 6 where
// that (and not 4) holds the whole launch in one wave (72 x 64 x 80: 12.5 us
// against 14.7).  4 (at most 128 registers, from 136, with a 36-byte spill):
// 0.333 ms against 0.345 at 256^3 L=2 on a B200, 0.295 since.  5 CTAs (102
// registers) is slower again, and a component-at-a-time update with 80
// registers slower still (0.37 ms): the kernel is bound by the stencil loads
// each thread keeps in flight.  CTAs of 256 or 512 threads: 0.323-0.343 ms.
// Taking the x planes in the reverse of the stress kernel's order (each
// kernel starting on the planes the other has just written) was measured
// and is not faster: 16.96 against 17.00 Gcell/s at 256^3, L=2.
template <int R, int NB = 4>
__global__ void __launch_bounds__(128, NB) k_v3d_q4_b(Grid g, Fields f)
{
    constexpr int F = half_width(R);
    constexpr bool MB = false;
    CELL3D_Q4
    v3d_q4_at<R, float, 0>(g, f, gz0, gy, gx, iv, ip);
}

// CPML corrections of cpml_s3d (forward form) for a quad of z cells
template <bool DIV>
__device__ __forceinline__ void cpml_s3d_q4(const Grid &g, const Fields &f, int gz0, int gy, int gx, Q4 &vxx,
                                            Q4 &vxy, Q4 &vxz, Q4 &vyx, Q4 &vyy, Q4 &vyz, Q4 &vzx, Q4 &vzy, Q4 &vzz)
{
    const int F = g.F, NAB = g.nab, NZ = g.NZl, NY = g.NY, NX = g.NX;
    const i64 nz = g.nz, ny = g.ny;
    // side-merged forms where the slabs are apart: far-side profile indices are
    // 2 nab - k (integer grid) and 2 nab - 1 - k (half grid) of the slab-local
    // index k.  zq: a quad lies wholly inside or outside a z slab
    const bool apart = cpml_slabs_apart(g), zq = z_quads(g);
    const int zpad = g.zpad;
    const i64 k0 = gz0 - F;
    if (apart && !zpad) {
        const bool zhi = gz0 > NZ - NAB - F - 1, zlo = !g.freesurf && gz0 - F < NAB;
        if (zhi || zlo) {
            const int k = zhi ? gz0 - NZ + 2 * NAB + F : gz0 - F;
            const int st = zhi ? -1 : 1, cf = zhi ? 2 * NAB - k : k, ch = zhi ? 2 * NAB - 1 - k : k;
            const i64 q = ((i64)(gx - F) * ny + (gy - F)) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ch, st, vxz);
            cpml_zq<DIV>(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ch, st, vyz);
            cpml_zq<DIV>(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], cf, st, vzz);
        }
    } else {
        if (zq && !zpad && gz0 > NZ - NAB - F - 1) {
            i64 i = gx - F, jj = gy - F, k = gz0 - NZ + NAB + F + NAB;
            int ind = 2 * NAB - 1 - (int)k;
            i64 q = (i * ny + jj) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, -1, vxz);
            cpml_zq<DIV>(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, -1, vyz);
            cpml_zq<DIV>(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, -1, vzz);
        } else if (zq && !g.freesurf && gz0 - F < NAB) {
            i64 i = gx - F, jj = gy - F, k = gz0 - F;
            i64 q = (i * ny + jj) * (2 * NAB) + k;
            cpml_zq<DIV>(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, 1, vxz);
            cpml_zq<DIV>(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, 1, vyz);
            cpml_zq<DIV>(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, 1, vzz);
        } else if (gz0 + 3 > NZ - NAB - F - 1 || (!zq && !g.freesurf && gz0 - F < NAB)) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int gz = gz0 + j;
                if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
                    i64 i = gx - F, jj = gy - F, k = gz - NZ + NAB + F + NAB;
                    int ind = 2 * NAB - 1 - (int)k;
                    i64 q = (i * ny + jj) * (2 * NAB) + k;
                    cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vxz.v[j]);
                    cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vyz.v[j]);
                    cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, vzz.v[j]);
                }
                if (!g.freesurf && gz - F < NAB) {
                    i64 i = gx - F, jj = gy - F, k = gz - F;
                    i64 q = (i * ny + jj) * (2 * NAB) + k;
                    cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vxz.v[j]);
                    cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vyz.v[j]);
                    cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, vzz.v[j]);
                }
            }
        }
    }
    if (apart) {
        const bool ylo = gy - F < NAB, yhi = gy > NY - NAB - F - 1;
        if (ylo || yhi) {
            const int j = ylo ? gy - F : gy - NY + 2 * NAB + F;
            const int cf = ylo ? j : 2 * NAB - j, ch = ylo ? j : 2 * NAB - 1 - j;
            const i64 q = ((i64)(gx - F) * (2 * NAB) + j) * nz + k0;
            cpml_q<DIV>(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ch, vxy);
            cpml_q<DIV>(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], cf, vyy);
            cpml_q<DIV>(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ch, vzy);
        }
        const bool xlo = gx - F < NAB, xhi = gx > NX - NAB - F - 1;
        if (xlo || xhi) {
            const int i = xlo ? gx - F : gx - NX + 2 * NAB + F;
            const int cf = xlo ? i : 2 * NAB - i, ch = xlo ? i : 2 * NAB - 1 - i;
            const i64 q = ((i64)i * ny + (gy - F)) * nz + k0;
            cpml_q<DIV>(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], cf, vxx);
            cpml_q<DIV>(f.psi[PVY_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ch, vyx);
            cpml_q<DIV>(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ch, vzx);
        }
        return;
    }
    if (gy - F < NAB) {
        i64 i = gx - F, j = gy - F;
        i64 q = (i * (2 * NAB) + j) * nz + k0;
        cpml_q<DIV>(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vxy);
        cpml_q<DIV>(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, vyy);
        cpml_q<DIV>(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vzy);
    }
    if (gy > NY - NAB - F - 1) {
        i64 i = gx - F, j = gy - NY + NAB + F + NAB;
        int ind = 2 * NAB - 1 - (int)j;
        i64 q = (i * (2 * NAB) + j) * nz + k0;
        cpml_q<DIV>(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, vxy);
        cpml_q<DIV>(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, vyy);
        cpml_q<DIV>(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, vzy);
    }
    if (gx - F < NAB) {
        i64 i = gx - F, j = gy - F;
        i64 q = (i * ny + j) * nz + k0;
        cpml_q<DIV>(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, vxx);
        cpml_q<DIV>(f.psi[PVY_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, vyx);
        cpml_q<DIV>(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, vzx);
    }
    if (gx > NX - NAB - F - 1) {
        i64 i = gx - NX + NAB + F + NAB, j = gy - F;
        int ind = 2 * NAB - 1 - (int)i;
        i64 q = (i * ny + j) * nz + k0;
        cpml_q<DIV>(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, vxx);
        cpml_q<DIV>(f.psi[PVY_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vyx);
        cpml_q<DIV>(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vzx);
    }
}

// the strains (vxx, vyy, vzz) the free surface takes at the top cell iv, as
// k_surf3d forms them: derivatives times 1/K plus the memory of this step
template <int F, class T>
__device__ __forceinline__ void surf_strain(const Grid &g, const Fields &f, int gy, int gx, i64 iv, float (&v)[3])
{
    const int NAB = g.nab;
    v[0] = dbwT<F>(fld<T>(f.w[VX]), iv, (i64)g.NY * g.NZ, g.hc);
    v[1] = dbwT<F>(fld<T>(f.w[VY]), iv, (i64)g.NZ, g.hc);
    v[2] = dbwT<F>(fld<T>(f.w[VZ]), iv, 1, g.hc);
    if (g.abs_type != 1) return;
    const i64 nz = g.nz, ny = g.ny, i = gx - F, j = gy - F;
    if (j < NAB) {
        v[1] = __fmaf_rn(v[1], f.kinv[1][0][j], f.psi[PVY_Y][(i * (2 * NAB) + j) * nz]);
    } else if (j >= ny - NAB) {
        const i64 k = j - ny + 2 * NAB;
        v[1] = __fmaf_rn(v[1], f.kinv[1][0][2 * NAB - k], f.psi[PVY_Y][(i * (2 * NAB) + k) * nz]);
    }
    if (i < NAB) v[0] = __fmaf_rn(v[0], f.kinv[0][0][i], f.psi[PVX_X][(i * ny + j) * nz]);
    if (i >= g.nx - NAB) {
        const i64 k = i - g.nx + 2 * NAB;
        v[0] = __fmaf_rn(v[0], f.kinv[0][0][2 * NAB - k], f.psi[PVX_X][(k * ny + j) * nz]);
    }
}
// whether a folded surface takes the roundings of the separate launch
// (k_surf3d): where the call asks for it (SURF_APART), and on grids and
// storage types that otherwise run that launch
template <int R, class T>
__device__ __forceinline__ bool surf_apart(Surf surf)
{
    return surf == SURF_APART || !whole_rows(R) || sizeof(T) == 2;
}
// a value as storage type T keeps it
template <class T> __device__ __forceinline__ float stored(float v) { return to_f<T>(from_f<T>(v)); }

// shell indices of a quad's cells (-1: none).  Most quads lie wholly inside
// or outside the shell: one comparison per axis settles them, against some
// forty integer operations a cell.
__device__ __forceinline__ bool shell_quad3d(const Grid &g, int gz0, int gy, int gx, int (&m)[4])
{
    const BndDims b = bnd_dims(g);
    const int F = g.F, i = gx - b.lbnd, j = gy - b.lbnd, k = gz0 - b.lbnds;
    if (i < 0 || i >= b.NXbnd || j < 0 || j >= b.NYbnd || k + 3 < 0 || k >= b.NZbnd) return false;
    if (i >= F && i < b.NXbnd - F && j >= F && j < b.NYbnd - F && k >= F && k + 3 < b.NZbnd - F) return false;
#pragma unroll
    for (int q = 0; q < 4; q++) m[q] = inject_ind3d(g, gz0 + q, gy, gx);
    return true;
}

// the boundary shells a stress update saves: stores, offset of the step's
// slice, shell indices of the quad's cells (none: the quad has none)
struct BndQuad {
    const BndSlot *b;
    i64 at;
    int m[4];
    bool any;
};
template <class TB>
__device__ __forceinline__ void bnd_save(const Grid &g, const BndQuad &q, int w, const Q4 &v)
{
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (q.m[j] >= 0) ((TB *)q.b->p[w])[q.at + q.m[j]] = from_f<TB>(v.v[j] * g.bsc[w]);
}

// Stress and memory-variable update of four z cells (the arithmetic of
// k_s3d_stream per cell).  The per-cell work runs in two phases -- normal
// stresses (sxx, syy, szz with rxx, ryy, rzz) then shear stresses (sxy, syz,
// sxz with rxy, ryz, rxz) -- each loading only its own memory variables and
// parameters, so the live state fits in registers; the components are
// independent, so the split changes no result.
//
// surf: the free surface of the same step follows the update in registers
// (k_surf3d at z = F, forward direction): the quad at gz0 = F zeroes szz and
// rzz there, corrects sxx, syy, rxx, ryy and writes the images
// szz(F-m) = -szz(F+m), sxz(F-m) = -sxz(F+m-1) and syz(F-m) = -syz(F+m-1) that
// its own cells give; at order 8 the quad at gz0 = F+4 writes szz(F-4).
template <int R, int L, class T, class TR = T, class TB = void>
__device__ __forceinline__ void s_normal_q4(const Grid &g, const Fields &f, int gz0, int gy, int gx, i64 iv, i64 ip,
                                            const Q4 &vxx, const Q4 &vyy, const Q4 &vzz, Surf surf = SURF_NONE,
                                            const BndQuad *bq = nullptr)
{
    constexpr int F = half_width(R);
    T *const ws[3] = {fld<T>(f.w[SXX]), fld<T>(f.w[SYY]), fld<T>(f.w[SZZ])};
    TR *const wr[3] = {fld<TR>(f.r[RXX]), fld<TR>(f.r[RYY]), fld<TR>(f.r[RZZ])};
    Q4 sq[3];
#pragma unroll
    for (int q = 0; q < 3; q++) sq[q] = ldq_rw(ws[q] + iv);
    const Q4 qM = ldq(f.p[PM] + ip), qmu = ldq(f.p[PMU] + ip);
    Q4 rq[3][L > 0 ? L : 1];
    S2dMat m0;   // material of the first cell, for the surface
    if constexpr (L == 0) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float tr = __fadd_rn(__fadd_rn(vxx.v[j], vyy.v[j]), vzz.v[j]);
            const float pr[3] = {__fadd_rn(vyy.v[j], vzz.v[j]), __fadd_rn(vxx.v[j], vzz.v[j]), __fadd_rn(vxx.v[j], vyy.v[j])};
            const S2dMat m = s2d_elastic(qM.v[j], qmu.v[j], 0.0f);
            if (j == 0) m0 = m;
#pragma unroll
            for (int q = 0; q < 3; q++) sq[q].v[j] = __fadd_rn(sq[q].v[j], s2d_normal(m.gm, tr, m.fm, pr[q]));
        }
    } else {
        const Q4 qtaup = ldq(f.p[PTAUP] + ip), qtaus = ldq(f.p[PTAUS] + ip);
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) rq[q][l] = ldr_q<T>(g, wr[q] + l * g.nvol + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float tr = __fadd_rn(__fadd_rn(vxx.v[j], vyy.v[j]), vzz.v[j]);
            const float pr[3] = {__fadd_rn(vyy.v[j], vzz.v[j]), __fadd_rn(vxx.v[j], vzz.v[j]), __fadd_rn(vxx.v[j], vyy.v[j])};
            const S2dMat m = s2d_visco(L, g.dt, qM.v[j], qmu.v[j], 0.0f, qtaup.v[j], qtaus.v[j], 0.0f);
            if (j == 0) m0 = m;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const float x = s2d_normal(m.e, tr, m.d, pr[q]);
                float o = 0, n = 0;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    o += rq[q][l].v[j];
                    rq[q][l].v[j] = s2d_memory(rq[q][l].v[j], g.eta[l], g.eta_b[l], g.eta_c[l], x);
                    n += rq[q][l].v[j];
                }
                sq[q].v[j] = s2d_add(sq[q].v[j], __fmaf_rn(g.dt2, o, s2d_normal(m.gm, tr, m.fm, pr[q])), g.dt2, n);
            }
        }
    }
    if (g.abs_type == 2) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float v3[3] = {sq[0].v[j], sq[1].v[j], sq[2].v[j]};
            taper_regs<3>(g, f.taper, gz0 + j, gy, gx, v3);
#pragma unroll
            for (int q = 0; q < 3; q++) sq[q].v[j] = v3[q];
        }
    }
    if constexpr (!std::is_void<TB>::value) {   // before the free surface
        if (bq->any) {
            const int id[3] = {SXX, SYY, SZZ};
#pragma unroll
            for (int q = 0; q < 3; q++) bnd_save<TB>(g, *bq, id[q], sq[q]);
        }
    }
    if (F == 4 && surf && gz0 == F + 4) stv(ws[2] + iv - 8, -sq[2].v[0]);
    if (surf && gz0 == F) {
        // the arithmetic of k_surf3d, forward
        const Surf2d su = surf2d_of(m0);
        float v1[3] = {vxx.v[0], vyy.v[0], vzz.v[0]};
        // whole rows: the update's own CPML multiplies by 1/K
        if constexpr (!whole_rows(R)) surf_strain<F, T>(g, f, gy, gx, iv, v1);
        const float vh = __fadd_rn(v1[0], v1[1]), vz0 = v1[2], h = L == 0 || !surf_apart<R, T>(surf) ? surf2d_h<true>(su, vh, vz0) : surf2d_h<false>(su, vh, vz0);
        // FP16 fields: k_surf3d reads what the update has stored
        if constexpr (sizeof(T) == 2) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                sq[q].v[0] = stored<T>(sq[q].v[0]);
#pragma unroll
                for (int l = 0; l < L; l++) rq[q][l].v[0] = stored<T>(rq[q][l].v[0]);
            }
        }
        sq[2].v[0] = 0.0f;
        if constexpr (L == 0) {
            sq[0].v[0] = __fadd_rn(sq[0].v[0], h);
            sq[1].v[0] = __fadd_rn(sq[1].v[0], h);
        } else {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                float sum = 0;
#pragma unroll
                for (int l = 0; l < L; l++) sum += rq[q][l].v[0];
                const float t = stored<T>(__fadd_rn(sq[q].v[0], __fmaf_rn(-g.dt2, sum, h)));
                sum = 0;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    const float b = surf2d_b(g.eta[l]), hr = surf2d_hr(su, vh, vz0);
                    rq[q][l].v[0] = q == 0 && sizeof(T) == 4 && surf_apart<R, T>(surf) ? __fadd_rn(rq[q][l].v[0], __fmul_rn(b, hr)) : __fmaf_rn(b, hr, rq[q][l].v[0]);
                    sum += rq[q][l].v[0];
                }
                sq[q].v[0] = __fmaf_rn(g.dt2, sum, t);
            }
#pragma unroll
            for (int l = 0; l < L; l++) rq[2][l].v[0] = 0.0f;
        }
#pragma unroll
        for (int m = 1; m <= (F < 4 ? F : 3); m++) stv(ws[2] + iv - m, -sq[2].v[m]);
    }
    if constexpr (L > 0) {
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) str_q<T>(g, wr[q] + l * g.nvol + iv, rq[q][l]);
    }
#pragma unroll
    for (int q = 0; q < 3; q++) stq(ws[q] + iv, sq[q]);
}

template <int R, int L, class T, class TR = T, class TB = void>
__device__ __forceinline__ void s_shear_q4(const Grid &g, const Fields &f, int gz0, int gy, int gx, i64 iv, i64 ip,
                                           const Q4 &vxyyx, const Q4 &vyzzy, const Q4 &vxzzx, Surf surf = SURF_NONE,
                                           const BndQuad *bq = nullptr)
{
    constexpr int F = half_width(R);
    T *const ws[3] = {fld<T>(f.w[SXY]), fld<T>(f.w[SYZ]), fld<T>(f.w[SXZ])};
    TR *const wr[3] = {fld<TR>(f.r[RXY]), fld<TR>(f.r[RYZ]), fld<TR>(f.r[RXZ])};
    Q4 sq[3];
#pragma unroll
    for (int q = 0; q < 3; q++) sq[q] = ldq_rw(ws[q] + iv);
    const Q4 qmuipjp = ldq(f.p[PMUIPJP] + ip), qmujpkp = ldq(f.p[PMUJPKP] + ip), qmuipkp = ldq(f.p[PMUIPKP] + ip);
    if constexpr (L == 0) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            sq[0].v[j] = __fmaf_rn(qmuipjp.v[j], vxyyx.v[j], sq[0].v[j]);
            sq[1].v[j] = __fmaf_rn(qmujpkp.v[j], vyzzy.v[j], sq[1].v[j]);
            sq[2].v[j] = __fmaf_rn(qmuipkp.v[j], vxzzx.v[j], sq[2].v[j]);
        }
    } else {
        const Q4 qt[3] = {ldq(f.p[PTAUSIPJP] + ip), ldq(f.p[PTAUSJPKP] + ip), ldq(f.p[PTAUSIPKP] + ip)};
        Q4 rq[3][L];
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) rq[q][l] = ldr_q<T>(g, wr[q] + l * g.nvol + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float mu[3] = {qmuipjp.v[j], qmujpkp.v[j], qmuipkp.v[j]}, v[3] = {vxyyx.v[j], vyzzy.v[j], vxzzx.v[j]};
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const float fc = __fmul_rn(mu[q], __fmaf_rn((float)L, qt[q].v[j], 1.0f));
                const float x = __fmul_rn(__fdiv_rn(__fmul_rn(mu[q], qt[q].v[j]), g.dt), v[q]);
                float o = 0, n = 0;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    o += rq[q][l].v[j];
                    rq[q][l].v[j] = s2d_memory(rq[q][l].v[j], g.eta[l], g.eta_b[l], g.eta_c[l], x);
                    n += rq[q][l].v[j];
                }
                sq[q].v[j] = s2d_add(sq[q].v[j], __fmaf_rn(fc, v[q], __fmul_rn(g.dt2, o)), g.dt2, n);
            }
        }
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) str_q<T>(g, wr[q] + l * g.nvol + iv, rq[q][l]);
    }
    if (g.abs_type == 2) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float v3[3] = {sq[0].v[j], sq[1].v[j], sq[2].v[j]};
            taper_regs<3>(g, f.taper, gz0 + j, gy, gx, v3);
#pragma unroll
            for (int q = 0; q < 3; q++) sq[q].v[j] = v3[q];
        }
    }
    if constexpr (!std::is_void<TB>::value) {
        if (bq->any) {
            const int id[3] = {SXY, SYZ, SXZ};
#pragma unroll
            for (int q = 0; q < 3; q++) bnd_save<TB>(g, *bq, id[q], sq[q]);
        }
    }
    if (surf && gz0 == F) {
#pragma unroll
        for (int m = 1; m <= F; m++) {
            stv(ws[2] + iv - m, -sq[2].v[m - 1]);   // sxz
            stv(ws[1] + iv - m, -sq[1].v[m - 1]);   // syz
        }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) stq(ws[q] + iv, sq[q]);
}

// stress update of the quad (gz0..gz0+3, gy, gx); LP: load policy of the
// velocity reads; surf: free surface folded in (see s_normal_q4); PF: first
// ask L2 for the quad's per-cell streams
template <int R, int L, class T, int LP = 0, bool PF = false, class TR = T, class TB = void>
__device__ __forceinline__ void s3d_q4_at(const Grid &g, const Fields &f, int gz0, int gy, int gx, i64 iv, i64 ip,
                                          Surf surf = SURF_NONE, const BndQuad *bq = nullptr)
{
    constexpr int F = half_width(R);
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    const float *hc = g.hc;
    if constexpr (PF) {
#pragma unroll
        for (int q = SXX; q <= SXZ; q++) asm volatile("prefetch.global.L2 [%0];" ::"l"(fld<T>(f.w[q]) + iv));
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < NR; q++)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(fld<TR>(f.r[q]) + l * g.nvol + iv));
        constexpr int np = L > 0 ? 10 : 5;
        constexpr int pid[10] = {PM, PMU, PMUIPJP, PMUJPKP, PMUIPKP, PTAUP, PTAUS, PTAUSIPJP, PTAUSJPKP, PTAUSIPKP};
#pragma unroll
        for (int k = 0; k < np; k++) asm volatile("prefetch.global.L2 [%0];" ::"l"(f.p[pid[k]] + ip));
    }
    const T *Vx = fld<T>(f.w[VX]), *Vy = fld<T>(f.w[VY]), *Vz = fld<T>(f.w[VZ]);
    Q4 vzz = dbw_z<F>(ldw<T, LP>(Vz, iv), hc);
    Q4 vyz = dfw_z<F>(ldw<T, LP>(Vy, iv), hc);
    Q4 vxz = dfw_z<F>(ldw<T, LP>(Vx, iv), hc);
    Q4 vzx = dfw_q<F, T, LP>(Vz, iv, sx, hc), vzy = dfw_q<F, T, LP>(Vz, iv, sy, hc);
    Q4 vyx = dfw_q<F, T, LP>(Vy, iv, sx, hc), vyy = dbw_q<F, T, LP>(Vy, iv, sy, hc);
    Q4 vxx = dbw_q<F, T, LP>(Vx, iv, sx, hc), vxy = dfw_q<F, T, LP>(Vx, iv, sy, hc);
    if (g.abs_type == 1) cpml_s3d_q4<!whole_rows(R)>(g, f, gz0, gy, gx, vxx, vxy, vxz, vyx, vyy, vyz, vzx, vzy, vzz);
    Q4 vxyyx, vyzzy, vxzzx;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        vxyyx.v[j] = __fadd_rn(vxy.v[j], vyx.v[j]);
        vyzzy.v[j] = __fadd_rn(vyz.v[j], vzy.v[j]);
        vxzzx.v[j] = __fadd_rn(vxz.v[j], vzx.v[j]);
    }
    s_normal_q4<R, L, T, TR, TB>(g, f, gz0, gy, gx, iv, ip, vxx, vyy, vzz, surf, bq);
    s_shear_q4<R, L, T, TR, TB>(g, f, gz0, gy, gx, iv, ip, vxyyx, vyzzy, vxzzx, surf, bq);
}

// surf: the free surface of the step applied in the same launch (single-shot
// modelling runs; see s_normal_q4).  Elastic launches ask for 6 CTAs per SM,
// viscoelastic ones for 4: 100 x 200 x 200 elastic 115 us at 4, 109 at 5, 106
// at 6; 128 x 160 x 160 84, 79, 79; 72 x 64 x 80 (6 make it one wave) 15.4 and
// 12.6.
template <int R, int L, class T, bool MB = false>
__global__ void __launch_bounds__(128, L == 0 && sizeof(T) == 4 ? 6 : 4) k_s3d_q4(Grid g, Fields f, Surf surf)
{
    constexpr int F = half_width(R);
    CELL3D_Q4
    s3d_q4_at<R, L, T, 0>(g, f, gz0, gy, gx, iv, ip, surf);
}

// Elastic single-shot gradient runs: the update also saves the boundary
// shells (stores b in type TB, step offset tofs) and then applies the free
// surface, which the separate launches did in 15 + 15 us of a 237 us step at
// 100 x 200 x 200.
template <int R, class TB>
__global__ void __launch_bounds__(128, 5) k_s3d_q4_bnd(Grid g, Fields f, BndSlot b, i64 tofs, Surf surf)
{
    constexpr int F = half_width(R);
    constexpr bool MB = false;
    CELL3D_Q4
    BndQuad bq;
    bq.b = &b;
    bq.at = tofs;
    bq.any = shell_quad3d(g, gz0, gy, gx, bq.m);
    if (bq.any) {
#pragma unroll
        for (int w = VX; w <= VZ; w++) bnd_save<TB>(g, bq, w, ldq(f.w[w] + iv));
    }
    s3d_q4_at<R, 0, float, 0, false, float, TB>(g, f, gz0, gy, gx, iv, ip, surf, &bq);
}

// Single-shot launches of the default selection: each thread first asks L2
// for its own per-cell streams (prefetch.global.L2 of its stresses, memory
// variables and parameters), so they are on their way while the velocity
// stencils load, and the launch takes 3 CTAs per SM (168 registers) so that
// more stencil loads stay in flight.  256^3, L=2, CPML 20, FP32 on a B200:
// 0.651 ms against 0.695 for k_s3d_q4 (0.571 against 0.601 without
// absorbing boundary); the prefetch at 4 CTAs per SM gave 0.674, 3 CTAs
// without it 0.713.
// An ordinary launch that lets the receivers' kernel launch early.  Launched
// with programmatic serialization itself, with the prefetch ahead of its
// wait, it has to read the velocities with plain loads (a read-only-path load
// counts as invariant, and the compiler may move it above the wait): 0.637 ms
// against 0.622, and 919 us a step against 911 (0.625 and 919 with the general
// kernels' roundings); 122 x 131 x 117, L = 1 143.9 against 142.9.  256 and 384 threads a CTA: 0.686-0.721 ms.
// TR: storage type of the memory variables (FP16 under FP32 wave fields
// with Grid::rhalf)
template <int R, int L, class T, class TR = T>
__global__ void __launch_bounds__(128, 3) k_s3d_q4_pf(Grid g, Fields f, Surf surf)
{
    constexpr int F = half_width(R);
    constexpr bool MB = false;
    pdl_trigger();
    CELL3D_Q4
    s3d_q4_at<R, L, T, 0, true, TR>(g, f, gz0, gy, gx, iv, ip, surf);
}

// ------------------------------------------------------------- launchers
// CTA shape (quads x y rows x x planes) of a 4-cell launch: the preferred
// shape, half as many quads along z and twice the rows where that leaves fewer
// threads without a quad, or -- where both leave more than 6 % -- rows of the
// whole column or an even part of it.  nz = 100 (25 quads), 200 x 200,
// elastic: velocity 93.7 us with 25 x 5 x 1 against 95.6 with 16 x 4 x 2, stress
// 110 against 115, an adjoint step 478 against 519; 128 x 160 x 160 (32 quads)
// keeps the preferred shape (adjoint step 361 against 366 with 16 x 8 x 1).
static dim3 q4_block(const Grid &g, unsigned bx, unsigned by, unsigned bz)
{
    const unsigned nq = (unsigned)(g.nz / 4);
    dim3 b(bx, by, bz);
    if (bx >= 16 && cdiv(nq, bx / 2) * (bx / 2) < cdiv(nq, bx) * bx) b = dim3(bx / 2, by * 2, bz);
    const unsigned slots = cdiv(nq, b.x) * b.x, part = cdiv(nq, cdiv(nq, 32));
    if (nq >= 12 && slots * 100 > nq * 106 && cdiv(nq, part) * part < slots) b = dim3(part, 128 / part, 1);
    return b;
}
// whether a launch's threads fit the chip at once with `ctas` CTAs of 128
// threads an SM
static bool one_wave(const Grid &g, int ctas)
{
    return (int64_t)(g.nz / 4) * g.ny * g.nx * g.nb <= (int64_t)148 * 128 * ctas;
}
static dim3 q4_grid(const Grid &g, dim3 b)
{
    return dim3(cdiv(g.nz / 4, b.x), cdiv(g.ny, b.y), cdiv(g.nx, b.z) * g.nb);
}


template <int R>
void quad_update_v(const Grid &g, const Fields &f, cudaStream_t st)
{
    if (g.fhalf) {
        const dim3 b = q4_block(g, 8, 4, 4), gr = q4_grid(g, b);
        k_v3d_q4<R, __half><<<gr, b, 0, st>>>(g, f);
        return;
    }
    // 16 quads (64 z cells) x 4 y x 2 x per CTA: the y and x stencil
    // rows of neighbouring threads share L1 lines.  Interior-only
    // timing at 256^3 on a B200: 0.268 ms, against 0.275 for 8 x 4 x
    // 4, 0.284 for 8 x 2 x 8 and 0.34 for 4 x 8 x 4 quads x y x x
    const dim3 b = q4_block(g, 16, 4, 2), gr = q4_grid(g, b);
    if (g.nb > 1) k_v3d_q4<R, float, true><<<gr, b, 0, st>>>(g, f);
    else if (one_wave(g, 6) && !one_wave(g, 4)) k_v3d_q4_b<R, 6><<<gr, b, 0, st>>>(g, f);
    else k_v3d_q4_b<R><<<gr, b, 0, st>>>(g, f);
}

template <int R, int L>
static void quad_update_s_l(const Grid &g, const Fields &f, dim3 g4, dim3 b4, cudaStream_t st, Surf surf)
{
    // the stream prefetch pays where memory variables add per-cell
    // streams: 256^3, L=2: 0.654 ms against 0.706; elastic (L=0):
    // 0.376 against 0.366 without it.  kernels 5 keeps k_s3d_q4.
    if constexpr (L > 0) {
        if (g.nb == 1 && g.kernels == 0) {
            if (g.fhalf) k_s3d_q4_pf<R, L, __half><<<g4, b4, 0, st>>>(g, f, surf);
            else if (g.rhalf) k_s3d_q4_pf<R, L, float, __half><<<g4, b4, 0, st>>>(g, f, surf);
            else k_s3d_q4_pf<R, L, float><<<g4, b4, 0, st>>>(g, f, surf);
            return;
        }
    }
    if (g.fhalf) { k_s3d_q4<R, L, __half><<<g4, b4, 0, st>>>(g, f, surf); return; }
    MB_DISPATCH(g, k_s3d_q4<R, L, float, MBV><<<g4, b4, 0, st>>>(g, f, surf))
}

template <int R>
bool quad_update_s(const Grid &g, const Fields &f, cudaStream_t st, Surf surf)
{
    const dim3 b4 = q4_block(g, 16, 8, 1), g4 = q4_grid(g, b4);  // 0.70 ms vs 0.71 (32 x 2 x 2)
    switch (g.L) {
    case 0: quad_update_s_l<R, 0>(g, f, g4, b4, st, surf); break;
    case 1: quad_update_s_l<R, 1>(g, f, g4, b4, st, surf); break;
    case 2: quad_update_s_l<R, 2>(g, f, g4, b4, st, surf); break;
    default: quad_update_s_l<R, 3>(g, f, g4, b4, st, surf); break;
    }
    return surf != SURF_NONE;
}

template <int R>
void quad_update_s_bnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, bool surface, cudaStream_t st)
{
    const Surf surf = surface ? SURF_APART : SURF_NONE;
    const dim3 b4 = q4_block(g, 16, 8, 1), g4 = q4_grid(g, b4);
    if (prec == SFD_PREC_FP16) k_s3d_q4_bnd<R, __half><<<g4, b4, 0, st>>>(g, f, b, tofs, surf);
    else if (prec == SFD_PREC_BF16) k_s3d_q4_bnd<R, __nv_bfloat16><<<g4, b4, 0, st>>>(g, f, b, tofs, surf);
    else k_s3d_q4_bnd<R, float><<<g4, b4, 0, st>>>(g, f, b, tofs, surf);
}

}  // namespace sfd
