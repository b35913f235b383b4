// sfd_device.cuh -- device functions shared by the stencil kernels:
// differences, storage access, CPML, saved-boundary indices, and the P-SV
// cell arithmetic.
//
// The arithmetic of a 2D cell is written with explicit roundings (__fmaf_rn,
// __fmul_rn, __fadd_rn): every 2D kernel gives the same bits, whatever the
// compiler would contract in each.
#pragma once

#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "sfd_internal.h"

namespace sfd {

typedef int64_t i64;

// ---------------------------------------------------------------- helpers
// forward difference c1 (v[i+1]-v[i]) + c2 (v[i+2]-v[i-1]) + ...  (Dxp)
template <int F>
__device__ __forceinline__ float dfw(const float *__restrict__ v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], __ldg(v + i + st) - __ldg(v + i));
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], __ldg(v + i + m * st) - __ldg(v + i - (m - 1) * st), acc);
    return acc;
}
// backward difference c1 (v[i]-v[i-1]) + c2 (v[i+1]-v[i-2]) + ...  (Dxm)
template <int F>
__device__ __forceinline__ float dbw(const float *__restrict__ v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], __ldg(v + i) - __ldg(v + i - st));
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], __ldg(v + i + (m - 1) * st) - __ldg(v + i - m * st), acc);
    return acc;
}
// non-cached variants for arrays written by the same kernel
template <int F>
__device__ __forceinline__ float dfw_rw(const float *v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], v[i + st] - v[i]);
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], v[i + m * st] - v[i - (m - 1) * st], acc);
    return acc;
}
template <int F>
__device__ __forceinline__ float dbw_rw(const float *v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], v[i] - v[i - st]);
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], v[i + (m - 1) * st] - v[i - m * st], acc);
    return acc;
}

// Wave-field storage access: FP32, or FP16 holding the field times a power
// of two (the kernels compute in FP32 either way).
template <class T> __device__ __forceinline__ float ldv(const T *p);
template <> __device__ __forceinline__ float ldv<float>(const float *p) { return *p; }
template <> __device__ __forceinline__ float ldv<__half>(const __half *p) { return __half2float(*p); }
template <class T> __device__ __forceinline__ float ldgv(const T *p);
template <> __device__ __forceinline__ float ldgv<float>(const float *p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldgv<__half>(const __half *p) { return __half2float(__ldg(p)); }
template <class T> __device__ __forceinline__ void stv(T *p, float v);
template <> __device__ __forceinline__ void stv<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void stv<__half>(__half *p, float v) { *p = __float2half_rn(v); }
template <class T> __device__ __forceinline__ T *fld(float *p) { return reinterpret_cast<T *>(p); }

template <int F, class T>
__device__ __forceinline__ float dfwT(const T *__restrict__ v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], ldgv(v + i + st) - ldgv(v + i));
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], ldgv(v + i + m * st) - ldgv(v + i - (m - 1) * st), acc);
    return acc;
}
template <int F, class T>
__device__ __forceinline__ float dbwT(const T *__restrict__ v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], ldgv(v + i) - ldgv(v + i - st));
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], ldgv(v + i + (m - 1) * st) - ldgv(v + i - m * st), acc);
    return acc;
}
template <int F, class T>
__device__ __forceinline__ float dbw_rwT(const T *v, i64 i, i64 st, const float *hc)
{
    float acc = __fmul_rn(hc[0], ldv(v + i) - ldv(v + i - st));
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], ldv(v + i + (m - 1) * st) - ldv(v + i - m * st), acc);
    return acc;
}

// psi = b psi + a d ; d = d/K + psi    (the CPML recursion).  The 4-cell
// kernels of 3D grids whose rows are whole quads multiply by 1/K in FP32
// instead (cpml_q); everything else takes the quotient.
__device__ __forceinline__ float cpml_psi(float psi, float a, float b, float d)
{
    return __fmaf_rn(b, psi, __fmul_rn(a, d));
}
struct KTab {           // 1/K of a profile: of the FP32 value in FP64, and in FP32
    const double *kq;
    const float *kinv;
};
__device__ __forceinline__ KTab ktab(const Fields &f, int axis, int half) { return KTab{f.kq[axis][half], f.kinv[axis][half]}; }
// d / K + psi with the bits of FP32 division: the FP64 product is within 2^-52
// of the quotient, and a quotient of two 24-bit significands is 2^-49 or more
// away from where its rounding to FP32 would change.  With division
// instructions instead, a run of 130 x 121 x 147, order 4, took 39 ms against
// 26, and one of 100 x 150 2.2 against 1.6.
__device__ __forceinline__ float cpml_quot(float d, double kq, float psi)
{
    return __fadd_rn(__double2float_rn(__dmul_rn((double)d, kq)), psi);
}
__device__ __forceinline__ void cpml(float *psi, i64 q, KTab k, const float *a, const float *b, int ci, float &d)
{
    const float ps = cpml_psi(psi[q], __ldg(a + ci), __ldg(b + ci), d);
    psi[q] = ps;
    d = cpml_quot(d, __ldg(k.kq + ci), ps);
}

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Programmatic dependent launch (the 3D modelling loop's kernels, see
// pdl_enabled): a kernel launched with programmatic stream serialization may
// be resident before the previous kernel of the stream has finished.
// pdl_wait returns once that kernel has completed and its stores are
// visible (at once for an ordinary launch); nothing it writes may be read,
// and nothing at all written, before it.  pdl_trigger lets the next
// kernel's CTAs launch once every CTA of this grid has passed it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// batched shots: shot b of a launch (blockIdx.z) works on copy b of every
// per-shot array
__device__ __forceinline__ void shot_fields(const Grid &g, Fields &f, int b)
{
#pragma unroll
    for (int w = 0; w < NW; w++)
        if (f.w[w]) f.w[w] += b * g.sb_w;
#pragma unroll
    for (int r = 0; r < NR; r++)
        if (f.r[r]) f.r[r] += b * g.sb_r;
#pragma unroll
    for (int i = 0; i < NPSI; i++)
        if (f.psi[i]) f.psi[i] += b * g.sb_psi;
}
__device__ __forceinline__ void shot_adj(const Grid &g, AdjFields &a, int b)
{
#pragma unroll
    for (int w = 0; w < NW; w++) {
        if (a.wr[w]) a.wr[w] += b * g.sb_w;
        if (a.bnd[w]) a.bnd[w] = (const char *)a.bnd[w] + b * g.sb_bnd;
    }
#pragma unroll
    for (int r = 0; r < NR; r++)
        if (a.rr[r]) a.rr[r] += b * g.sb_r;
#pragma unroll
    for (int k = 0; k < NG; k++) {
        if (a.grad[k]) a.grad[k] += b * g.sb_g;
        if (a.hess[k]) a.hess[k] += b * g.sb_g;
    }
}
#define SHOT_F  if (g.nb > 1) shot_fields(g, f, blockIdx.z);
#define SHOT_FA if (g.nb > 1) { shot_fields(g, f, blockIdx.z); shot_adj(g, a, blockIdx.z); }

// a saved boundary value (slice t-1) back in field units: FP16 stores carry
// a power-of-two scale (exact; 1 for FP32 and BF16 stores)
template <class T>
__device__ __forceinline__ float bnd_at(const Grid &g, const AdjFields &a, int w, i64 m)
{
    return to_f<T>(((const T *)a.bnd[w])[m]) * g.bsci[w];
}

// checkpointed gradients (g.ckpt): the forward wave field of the adjoint
// step, stored when the forward run was recomputed from a snapshot (same
// storage type and scales as the saved boundaries)
template <class T>
__device__ __forceinline__ float fwd_at(const Grid &g, const AdjFields &a, int w, i64 iv)
{
    return to_f<T>(((const T *)a.fwd[w])[iv]) * g.bsci[w];
}

// ------------------------------------------------------- boundary shells
struct BndDims {
    int NXbnd, NYbnd, NZbnd, lbnd, lbnds;
};
__device__ __host__ inline BndDims bnd_dims(const Grid &g)
{
    BndDims b;
    b.NXbnd = g.NX - 2 * g.F - 2 * g.nab;
    b.NYbnd = g.nd == 3 ? g.NY - 2 * g.F - 2 * g.nab : 1;
    if (!g.freesurf) {
        b.NZbnd = g.NZl - 2 * g.F - 2 * g.nab;
        b.lbnd = g.F + g.nab;
        b.lbnds = g.F + g.nab;
    } else {
        b.NZbnd = g.NZl - 2 * g.F - g.nab;
        b.lbnd = g.F + g.nab;
        b.lbnds = g.F;
    }
    return b;
}

// index of cell (k, i) in the saved shell, -1 if not a shell cell
// (src/header_injectbnd.cl:238-283)
__device__ __forceinline__ int inject_ind2d(const Grid &g, int k, int i)
{
    BndDims b = bnd_dims(g);
    int F = g.F, m = -1;
    i -= b.lbnd;
    k -= b.lbnds;
    if ((k > F - 1 && k < b.NZbnd - F) && (i > F - 1 && i < b.NXbnd - F)) m = -1;
    else if (k < 0 || k > b.NZbnd - 1 || i < 0 || i > b.NXbnd - 1) m = -1;
    else if (i < F) m = i * b.NZbnd + k;
    else if (i > b.NXbnd - 1 - F) { i = i - b.NXbnd + F; m = b.NZbnd * F + i * b.NZbnd + k; }
    else if (k < F) { i = i - F; m = b.NZbnd * F * 2 + (b.NXbnd - 2 * F) * F + i + k * (b.NXbnd - 2 * F); }
    else { i = i - F; k = k - b.NZbnd + F; m = b.NZbnd * F * 2 + i + k * (b.NXbnd - 2 * F); }
    return m;
}
// (src/header_injectbnd.cl:25-84)
__device__ __forceinline__ int inject_ind3d(const Grid &g, int k, int j, int i)
{
    BndDims b = bnd_dims(g);
    int F = g.F, m = -1;
    i -= b.lbnd; j -= b.lbnd; k -= b.lbnds;
    int NX = b.NXbnd, NY = b.NYbnd, NZ = b.NZbnd;
    if ((k > F - 1 && k < NZ - F) && (j > F - 1 && j < NY - F) && (i > F - 1 && i < NX - F)) m = -1;
    else if (k < 0 || k > NZ - 1 || j < 0 || j > NY - 1 || i < 0 || i > NX - 1) m = -1;
    else if (i < F) m = i * NY * NZ + j * NZ + k;
    else if (i > NX - 1 - F) { i = i - NX + F; m = NY * NZ * F + i * NY * NZ + j * NZ + k; }
    else if (j < F) { i = i - F; m = NY * NZ * F * 2 + i * F * NZ + j * NZ + k; }
    else if (j > NY - 1 - F) { i = i - F; j = j - NY + F; m = NY * NZ * F * 2 + (NX - 2 * F) * NZ * F + i * F * NZ + j * NZ + k; }
    else if (k < F) {
        i = i - F; j = j - F;
        m = NY * NZ * F * 2 + (NX - 2 * F) * NZ * F * 2 + (NX - 2 * F) * (NY - 2 * F) * F + i * (NY - 2 * F) * F + j * F + k;
    } else {
        i = i - F; j = j - F; k = k - NZ + F;
        m = NY * NZ * F * 2 + (NX - 2 * F) * NZ * F * 2 + i * (NY - 2 * F) * F + j * F + k;
    }
    return m;
}

// shell cell of saved index gid (src/savebnd2D.cl:52-93, savebnd3D.cl:46-103)
__device__ __forceinline__ bool shell_cell(const Grid &g, int gid, int &i, int &j, int &k)
{
    BndDims b = bnd_dims(g);
    int F = g.F, NAB = g.nab, gidf;
    if (g.nd != 3) {
        j = 0;
        int NZ = b.NZbnd, NX = b.NXbnd;
        if (gid < NZ * F) { gidf = gid; i = gidf / NZ + b.lbnd; k = gidf % NZ + b.lbnds; }
        else if (gid < NZ * F * 2) { gidf = gid - NZ * F; i = gidf / NZ + NX + NAB; k = gidf % NZ + b.lbnds; }
        else if (gid < NZ * F * 2 + (NX - 2 * F) * F) {
            gidf = gid - NZ * F * 2; i = gidf % (NX - 2 * F) + b.lbnd + F; k = gidf / (NX - 2 * F) + NZ + b.lbnds - F;
        } else if (gid < NZ * F * 2 + (NX - 2 * F) * 2 * F) {
            gidf = gid - NZ * F * 2 - (NX - 2 * F) * F; i = gidf % (NX - 2 * F) + b.lbnd + F; k = gidf / (NX - 2 * F) + b.lbnds;
        } else return false;
        return true;
    }
    int NX = b.NXbnd, NY = b.NYbnd, NZ = b.NZbnd;
    int a0 = NY * NZ * F, a1 = NZ * (NX - 2 * F) * F, a2 = (NY - 2 * F) * (NX - 2 * F) * F;
    if (gid < a0) { gidf = gid; i = gidf / (NY * NZ) + b.lbnd; j = (gidf / NZ) % NY + b.lbnd; k = gidf % NZ + b.lbnds; }
    else if (gid < 2 * a0) { gidf = gid - a0; i = gidf / (NY * NZ) + NX + NAB; j = (gidf / NZ) % NY + b.lbnd; k = gidf % NZ + b.lbnds; }
    else if (gid < 2 * a0 + a1) { gidf = gid - 2 * a0; i = gidf / (NZ * F) + b.lbnd + F; j = (gidf / NZ) % F + b.lbnd; k = gidf % NZ + b.lbnds; }
    else if (gid < 2 * a0 + 2 * a1) { gidf = gid - 2 * a0 - a1; i = gidf / (NZ * F) + b.lbnd + F; j = (gidf / NZ) % F + NY + NAB; k = gidf % NZ + b.lbnds; }
    else if (gid < 2 * a0 + 2 * a1 + a2) {
        gidf = gid - 2 * a0 - 2 * a1;
        i = gidf / (F * (NY - 2 * F)) + b.lbnd + F; j = (gidf / F) % (NY - 2 * F) + b.lbnd + F; k = gidf % F + NZ + b.lbnds - F;
    } else if (gid < 2 * a0 + 2 * a1 + 2 * a2) {
        gidf = gid - 2 * a0 - 2 * a1 - a2;
        i = gidf / (F * (NY - 2 * F)) + b.lbnd + F; j = (gidf / F) % (NY - 2 * F) + b.lbnd + F; k = gidf % F + b.lbnds;
    } else return false;
    return true;
}

// ------------------------------------------------------------------ taper
template <int NF, class T = float>
__device__ __forceinline__ void apply_taper(const Grid &g, const float *taper, int gz, int gy, int gx,
                                            T *const *fs, i64 iv)
{
    int F = g.F, NAB = g.nab;
    auto mul = [&](float t) {
        for (int q = 0; q < NF; q++) stv(fs[q] + iv, ldv(fs[q] + iv) * t);
    };
    if (!g.freesurf && gz - F < NAB) mul(__ldg(taper + gz - F));
    if (gz > g.NZl - NAB - F - 1 && gz < g.NZl - F) mul(__ldg(taper + g.NZl - F - gz - 1));
    if (g.nd == 3) {
        if (gy - F < NAB) mul(__ldg(taper + gy - F));
        if (gy > g.NY - NAB - F - 1) mul(__ldg(taper + g.NY - F - gy - 1));
    }
    if (gx - F < NAB) mul(__ldg(taper + gx - F));
    if (gx > g.NX - NAB - F - 1) mul(__ldg(taper + g.NX - F - gx - 1));
}

template <int NF>
__device__ __forceinline__ void taper_regs(const Grid &g, const float *taper, int gz, int gy, int gx, float (&v)[NF])
{
    const int F = g.F, NAB = g.nab;
    auto mul = [&](float t) {
#pragma unroll
        for (int q = 0; q < NF; q++) v[q] *= t;
    };
    if (!g.freesurf && gz - F < NAB) mul(__ldg(taper + gz - F));
    if (gz > g.NZl - NAB - F - 1 && gz < g.NZl - F) mul(__ldg(taper + g.NZl - F - gz - 1));
    if (gy - F < NAB) mul(__ldg(taper + gy - F));
    if (gy > g.NY - NAB - F - 1) mul(__ldg(taper + g.NY - F - gy - 1));
    if (gx - F < NAB) mul(__ldg(taper + gx - F));
    if (gx > g.NX - NAB - F - 1) mul(__ldg(taper + g.NX - F - gx - 1));
}

// ===================================================================== 2D
// CPML on the stress derivatives (update_v2D.cl:146-207)
__device__ __forceinline__ void cpml_v2d(const Grid &g, const Fields &f, int gz, int gx, float &sxx_x,
                                         float &szz_z, float &sxz_x, float &sxz_z)
{
    int F = g.F, NAB = g.nab, NZ = g.NZl, NX = g.NX;
    if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
        int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
        i64 q = (i64)i * (2 * NAB) + k;
        cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, sxz_z);
        cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, szz_z);
    } else if (!g.freesurf && gz - F < NAB && gz < NZ - F) {
        int i = gx - F, k = gz - F;
        i64 q = (i64)i * (2 * NAB) + k;
        cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, sxz_z);
        cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, szz_z);
    }
    if (gx - F < NAB) {
        int i = gx - F, k = gz - F;
        i64 q = (i64)i * g.nz + k;
        cpml(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], i, sxx_x);
        cpml(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], i, sxz_x);
    }
    if (gx > NX - NAB - F - 1) {
        int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
        i64 q = (i64)i * g.nz + k;
        cpml(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, sxx_x);
        cpml(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, sxz_x);
    }
}

// CPML on the velocity derivatives (update_s2D.cl:145-208)
__device__ __forceinline__ void cpml_s2d(const Grid &g, const Fields &f, int gz, int gx, float &vxx, float &vxz,
                                         float &vzx, float &vzz)
{
    int F = g.F, NAB = g.nab, NZ = g.NZl, NX = g.NX;
    if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
        int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
        i64 q = (i64)i * (2 * NAB) + k;
        cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vxz);
        cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, vzz);
    } else if (!g.freesurf && gz - F < NAB && gz < NZ - F) {
        int i = gx - F, k = gz - F;
        i64 q = (i64)i * (2 * NAB) + k;
        cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, vxz);
        cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, vzz);
    }
    if (gx - F < NAB) {
        int i = gx - F, k = gz - F;
        i64 q = (i64)i * g.nz + k;
        cpml(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], i, vxx);
        cpml(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], i, vzx);
    }
    if (gx > NX - NAB - F - 1) {
        int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
        i64 q = (i64)i * g.nz + k;
        cpml(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, vxx);
        cpml(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vzx);
    }
}

// ------------------------------------------------- P-SV cell arithmetic
__device__ __forceinline__ float v2d_math(float v, float dn, float ds, float buoy)
{
    return __fmaf_rn(__fadd_rn(dn, ds), buoy, v);
}

// material of a cell's stress update; elastic cells use fipkp, gm, fm only
struct S2dMat {
    float fipkp, gm, fm, dipkp, d, e;
};
__device__ __forceinline__ S2dMat s2d_elastic(float M, float mu, float muipkp)
{
    return S2dMat{muipkp, M, __fmul_rn(2.0f, mu), 0.0f, 0.0f, 0.0f};
}
__device__ __forceinline__ S2dMat s2d_visco(int L, float dt, float M, float mu, float muipkp, float taup, float taus,
                                            float tausipkp)
{
    S2dMat m;
    const float fl = (float)L;
    m.fipkp = __fmul_rn(muipkp, __fmaf_rn(fl, tausipkp, 1.0f));
    m.gm = __fmul_rn(M, __fmaf_rn(fl, taup, 1.0f));
    m.fm = __fmul_rn(__fmul_rn(2.0f, mu), __fmaf_rn(fl, taus, 1.0f));
    m.dipkp = __fdiv_rn(__fmul_rn(muipkp, tausipkp), dt);
    m.d = __fdiv_rn(__fmul_rn(__fmul_rn(2.0f, mu), taus), dt);
    m.e = __fdiv_rn(__fmul_rn(M, taup), dt);
    return m;
}
// a (vxx + vzz) - b v
__device__ __forceinline__ float s2d_normal(float a, float tr, float b, float v)
{
    return __fmaf_rn(-b, v, __fmul_rn(a, tr));
}
// one memory variable: b (r c - el x), b = Grid::eta_b, c = Grid::eta_c
__device__ __forceinline__ float s2d_memory(float r, float el, float b, float c, float x)
{
    return __fmul_rn(b, __fmaf_rn(r, c, -__fmul_rn(el, x)));
}
// stress increment without (elastic) / with the relaxed part: s + (rate + dt2 a)
__device__ __forceinline__ float s2d_add(float s, float rate, float dt2, float a)
{
    return __fadd_rn(s, __fmaf_rn(dt2, a, rate));
}
// free surface (surface2D.cl, surface3D.cl): what a column's correction of sxx
// (h) and of its memory variables (b hr) needs of its material and mechanisms
struct Surf2d {
    float q, qq, gm, c, de;   // gm - fm, its square, gm, (d - e)(fm / gm - 1), d - e
};
__device__ __forceinline__ Surf2d surf2d_of(const S2dMat &m)
{
    Surf2d s;
    s.q = __fsub_rn(m.gm, m.fm);
    s.qq = __fmul_rn(s.q, s.q);
    s.gm = m.gm;
    s.de = __fsub_rn(m.d, m.e);
    s.c = __fmul_rn(s.de, __fsub_rn(__fdiv_rn(m.fm, m.gm), 1.0f));
    return s;
}
__device__ __forceinline__ float surf2d_b(float eta) { return __fdiv_rn(eta, __fmaf_rn(eta, 0.5f, 1.0f)); }
// FMA: whether the second product is added in one rounding: elastic media, and
// the surface folded into the 3D stress update of whole rows
template <bool FMA>
__device__ __forceinline__ float surf2d_h(const Surf2d &s, float vxx, float vzz)
{
    const float t = __fdiv_rn(__fmul_rn(s.qq, vxx), s.gm);
    return FMA ? __fmaf_rn(-s.q, vzz, -t) : __fsub_rn(-t, __fmul_rn(s.q, vzz));
}
// what a mechanism's memory variable gains is b (surf2d_b) times this
__device__ __forceinline__ float surf2d_hr(const Surf2d &s, float vxx, float vzz)
{
    return __fmaf_rn(s.c, vxx, -__fmul_rn(s.de, vzz));
}

// elastic P-SV gradient terms of a cell: coefficients of its material, then
// the terms from the forward stresses and the adjoint increments
struct Adj2dCoef {
    float c1, c3;
};
__device__ __forceinline__ Adj2dCoef adj2d_coef(float M, float mu)
{
    const float q = __fmul_rn(2.0f, __fsub_rn(M, mu));
    return Adj2dCoef{__fdiv_rn(1.0f, __fmul_rn(q, q)), __fdiv_rn(1.0f, __fmul_rn(mu, mu))};
}
struct Adj2dGrad {
    float M, mu;
};
__device__ __forceinline__ Adj2dGrad adj2d_terms(int restype, Adj2dCoef k, float sxx, float szz, float sxz, float lsxx,
                                                 float lszz, float lsxz)
{
    const float p = __fadd_rn(sxx, szz), lp = __fadd_rn(lsxx, lszz);
    if (restype != 0) return Adj2dGrad{-__fmul_rn(p, lp), 0.0f};
    const float dM = __fmul_rn(__fmul_rn(k.c1, p), lp);
    const float sh = __fmaf_rn(-k.c3, __fmul_rn(sxz, lsxz), dM);
    return Adj2dGrad{-dM, __fmaf_rn(-__fmul_rn(0.25f, k.c3), __fmul_rn(__fsub_rn(sxx, szz), __fsub_rn(lsxx, lszz)), sh)};
}
__device__ __forceinline__ Adj2dGrad adj2d_grad(int restype, float M, float mu, float sxx, float szz, float sxz,
                                                float lsxx, float lszz, float lsxz)
{
    return adj2d_terms(restype, adj2d_coef(M, mu), sxx, szz, sxz, lsxx, lszz, lsxz);
}

}  // namespace sfd
