// sfd_kernels.cu -- general sm_100a kernels of the staggered-grid FDTD engine.
//
// One thread per grid cell; z (fastest) runs along the warp so every stencil
// tap is a coalesced row load served from L1/L2.  These kernels cover every
// configuration the engine accepts (2D P-SV and 3D, FDORDER 2..12, elastic
// and viscoelastic, CPML or Cerjan taper, free surface) and are the
// reference implementation inside the product; sfd_kernels3d_fast.cu holds
// the register-blocked 3D kernels used on the hot configurations.
//
// Semantics follow the reference kernels cell for cell:
//   update_v  src/update_v2D.cl:32-246,  src/update_v3D.cl:34-369
//   update_s  src/update_s2D.cl:30-327,  src/update_s3D.cl:35-489
//   surface   src/surface2D.cl:30-193,   src/surface3D.cl:39-271
//   adjoint   src/update_adj{v,s}{2D,3D}.cl, src/surface{2D,3D}_adj.cl
//   boundary  src/savebnd{2D,3D}.cl, src/header_injectbnd.cl
// Arithmetic is FP32 with FMA; gradients accumulate in FP64.
#include <algorithm>
#include <cstring>
#include <cstdlib>
#include <utility>
#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "sfd_device.cuh"
#include "sfd_internal.h"
#include "sfd_kernels.h"
#include "sfd_launch.cuh"

namespace sfd {

// T: storage of the wave fields and memory variables (float, or __half
// holding them times power-of-two scales; the arithmetic is FP32)
template <int F, class T = float>
__global__ void __launch_bounds__(256) k_v2d(Grid g, Fields f)
{
    SHOT_F
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    const float *hc = g.hc;
    T *vx = fld<T>(f.w[VX]), *vz = fld<T>(f.w[VZ]);
    float sxx_x = dfwT<F>(fld<T>(f.w[SXX]), iv, g.NZ, hc);
    float szz_z = dfwT<F>(fld<T>(f.w[SZZ]), iv, 1, hc);
    float sxz_z = dbwT<F>(fld<T>(f.w[SXZ]), iv, 1, hc);
    float sxz_x = dbwT<F>(fld<T>(f.w[SXZ]), iv, g.NZ, hc);
    if (g.abs_type == 1) cpml_v2d(g, f, gz, gx, sxx_x, szz_z, sxz_x, sxz_z);
    stv(vx + iv, v2d_math(ldv(vx + iv), sxx_x, sxz_z, __ldg(f.p[PRIP] + ip)));
    stv(vz + iv, v2d_math(ldv(vz + iv), szz_z, sxz_x, __ldg(f.p[PRKP] + ip)));
    if (g.abs_type == 2) {
        T *fs[2] = {vx, vz};
        apply_taper<2>(g, f.taper, gz, 0, gx, fs, iv);
    }
}

// one cell of the P-SV stress update (update_s2D.cl:30-327)
template <int F, class T = float>
__device__ __forceinline__ void s2d_cell(const Grid &g, const Fields &f, int gz, int gx)
{
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    const float *hc = g.hc;
    T *wsxx = fld<T>(f.w[SXX]), *wszz = fld<T>(f.w[SZZ]), *wsxz = fld<T>(f.w[SXZ]);
    float vxx = dbwT<F>(fld<T>(f.w[VX]), iv, g.NZ, hc);
    float vxz = dfwT<F>(fld<T>(f.w[VX]), iv, 1, hc);
    float vzz = dbwT<F>(fld<T>(f.w[VZ]), iv, 1, hc);
    float vzx = dfwT<F>(fld<T>(f.w[VZ]), iv, g.NZ, hc);
    if (g.abs_type == 1) cpml_s2d(g, f, gz, gx, vxx, vxz, vzx, vzz);
    const int L = g.L;
    const float tr = __fadd_rn(vxx, vzz), sh = __fadd_rn(vxz, vzx);
    if (L == 0) {
        const S2dMat m = s2d_elastic(__ldg(f.p[PM] + ip), __ldg(f.p[PMU] + ip), __ldg(f.p[PMUIPKP] + ip));
        stv(wsxz + iv, __fmaf_rn(m.fipkp, sh, ldv(wsxz + iv)));
        stv(wsxx + iv, __fadd_rn(ldv(wsxx + iv), s2d_normal(m.gm, tr, m.fm, vzz)));
        stv(wszz + iv, __fadd_rn(ldv(wszz + iv), s2d_normal(m.gm, tr, m.fm, vxx)));
    } else {
        const S2dMat m = s2d_visco(L, g.dt, __ldg(f.p[PM] + ip), __ldg(f.p[PMU] + ip), __ldg(f.p[PMUIPKP] + ip),
                                   __ldg(f.p[PTAUP] + ip), __ldg(f.p[PTAUS] + ip), __ldg(f.p[PTAUSIPKP] + ip));
        T *rxx = fld<T>(f.r[RXX]), *rzz = fld<T>(f.r[RZZ]), *rxz = fld<T>(f.r[RXZ]);
        float sxz_ = 0, sxx_ = 0, szz_ = 0;
        for (int l = 0; l < L; l++) {
            i64 ir = l * g.nvol + iv;
            sxz_ += ldv(rxz + ir); sxx_ += ldv(rxx + ir); szz_ += ldv(rzz + ir);
        }
        const float lsxz = __fmaf_rn(m.fipkp, sh, __fmul_rn(g.dt2, sxz_));
        const float lsxx = __fmaf_rn(g.dt2, sxx_, s2d_normal(m.gm, tr, m.fm, vzz));
        const float lszz = __fmaf_rn(g.dt2, szz_, s2d_normal(m.gm, tr, m.fm, vxx));
        sxz_ = sxx_ = szz_ = 0;
        for (int l = 0; l < L; l++) {
            const float el = g.eta[l];
            i64 ir = l * g.nvol + iv;
            float a1 = s2d_memory(ldv(rxz + ir), el, g.eta_b[l], g.eta_c[l], __fmul_rn(m.dipkp, sh));
            float a2 = s2d_memory(ldv(rxx + ir), el, g.eta_b[l], g.eta_c[l], s2d_normal(m.e, tr, m.d, vzz));
            float a3 = s2d_memory(ldv(rzz + ir), el, g.eta_b[l], g.eta_c[l], s2d_normal(m.e, tr, m.d, vxx));
            stv(rxz + ir, a1); stv(rxx + ir, a2); stv(rzz + ir, a3);
            // the stored values (rounded to T) are what the next step reads;
            // the sums use the FP32 ones, as the FP32 build does
            sxz_ += a1; sxx_ += a2; szz_ += a3;
        }
        stv(wsxz + iv, s2d_add(ldv(wsxz + iv), lsxz, g.dt2, sxz_));
        stv(wsxx + iv, s2d_add(ldv(wsxx + iv), lsxx, g.dt2, sxx_));
        stv(wszz + iv, s2d_add(ldv(wszz + iv), lszz, g.dt2, szz_));
    }
    if (g.abs_type == 2) {
        T *fs[3] = {wsxx, wszz, wsxz};
        apply_taper<3>(g, f.taper, gz, 0, gx, fs, iv);
    }
}

// free surface of one column (surface2D.cl:30-193)
template <int F, class T = float>
__device__ __forceinline__ void surf2d_column(const Grid &g, const Fields &f, int gx, int pdir)
{
    int gz = F, NZ = g.NZ, L = g.L, NAB = g.nab;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * NZ + gz;
    T *vx = fld<T>(f.w[VX]), *vz = fld<T>(f.w[VZ]), *sxx = fld<T>(f.w[SXX]), *szz = fld<T>(f.w[SZZ]),
      *sxz = fld<T>(f.w[SXZ]);
    T *rxx = fld<T>(f.r[RXX]), *rzz = fld<T>(f.r[RZZ]);
    stv(szz + iv, 0.0f);
    for (int l = 0; l < L; l++) stv(rzz + l * g.nvol + iv, 0.0f);
#pragma unroll
    for (int m = 1; m <= F; m++) {
        stv(szz + iv - m, -ldv(szz + iv + m));
        stv(sxz + iv - m, -ldv(sxz + iv + m - 1));
    }
    float vxx = dbw_rwT<F>(vx, iv, NZ, g.hc);
    float vzz = dbw_rwT<F>(vz, iv, 1, g.hc);
    if (g.abs_type == 1) {
        if (gx - F < NAB) {
            int i = gx - F;
            vxx = cpml_quot(vxx, f.kq[0][0][i], f.psi[PVX_X][(i64)i * g.nz + (gz - F)]);
        }
        if (gx > g.NX - NAB - F - 1) {
            int i = gx - g.NX + NAB + F + NAB, ind = 2 * NAB - 1 - i;
            vxx = cpml_quot(vxx, f.kq[0][0][ind + 1], f.psi[PVX_X][(i64)i * g.nz + (gz - F)]);
        }
    }
    const float sg = (float)pdir;
    if (L == 0) {
        const S2dMat m = s2d_elastic(f.p[PM][ip], f.p[PMU][ip], 0.0f);
        stv(sxx + iv, __fmaf_rn(sg, surf2d_h<true>(surf2d_of(m), vxx, vzz), ldv(sxx + iv)));
    } else {
        const S2dMat m = s2d_visco(L, g.dt, f.p[PM][ip], f.p[PMU][ip], 0.0f, f.p[PTAUP][ip], f.p[PTAUS][ip], 0.0f);
        float sump = 0;
        for (int l = 0; l < L; l++) sump += ldv(rxx + l * g.nvol + iv);
        const Surf2d su = surf2d_of(m);
        const float h = __fmaf_rn(-g.dt2, sump, surf2d_h<false>(su, vxx, vzz));
        stv(sxx + iv, __fmaf_rn(sg, h, ldv(sxx + iv)));
        sump = 0;
        for (int l = 0; l < L; l++) {
            const float hh = __fmul_rn(surf2d_b(g.eta[l]), surf2d_hr(su, vxx, vzz));
            float r = __fmaf_rn(sg, hh, ldv(rxx + l * g.nvol + iv));
            stv(rxx + l * g.nvol + iv, r);
            sump += r;
        }
        stv(sxx + iv, __fmaf_rn(sg, __fmul_rn(g.dt2, sump), ldv(sxx + iv)));
    }
}

// free surface, one thread per surface column
template <int F, class T = float>
__global__ void k_surf2d(Grid g, Fields f, int pdir)
{
    SHOT_F
    int gx = blockIdx.x * blockDim.x + threadIdx.x + F;
    if (gx <= g.NX - F - 1) surf2d_column<F, T>(g, f, gx, pdir);
}

template <int F, class T = float>
__global__ void __launch_bounds__(256) k_s2d(Grid g, Fields f)
{
    SHOT_F
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz <= g.NZ - F - 1 && gx <= g.NX - F - 1) s2d_cell<F, T>(g, f, gz, gx);
}

// ===================================================================== 3D
__device__ __forceinline__ void cpml_v3d(const Grid &g, const Fields &f, int gz, int gy, int gx, float &sxx_x,
                                         float &syy_y, float &szz_z, float &sxy_y, float &sxy_x, float &syz_y,
                                         float &syz_z, float &sxz_x, float &sxz_z)
{
    int F = g.F, NAB = g.nab, NZ = g.NZl, NY = g.NY, NX = g.NX;
    i64 nz = g.nz, ny = g.ny;
    if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
        i64 i = gx - F, j = gy - F, k = gz - NZ + NAB + F + NAB;
        int ind = 2 * NAB - 1 - (int)k;
        i64 q = (i * ny + j) * (2 * NAB) + k;
        cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, sxz_z);
        cpml(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, syz_z);
        cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, szz_z);
    } else if (!g.freesurf && gz - F < NAB) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * ny + j) * (2 * NAB) + k;
        cpml(f.psi[PSXZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, sxz_z);
        cpml(f.psi[PSYZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, syz_z);
        cpml(f.psi[PSZZ_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, szz_z);
    }
    if (gy - F < NAB) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * (2 * NAB) + j) * nz + k;
        cpml(f.psi[PSXY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, sxy_y);
        cpml(f.psi[PSYY_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, syy_y);
        cpml(f.psi[PSYZ_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, syz_y);
    } else if (gy > NY - NAB - F - 1) {
        i64 i = gx - F, j = gy - NY + NAB + F + NAB, k = gz - F;
        int ind = 2 * NAB - 1 - (int)j;
        i64 q = (i * (2 * NAB) + j) * nz + k;
        cpml(f.psi[PSXY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, sxy_y);
        cpml(f.psi[PSYY_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, syy_y);
        cpml(f.psi[PSYZ_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, syz_y);
    }
    if (gx - F < NAB) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * ny + j) * nz + k;
        cpml(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, sxx_x);
        cpml(f.psi[PSXY_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, sxy_x);
        cpml(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, sxz_x);
    }
    if (gx > NX - NAB - F - 1) {
        i64 i = gx - NX + NAB + F + NAB, j = gy - F, k = gz - F;
        int ind = 2 * NAB - 1 - (int)i;
        i64 q = (i * ny + j) * nz + k;
        cpml(f.psi[PSXX_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, sxx_x);
        cpml(f.psi[PSXY_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, sxy_x);
        cpml(f.psi[PSXZ_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, sxz_x);
    }
}

// update_s3D.cl:190-298 (plain "if"s); the adjoint form uses "else if" for the
// z-top and y-far branches (update_adjs3D.cl)
__device__ __forceinline__ void cpml_s3d(const Grid &g, const Fields &f, int gz, int gy, int gx, float &vxx,
                                         float &vxy, float &vxz, float &vyx, float &vyy, float &vyz, float &vzx,
                                         float &vzy, float &vzz, bool adjoint_form)
{
    int F = g.F, NAB = g.nab, NZ = g.NZl, NY = g.NY, NX = g.NX;
    i64 nz = g.nz, ny = g.ny;
    bool zb = gz > NZ - NAB - F - 1 && gz < NZ - F;
    if (zb) {
        i64 i = gx - F, j = gy - F, k = gz - NZ + NAB + F + NAB;
        int ind = 2 * NAB - 1 - (int)k;
        i64 q = (i * ny + j) * (2 * NAB) + k;
        cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vxz);
        cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vyz);
        cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, vzz);
    }
    if (!g.freesurf && gz - F < NAB && !(adjoint_form && zb)) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * ny + j) * (2 * NAB) + k;
        cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vxz);
        cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vyz);
        cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, vzz);
    }
    bool yb = gy - F < NAB;
    if (yb) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * (2 * NAB) + j) * nz + k;
        cpml(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vxy);
        cpml(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, vyy);
        cpml(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vzy);
    }
    if (gy > NY - NAB - F - 1 && !(adjoint_form && yb)) {
        i64 i = gx - F, j = gy - NY + NAB + F + NAB, k = gz - F;
        int ind = 2 * NAB - 1 - (int)j;
        i64 q = (i * (2 * NAB) + j) * nz + k;
        cpml(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, vxy);
        cpml(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], ind + 1, vyy);
        cpml(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], ind, vzy);
    }
    if (gx - F < NAB) {
        i64 i = gx - F, j = gy - F, k = gz - F;
        i64 q = (i * ny + j) * nz + k;
        cpml(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], (int)i, vxx);
        cpml(f.psi[PVY_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, vyx);
        cpml(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], (int)i, vzx);
    }
    if (gx > NX - NAB - F - 1) {
        i64 i = gx - NX + NAB + F + NAB, j = gy - F, k = gz - F;
        int ind = 2 * NAB - 1 - (int)i;
        i64 q = (i * ny + j) * nz + k;
        cpml(f.psi[PVX_X], q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, vxx);
        cpml(f.psi[PVY_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vyx);
        cpml(f.psi[PVZ_X], q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vzx);
    }
}

// grid z: the x blocks of each shot of the launch, shot after shot
#define SHOT3D                                                                         \
    int shot = 0, xb_ = blockIdx.z;                                                    \
    if (MB) {                                                                          \
        const int nxb_ = gridDim.z / g.nb;                                             \
        shot = blockIdx.z / nxb_;                                                      \
        xb_ = blockIdx.z - shot * nxb_;                                                \
    }
#define CELL3D                                                                         \
    SHOT3D                                                                             \
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;                                \
    int gy = blockIdx.y * blockDim.y + threadIdx.y + F;                                \
    int gx = xb_ * blockDim.z + threadIdx.z + F;                                       \
    if (gz > g.NZ - F - 1 || gy > g.NY - F - 1 || gx > g.NX - F - 1) return;           \
    if (MB) shot_fields(g, f, shot);                                                   \
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;                                        \
    i64 iv = gx * sx + (i64)gy * sy + gz;                                              \
    i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz - F);

template <int F, bool MB = false>
__global__ void __launch_bounds__(256) k_v3d(Grid g, Fields f)
{
    CELL3D
    const float *hc = g.hc;
    float szz_z = dfw<F>(f.w[SZZ], iv, 1, hc);
    float sxx_x = dfw<F>(f.w[SXX], iv, sx, hc);
    float sxz_x = dbw<F>(f.w[SXZ], iv, sx, hc);
    float sxz_z = dbw<F>(f.w[SXZ], iv, 1, hc);
    float syz_y = dbw<F>(f.w[SYZ], iv, sy, hc);
    float syz_z = dbw<F>(f.w[SYZ], iv, 1, hc);
    float syy_y = dfw<F>(f.w[SYY], iv, sy, hc);
    float sxy_x = dbw<F>(f.w[SXY], iv, sx, hc);
    float sxy_y = dbw<F>(f.w[SXY], iv, sy, hc);
    if (g.abs_type == 1) cpml_v3d(g, f, gz, gy, gx, sxx_x, syy_y, szz_z, sxy_y, sxy_x, syz_y, syz_z, sxz_x, sxz_z);
    f.w[VX][iv] += (sxx_x + sxy_y + sxz_z) * __ldg(f.p[PRIP] + ip);
    f.w[VY][iv] += (syy_y + sxy_x + syz_z) * __ldg(f.p[PRJP] + ip);
    f.w[VZ][iv] += (szz_z + sxz_x + syz_y) * __ldg(f.p[PRKP] + ip);
    if (g.abs_type == 2) {
        float *fs[3] = {f.w[VX], f.w[VY], f.w[VZ]};
        apply_taper<3>(g, f.taper, gz, gy, gx, fs, iv);
    }
}

template <int F, bool MB = false>
__global__ void __launch_bounds__(256) k_s3d(Grid g, Fields f)
{
    CELL3D
    const float *hc = g.hc;
    float vzx = dfw<F>(f.w[VZ], iv, sx, hc), vzy = dfw<F>(f.w[VZ], iv, sy, hc), vzz = dbw<F>(f.w[VZ], iv, 1, hc);
    float vyx = dfw<F>(f.w[VY], iv, sx, hc), vyy = dbw<F>(f.w[VY], iv, sy, hc), vyz = dfw<F>(f.w[VY], iv, 1, hc);
    float vxx = dbw<F>(f.w[VX], iv, sx, hc), vxy = dfw<F>(f.w[VX], iv, sy, hc), vxz = dfw<F>(f.w[VX], iv, 1, hc);
    if (g.abs_type == 1) cpml_s3d(g, f, gz, gy, gx, vxx, vxy, vxz, vyx, vyy, vyz, vzx, vzy, vzz, false);
    float vxyyx = vxy + vyx, vyzzy = vyz + vzy, vxzzx = vxz + vzx;
    float vxxyyzz = vxx + vyy + vzz, vyyzz = vyy + vzz, vxxzz = vxx + vzz, vxxyy = vxx + vyy;
    const int L = g.L;
    if (L == 0) {
        float fipjp = __ldg(f.p[PMUIPJP] + ip), fjpkp = __ldg(f.p[PMUJPKP] + ip), fipkp = __ldg(f.p[PMUIPKP] + ip);
        float gm = __ldg(f.p[PM] + ip), fm = 2.0f * __ldg(f.p[PMU] + ip);
        f.w[SXY][iv] += fipjp * vxyyx;
        f.w[SYZ][iv] += fjpkp * vyzzy;
        f.w[SXZ][iv] += fipkp * vxzzx;
        f.w[SXX][iv] += gm * vxxyyzz - fm * vyyzz;
        f.w[SYY][iv] += gm * vxxyyzz - fm * vxxzz;
        f.w[SZZ][iv] += gm * vxxyyzz - fm * vxxyy;
    } else {
        float lM = __ldg(f.p[PM] + ip), lmu = __ldg(f.p[PMU] + ip);
        float lmuipkp = __ldg(f.p[PMUIPKP] + ip), lmuipjp = __ldg(f.p[PMUIPJP] + ip), lmujpkp = __ldg(f.p[PMUJPKP] + ip);
        float ltaup = __ldg(f.p[PTAUP] + ip), ltaus = __ldg(f.p[PTAUS] + ip);
        float ltausipkp = __ldg(f.p[PTAUSIPKP] + ip), ltausipjp = __ldg(f.p[PTAUSIPJP] + ip),
              ltausjpkp = __ldg(f.p[PTAUSJPKP] + ip);
        float fipjp = lmuipjp * (1.0f + (float)L * ltausipjp);
        float fjpkp = lmujpkp * (1.0f + (float)L * ltausjpkp);
        float fipkp = lmuipkp * (1.0f + (float)L * ltausipkp);
        float gm = lM * (1.0f + (float)L * ltaup);
        float fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
        float dipjp = lmuipjp * ltausipjp / g.dt, djpkp = lmujpkp * ltausjpkp / g.dt, dipkp = lmuipkp * ltausipkp / g.dt;
        float d = 2.0f * lmu * ltaus / g.dt, e = lM * ltaup / g.dt;
        float a[6] = {0, 0, 0, 0, 0, 0};
        float *const *r = f.r;
        for (int l = 0; l < L; l++) {
            i64 ir = l * g.nvol + iv;
            a[0] += r[RXY][ir]; a[1] += r[RYZ][ir]; a[2] += r[RXZ][ir];
            a[3] += r[RXX][ir]; a[4] += r[RYY][ir]; a[5] += r[RZZ][ir];
        }
        float lsxy = fipjp * vxyyx + g.dt2 * a[0];
        float lsyz = fjpkp * vyzzy + g.dt2 * a[1];
        float lsxz = fipkp * vxzzx + g.dt2 * a[2];
        float lsxx = (gm * vxxyyzz - fm * vyyzz) + g.dt2 * a[3];
        float lsyy = (gm * vxxyyzz - fm * vxxzz) + g.dt2 * a[4];
        float lszz = (gm * vxxyyzz - fm * vxxyy) + g.dt2 * a[5];
        for (int q = 0; q < 6; q++) a[q] = 0;
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
            i64 ir = l * g.nvol + iv;
            float n0 = b * (r[RXY][ir] * c - el * (dipjp * vxyyx));
            float n1 = b * (r[RYZ][ir] * c - el * (djpkp * vyzzy));
            float n2 = b * (r[RXZ][ir] * c - el * (dipkp * vxzzx));
            float n3 = b * (r[RXX][ir] * c - el * (e * vxxyyzz - d * vyyzz));
            float n4 = b * (r[RYY][ir] * c - el * (e * vxxyyzz - d * vxxzz));
            float n5 = b * (r[RZZ][ir] * c - el * (e * vxxyyzz - d * vxxyy));
            r[RXY][ir] = n0; r[RYZ][ir] = n1; r[RXZ][ir] = n2; r[RXX][ir] = n3; r[RYY][ir] = n4; r[RZZ][ir] = n5;
            a[0] += n0; a[1] += n1; a[2] += n2; a[3] += n3; a[4] += n4; a[5] += n5;
        }
        f.w[SXY][iv] += lsxy + g.dt2 * a[0];
        f.w[SYZ][iv] += lsyz + g.dt2 * a[1];
        f.w[SXZ][iv] += lsxz + g.dt2 * a[2];
        f.w[SXX][iv] += lsxx + g.dt2 * a[3];
        f.w[SYY][iv] += lsyy + g.dt2 * a[4];
        f.w[SZZ][iv] += lszz + g.dt2 * a[5];
    }
    if (g.abs_type == 2) {
        float *fs[6] = {f.w[SXY], f.w[SYZ], f.w[SXZ], f.w[SXX], f.w[SYY], f.w[SZZ]};
        apply_taper<6>(g, f.taper, gz, gy, gx, fs, iv);
    }
}

// ----------------------------------------------------- streaming 3D kernels
// Same arithmetic as k_v3d / k_s3d, one thread per cell, but every per-cell
// stream (the updated fields, memory variables and parameters) is loaded
// into registers before the stencil work starts, so each thread has all of
// its independent DRAM loads in flight at once; the updated values are
// stored once at the end (taper applied in registers, in the reference's
// factor order).  L is a template parameter so the memory variables stay in
// registers.  The stencil taps go through the read-only cache as in the
// general kernels.
template <int F, class T = float, bool MB = false>
__global__ void __launch_bounds__(256, 3) k_v3d_stream(Grid g, Fields f)
{
    CELL3D
    const float *hc = g.hc;
    T *wvx = fld<T>(f.w[VX]), *wvy = fld<T>(f.w[VY]), *wvz = fld<T>(f.w[VZ]);
    float v[3] = {ldgv(wvx + iv), ldgv(wvy + iv), ldgv(wvz + iv)};
    const float rip = __ldg(f.p[PRIP] + ip), rjp = __ldg(f.p[PRJP] + ip), rkp = __ldg(f.p[PRKP] + ip);
    const T *Sxx = fld<T>(f.w[SXX]), *Syy = fld<T>(f.w[SYY]), *Szz = fld<T>(f.w[SZZ]);
    const T *Sxy = fld<T>(f.w[SXY]), *Syz = fld<T>(f.w[SYZ]), *Sxz = fld<T>(f.w[SXZ]);
    float szz_z = dfwT<F>(Szz, iv, 1, hc);
    float sxx_x = dfwT<F>(Sxx, iv, sx, hc);
    float sxz_x = dbwT<F>(Sxz, iv, sx, hc);
    float sxz_z = dbwT<F>(Sxz, iv, 1, hc);
    float syz_y = dbwT<F>(Syz, iv, sy, hc);
    float syz_z = dbwT<F>(Syz, iv, 1, hc);
    float syy_y = dfwT<F>(Syy, iv, sy, hc);
    float sxy_x = dbwT<F>(Sxy, iv, sx, hc);
    float sxy_y = dbwT<F>(Sxy, iv, sy, hc);
    if (g.abs_type == 1) cpml_v3d(g, f, gz, gy, gx, sxx_x, syy_y, szz_z, sxy_y, sxy_x, syz_y, syz_z, sxz_x, sxz_z);
    v[0] += (sxx_x + sxy_y + sxz_z) * rip;
    v[1] += (syy_y + sxy_x + syz_z) * rjp;
    v[2] += (szz_z + sxz_x + syz_y) * rkp;
    if (g.abs_type == 2) taper_regs<3>(g, f.taper, gz, gy, gx, v);
    stv(wvx + iv, v[0]);
    stv(wvy + iv, v[1]);
    stv(wvz + iv, v[2]);
}

template <int F, int L, class T = float, bool MB = false>
__global__ void __launch_bounds__(256, 2) k_s3d_stream(Grid g, Fields f)
{
    CELL3D
    const float *hc = g.hc;
    // per-cell streams first: stresses, memory variables, parameters
    T *ws[6] = {fld<T>(f.w[SXY]), fld<T>(f.w[SYZ]), fld<T>(f.w[SXZ]),
                fld<T>(f.w[SXX]), fld<T>(f.w[SYY]), fld<T>(f.w[SZZ])};
    T *wr[6] = {fld<T>(f.r[RXY]), fld<T>(f.r[RYZ]), fld<T>(f.r[RXZ]),
                fld<T>(f.r[RXX]), fld<T>(f.r[RYY]), fld<T>(f.r[RZZ])};
    float s[6];
#pragma unroll
    for (int q = 0; q < 6; q++) s[q] = ldgv(ws[q] + iv);
    float r[6][L > 0 ? L : 1];
#pragma unroll
    for (int l = 0; l < L; l++) {
        const i64 ir = l * g.nvol + iv;
#pragma unroll
        for (int q = 0; q < 6; q++) r[q][l] = ldgv(wr[q] + ir);
    }
    const float lM = __ldg(f.p[PM] + ip), lmu = __ldg(f.p[PMU] + ip);
    const float lmuipkp = __ldg(f.p[PMUIPKP] + ip), lmuipjp = __ldg(f.p[PMUIPJP] + ip),
                lmujpkp = __ldg(f.p[PMUJPKP] + ip);
    float ltaup = 0, ltaus = 0, ltausipkp = 0, ltausipjp = 0, ltausjpkp = 0;
    if (L > 0) {
        ltaup = __ldg(f.p[PTAUP] + ip); ltaus = __ldg(f.p[PTAUS] + ip);
        ltausipkp = __ldg(f.p[PTAUSIPKP] + ip); ltausipjp = __ldg(f.p[PTAUSIPJP] + ip);
        ltausjpkp = __ldg(f.p[PTAUSJPKP] + ip);
    }
    const T *Vx = fld<T>(f.w[VX]), *Vy = fld<T>(f.w[VY]), *Vz = fld<T>(f.w[VZ]);
    float vzx = dfwT<F>(Vz, iv, sx, hc), vzy = dfwT<F>(Vz, iv, sy, hc), vzz = dbwT<F>(Vz, iv, 1, hc);
    float vyx = dfwT<F>(Vy, iv, sx, hc), vyy = dbwT<F>(Vy, iv, sy, hc), vyz = dfwT<F>(Vy, iv, 1, hc);
    float vxx = dbwT<F>(Vx, iv, sx, hc), vxy = dfwT<F>(Vx, iv, sy, hc), vxz = dfwT<F>(Vx, iv, 1, hc);
    if (g.abs_type == 1) cpml_s3d(g, f, gz, gy, gx, vxx, vxy, vxz, vyx, vyy, vyz, vzx, vzy, vzz, false);
    float vxyyx = vxy + vyx, vyzzy = vyz + vzy, vxzzx = vxz + vzx;
    float vxxyyzz = vxx + vyy + vzz, vyyzz = vyy + vzz, vxxzz = vxx + vzz, vxxyy = vxx + vyy;
    if (L == 0) {
        float gm = lM, fm = 2.0f * lmu;
        s[0] += lmuipjp * vxyyx;
        s[1] += lmujpkp * vyzzy;
        s[2] += lmuipkp * vxzzx;
        s[3] += gm * vxxyyzz - fm * vyyzz;
        s[4] += gm * vxxyyzz - fm * vxxzz;
        s[5] += gm * vxxyyzz - fm * vxxyy;
    } else {
        float fipjp = lmuipjp * (1.0f + (float)L * ltausipjp);
        float fjpkp = lmujpkp * (1.0f + (float)L * ltausjpkp);
        float fipkp = lmuipkp * (1.0f + (float)L * ltausipkp);
        float gm = lM * (1.0f + (float)L * ltaup);
        float fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
        float dipjp = lmuipjp * ltausipjp / g.dt, djpkp = lmujpkp * ltausjpkp / g.dt, dipkp = lmuipkp * ltausipkp / g.dt;
        float d = 2.0f * lmu * ltaus / g.dt, e = lM * ltaup / g.dt;
        float a[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 6; q++) a[q] += r[q][l];
        float ls[6] = {fipjp * vxyyx + g.dt2 * a[0], fjpkp * vyzzy + g.dt2 * a[1], fipkp * vxzzx + g.dt2 * a[2],
                       (gm * vxxyyzz - fm * vyyzz) + g.dt2 * a[3], (gm * vxxyyzz - fm * vxxzz) + g.dt2 * a[4],
                       (gm * vxxyyzz - fm * vxxyy) + g.dt2 * a[5]};
#pragma unroll
        for (int q = 0; q < 6; q++) a[q] = 0;
#pragma unroll
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
            r[0][l] = b * (r[0][l] * c - el * (dipjp * vxyyx));
            r[1][l] = b * (r[1][l] * c - el * (djpkp * vyzzy));
            r[2][l] = b * (r[2][l] * c - el * (dipkp * vxzzx));
            r[3][l] = b * (r[3][l] * c - el * (e * vxxyyzz - d * vyyzz));
            r[4][l] = b * (r[4][l] * c - el * (e * vxxyyzz - d * vxxzz));
            r[5][l] = b * (r[5][l] * c - el * (e * vxxyyzz - d * vxxyy));
#pragma unroll
            for (int q = 0; q < 6; q++) a[q] += r[q][l];
            const i64 ir = l * g.nvol + iv;
#pragma unroll
            for (int q = 0; q < 6; q++) stv(wr[q] + ir, r[q][l]);
        }
#pragma unroll
        for (int q = 0; q < 6; q++) s[q] += ls[q] + g.dt2 * a[q];
    }
    if (g.abs_type == 2) taper_regs<6>(g, f.taper, gz, gy, gx, s);
#pragma unroll
    for (int q = 0; q < 6; q++) stv(ws[q] + iv, s[q]);
}

// free surface 3D, one thread per (y, x) column (surface3D.cl:39-271)
// TR: storage type of the memory variables; values are read times
// g.rsci and stored times g.rsc (1 except with Grid::rhalf)
template <int F, class T = float, class TR = T>
__global__ void k_surf3d(Grid g, Fields f, int pdir)
{
    SHOT_F
    int gy = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gy > g.NY - F - 1 || gx > g.NX - F - 1) return;
    int gz = F, NAB = g.nab, L = g.L;
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    i64 iv = gx * sx + (i64)gy * sy + gz;
    i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz - F);
    T *sxx = fld<T>(f.w[SXX]), *syy = fld<T>(f.w[SYY]), *szz = fld<T>(f.w[SZZ]), *syz = fld<T>(f.w[SYZ]),
      *sxz = fld<T>(f.w[SXZ]);
    TR *rxx = fld<TR>(f.r[RXX]), *ryy = fld<TR>(f.r[RYY]), *rzz = fld<TR>(f.r[RZZ]);
    stv(szz + iv, 0.0f);
    for (int l = 0; l < L; l++) stv(rzz + l * g.nvol + iv, 0.0f);
#pragma unroll
    for (int m = 1; m <= F; m++) {
        stv(szz + iv - m, -ldv(szz + iv + m));
        stv(sxz + iv - m, -ldv(sxz + iv + m - 1));
        stv(syz + iv - m, -ldv(syz + iv + m - 1));
    }
    float vxx = dbw_rwT<F>(fld<T>(f.w[VX]), iv, sx, g.hc);
    float vyy = dbw_rwT<F>(fld<T>(f.w[VY]), iv, sy, g.hc);
    float vzz = dbw_rwT<F>(fld<T>(f.w[VZ]), iv, 1, g.hc);
    if (g.abs_type == 1) {
        i64 nz = g.nz, ny = g.ny;
        if (gy - F < NAB) {
            i64 i = gx - F, j = gy - F;
            vyy = __fmaf_rn(vyy, f.kinv[1][0][j], f.psi[PVY_Y][(i * (2 * NAB) + j) * nz]);
        } else if (gy > g.NY - NAB - F - 1) {
            i64 i = gx - F, j = gy - g.NY + NAB + F + NAB;
            int ind = 2 * NAB - 1 - (int)j;
            vyy = __fmaf_rn(vyy, f.kinv[1][0][ind + 1], f.psi[PVY_Y][(i * (2 * NAB) + j) * nz]);
        }
        if (gx - F < NAB) {
            i64 i = gx - F, j = gy - F;
            vxx = __fmaf_rn(vxx, f.kinv[0][0][i], f.psi[PVX_X][(i * ny + j) * nz]);
        }
        if (gx > g.NX - NAB - F - 1) {
            i64 i = gx - g.NX + NAB + F + NAB, j = gy - F;
            int ind = 2 * NAB - 1 - (int)i;
            vxx = __fmaf_rn(vxx, f.kinv[0][0][ind + 1], f.psi[PVX_X][(i * ny + j) * nz]);
        }
    }
    const float vh = __fadd_rn(vxx, vyy), sg = (float)pdir;
    if (L == 0) {
        // the reference adds h without the propagation direction (surface3D.cl:172-173)
        const float h = surf2d_h<true>(surf2d_of(s2d_elastic(f.p[PM][ip], f.p[PMU][ip], 0.0f)), vh, vzz);
        stv(sxx + iv, __fadd_rn(ldv(sxx + iv), h));
        stv(syy + iv, __fadd_rn(ldv(syy + iv), h));
    } else {
        const Surf2d su = surf2d_of(s2d_visco(L, g.dt, f.p[PM][ip], f.p[PMU][ip], 0.0f, f.p[PTAUP][ip], f.p[PTAUS][ip], 0.0f));
        const float h = surf2d_h<false>(su, vh, vzz);
        float sumx = 0, sumy = 0;
        for (int l = 0; l < L; l++) {
            sumx += ldv(rxx + l * g.nvol + iv) * g.rsci;
            sumy += ldv(ryy + l * g.nvol + iv) * g.rsci;
        }
        stv(sxx + iv, __fmaf_rn(sg, __fmaf_rn(-g.dt2, sumx, h), ldv(sxx + iv)));
        stv(syy + iv, __fmaf_rn(sg, __fmaf_rn(-g.dt2, sumy, h), ldv(syy + iv)));
        sumx = 0; sumy = 0;
        for (int l = 0; l < L; l++) {
            const float b = surf2d_b(g.eta[l]), hr = surf2d_hr(su, vh, vzz);
            const float x = __fmul_rn(ldv(rxx + l * g.nvol + iv), g.rsci), y = __fmul_rn(ldv(ryy + l * g.nvol + iv), g.rsci);
            const float rx = sizeof(T) == 2 ? __fmaf_rn(b, hr, x) : __fadd_rn(x, __fmul_rn(b, hr)), ry = __fmaf_rn(b, hr, y);
            stv(rxx + l * g.nvol + iv, rx * g.rsc);
            stv(ryy + l * g.nvol + iv, ry * g.rsc);
            sumx += rx; sumy += ry;
        }
        stv(sxx + iv, __fmaf_rn(g.dt2, sumx, ldv(sxx + iv)));
        stv(syy + iv, __fmaf_rn(g.dt2, sumy, ldv(syy + iv)));
    }
}


// ============================================================ 2D acoustic
// src/update_v2D_acc.cl:80-324, src/update_s2D_acc.cl:79-402; the pressure
// lives in the SXX slot, its memory variable in RXX, psi_p_x / psi_p_z in the
// PSXX_X / PSZZ_Z slots.
template <int F>
__global__ void __launch_bounds__(256) k_v2d_acc(Grid g, Fields f)
{
    SHOT_F
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    int NAB = g.nab, NZ = g.NZ, NX = g.NX;
    float p_x = dfw<F>(f.w[SXX], iv, NZ, g.hc);
    float p_z = dfw<F>(f.w[SXX], iv, 1, g.hc);
    if (g.abs_type == 1) {
        if (gz > NZ - NAB - F - 1) {
            int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
            cpml(f.psi[PSZZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, p_z);
        } else if (!g.freesurf && gz - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PSZZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, p_z);
        }
        if (gx - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PSXX_X], (i64)i * g.nz + k, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], i, p_x);
        }
        if (gx > NX - NAB - F - 1) {
            int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
            cpml(f.psi[PSXX_X], (i64)i * g.nz + k, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, p_x);
        }
    }
    float vx = f.w[VX][iv] + p_x * __ldg(f.p[PRIP] + ip);
    float vz = f.w[VZ][iv] + p_z * __ldg(f.p[PRKP] + ip);
    if (g.abs_type == 2) {
        // the acoustic kernels taper the top even with a free surface
        const float *tp = f.taper;
        if (gz - F < NAB) { vx *= tp[gz - F]; vz *= tp[gz - F]; }
        if (gz > NZ - NAB - F - 1) { vx *= tp[NZ - F - gz - 1]; vz *= tp[NZ - F - gz - 1]; }
        if (gx - F < NAB) { vx *= tp[gx - F]; vz *= tp[gx - F]; }
        if (gx > NX - NAB - F - 1) { vx *= tp[NX - F - gx - 1]; vz *= tp[NX - F - gx - 1]; }
    }
    f.w[VX][iv] = vx;
    f.w[VZ][iv] = vz;
}

// one cell of the acoustic pressure update (update_s2D_acc.cl:79-402)
template <int F>
__device__ __forceinline__ void s2d_acc_cell(const Grid &g, const Fields &f, int gz, int gx)
{
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    int NAB = g.nab, NZ = g.NZ, NX = g.NX, L = g.L;
    float vxx = dbw<F>(f.w[VX], iv, NZ, g.hc);
    float vzz = dbw<F>(f.w[VZ], iv, 1, g.hc);
    if (g.abs_type == 1) {
        if (gz > NZ - NAB - F - 1) {
            int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
            cpml(f.psi[PVZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, vzz);
        } else if (!g.freesurf && gz - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PVZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, vzz);
        }
        if (gx - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PVX_X], (i64)i * g.nz + k, ktab(f, 0, 0), f.cx[CA], f.cx[CB], i, vxx);
        }
        if (gx > NX - NAB - F - 1) {
            int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
            cpml(f.psi[PVX_X], (i64)i * g.nz + k, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind + 1, vxx);
        }
    }
    float p = f.w[SXX][iv];
    if (L == 0) {
        p += __ldg(f.p[PM] + ip) * (vxx + vzz);
    } else {
        float lM = __ldg(f.p[PM] + ip), ltaup = __ldg(f.p[PTAUP] + ip);
        float gm = lM * (1.0f + (float)L * ltaup);
        float e = lM * ltaup;  // no 1/dt, as update_s2D_acc.cl:333
        float sumrp = 0;
        for (int l = 0; l < L; l++) sumrp += f.r[RXX][l * g.nvol + iv];
        float lp = gm * (vxx + vzz) + g.dt2 * sumrp;
        sumrp = 0;
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
            i64 ir = l * g.nvol + iv;
            float r = b * (f.r[RXX][ir] * c - el * e * (vxx + vzz));
            f.r[RXX][ir] = r;
            sumrp += r;
        }
        p += lp + g.dt2 * sumrp;
    }
    if (g.abs_type == 2) {
        const float *tp = f.taper;
        if (gz - F < NAB) p *= tp[gz - F];
        if (gz > NZ - NAB - F - 1) p *= tp[NZ - F - gz - 1];
        if (gx - F < NAB) p *= tp[gx - F];
        if (gx > NX - NAB - F - 1) p *= tp[NX - F - gx - 1];
    }
    f.w[SXX][iv] = p;
}

template <int F>
__global__ void __launch_bounds__(256) k_s2d_acc(Grid g, Fields f)
{
    SHOT_F
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz <= g.NZ - F - 1 && gx <= g.NX - F - 1) s2d_acc_cell<F>(g, f, gz, gx);
}

// ================================================================== 2D SH
// src/update_v2D_SH.cl:106-356, src/update_s2D_SH.cl:109-421 (elastic).
// Buoyancy and shear modulus at the cell, unaveraged; the far-x CPML of the
// velocity uses the full-node coefficients at ind; at FDOH=1 the stress
// differences carry no coefficient; stresses are not tapered.
template <int F>
__global__ void __launch_bounds__(256) k_v2d_sh(Grid g, Fields f)
{
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    int NAB = g.nab, NZ = g.NZ, NX = g.NX;
    float sxy_x = dbw<F>(f.w[SXY], iv, NZ, g.hc);
    float syz_z = dbw<F>(f.w[SYZ], iv, 1, g.hc);
    if (g.abs_type == 1) {
        if (gz > NZ - NAB - F - 1) {
            int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
            cpml(f.psi[PSYZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, syz_z);
        } else if (!g.freesurf && gz - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PSYZ_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, syz_z);
        }
        if (gx - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PSXY_X], (i64)i * g.nz + k, ktab(f, 0, 0), f.cx[CA], f.cx[CB], i, sxy_x);
        }
        if (gx > NX - NAB - F - 1) {
            int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
            cpml(f.psi[PSXY_X], (i64)i * g.nz + k, ktab(f, 0, 0), f.cx[CA], f.cx[CB], ind, sxy_x);
        }
    }
    float vy = f.w[VY][iv] + (sxy_x + syz_z) * __ldg(f.p[PRHO] + ip);
    if (g.abs_type == 2) {
        const float *tp = f.taper;
        if (!g.freesurf && gz - F < NAB) vy *= tp[gz - F];
        if (gz > NZ - NAB - F - 1) vy *= tp[NZ - F - gz - 1];
        if (gx - F < NAB) vy *= tp[gx - F];
        if (gx > NX - NAB - F - 1) vy *= tp[NX - F - gx - 1];
    }
    f.w[VY][iv] = vy;
}

template <int F>
__global__ void __launch_bounds__(256) k_s2d_sh(Grid g, Fields f)
{
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    int NAB = g.nab, NZ = g.NZ, NX = g.NX;
    float hone[6] = {1.0f, 0, 0, 0, 0, 0};
    const float *h = F == 1 ? hone : g.hc;
    float vyx = dfw<F>(f.w[VY], iv, NZ, h);
    float vyz = dfw<F>(f.w[VY], iv, 1, h);
    if (g.abs_type == 1) {
        if (gz > NZ - NAB - F - 1) {
            int i = gx - F, k = gz - NZ + NAB + F + NAB, ind = 2 * NAB - 1 - k;
            cpml(f.psi[PVY_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vyz);
        } else if (!g.freesurf && gz - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PVY_Z], (i64)i * (2 * NAB) + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, vyz);
        }
        if (gx - F < NAB) {
            int i = gx - F, k = gz - F;
            cpml(f.psi[PVY_X], (i64)i * g.nz + k, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], i, vyx);
        }
        if (gx > NX - NAB - F - 1) {
            int i = gx - NX + NAB + F + NAB, k = gz - F, ind = 2 * NAB - 1 - i;
            cpml(f.psi[PVY_X], (i64)i * g.nz + k, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], ind, vyx);
        }
    }
    float mu = __ldg(f.p[PMU] + ip);
    f.w[SXY][iv] += mu * vyx;
    f.w[SYZ][iv] += mu * vyz;
}

// SH free surface: image syz above the surface (src/surface2D_SH.cl:37-39)
template <int F>
__global__ void k_surf_sh(Grid g, Fields f)
{
    int gx = blockIdx.x * blockDim.x + threadIdx.x + F;
    if (gx > g.NX - F - 1) return;
    i64 iv = (i64)gx * g.NZ + F;
#pragma unroll
    for (int m = 1; m <= F; m++) f.w[SYZ][iv - m] = -f.w[SYZ][iv + m - 1];
}

// ---------------------------------------------------- boundary save (forward)
template <typename T>
__global__ void k_savebnd(Grid g, Fields f, BndSlot b, i64 tofs)
{
    SHOT_F
    int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= g.nbnd) return;
    const i64 sh = (i64)blockIdx.z * (g.sb_bnd / (i64)sizeof(T));
    int i, j, k;
    if (!shell_cell(g, gid, i, j, k)) return;
    i64 iv = ((i64)i * g.NY + j) * g.NZ + k;
    // every field index is a compile-time constant (a saved field has its
    // store in b.p[w]): indexing the parameter structs with a run-time field
    // id made each thread copy them to local memory (a 688-byte stack frame);
    // all loads go out before the stores
    float v[NW];
#pragma unroll
    for (int w = 0; w < NW; w++)
        if (b.p[w]) v[w] = f.w[w][iv];
#pragma unroll
    for (int w = 0; w < NW; w++)
        if (b.p[w]) ((T *)b.p[w])[sh + tofs + gid] = from_f<T>(v[w] * g.bsc[w]);
}

// ------------------------------------------------------- adjoint kernels 2D
template <int F, typename T>
__global__ void __launch_bounds__(256) k_adjv2d(Grid g, Fields f, AdjFields a)
{
    SHOT_FA
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    const float *hc = g.hc;
    float rip = __ldg(f.p[PRIP] + ip), rkp = __ldg(f.p[PRKP] + ip);
    float vx = 0.0f, vz = 0.0f;
    if (g.ckpt) {
        vx = fwd_at<T>(g, a, VX, iv);
        vz = fwd_at<T>(g, a, VZ, iv);
    } else if (!g.bp2) {  // backpropagate the forward velocities (update_adjv2D.cl:205-240)
        float sxx_x = dfw<F>(f.w[SXX], iv, g.NZ, hc);
        float szz_z = dfw<F>(f.w[SZZ], iv, 1, hc);
        float sxz_z = dbw<F>(f.w[SXZ], iv, 1, hc);
        float sxz_x = dbw<F>(f.w[SXZ], iv, g.NZ, hc);
        vx = __fmaf_rn(-__fadd_rn(sxx_x, sxz_z), rip, f.w[VX][iv]);
        vz = __fmaf_rn(-__fadd_rn(szz_z, sxz_x), rkp, f.w[VZ][iv]);
        int m = inject_ind2d(g, gz, gx);
        if (m != -1) {
            vx = bnd_at<T>(g, a, VX, m);
            vz = bnd_at<T>(g, a, VZ, m);
        }
        f.w[VX][iv] = vx;
        f.w[VZ][iv] = vz;
    }
    float sxx_xr = dfw<F>(a.wr[SXX], iv, g.NZ, hc);
    float szz_zr = dfw<F>(a.wr[SZZ], iv, 1, hc);
    float sxz_zr = dbw<F>(a.wr[SXZ], iv, 1, hc);
    float sxz_xr = dbw<F>(a.wr[SXZ], iv, g.NZ, hc);
    if (g.abs_type == 1) cpml_v2d(g, f, gz, gx, sxx_xr, szz_zr, sxz_xr, sxz_zr);
    float lvx = __fmul_rn(__fadd_rn(sxx_xr, sxz_zr), rip);
    float lvz = __fmul_rn(__fadd_rn(szz_zr, sxz_xr), rkp);
    a.wr[VX][iv] += lvx;
    a.wr[VZ][iv] += lvz;
    if (g.abs_type == 2) {
        float *fs[2] = {a.wr[VX], a.wr[VZ]};
        apply_taper<2>(g, f.taper, gz, 0, gx, fs, iv);
    }
    if (!g.bp2) a.grad[GRHO][ip] += (double)__fmaf_rn(-vx, lvx, -__fmul_rn(vz, lvz));
}

template <int F, typename T>
__global__ void __launch_bounds__(256) k_adjs2d(Grid g, Fields f, AdjFields a)
{
    SHOT_FA
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gz > g.NZ - F - 1 || gx > g.NX - F - 1) return;
    i64 ip = (i64)(gx - F) * g.nz + (gz - F), iv = (i64)gx * g.NZ + gz;
    const float *hc = g.hc;
    float vxx = 0.0f, vxz = 0.0f, vzz = 0.0f, vzx = 0.0f;
    if (!g.bp2 && !g.ckpt) {
        vxx = dbw<F>(f.w[VX], iv, g.NZ, hc); vxz = dfw<F>(f.w[VX], iv, 1, hc);
        vzz = dbw<F>(f.w[VZ], iv, 1, hc); vzx = dfw<F>(f.w[VZ], iv, g.NZ, hc);
    }
    float vxxr = dbw<F>(a.wr[VX], iv, g.NZ, hc), vxzr = dfw<F>(a.wr[VX], iv, 1, hc);
    float vzzr = dbw<F>(a.wr[VZ], iv, 1, hc), vzxr = dfw<F>(a.wr[VZ], iv, g.NZ, hc);
    const int L = g.L;
    float lM = __ldg(f.p[PM] + ip), lmu = __ldg(f.p[PMU] + ip), fipkp, fm, gm, dipkp = 0, d = 0, e = 0;
    if (L == 0) {
        fipkp = __ldg(f.p[PMUIPKP] + ip);
        fm = 2.0f * lmu;
        gm = lM;
    } else {
        float lmuipkp = __ldg(f.p[PMUIPKP] + ip), ltaup = __ldg(f.p[PTAUP] + ip), ltaus = __ldg(f.p[PTAUS] + ip);
        float ltausipkp = __ldg(f.p[PTAUSIPKP] + ip);
        fipkp = lmuipkp * (1.0f + (float)L * ltausipkp);
        gm = lM * (1.0f + (float)L * ltaup);
        fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
        dipkp = lmuipkp * ltausipkp / g.dt;
        d = 2.0f * lmu * ltaus / g.dt;
        e = lM * ltaup / g.dt;
    }
    float sxx = 0.0f, szz = 0.0f, sxz = 0.0f;
    // reconstruct the forward stresses (update_adjs2D.cl:222-278)
    if (g.bp2) {
    } else if (g.ckpt) {
        sxx = fwd_at<T>(g, a, SXX, iv); szz = fwd_at<T>(g, a, SZZ, iv); sxz = fwd_at<T>(g, a, SXZ, iv);
    } else if (L == 0) {
        sxx = f.w[SXX][iv]; szz = f.w[SZZ][iv]; sxz = f.w[SXZ][iv];
        const float tr = __fadd_rn(vxx, vzz);
        sxz = __fmaf_rn(-fipkp, __fadd_rn(vxz, vzx), sxz);
        sxx = __fsub_rn(sxx, s2d_normal(gm, tr, fm, vzz));
        szz = __fsub_rn(szz, s2d_normal(gm, tr, fm, vxx));
    } else {
        sxx = f.w[SXX][iv]; szz = f.w[SZZ][iv]; sxz = f.w[SXZ][iv];
        float *rxx = f.r[RXX], *rzz = f.r[RZZ], *rxz = f.r[RXZ];
        float s1 = 0, s2 = 0, s3 = 0;
        for (int l = 0; l < L; l++) { i64 ir = l * g.nvol + iv; s1 += rxz[ir]; s2 += rxx[ir]; s3 += rzz[ir]; }
        float lsxz = fipkp * (vxz + vzx) + g.dt2 * s1;
        float lsxx = (gm * (vxx + vzz) - fm * vzz) + g.dt2 * s2;
        float lszz = (gm * (vxx + vzz) - fm * vxx) + g.dt2 * s3;
        s1 = s2 = s3 = 0;
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f - el * 0.5f), c = 1.0f + el * 0.5f;
            i64 ir = l * g.nvol + iv;
            float n1 = b * (rxz[ir] * c - el * (dipkp * (vxz + vzx)));
            float n2 = b * (rxx[ir] * c - el * (e * (vxx + vzz) - d * vzz));
            float n3 = b * (rzz[ir] * c - el * (e * (vxx + vzz) - d * vxx));
            rxz[ir] = n1; rxx[ir] = n2; rzz[ir] = n3;
            s1 += n1; s2 += n2; s3 += n3;
        }
        sxz -= lsxz + g.dt2 * s1;
        sxx -= lsxx + g.dt2 * s2;
        szz -= lszz + g.dt2 * s3;
    }
    if (!g.bp2 && !g.ckpt) {
        int m = inject_ind2d(g, gz, gx);
        if (m != -1) {
            sxx = bnd_at<T>(g, a, SXX, m);
            szz = bnd_at<T>(g, a, SZZ, m);
            sxz = bnd_at<T>(g, a, SXZ, m);
        }
        f.w[SXX][iv] = sxx; f.w[SZZ][iv] = szz; f.w[SXZ][iv] = sxz;
    }
    if (g.abs_type == 1) cpml_s2d(g, f, gz, gx, vxxr, vxzr, vzxr, vzzr);
    float lsxz, lsxx, lszz;
    if (L == 0) {
        const float tr = __fadd_rn(vxxr, vzzr);
        lsxz = __fmul_rn(fipkp, __fadd_rn(vxzr, vzxr));
        lsxx = s2d_normal(gm, tr, fm, vzzr);
        lszz = s2d_normal(gm, tr, fm, vxxr);
        a.wr[SXZ][iv] += lsxz;
        a.wr[SXX][iv] += lsxx;
        a.wr[SZZ][iv] += lszz;
    } else {
        float *rxxr = a.rr[RXX], *rzzr = a.rr[RZZ], *rxzr = a.rr[RXZ];
        float s1 = 0, s2 = 0, s3 = 0;
        for (int l = 0; l < L; l++) { i64 ir = l * g.nvol + iv; s1 += rxzr[ir]; s2 += rxxr[ir]; s3 += rzzr[ir]; }
        lsxz = fipkp * (vxzr + vzxr) + g.dt2 * s1;
        lsxx = (gm * (vxxr + vzzr) - fm * vzzr) + g.dt2 * s2;
        lszz = (gm * (vxxr + vzzr) - fm * vxxr) + g.dt2 * s3;
        s1 = s2 = s3 = 0;
        // every iteration updates the last mechanism's slot, as the reference
        // does (update_adjs2D.cl:379-391)
        i64 ir = (L - 1) * g.nvol + iv;
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
            float n1 = b * (rxzr[ir] * c - el * (dipkp * (vxzr + vzxr)));
            float n2 = b * (rxxr[ir] * c - el * (e * (vxxr + vzzr) - d * vzzr));
            float n3 = b * (rzzr[ir] * c - el * (e * (vxxr + vzzr) - d * vxxr));
            rxzr[ir] = n1; rxxr[ir] = n2; rzzr[ir] = n3;
            s1 += n1; s2 += n2; s3 += n3;
        }
        a.wr[SXZ][iv] += lsxz + g.dt2 * s1;
        a.wr[SXX][iv] += lsxx + g.dt2 * s2;
        a.wr[SZZ][iv] += lszz + g.dt2 * s3;
    }
    if (g.abs_type == 2) {
        float *fs[3] = {a.wr[SXZ], a.wr[SXX], a.wr[SZZ]};
        apply_taper<3>(g, f.taper, gz, 0, gx, fs, iv);
    }
    if (g.bp2) {
    } else if (g.restype == 0) {
        const Adj2dGrad q = adj2d_grad(0, lM, lmu, sxx, szz, sxz, lsxx, lszz, lsxz);
        a.grad[GM][ip] += (double)q.M;
        a.grad[GMU][ip] += (double)q.mu;
        if (g.hout) {
            float c1 = 1.0f / ((2.0f * lM - 2.0f * lmu) * (2.0f * lM - 2.0f * lmu));
            float c3 = 1.0f / (lmu * lmu);
            float c5 = 0.25f * c3;
            const float dM = -q.M;
            // update_adjs2D.cl:453-457 (the mu term subtracts the gradient's dM)
            float dMH = c1 * (sxx + szz) * (sxx + szz);
            a.hess[GM][ip] += (double)dMH;
            a.hess[GMU][ip] += (double)(c3 * sxz * sxz - dM + c5 * (sxx - szz) * (sxx - szz));
        }
    } else {
        a.grad[GM][ip] += (double)adj2d_grad(1, lM, lmu, sxx, szz, sxz, lsxx, lszz, lsxz).M;
        if (g.hout) a.hess[GM][ip] += (double)((sxx + szz) * (sxx + szz));
    }
}

// surface adjoint, split in two passes so no thread updates another
// column's cell (surface2D_adj.cl:35-148 lets neighbouring work-items add
// into the same vxr cells).  Pass 1: per column, the L transform, the vzr
// update of its own column, and q = hx * lsxx for pass 2.
template <int F>
__global__ void k_surfadj2d_a(Grid g, Fields f, AdjFields a, float *q)
{
    SHOT_FA
    q += blockIdx.z * g.sb_q;
    int gx = blockIdx.x * blockDim.x + threadIdx.x + F;
    if (gx > g.NX - F - 1) return;
    int gz = F;
    i64 iv = (i64)gx * g.NZ + gz, ip = (i64)(gx - F) * g.nz + (gz - F);
    float lszz = a.wr[SZZ][iv], lsxx = a.wr[SXX][iv];
    float lmu = f.p[PMU][ip], lM = f.p[PM][ip];
    float t1 = lsxx, t2 = lszz;
    float aa = 1.0f / (4.0f * lM * lmu - 4.0f * lmu * lmu);
    lsxx = -aa * (lM * t1 + (-lM + 2.0f * lmu) * t2);
    lszz = 0.0f;
    float hx = -((lM - lmu * 2.0f) * (lM - lmu * 2.0f) / lM);
    float hz = -(lM - lmu * 2.0f);
    for (int m = 0; m < F; m++)
        a.wr[VZ][iv + m] += g.hc[m] * hz * lsxx * f.p[PRKP][ip + m];
    q[gx - F] = hx * lsxx;
    a.wr[SZZ][iv] = -(lM * lszz + (lM - 2.0f * lmu) * lsxx);
    a.wr[SXX][iv] = -(lM * lsxx + (lM - 2.0f * lmu) * lszz);
}
// Pass 2: each column gathers the contributions of its neighbours.
template <int F>
__global__ void k_surfadj2d_b(Grid g, Fields f, AdjFields a, const float *q)
{
    SHOT_FA
    q += blockIdx.z * g.sb_q;
    int gx = blockIdx.x * blockDim.x + threadIdx.x + F;
    if (gx > g.NX - F - 1) return;
    int gz = F, x = gx - F, nx = g.nx;
    i64 iv = (i64)gx * g.NZ + gz, ip = (i64)(gx - F) * g.nz + (gz - F);
    float rip = f.p[PRIP][ip], acc = 0.0f;
    for (int m = 0; m < F; m++) {
        if (x - m >= 0) acc += g.hc[m] * q[x - m];
        if (x + m + 1 < nx) acc -= g.hc[m] * q[x + m + 1];
    }
    a.wr[VX][iv] += acc * rip;
}

// ------------------------------------------------------- adjoint kernels 3D
template <int F, typename T, bool MB = false>
__global__ void __launch_bounds__(256) k_adjv3d(Grid g, Fields f, AdjFields a)
{
    CELL3D
    if (MB) shot_adj(g, a, shot);
    const float *hc = g.hc;
    float rip = __ldg(f.p[PRIP] + ip), rjp = __ldg(f.p[PRJP] + ip), rkp = __ldg(f.p[PRKP] + ip);
    float vx = 0.0f, vy = 0.0f, vz = 0.0f;
    if (g.ckpt) {
        vx = fwd_at<T>(g, a, VX, iv); vy = fwd_at<T>(g, a, VY, iv); vz = fwd_at<T>(g, a, VZ, iv);
    } else if (!g.bp2) {  // backpropagate the forward velocities (update_adjv3D.cl:297-340)
        float szz_z = dfw<F>(f.w[SZZ], iv, 1, hc), sxx_x = dfw<F>(f.w[SXX], iv, sx, hc);
        float sxz_x = dbw<F>(f.w[SXZ], iv, sx, hc), sxz_z = dbw<F>(f.w[SXZ], iv, 1, hc);
        float syz_y = dbw<F>(f.w[SYZ], iv, sy, hc), syz_z = dbw<F>(f.w[SYZ], iv, 1, hc);
        float syy_y = dfw<F>(f.w[SYY], iv, sy, hc);
        float sxy_x = dbw<F>(f.w[SXY], iv, sx, hc), sxy_y = dbw<F>(f.w[SXY], iv, sy, hc);
        vx = f.w[VX][iv] - (sxx_x + sxy_y + sxz_z) * rip;
        vy = f.w[VY][iv] - (syy_y + sxy_x + syz_z) * rjp;
        vz = f.w[VZ][iv] - (szz_z + sxz_x + syz_y) * rkp;
        int m = inject_ind3d(g, gz, gy, gx);
        if (m != -1) {
            vx = bnd_at<T>(g, a, VX, m);
            vy = bnd_at<T>(g, a, VY, m);
            vz = bnd_at<T>(g, a, VZ, m);
        }
        f.w[VX][iv] = vx; f.w[VY][iv] = vy; f.w[VZ][iv] = vz;
    }
    float szz_zr = dfw<F>(a.wr[SZZ], iv, 1, hc), sxx_xr = dfw<F>(a.wr[SXX], iv, sx, hc);
    float sxz_xr = dbw<F>(a.wr[SXZ], iv, sx, hc), sxz_zr = dbw<F>(a.wr[SXZ], iv, 1, hc);
    float syz_yr = dbw<F>(a.wr[SYZ], iv, sy, hc), syz_zr = dbw<F>(a.wr[SYZ], iv, 1, hc);
    float syy_yr = dfw<F>(a.wr[SYY], iv, sy, hc);
    float sxy_xr = dbw<F>(a.wr[SXY], iv, sx, hc), sxy_yr = dbw<F>(a.wr[SXY], iv, sy, hc);
    if (g.abs_type == 1)
        cpml_v3d(g, f, gz, gy, gx, sxx_xr, syy_yr, szz_zr, sxy_yr, sxy_xr, syz_yr, syz_zr, sxz_xr, sxz_zr);
    float lvx = (sxx_xr + sxy_yr + sxz_zr) * rip;
    float lvy = (syy_yr + sxy_xr + syz_zr) * rjp;
    float lvz = (szz_zr + sxz_xr + syz_yr) * rkp;
    a.wr[VX][iv] += lvx; a.wr[VY][iv] += lvy; a.wr[VZ][iv] += lvz;
    if (g.abs_type == 2) {
        float *fs[3] = {a.wr[VX], a.wr[VY], a.wr[VZ]};
        apply_taper<3>(g, f.taper, gz, gy, gx, fs, iv);
    }
    if (!g.bp2) a.grad[GRHO][ip] += (double)(-vx * lvx - vy * lvy - vz * lvz);
}

template <int F, typename T, bool MB = false>
__global__ void __launch_bounds__(256) k_adjs3d(Grid g, Fields f, AdjFields a)
{
    CELL3D
    if (MB) shot_adj(g, a, shot);
    const float *hc = g.hc;
    float vzx = 0.0f, vzy = 0.0f, vzz = 0.0f, vyx = 0.0f, vyy = 0.0f, vyz = 0.0f, vxx = 0.0f, vxy = 0.0f, vxz = 0.0f;
    if (!g.bp2 && !g.ckpt) {
        vzx = dfw<F>(f.w[VZ], iv, sx, hc); vzy = dfw<F>(f.w[VZ], iv, sy, hc); vzz = dbw<F>(f.w[VZ], iv, 1, hc);
        vyx = dfw<F>(f.w[VY], iv, sx, hc); vyy = dbw<F>(f.w[VY], iv, sy, hc); vyz = dfw<F>(f.w[VY], iv, 1, hc);
        vxx = dbw<F>(f.w[VX], iv, sx, hc); vxy = dfw<F>(f.w[VX], iv, sy, hc); vxz = dfw<F>(f.w[VX], iv, 1, hc);
    }
    float vzxr = dfw<F>(a.wr[VZ], iv, sx, hc), vzyr = dfw<F>(a.wr[VZ], iv, sy, hc), vzzr = dbw<F>(a.wr[VZ], iv, 1, hc);
    float vyxr = dfw<F>(a.wr[VY], iv, sx, hc), vyyr = dbw<F>(a.wr[VY], iv, sy, hc), vyzr = dfw<F>(a.wr[VY], iv, 1, hc);
    float vxxr = dbw<F>(a.wr[VX], iv, sx, hc), vxyr = dfw<F>(a.wr[VX], iv, sy, hc), vxzr = dfw<F>(a.wr[VX], iv, 1, hc);
    const int L = g.L;
    float lM = __ldg(f.p[PM] + ip), lmu = __ldg(f.p[PMU] + ip);
    float fipjp, fjpkp, fipkp, gm, fm, dipjp = 0, djpkp = 0, dipkp = 0, d = 0, e = 0;
    if (L == 0) {
        fipjp = __ldg(f.p[PMUIPJP] + ip); fjpkp = __ldg(f.p[PMUJPKP] + ip); fipkp = __ldg(f.p[PMUIPKP] + ip);
        gm = lM; fm = 2.0f * lmu;
    } else {
        float lmuipkp = __ldg(f.p[PMUIPKP] + ip), lmuipjp = __ldg(f.p[PMUIPJP] + ip), lmujpkp = __ldg(f.p[PMUJPKP] + ip);
        float ltaup = __ldg(f.p[PTAUP] + ip), ltaus = __ldg(f.p[PTAUS] + ip);
        float ltausipkp = __ldg(f.p[PTAUSIPKP] + ip), ltausipjp = __ldg(f.p[PTAUSIPJP] + ip),
              ltausjpkp = __ldg(f.p[PTAUSJPKP] + ip);
        fipjp = lmuipjp * (1.0f + (float)L * ltausipjp);
        fjpkp = lmujpkp * (1.0f + (float)L * ltausjpkp);
        fipkp = lmuipkp * (1.0f + (float)L * ltausipkp);
        gm = lM * (1.0f + (float)L * ltaup);
        fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
        dipjp = lmuipjp * ltausipjp / g.dt; djpkp = lmujpkp * ltausjpkp / g.dt; dipkp = lmuipkp * ltausipkp / g.dt;
        d = 2.0f * lmu * ltaus / g.dt; e = lM * ltaup / g.dt;
    }
    float vxyyx = vxy + vyx, vyzzy = vyz + vzy, vxzzx = vxz + vzx;
    float vxxyyzz = vxx + vyy + vzz, vyyzz = vyy + vzz, vxxzz = vxx + vzz, vxxyy = vxx + vyy;
    float s[6] = {0, 0, 0, 0, 0, 0};
    if (g.ckpt) {
        s[0] = fwd_at<T>(g, a, SXY, iv); s[1] = fwd_at<T>(g, a, SYZ, iv); s[2] = fwd_at<T>(g, a, SXZ, iv);
        s[3] = fwd_at<T>(g, a, SXX, iv); s[4] = fwd_at<T>(g, a, SYY, iv); s[5] = fwd_at<T>(g, a, SZZ, iv);
    } else if (!g.bp2) {
        s[0] = f.w[SXY][iv]; s[1] = f.w[SYZ][iv]; s[2] = f.w[SXZ][iv];
        s[3] = f.w[SXX][iv]; s[4] = f.w[SYY][iv]; s[5] = f.w[SZZ][iv];
    }
    float *const *r = f.r;
    if (g.bp2 || g.ckpt) {
    } else if (L == 0) {
        s[0] -= fipjp * vxyyx; s[1] -= fjpkp * vyzzy; s[2] -= fipkp * vxzzx;
        s[3] -= gm * vxxyyzz - fm * vyyzz; s[4] -= gm * vxxyyzz - fm * vxxzz; s[5] -= gm * vxxyyzz - fm * vxxyy;
    } else {
        float aa[6] = {0, 0, 0, 0, 0, 0};
        for (int l = 0; l < L; l++) {
            i64 ir = l * g.nvol + iv;
            aa[0] += r[RXY][ir]; aa[1] += r[RYZ][ir]; aa[2] += r[RXZ][ir];
            aa[3] += r[RXX][ir]; aa[4] += r[RYY][ir]; aa[5] += r[RZZ][ir];
        }
        float ls[6] = {fipjp * vxyyx + g.dt2 * aa[0], fjpkp * vyzzy + g.dt2 * aa[1], fipkp * vxzzx + g.dt2 * aa[2],
                       (gm * vxxyyzz - fm * vyyzz) + g.dt2 * aa[3], (gm * vxxyyzz - fm * vxxzz) + g.dt2 * aa[4],
                       (gm * vxxyyzz - fm * vxxyy) + g.dt2 * aa[5]};
        for (int q = 0; q < 6; q++) aa[q] = 0;
        // 3D reconstruction keeps the forward-time coefficients (update_adjs3D.cl:357-359)
        for (int l = 0; l < L; l++) {
            float el = g.eta[l];
            float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
            i64 ir = l * g.nvol + iv;
            float n0 = b * (r[RXY][ir] * c - el * (dipjp * vxyyx));
            float n1 = b * (r[RYZ][ir] * c - el * (djpkp * vyzzy));
            float n2 = b * (r[RXZ][ir] * c - el * (dipkp * vxzzx));
            float n3 = b * (r[RXX][ir] * c - el * (e * vxxyyzz - d * vyyzz));
            float n4 = b * (r[RYY][ir] * c - el * (e * vxxyyzz - d * vxxzz));
            float n5 = b * (r[RZZ][ir] * c - el * (e * vxxyyzz - d * vxxyy));
            r[RXY][ir] = n0; r[RYZ][ir] = n1; r[RXZ][ir] = n2; r[RXX][ir] = n3; r[RYY][ir] = n4; r[RZZ][ir] = n5;
            aa[0] += n0; aa[1] += n1; aa[2] += n2; aa[3] += n3; aa[4] += n4; aa[5] += n5;
        }
        for (int q = 0; q < 6; q++) s[q] -= ls[q] + g.dt2 * aa[q];
    }
    if (!g.bp2 && !g.ckpt) {
        int m = inject_ind3d(g, gz, gy, gx);
        if (m != -1) {
            s[3] = bnd_at<T>(g, a, SXX, m); s[4] = bnd_at<T>(g, a, SYY, m);
            s[5] = bnd_at<T>(g, a, SZZ, m); s[0] = bnd_at<T>(g, a, SXY, m);
            s[1] = bnd_at<T>(g, a, SYZ, m); s[2] = bnd_at<T>(g, a, SXZ, m);
        }
        f.w[SXY][iv] = s[0]; f.w[SYZ][iv] = s[1]; f.w[SXZ][iv] = s[2];
        f.w[SXX][iv] = s[3]; f.w[SYY][iv] = s[4]; f.w[SZZ][iv] = s[5];
    }
    if (g.abs_type == 1) cpml_s3d(g, f, gz, gy, gx, vxxr, vxyr, vxzr, vyxr, vyyr, vyzr, vzxr, vzyr, vzzr, true);
    float vxyyxr = vxyr + vyxr, vyzzyr = vyzr + vzyr, vxzzxr = vxzr + vzxr;
    float vxxyyzzr = vxxr + vyyr + vzzr, vyyzzr = vyyr + vzzr, vxxzzr = vxxr + vzzr, vxxyyr = vxxr + vyyr;
    float ls[6];
    ls[0] = fipjp * vxyyxr; ls[1] = fjpkp * vyzzyr; ls[2] = fipkp * vxzzxr;
    ls[3] = gm * vxxyyzzr - fm * vyyzzr; ls[4] = gm * vxxyyzzr - fm * vxxzzr; ls[5] = gm * vxxyyzzr - fm * vxxyyr;
    float *const *wr = a.wr;
    const int sid[6] = {SXY, SYZ, SXZ, SXX, SYY, SZZ};
    if (L == 0) {
        for (int q = 0; q < 6; q++) wr[sid[q]][iv] += ls[q];
    } else {
        float *const *rr = a.rr;
        const int rid[6] = {RXY, RYZ, RXZ, RXX, RYY, RZZ};
        float aa[6] = {0, 0, 0, 0, 0, 0};
        for (int l = 0; l < L; l++) {
            i64 ir = l * g.nvol + iv;
            for (int q = 0; q < 6; q++) aa[q] += rr[rid[q]][ir];
        }
        for (int q = 0; q < 6; q++) ls[q] += g.dt2 * aa[q];
        // the reference stores these into the forward memory variables and
        // keeps only the last adjoint value of each sum (update_adjs3D.cl:566-583);
        // a checkpointed adjoint skips the stores (dead: the forward arrays are
        // reloaded from a snapshot before they are read)
        for (int l = 0; l < L; l++) {
            i64 ir = l * g.nvol + iv;
            if (!g.ckpt) {
                float el = g.eta[l];
                float b = 1.0f / (1.0f + el * 0.5f), c = 1.0f - el * 0.5f;
                r[RXY][ir] = b * (rr[RXY][ir] * c - el * (dipjp * vxyyxr));
                r[RYZ][ir] = b * (rr[RYZ][ir] * c - el * (djpkp * vyzzyr));
                r[RXZ][ir] = b * (rr[RXZ][ir] * c - el * (dipkp * vxzzxr));
                r[RXX][ir] = b * (rr[RXX][ir] * c - el * (e * vxxyyzzr - d * vyyzzr));
                r[RYY][ir] = b * (rr[RYY][ir] * c - el * (e * vxxyyzzr - d * vxxzzr));
                r[RZZ][ir] = b * (rr[RZZ][ir] * c - el * (e * vxxyyzzr - d * vxxyyr));
            }
            // after the stores: in the DFT adjoint r and rr are one buffer
            for (int q = 0; q < 6; q++) aa[q] = rr[rid[q]][ir];
        }
        for (int q = 0; q < 6; q++) wr[sid[q]][iv] += ls[q] + g.dt2 * aa[q];
    }
    if (g.abs_type == 2) {
        float *fs[6] = {wr[SXY], wr[SYZ], wr[SXZ], wr[SXX], wr[SYY], wr[SZZ]};
        apply_taper<6>(g, f.taper, gz, gy, gx, fs, iv);
    }
    float sxx = s[3], syy = s[4], szz = s[5], sxy = s[0], syz = s[1], sxz = s[2];
    float lsxy = ls[0], lsyz = ls[1], lsxz = ls[2], lsxx = ls[3], lsyy = ls[4], lszz = ls[5];
    if (g.bp2) {
    } else if (g.restype == 0) {
        float c1 = 1.0f / (3.0f * lM - 4.0f * lmu) / (3.0f * lM - 4.0f * lmu);
        float c3 = 1.0f / lmu / lmu;
        float c5 = 1.0f / 6.0f * c3;
        float dM = c1 * (sxx + syy + szz) * (lsxx + lsyy + lszz);
        a.grad[GM][ip] += (double)(-dM);
        a.grad[GMU][ip] += (double)(-c3 * (sxz * lsxz + sxy * lsxy + syz * lsyz) + 4.0f / 3.0f * dM -
                                    c5 * (lsxx * (2.0f * sxx - syy - szz) + lsyy * (2.0f * syy - sxx - szz) +
                                          lszz * (2.0f * szz - sxx - syy)));
    } else {
        float dM = (sxx + syy + szz) * (lsxx + lsyy + lszz);
        a.grad[GM][ip] += (double)(-dM);
    }
}

// surface adjoint 3D (surface3D_adj.cl:29-116), two passes like 2D.  The
// reference reads the syy component from sxxr (:62).
template <int F>
__global__ void k_surfadj3d_a(Grid g, Fields f, AdjFields a, float *q)
{
    SHOT_FA
    q += blockIdx.z * g.sb_q;
    int gy = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gy > g.NY - F - 1 || gx > g.NX - F - 1) return;
    int gz = F;
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    i64 iv = gx * sx + (i64)gy * sy + gz;
    i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz - F);
    float lszz = -a.wr[SZZ][iv], lsxx = -a.wr[SXX][iv], lsyy = -a.wr[SXX][iv];
    float lmu = f.p[PMU][ip], lM = f.p[PM][ip];
    float t1 = lsxx, t2 = lsyy, t3 = lszz;
    float aa = 1.0f / (6.0f * lM * lmu - 8.0f * lmu * lmu);
    lsxx = aa * (2.0f * (lM - lmu) * t1 + (-lM + 2.0f * lmu) * (t2 + t3));
    lsyy = aa * (2.0f * (lM - lmu) * t2 + (-lM + 2.0f * lmu) * (t1 + t3));
    lszz = 0.0f;
    float h = -((lM - lmu * 2.0f) * (lM - lmu * 2.0f) / lM);
    float hz = -(lM - lmu * 2.0f);
    for (int m = 0; m < F; m++) a.wr[VZ][iv + m] += g.hc[m] * hz * (lsxx + lsyy) * f.p[PRKP][ip + m];
    q[(i64)(gx - F) * g.ny + (gy - F)] = h * (lsxx + lsyy);
    a.wr[SXX][iv] = -(lM * lsxx + (lM - 2.0f * lmu) * (lsyy + lszz));
    a.wr[SYY][iv] = -(lM * lsyy + (lM - 2.0f * lmu) * (lsxx + lszz));
    a.wr[SZZ][iv] = -(lM * lszz + (lM - 2.0f * lmu) * (lsxx + lsyy));
}
template <int F>
__global__ void k_surfadj3d_b(Grid g, Fields f, AdjFields a, const float *q)
{
    SHOT_FA
    q += blockIdx.z * g.sb_q;
    int gy = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    if (gy > g.NY - F - 1 || gx > g.NX - F - 1) return;
    int gz = F, x = gx - F, y = gy - F, nx = g.nx, ny = g.ny;
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    i64 iv = gx * sx + (i64)gy * sy + gz;
    i64 ip = ((i64)x * g.ny + y) * g.nz;
    float accx = 0.0f, accy = 0.0f;
    for (int m = 0; m < F; m++) {
        if (x - m >= 0) accx += g.hc[m] * q[(i64)(x - m) * ny + y];
        if (x + m + 1 < nx) accx -= g.hc[m] * q[(i64)(x + m + 1) * ny + y];
        if (y - m >= 0) accy += g.hc[m] * q[(i64)x * ny + (y - m)];
        if (y + m + 1 < ny) accy -= g.hc[m] * q[(i64)x * ny + (y + m + 1)];
    }
    a.wr[VX][iv] += accx * f.p[PRIP][ip];
    a.wr[VY][iv] += accy * f.p[PRJP][ip];
}

// ------------------------------------------------ point kernels (per shot)
// src/automatic_kernels.c:394-629; several sources may share a cell
template <class T>
__device__ __forceinline__ void source_point(const Fields &f, const PointSet &s, const float *src, int nt_total,
                                             int t, int pdir, float dt, int freesurf, int F, const WScale &ws,
                                             int gid)
{
    i64 cell = s.cell[gid];
    if (cell < 0) return;
    if (freesurf && pdir == -1 && s.kz[gid] < 2 * F) return;
    float amp = (float)pdir * (dt * src[(i64)gid * nt_total + t]);
    for (int q = 0; q < s.ntarget[gid]; q++) {
        float dv = s.div[gid * 3 + q];
        float val = dv == 0.0f ? amp : amp / dv;
        const int w = s.field[gid * 3 + q];
        atomicAdd(fld<T>(f.w[w]) + cell, (T)(val * ws.w[w]));
    }
}

template <class T = float>
__global__ void k_sources(Fields f, PointSet s, const float *src, int nt_total, int t, int pdir, float dt,
                          int freesurf, int F, WScale ws)
{
    pdl_trigger();
    pdl_wait();
    int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid < s.n) source_point<T>(f, s, src, nt_total, t, pdir, dt, freesurf, F, ws, gid);
}

// src/automatic_kernels.c:22-219; out is [nsel][nrec][NT].  L2: the loads
// bypass L1 (values stored by other blocks of the running kernel).
template <class T> __device__ __forceinline__ float ldv_l2(const T *p);
template <> __device__ __forceinline__ float ldv_l2<float>(const float *p) { return __ldcg(p); }
template <> __device__ __forceinline__ float ldv_l2<__half>(const __half *p) { return __half2float(__ldcg(p)); }

template <class T, bool L2>
__device__ __forceinline__ void record_point(const Fields &f, const PointSet &r, float *out, int nt_total, int t,
                                             unsigned outmask, int nd, const WScale &ws, int gid)
{
    i64 cell = r.cell[gid];
    if (cell < 0) return;
    auto ld = [](const T *q) { return L2 ? ldv_l2<T>(q) : ldv(q); };
    int slot = 0;
    for (int o = 0; o < SFD_NOUT; o++) {
        if (!(outmask & (1u << o))) continue;
        float v;
        if (o == SFD_OUT_P) {
            const T *xx = fld<T>(f.w[SXX]), *zz = fld<T>(f.w[SZZ]);
            if (nd == 3) v = (ld(xx + cell) + ld(zz + cell) + ld(fld<T>(f.w[SYY]) + cell)) / 3.0f;
            else if (nd == 22) v = ld(xx + cell);
            else v = (ld(xx + cell) + ld(zz + cell)) / 2.0f;
            v /= ws.w[SXX];
        } else {
            v = ld(fld<T>(f.w[o]) + cell) / ws.w[o];
        }
        out[((i64)slot * r.n + gid) * nt_total + t] = v;
        slot++;
    }
}

template <class T = float>
__global__ void k_record(Fields f, PointSet r, float *out, int nt_total, int t, unsigned outmask, int nd, WScale ws)
{
    pdl_trigger();
    pdl_wait();
    int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid < r.n) record_point<T, false>(f, r, out, nt_total, t, outmask, nd, ws, gid);
}

// receivers of step t and sources of step tsrc, for shots without a receiver
// on a source's cell: the first `rblocks` blocks record, the rest inject
template <class T = float>
__global__ void k_record_sources(Fields f, PointSet r, float *out, int nt_total, int t, unsigned outmask, int nd,
                                 WScale ws, unsigned rblocks, PointSet s, const float *src, int tsrc, float dt,
                                 int freesurf, int F)
{
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x < rblocks) {
        const int gid = blockIdx.x * blockDim.x + threadIdx.x;
        if (gid < r.n) record_point<T, false>(f, r, out, nt_total, t, outmask, nd, ws, gid);
    } else {
        const int gid = (blockIdx.x - rblocks) * blockDim.x + threadIdx.x;
        if (gid < s.n) source_point<T>(f, s, src, nt_total, tsrc, 1, dt, freesurf, F, ws, gid);
    }
}

// ---------------------------------------------- fused 2D forward step tail
// The stress kernel of a fused 2D step ends with the receivers of step t
// and the sources of step t+1 (time_stepping.c:783-816 order: sources,
// update_v, update_s, surface, record), run by the block that finishes
// last: every block fences its stores and takes a ticket; the block with
// the last ticket sees all stores of the launch, records, adds the next
// step's sources and resets the ticket.  Nothing waits on another block.
template <class T = float>
__device__ __forceinline__ void step_tail(const Grid &g, const Fields &f, const StepTail &tl)
{
    __shared__ int s_last;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nth = blockDim.x * blockDim.y * blockDim.z;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(tl.ticket, 1) == (int)(gridDim.x * gridDim.y * gridDim.z) - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = tid; i < tl.rec.n; i += nth)
        record_point<T, true>(f, tl.rec, tl.out, tl.nt_total, tl.t, tl.outmask, g.nd, g.ws, i);
    __syncthreads();
    if (tl.tsrc >= 0)
        for (int i = tid; i < tl.src.n; i += nth)
            source_point<T>(f, tl.src, tl.stf, tl.nt_total, tl.tsrc, 1, g.dt, g.freesurf, g.F, g.ws, i);
    if (tid == 0) *tl.ticket = 0;
}

// P-SV stress update, free surface (blocks of the top row: their 32 z
// rows hold every stress the surface reads, rows F..2F) and step tail.
// pdir (1) is a launch argument, as for the separate surface kernel, so
// that both contract and round alike.
template <int F, class T = float>
__global__ void __launch_bounds__(256) k_s2d_step(Grid g, Fields f, StepTail tl, int pdir)
{
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    Fields fs = f;   // this block's shot; the tail's points carry their shot in their cells
    if (g.nb > 1) shot_fields(g, fs, blockIdx.z);
    if (gz <= g.NZ - F - 1 && gx <= g.NX - F - 1) s2d_cell<F, T>(g, fs, gz, gx);
    if (g.freesurf && blockIdx.x == 0) {
        __syncthreads();
        if (threadIdx.x == 0 && gx <= g.NX - F - 1) surf2d_column<F, T>(g, fs, gx, pdir);
    }
    step_tail<T>(g, f, tl);
}

// acoustic pressure update and step tail (no free-surface kernel)
template <int F>
__global__ void __launch_bounds__(256) k_s2d_acc_step(Grid g, Fields f, StepTail tl)
{
    int gz = blockIdx.x * blockDim.x + threadIdx.x + F;
    int gx = blockIdx.y * blockDim.y + threadIdx.y + F;
    Fields fs = f;
    if (g.nb > 1) shot_fields(g, fs, blockIdx.z);
    if (gz <= g.NZ - F - 1 && gx <= g.NX - F - 1) s2d_acc_cell<F>(g, fs, gz, gx);
    step_tail(g, f, tl);
}

// src/automatic_kernels.c:631-836; res is [nsel][nrec][NT]
// (into the adjoint fields); the blocks after the first `rblocks` take the
// sources of step tsrc out of the forward fields
__global__ void k_residuals(AdjFields a, PointSet r, const float *res, int nt_total, int t, unsigned outmask, int nd,
                            unsigned rblocks, Fields f, PointSet s, const float *src, int tsrc, float dt, int freesurf,
                            int F, WScale ws)
{
    if (blockIdx.x >= rblocks) {
        const int q = (blockIdx.x - rblocks) * blockDim.x + threadIdx.x;
        if (q < s.n) source_point<float>(f, s, src, nt_total, tsrc, -1, dt, freesurf, F, ws, q);
        return;
    }
    int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= r.n) return;
    i64 cell = r.cell[gid];
    if (cell < 0) return;
    int slot = 0;
    for (int o = 0; o < SFD_NOUT; o++) {
        if (!(outmask & (1u << o))) continue;
        float v = res[((i64)slot * r.n + gid) * nt_total + t];
        if (o == SFD_OUT_P) {
            float n2 = nd == 3 ? 3.0f : 2.0f;
            atomicAdd(a.wr[SXX] + cell, v / n2);
            atomicAdd(a.wr[SZZ] + cell, v / n2);
            if (nd == 3) atomicAdd(a.wr[SYY] + cell, v / n2);
        } else {
            atomicAdd(a.wr[o] + cell, v);
        }
        slot++;
    }
}

// ------------------------------------------------------------- launchers
// true when the 4-cell kernels apply to this grid (rows of whole quads whose
// first cell is aligned, see init_grid)
static inline bool q4_ok(const Grid &g)
{
    return g.nd == 3 && g.nz % 4 == 0 && (g.F == 4 || g.F == 2) && (g.F + g.zshift) % 4 == 0;
}

// the instances of a grid's rows (grids that q4_ok accepts)
#define ROWS_DISPATCH(g, ...)                                                   \
    if ((g).F != 4) { constexpr int R = ROWS_O4; __VA_ARGS__; }                  \
    else if ((g).zpad) { constexpr int R = ROWS_FILLED; __VA_ARGS__; }           \
    else { constexpr int R = ROWS_WHOLE; __VA_ARGS__; }

#define DISPATCH_F(F, ...)                                                      \
    switch (F) {                                                               \
    case 1: { constexpr int FF = 1; __VA_ARGS__; } break;                      \
    case 2: { constexpr int FF = 2; __VA_ARGS__; } break;                      \
    case 3: { constexpr int FF = 3; __VA_ARGS__; } break;                      \
    case 4: { constexpr int FF = 4; __VA_ARGS__; } break;                      \
    case 5: { constexpr int FF = 5; __VA_ARGS__; } break;                      \
    case 6: { constexpr int FF = 6; __VA_ARGS__; } break;                      \
    default: break;                                                            \
    }

void launch_update_v(const Grid &g, const Fields &f, cudaStream_t st)
{
    if (g.fhalf && g.nd == 3) {   // FP16 storage: the vectorised or the streaming kernels
        if (q4_ok(g)) {
            ROWS_DISPATCH(g, quad_update_v<R>(g, f, st))
            return;
        }
        dim3 b(32, 4, 2), gr(cdiv(g.nz, 32), cdiv(g.ny, 4), cdiv(g.nx, 2) * g.nb);
        DISPATCH_F(g.F, k_v3d_stream<FF, __half><<<gr, b, 0, st>>>(g, f));
        return;
    }
    // kernels 0 takes the 4-cell vectorised kernel where it applies (0.43 ms
    // at 256^3, against 0.57 streaming, 0.58 general and 0.63 TMA), else the
    // streaming one; only kernels 3 takes the TMA path
    if (g.kernels == 3 && launch_update_v_tma(g, f, st)) return;
    if (g.kernels == 2 && launch_update_v_fast(g, f, st)) return;
    if (g.vasync && launch_update_v_async(g, f, st)) return;
    if (g.nd == 21 || g.nd == 22) {
        dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);
        if (g.nd == 21) DISPATCH_F(g.F, k_v2d_sh<FF><<<gr, b, 0, st>>>(g, f))
        else DISPATCH_F(g.F, k_v2d_acc<FF><<<gr, b, 0, st>>>(g, f))
        return;
    }
    if (g.nd == 3) {
        if ((g.kernels == 0 || g.kernels == 5) && q4_ok(g)) {
            ROWS_DISPATCH(g, quad_update_v<R>(g, f, st))
            return;
        }
        dim3 b(32, 4, 2), gr(cdiv(g.nz, 32), cdiv(g.ny, 4), cdiv(g.nx, 2) * g.nb);
        if (g.kernels == 0 || g.kernels == 4 || g.kernels == 5) {
            DISPATCH_F(g.F, MB_DISPATCH(g, k_v3d_stream<FF, float, MBV><<<gr, b, 0, st>>>(g, f)));
            return;
        }
        DISPATCH_F(g.F, MB_DISPATCH(g, k_v3d<FF, MBV><<<gr, b, 0, st>>>(g, f)));
    } else if (quad2d_ok(g)) {
        launch_quad2d_v(g, f, st);
    } else {
        dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);
        if (g.fhalf) DISPATCH_F(g.F, k_v2d<FF, __half><<<gr, b, 0, st>>>(g, f))
        else DISPATCH_F(g.F, k_v2d<FF><<<gr, b, 0, st>>>(g, f));
    }
}

bool launch_update_s(const Grid &g, const Fields &f, cudaStream_t st, Surf fold)
{
    if (g.fhalf && g.nd == 3 && g.L <= 3) {   // FP16 storage: the vectorised or the streaming kernels
        if (q4_ok(g)) {
            const Surf surf = g.freesurf && g.nb == 1 ? fold : SURF_NONE;
            ROWS_DISPATCH(g, return quad_update_s<R>(g, f, st, surf))
        }
        dim3 b(32, 4, 2), gr(cdiv(g.nz, 32), cdiv(g.ny, 4), cdiv(g.nx, 2) * g.nb);
        switch (g.L) {
        case 0: DISPATCH_F(g.F, k_s3d_stream<FF, 0, __half><<<gr, b, 0, st>>>(g, f)); break;
        case 1: DISPATCH_F(g.F, k_s3d_stream<FF, 1, __half><<<gr, b, 0, st>>>(g, f)); break;
        case 2: DISPATCH_F(g.F, k_s3d_stream<FF, 2, __half><<<gr, b, 0, st>>>(g, f)); break;
        default: DISPATCH_F(g.F, k_s3d_stream<FF, 3, __half><<<gr, b, 0, st>>>(g, f)); break;
        }
        return false;
    }
    // kernels 0: the 4-cell vectorised kernel where it applies (0.74 ms at
    // 256^3, against 0.96 TMA and 0.98 streaming), else the streaming one
    if (g.kernels == 3 && launch_update_s_tma(g, f, st)) return false;
    if (g.kernels == 2 && launch_update_s_fast(g, f, st)) return false;
    // single-shot FP32 4-cell kernels apply the free surface in the same launch
    const Surf surf = g.freesurf && g.nb == 1 ? fold : SURF_NONE;
    if (g.nd == 21 || g.nd == 22) {
        dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);
        if (g.nd == 21) DISPATCH_F(g.F, k_s2d_sh<FF><<<gr, b, 0, st>>>(g, f))
        else DISPATCH_F(g.F, k_s2d_acc<FF><<<gr, b, 0, st>>>(g, f))
        return false;
    }
    if (g.nd == 3) {
        dim3 b(32, 4, 2), gr(cdiv(g.nz, 32), cdiv(g.ny, 4), cdiv(g.nx, 2) * g.nb);
        if ((g.kernels == 0 || g.kernels == 5) && q4_ok(g) && g.L <= 3) {
            ROWS_DISPATCH(g, return quad_update_s<R>(g, f, st, surf))
        }
        if ((g.kernels == 0 || g.kernels == 4 || g.kernels == 5) && g.L <= 3) {
            switch (g.L) {
            case 0: DISPATCH_F(g.F, MB_DISPATCH(g, k_s3d_stream<FF, 0, float, MBV><<<gr, b, 0, st>>>(g, f))); break;
            case 1: DISPATCH_F(g.F, MB_DISPATCH(g, k_s3d_stream<FF, 1, float, MBV><<<gr, b, 0, st>>>(g, f))); break;
            case 2: DISPATCH_F(g.F, MB_DISPATCH(g, k_s3d_stream<FF, 2, float, MBV><<<gr, b, 0, st>>>(g, f))); break;
            default: DISPATCH_F(g.F, MB_DISPATCH(g, k_s3d_stream<FF, 3, float, MBV><<<gr, b, 0, st>>>(g, f))); break;
            }
            return false;
        }
        DISPATCH_F(g.F, MB_DISPATCH(g, k_s3d<FF, MBV><<<gr, b, 0, st>>>(g, f)));
    } else if (quad2d_ok(g)) {
        BndSlot none;
        memset(&none, 0, sizeof none);
        const bool surf2d = fold != SURF_NONE && g.freesurf;
        launch_quad2d_s(g, f, none, SFD_PREC_FP32, 0, surf2d, st);
        return surf2d;
    } else {
        dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);
        if (g.fhalf) DISPATCH_F(g.F, k_s2d<FF, __half><<<gr, b, 0, st>>>(g, f))
        else DISPATCH_F(g.F, k_s2d<FF><<<gr, b, 0, st>>>(g, f));
    }
    return false;
}

bool launch_update_s_bnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, cudaStream_t st)
{
    if (!q4_ok(g) || g.kernels != 0 || g.L > 0 || g.nb > 1 || g.fhalf || g.fused || g.vasync) return false;
    ROWS_DISPATCH(g, quad_update_s_bnd<R>(g, f, b, prec, tofs, g.freesurf != 0, st))
    return true;
}

// movie snapshot (time_stepping.c:272-350): padded field -> [nx][ny][nz]
template <class T>
__global__ void k_movie(Grid g, const T *fld, float inv_scale, float *dst)
{
    const int nz = g.nz - g.zpad;
    const i64 n = (i64)nz * g.ny * g.nx;
    for (i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(idx % nz);
        const i64 r = idx / nz;
        const int j = (int)(r % g.ny), i = (int)(r / g.ny);
        const i64 iv = ((i64)(i + g.F) * g.NY + (g.nd == 3 ? j + g.F : 0)) * g.NZ + (k + g.F);
        dst[idx] = to_f<T>(fld[iv]) * inv_scale;
    }
}

// One wave field scanned for non-finite values (the reference tests the
// misfit for NaN once per run, src/residuals.c:444-448; here the field is
// tested every FINITE_CHECK_EVERY steps so a run reports the step near which
// it diverged).
template <class T>
__global__ void __launch_bounds__(256) k_finite(const T *__restrict__ v, i64 n, int t, int *first)
{
    bool bad = false;
    for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        bad |= !isfinite(to_f<T>(v[i]));
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicMin(first, t);
}
__global__ void __launch_bounds__(256) k_finite4(const float4 *__restrict__ v, i64 n4, int t, int *first)
{
    bool bad = false;
    for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n4; i += (i64)gridDim.x * blockDim.x) {
        const float4 q = __ldg(v + i);
        bad |= !(isfinite(q.x) && isfinite(q.y) && isfinite(q.z) && isfinite(q.w));
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicMin(first, t);
}

void launch_finite_check(const Grid &g, const float *fld, int64_t n, int t, int *first, cudaStream_t st)
{
    if (!fld || n <= 0) return;
    const unsigned blocks = (unsigned)std::min<i64>((n + 1023) / 1024, 148 * 8);
    if (g.fhalf) k_finite<__half><<<blocks, 256, 0, st>>>(reinterpret_cast<const __half *>(fld), n, t, first);
    else if (n % 4 == 0 && ((uintptr_t)fld & 15) == 0)
        k_finite4<<<blocks, 256, 0, st>>>(reinterpret_cast<const float4 *>(fld), n / 4, t, first);
    else k_finite<float><<<blocks, 256, 0, st>>>(fld, n, t, first);
}

void launch_movie(const Grid &g, const float *fld, float inv_scale, float *dst, cudaStream_t st)
{
    const i64 n = (i64)(g.nz - g.zpad) * g.ny * g.nx;
    unsigned blocks = (unsigned)std::min<i64>((n + 255) / 256, 148 * 16);
    if (g.fhalf) k_movie<__half><<<blocks, 256, 0, st>>>(g, reinterpret_cast<const __half *>(fld), inv_scale, dst);
    else k_movie<float><<<blocks, 256, 0, st>>>(g, fld, inv_scale, dst);
}

int stress_family(const Grid &g, const Fields &f)
{
    // the same selection as launch_update_s; 4-cell kernels on a grid that
    // needs padded rows (Grid::zpad) or a shifted base (Grid::zshift) count as
    // the streaming family's form for that grid
    const bool plain = q4_ok(g) && g.zpad == 0 && g.F == 4;
    if (g.nd != 3) return 0;
    if (g.fhalf && g.L <= 3) return plain ? 5 : 4;
    if (g.kernels == 3 && tma_ready(g, f)) return 3;
    if (g.kernels == 2) return 2;
    if ((g.kernels == 0 || g.kernels == 5) && plain && g.L <= 3) return 5;
    if ((g.kernels == 0 || g.kernels == 4 || g.kernels == 5) && g.L <= 3) return 4;
    return 1;
}

bool launch_update_s_step(const Grid &g, const Fields &f, const StepTail &tl, cudaStream_t st)
{
    if (g.nd != 2 && g.nd != 22) return false;
    dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);   // 32 z rows >= 2F + 1: the surface stays in its block
    if (g.nd == 2 && g.fhalf) DISPATCH_F(g.F, k_s2d_step<FF, __half><<<gr, b, 0, st>>>(g, f, tl, 1))
    else if (g.nd == 2) DISPATCH_F(g.F, k_s2d_step<FF><<<gr, b, 0, st>>>(g, f, tl, 1))
    else DISPATCH_F(g.F, k_s2d_acc_step<FF><<<gr, b, 0, st>>>(g, f, tl))
    return true;
}

void launch_surface(const Grid &g, const Fields &f, int pdir, cudaStream_t st)
{
    if (g.nd == 21) {
        DISPATCH_F(g.F, k_surf_sh<FF><<<cdiv(g.nx, 128), 128, 0, st>>>(g, f));
        return;
    }
    if (g.nd == 22) return;
    if (g.nd == 3) {
        dim3 b(32, 4), gr(cdiv(g.ny, 32), cdiv(g.nx, 4), g.nb);
        if (g.fhalf) DISPATCH_F(g.F, k_surf3d<FF, __half><<<gr, b, 0, st>>>(g, f, pdir))
        else if (g.rhalf) DISPATCH_F(g.F, (k_surf3d<FF, float, __half><<<gr, b, 0, st>>>(g, f, pdir)))
        else DISPATCH_F(g.F, k_surf3d<FF><<<gr, b, 0, st>>>(g, f, pdir))
    } else {
        if (g.fhalf) DISPATCH_F(g.F, k_surf2d<FF, __half><<<dim3(cdiv(g.nx, 128), 1, g.nb), 128, 0, st>>>(g, f, pdir))
        else DISPATCH_F(g.F, k_surf2d<FF><<<dim3(cdiv(g.nx, 128), 1, g.nb), 128, 0, st>>>(g, f, pdir));
    }
}

// S arrays (FP32 or FP16 wave fields) to T stores (pack) or FP32 arrays
// back from T stores (unpack), value times scale; one grid row per array, a
// grid-stride loop over its elements
//
// FP32 to FP32 moves as 128-bit words where source and destination are
// equally aligned: 9 arrays of 1.2 M cells took 23.5 us one value at a time.
template <class T, bool UNPACK, class S = float>
__global__ void k_pack(PackSet ps)
{
    const int q = blockIdx.y;
    i64 n = ps.n[q];
    const float sc = ps.scale[q];
    if constexpr (std::is_same<T, float>::value && std::is_same<S, float>::value) {
        const float *src = (const float *)ps.src[q];
        float *dst = (float *)ps.dst[q];
        if ((((uintptr_t)src ^ (uintptr_t)dst) & 15) == 0) {
            const int head = (int)((16 - ((uintptr_t)src & 15)) / 4) & 3;   // values before the first aligned word
            const i64 words = n > head ? (n - head) / 4 : 0;
            for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (i64)gridDim.x * blockDim.x) {
                float4 v = *reinterpret_cast<const float4 *>(src + head + 4 * i);
                v.x *= sc; v.y *= sc; v.z *= sc; v.w *= sc;
                *reinterpret_cast<float4 *>(dst + head + 4 * i) = v;
            }
            // the ends: at most three values each
            if (blockIdx.x == 0 && threadIdx.x < 8) {
                const i64 i = threadIdx.x < 4 ? threadIdx.x : head + 4 * words + threadIdx.x - 4;
                if (i < n && (i < head || i >= head + 4 * words)) dst[i] = src[i] * sc;
            }
            return;
        }
    }
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        if (UNPACK) ((float *)ps.dst[q])[i] = to_f<T>(((const T *)ps.src[q])[i]) * sc;
        else ((T *)ps.dst[q])[i] = from_f<T>(to_f<S>(((const S *)ps.src[q])[i]) * sc);
    }
}

void launch_pack(const PackSet &ps, int prec, bool unpack, cudaStream_t st, bool half_src)
{
    if (ps.narr <= 0) return;
    i64 nmax = 0;
    for (int q = 0; q < ps.narr; q++) nmax = ps.n[q] > nmax ? ps.n[q] : nmax;
    dim3 gr((unsigned)std::min<i64>((nmax + 255) / 256, 148 * 8), (unsigned)ps.narr);
    if (gr.x == 0) return;
    if (half_src && !unpack) {
        if (prec == SFD_PREC_FP16) k_pack<__half, false, __half><<<gr, 256, 0, st>>>(ps);
        else if (prec == SFD_PREC_BF16) k_pack<__nv_bfloat16, false, __half><<<gr, 256, 0, st>>>(ps);
        else k_pack<float, false, __half><<<gr, 256, 0, st>>>(ps);
    } else if (prec == SFD_PREC_FP16) {
        if (unpack) k_pack<__half, true><<<gr, 256, 0, st>>>(ps);
        else k_pack<__half, false><<<gr, 256, 0, st>>>(ps);
    } else if (prec == SFD_PREC_BF16) {
        if (unpack) k_pack<__nv_bfloat16, true><<<gr, 256, 0, st>>>(ps);
        else k_pack<__nv_bfloat16, false><<<gr, 256, 0, st>>>(ps);
    } else {
        if (unpack) k_pack<float, true><<<gr, 256, 0, st>>>(ps);
        else k_pack<float, false><<<gr, 256, 0, st>>>(ps);
    }
}

void launch_savebnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, cudaStream_t st)
{
    dim3 gr(cdiv(g.nbnd, 256), 1, g.nb);
    if (gr.x == 0) return;
    if (prec == SFD_PREC_FP16) k_savebnd<__half><<<gr, 256, 0, st>>>(g, f, b, tofs);
    else if (prec == SFD_PREC_BF16) k_savebnd<__nv_bfloat16><<<gr, 256, 0, st>>>(g, f, b, tofs);
    else k_savebnd<float><<<gr, 256, 0, st>>>(g, f, b, tofs);
}

template <typename T>
static void launch_adj_t(const Grid &g, const Fields &f, const AdjFields &a, bool stress, cudaStream_t st)
{
    if (g.nd == 3) {
        dim3 b(32, 4, 2), gr(cdiv(g.nz, 32), cdiv(g.ny, 4), cdiv(g.nx, 2) * g.nb);
        if (stress) DISPATCH_F(g.F, MB_DISPATCH(g, k_adjs3d<FF, T, MBV><<<gr, b, 0, st>>>(g, f, a)))
        else DISPATCH_F(g.F, MB_DISPATCH(g, k_adjv3d<FF, T, MBV><<<gr, b, 0, st>>>(g, f, a)))
    } else {
        dim3 b(32, 8), gr(cdiv(g.nz, 32), cdiv(g.nx, 8), g.nb);
        if (stress) DISPATCH_F(g.F, k_adjs2d<FF, T><<<gr, b, 0, st>>>(g, f, a))
        else DISPATCH_F(g.F, k_adjv2d<FF, T><<<gr, b, 0, st>>>(g, f, a))
    }
}

void launch_update_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st)
{
    if (g.nd == 3 && (g.kernels == 0 || g.kernels == 5) && q4_ok(g) && g.L <= 3) {
        ROWS_DISPATCH(g, quad_update_adj<R>(g, f, a, stress, prec, st))
        return;
    }
    if (launch_quad2d_adj(g, f, a, stress, prec, st)) return;
    if (prec == SFD_PREC_FP16) launch_adj_t<__half>(g, f, a, stress, st);
    else if (prec == SFD_PREC_BF16) launch_adj_t<__nv_bfloat16>(g, f, a, stress, st);
    else launch_adj_t<float>(g, f, a, stress, st);
}

void launch_surface_adj(const Grid &g, const Fields &f, const AdjFields &a, float *q, cudaStream_t st)
{
    if (g.nd == 3) {
        dim3 b(32, 4), gr(cdiv(g.ny, 32), cdiv(g.nx, 4), g.nb);
        DISPATCH_F(g.F, k_surfadj3d_a<FF><<<gr, b, 0, st>>>(g, f, a, q));
        DISPATCH_F(g.F, k_surfadj3d_b<FF><<<gr, b, 0, st>>>(g, f, a, q));
    } else {
        DISPATCH_F(g.F, k_surfadj2d_a<FF><<<dim3(cdiv(g.nx, 128), 1, g.nb), 128, 0, st>>>(g, f, a, q));
        DISPATCH_F(g.F, k_surfadj2d_b<FF><<<dim3(cdiv(g.nx, 128), 1, g.nb), 128, 0, st>>>(g, f, a, q));
    }
}

void launch_sources(const Grid &g, const Fields &f, const PointSet &s, const float *src, int nt_total, int t,
                    int pdir, cudaStream_t st)
{
    if (s.n == 0) return;
    const bool pdl = g.nd == 3 && g.nb == 1 && pdl_enabled();
    const dim3 gr(cdiv(s.n, 128)), b(128);
    if (g.fhalf)
        launch_maybe_pdl(pdl, k_sources<__half>, gr, b, st, f, s, src, nt_total, t, pdir, g.dt, g.freesurf, g.F, g.ws);
    else
        launch_maybe_pdl(pdl, k_sources<float>, gr, b, st, f, s, src, nt_total, t, pdir, g.dt, g.freesurf, g.F, g.ws);
}

void launch_record(const Grid &g, const Fields &f, const PointSet &r, float *out, int nt_total, int t,
                   unsigned outmask, cudaStream_t st)
{
    if (r.n == 0 || outmask == 0) return;
    const bool pdl = g.nd == 3 && g.nb == 1 && pdl_enabled();
    const dim3 gr(cdiv(r.n, 128)), b(128);
    if (g.fhalf) launch_maybe_pdl(pdl, k_record<__half>, gr, b, st, f, r, out, nt_total, t, outmask, g.nd, g.ws);
    else launch_maybe_pdl(pdl, k_record<float>, gr, b, st, f, r, out, nt_total, t, outmask, g.nd, g.ws);
}

void launch_record_sources(const Grid &g, const Fields &f, const PointSet &r, float *out, int nt_total, int t,
                           unsigned outmask, const PointSet &s, const float *src, int tsrc, cudaStream_t st)
{
    const unsigned rb = outmask ? cdiv(r.n, 128) : 0, sb = tsrc >= 0 ? cdiv(s.n, 128) : 0;
    if (rb + sb == 0) return;
    const bool pdl = g.nd == 3 && g.nb == 1 && pdl_enabled();
    if (g.fhalf)
        launch_maybe_pdl(pdl, k_record_sources<__half>, dim3(rb + sb), dim3(128), st, f, r, out, nt_total, t, outmask, g.nd,
                         g.ws, rb, s, src, tsrc, g.dt, g.freesurf, g.F);
    else
        launch_maybe_pdl(pdl, k_record_sources<float>, dim3(rb + sb), dim3(128), st, f, r, out, nt_total, t, outmask, g.nd,
                         g.ws, rb, s, src, tsrc, g.dt, g.freesurf, g.F);
}

void launch_residuals(const Grid &g, const Fields &f, const AdjFields &a, const PointSet &r, const float *res,
                      int nt_total, int t, unsigned outmask, const PointSet &s, const float *src, int tsrc,
                      cudaStream_t st)
{
    const unsigned rb = outmask ? cdiv(r.n, 128) : 0, sb = tsrc >= 0 ? cdiv(s.n, 128) : 0;
    if (rb + sb == 0) return;
    k_residuals<<<rb + sb, 128, 0, st>>>(a, r, res, nt_total, t, outmask, g.nd, rb, f, s, src, tsrc, g.dt, g.freesurf, g.F,
                                        g.ws);
}

}  // namespace sfd
