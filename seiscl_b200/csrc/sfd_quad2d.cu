// sfd_quad2d.cu -- 4-cell vectorised 2D P-SV kernels: forward velocity and
// stress updates and the elastic adjoint, orders 4 and 8.
//
// One thread updates four consecutive z cells of a column with 128-bit loads
// and stores: a z derivative takes one 12-value window (three loads) for four
// cells, an x derivative one load per tap for four cells, against eight and
// eight loads per cell in the one-cell kernels, which load issue and latency
// bound.  Rows are made of whole aligned quads by Grid::zpad and Grid::zshift
// (init_grid).  Per cell the arithmetic is that of k_v2d, k_s2d, k_surf2d,
// k_adjv2d and k_adjs2d, in the same order: the same bits.
//
// The stress update also saves the boundary shells of a gradient run and
// applies the free surface, in that order, so that a forward step is three
// launches: velocity, stress, receivers with the next step's sources.
//
// us per step on a B200, one-cell kernels / these: 602 x 1503 order 8, L = 2
// 47 / 29; 8 shots of 300 x 1000 order 4 with shells 65 / 35, their adjoint 221
// / 103 (stress 151 / 57, velocity 70 / 42).  The adjoint moves about 188 bytes a
// cell and step, 69 us at the copy rate; the forward step's fields stay in L2.
#include <cuda_runtime.h>

#include "sfd_quad3d.cuh"

namespace sfd {

namespace {

#define CELL2D_Q4                                                                      \
    const int gz0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4 + F;                   \
    const int gx = blockIdx.y * blockDim.y + threadIdx.y + F;                          \
    if (gz0 > g.NZ - F - 1 || gx > g.NX - F - 1) return;                               \
    const i64 ip = (i64)(gx - F) * g.nz + (gz0 - F), iv = (i64)gx * g.NZ + gz0, sx = g.NZ;

// z slabs (update_v2D.cl:146-170): the recursion with full-node coefficients
// on df, with half-node ones on dh
__device__ __forceinline__ void cpml2d_z(const Grid &g, const Fields &f, int gz0, int gx, float *pf, Q4 &df, float *ph,
                                         Q4 &dh)
{
    const int F = g.F, NAB = g.nab, NZ = g.NZl;
    const bool zq = z_quads(g);
    const i64 row = (i64)(gx - F) * (2 * NAB);
    if (zq && !g.zpad && gz0 > NZ - NAB - F - 1) {
        const int k = gz0 - NZ + 2 * NAB + F;
        cpml_zq<true>(pf, row + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], 2 * NAB - k, -1, df);
        cpml_zq<true>(ph, row + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], 2 * NAB - 1 - k, -1, dh);
    } else if (zq && !g.freesurf && gz0 - F < NAB) {
        const int k = gz0 - F;
        cpml_zq<true>(pf, row + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, 1, df);
        cpml_zq<true>(ph, row + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, 1, dh);
    } else if (gz0 + 3 > NZ - NAB - F - 1 || (!zq && !g.freesurf && gz0 - F < NAB)) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gz = gz0 + j;
            if (gz > NZ - NAB - F - 1 && gz < NZ - F) {
                const int k = gz - NZ + 2 * NAB + F;
                cpml(pf, row + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], 2 * NAB - k, df.v[j]);
                cpml(ph, row + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], 2 * NAB - 1 - k, dh.v[j]);
            } else if (!g.freesurf && gz - F < NAB && gz < NZ - F) {
                const int k = gz - F;
                cpml(pf, row + k, ktab(f, 2, 0), f.cz[CA], f.cz[CB], k, df.v[j]);
                cpml(ph, row + k, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], k, dh.v[j]);
            }
        }
    }
}
// x slabs, one profile index a quad
__device__ __forceinline__ void cpml2d_x(const Grid &g, const Fields &f, int gz0, int gx, float *pf, Q4 &df, float *ph,
                                         Q4 &dh)
{
    const int F = g.F, NAB = g.nab;
    if (gx - F < NAB) {
        const int i = gx - F;
        const i64 q = (i64)i * g.nz + (gz0 - F);
        cpml_q<true>(pf, q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], i, df);
        cpml_q<true>(ph, q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], i, dh);
    }
    if (gx > g.NX - NAB - F - 1) {
        const int i = gx - g.NX + 2 * NAB + F;
        const i64 q = (i64)i * g.nz + (gz0 - F);
        cpml_q<true>(pf, q, ktab(f, 0, 0), f.cx[CA], f.cx[CB], 2 * NAB - i, df);
        cpml_q<true>(ph, q, ktab(f, 0, 1), f.cx[CAH], f.cx[CBH], 2 * NAB - 1 - i, dh);
    }
}

// stress / velocity derivatives of a quad: {normal x, normal z, shear x, shear z}
struct Deriv {
    Q4 xx, zz, x, z;
};
template <int F>
__device__ __forceinline__ Deriv stress_diff(float *const *w, i64 iv, i64 sx, const float *hc)
{
    Deriv d;
    d.xx = dfw_q<F>(w[SXX], iv, sx, hc);
    d.x = dbw_q<F>(w[SXZ], iv, sx, hc);
    d.zz = dfw_z<F>(ldw(w[SZZ], iv), hc);
    d.z = dbw_z<F>(ldw(w[SXZ], iv), hc);
    return d;
}
// vxx, vzz, vzx (x), vxz (z)
template <int F>
__device__ __forceinline__ Deriv velocity_diff(float *const *w, i64 iv, i64 sx, const float *hc)
{
    Deriv d;
    d.xx = dbw_q<F>(w[VX], iv, sx, hc);
    d.x = dfw_q<F>(w[VZ], iv, sx, hc);
    d.z = dfw_z<F>(ldw(w[VX], iv), hc);
    d.zz = dbw_z<F>(ldw(w[VZ], iv), hc);
    return d;
}
__device__ __forceinline__ void cpml_stress(const Grid &g, const Fields &f, int gz0, int gx, Deriv &d)
{
    cpml2d_z(g, f, gz0, gx, f.psi[PSXZ_Z], d.z, f.psi[PSZZ_Z], d.zz);
    cpml2d_x(g, f, gz0, gx, f.psi[PSXZ_X], d.x, f.psi[PSXX_X], d.xx);
}
__device__ __forceinline__ void cpml_velocity(const Grid &g, const Fields &f, int gz0, int gx, Deriv &d)
{
    cpml2d_z(g, f, gz0, gx, f.psi[PVZ_Z], d.zz, f.psi[PVX_Z], d.z);
    cpml2d_x(g, f, gz0, gx, f.psi[PVX_X], d.xx, f.psi[PVZ_X], d.x);
}

// taper factors of apply_taper on NV quads
template <int NV>
__device__ __forceinline__ void taper2d_q(const Grid &g, const float *taper, int gz0, int gx, Q4 *const (&q)[NV])
{
    const int F = g.F, NAB = g.nab, NZ = g.NZl;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int gz = gz0 + j;
        auto mul = [&](float t) {
#pragma unroll
            for (int n = 0; n < NV; n++) q[n]->v[j] *= t;
        };
        if (!g.freesurf && gz - F < NAB) mul(__ldg(taper + gz - F));
        if (gz > NZ - NAB - F - 1 && gz < NZ - F) mul(__ldg(taper + NZ - F - gz - 1));
        if (gx - F < NAB) mul(__ldg(taper + gx - F));
        if (gx > g.NX - NAB - F - 1) mul(__ldg(taper + g.NX - F - gx - 1));
    }
}

template <typename T>
__device__ __forceinline__ void bnd_put(const Grid &g, const BndSlot &b, int w, i64 at, float v)
{
    ((T *)b.p[w])[at] = from_f<T>(v * g.bsc[w]);
}

// shell indices of a quad's cells (-1: none); most quads are inside or outside
__device__ __forceinline__ bool shell_quad(const Grid &g, int gz0, int gx, int (&m)[4])
{
    const BndDims b = bnd_dims(g);
    const int F = g.F, i = gx - b.lbnd, k = gz0 - b.lbnds;
    if (i < 0 || i >= b.NXbnd || k + 3 < 0 || k >= b.NZbnd ||
        (i >= F && i < b.NXbnd - F && k >= F && k + 3 < b.NZbnd - F))
        return false;
#pragma unroll
    for (int j = 0; j < 4; j++) m[j] = inject_ind2d(g, gz0 + j, gx);
    return true;
}

}  // namespace

template <int F>
__global__ void __launch_bounds__(128) k_v2d_q4(Grid g, Fields f)
{
    SHOT_F
    CELL2D_Q4
    Q4 vx = ldq_rw(f.w[VX] + iv), vz = ldq_rw(f.w[VZ] + iv);
    const Q4 rip = ldq(f.p[PRIP] + ip), rkp = ldq(f.p[PRKP] + ip);
    Deriv d = stress_diff<F>(f.w, iv, sx, g.hc);
    if (g.abs_type == 1) cpml_stress(g, f, gz0, gx, d);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        vx.v[j] = v2d_math(vx.v[j], d.xx.v[j], d.z.v[j], rip.v[j]);
        vz.v[j] = v2d_math(vz.v[j], d.zz.v[j], d.x.v[j], rkp.v[j]);
    }
    if (g.abs_type == 2) {
        Q4 *const q[2] = {&vx, &vz};
        taper2d_q<2>(g, f.taper, gz0, gx, q);
    }
    stq(f.w[VX] + iv, vx);
    stq(f.w[VZ] + iv, vz);
}

// b: boundary shells to save (nfield = 0: none) at step offset tofs, in type
// T; surf: apply the free surface
template <int F, int L, typename T>
__global__ void __launch_bounds__(128) k_s2d_q4(Grid g, Fields f, BndSlot b, i64 tofs, bool surf)
{
    SHOT_F
    CELL2D_Q4
    constexpr int LL = L > 0 ? L : 1;
    Q4 s[3] = {ldq_rw(f.w[SXX] + iv), ldq_rw(f.w[SZZ] + iv), ldq_rw(f.w[SXZ] + iv)};
    float *const wr[3] = {f.r[RXX], f.r[RZZ], f.r[RXZ]};
    Q4 r[3][LL], qtaup, qtaus, qtausipkp;
    const Q4 qM = ldq(f.p[PM] + ip), qmu = ldq(f.p[PMU] + ip), qmuipkp = ldq(f.p[PMUIPKP] + ip);
    if constexpr (L > 0) {
        qtaup = ldq(f.p[PTAUP] + ip); qtaus = ldq(f.p[PTAUS] + ip); qtausipkp = ldq(f.p[PTAUSIPKP] + ip);
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) r[q][l] = ldq_rw(wr[q] + l * g.nvol + iv);
    }
    Deriv d = velocity_diff<F>(f.w, iv, sx, g.hc);
    if (g.abs_type == 1) cpml_velocity(g, f, gz0, gx, d);
    S2dMat m0;   // material of the first cell, for the surface
#pragma unroll
    for (int j = 0; j < 4; j++) {
        S2dMat m;
        if constexpr (L == 0) m = s2d_elastic(qM.v[j], qmu.v[j], qmuipkp.v[j]);
        else m = s2d_visco(L, g.dt, qM.v[j], qmu.v[j], qmuipkp.v[j], qtaup.v[j], qtaus.v[j], qtausipkp.v[j]);
        if (j == 0) m0 = m;
        const float tr = __fadd_rn(d.xx.v[j], d.zz.v[j]), sh = __fadd_rn(d.z.v[j], d.x.v[j]);
        const float exx = s2d_normal(m.gm, tr, m.fm, d.zz.v[j]), ezz = s2d_normal(m.gm, tr, m.fm, d.xx.v[j]);
        if constexpr (L == 0) {
            s[2].v[j] = __fmaf_rn(m.fipkp, sh, s[2].v[j]);
            s[0].v[j] = __fadd_rn(s[0].v[j], exx);
            s[1].v[j] = __fadd_rn(s[1].v[j], ezz);
        } else {
            const float x[3] = {s2d_normal(m.e, tr, m.d, d.zz.v[j]), s2d_normal(m.e, tr, m.d, d.xx.v[j]),
                                __fmul_rn(m.dipkp, sh)};
            float o[3] = {0, 0, 0}, n[3] = {0, 0, 0};
#pragma unroll
            for (int l = 0; l < L; l++)
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    o[q] += r[q][l].v[j];
                    r[q][l].v[j] = s2d_memory(r[q][l].v[j], g.eta[l], g.eta_b[l], g.eta_c[l], x[q]);
                    n[q] += r[q][l].v[j];
                }
            s[2].v[j] = s2d_add(s[2].v[j], __fmaf_rn(m.fipkp, sh, __fmul_rn(g.dt2, o[2])), g.dt2, n[2]);
            s[0].v[j] = s2d_add(s[0].v[j], __fmaf_rn(g.dt2, o[0], exx), g.dt2, n[0]);
            s[1].v[j] = s2d_add(s[1].v[j], __fmaf_rn(g.dt2, o[1], ezz), g.dt2, n[1]);
        }
    }
    if (g.abs_type == 2) {
        Q4 *const q[3] = {&s[0], &s[1], &s[2]};
        taper2d_q<3>(g, f.taper, gz0, gx, q);
    }
    int m[4];
    if (b.nfield && shell_quad(g, gz0, gx, m)) {   // boundary shells, before the free surface
        const i64 at = (i64)blockIdx.z * (g.sb_bnd / (i64)sizeof(T)) + tofs;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (m[j] < 0) continue;
            bnd_put<T>(g, b, VX, at + m[j], f.w[VX][iv + j]);
            bnd_put<T>(g, b, VZ, at + m[j], f.w[VZ][iv + j]);
            bnd_put<T>(g, b, SXX, at + m[j], s[0].v[j]);
            bnd_put<T>(g, b, SZZ, at + m[j], s[1].v[j]);
            bnd_put<T>(g, b, SXZ, at + m[j], s[2].v[j]);
        }
    }
    if (surf && gz0 <= 2 * F) {   // the arithmetic of surf2d_column, forward
        if (F == 4 && gz0 == F + 4) f.w[SZZ][iv - 8] = -s[1].v[0];
        if (gz0 == F) {
            const Surf2d su = surf2d_of(m0);
            const float vxx = d.xx.v[0], vzz = d.zz.v[0], h = surf2d_h<L == 0>(su, vxx, vzz);
            s[1].v[0] = 0.0f;
            if constexpr (L == 0) {
                s[0].v[0] = __fadd_rn(h, s[0].v[0]);
            } else {
                float sump = 0;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    r[1][l].v[0] = 0.0f;
                    sump += r[0][l].v[0];
                }
                s[0].v[0] = __fadd_rn(__fmaf_rn(-g.dt2, sump, h), s[0].v[0]);
                sump = 0;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    r[0][l].v[0] = __fadd_rn(__fmul_rn(surf2d_b(g.eta[l]), surf2d_hr(su, vxx, vzz)), r[0][l].v[0]);
                    sump += r[0][l].v[0];
                }
                s[0].v[0] = __fadd_rn(__fmul_rn(g.dt2, sump), s[0].v[0]);
            }
#pragma unroll
            for (int k = 1; k <= (F < 4 ? F : 3); k++) f.w[SZZ][iv - k] = -s[1].v[k];
#pragma unroll
            for (int k = 1; k <= F; k++) f.w[SXZ][iv - k] = -s[2].v[k - 1];
        }
    }
    if constexpr (L > 0) {
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < 3; q++) stq(wr[q] + l * g.nvol + iv, r[q][l]);
    }
    stq(f.w[SXX] + iv, s[0]);
    stq(f.w[SZZ] + iv, s[1]);
    stq(f.w[SXZ] + iv, s[2]);
}

template <int F, typename T>
__global__ void __launch_bounds__(128) k_adjv2d_q4(Grid g, Fields f, AdjFields a)
{
    SHOT_FA
    CELL2D_Q4
    const float *hc = g.hc;
    const Q4 rip = ldq(f.p[PRIP] + ip), rkp = ldq(f.p[PRKP] + ip);
    Q4 vx = {{0, 0, 0, 0}}, vz = vx;
    if (g.ckpt) {
        vx = fwd_quad<T>(g, a, VX, iv);
        vz = fwd_quad<T>(g, a, VZ, iv);
    } else if (!g.bp2) {   // backpropagate the forward velocities (update_adjv2D.cl:205-240)
        const Deriv d = stress_diff<F>(f.w, iv, sx, hc);
        vx = ldq_rw(f.w[VX] + iv); vz = ldq_rw(f.w[VZ] + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            vx.v[j] = __fmaf_rn(-__fadd_rn(d.xx.v[j], d.z.v[j]), rip.v[j], vx.v[j]);
            vz.v[j] = __fmaf_rn(-__fadd_rn(d.zz.v[j], d.x.v[j]), rkp.v[j], vz.v[j]);
        }
        int m[4];
        if (shell_quad(g, gz0, gx, m)) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (m[j] < 0) continue;
                vx.v[j] = bnd_at<T>(g, a, VX, m[j]);
                vz.v[j] = bnd_at<T>(g, a, VZ, m[j]);
            }
        }
        stq(f.w[VX] + iv, vx);
        stq(f.w[VZ] + iv, vz);
    }
    Deriv d = stress_diff<F>(a.wr, iv, sx, hc);
    if (g.abs_type == 1) cpml_stress(g, f, gz0, gx, d);
    Q4 wx = ldq_rw(a.wr[VX] + iv), wz = ldq_rw(a.wr[VZ] + iv);
    float gr[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float lvx = __fmul_rn(__fadd_rn(d.xx.v[j], d.z.v[j]), rip.v[j]);
        const float lvz = __fmul_rn(__fadd_rn(d.zz.v[j], d.x.v[j]), rkp.v[j]);
        wx.v[j] = __fadd_rn(wx.v[j], lvx);
        wz.v[j] = __fadd_rn(wz.v[j], lvz);
        gr[j] = __fmaf_rn(-vx.v[j], lvx, -__fmul_rn(vz.v[j], lvz));
    }
    if (g.abs_type == 2) {
        Q4 *const q[2] = {&wx, &wz};
        taper2d_q<2>(g, f.taper, gz0, gx, q);
    }
    stq(a.wr[VX] + iv, wx);
    stq(a.wr[VZ] + iv, wz);
    if (!g.bp2) grad_add4(a.grad[GRHO], ip, gr);
}

// elastic media (L = 0), no Hessian
template <int F, typename T>
__global__ void __launch_bounds__(128) k_adjs2d_q4(Grid g, Fields f, AdjFields a)
{
    SHOT_FA
    CELL2D_Q4
    const float *hc = g.hc;
    const Q4 qM = ldq(f.p[PM] + ip), qmu = ldq(f.p[PMU] + ip), qmuipkp = ldq(f.p[PMUIPKP] + ip);
    Q4 s[3] = {{{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}};   // forward sxx, szz, sxz
    if (g.ckpt) {
        s[0] = fwd_quad<T>(g, a, SXX, iv); s[1] = fwd_quad<T>(g, a, SZZ, iv); s[2] = fwd_quad<T>(g, a, SXZ, iv);
    } else if (!g.bp2) {   // reconstruct the forward stresses (update_adjs2D.cl:222-278)
        const Deriv d = velocity_diff<F>(f.w, iv, sx, hc);
        s[0] = ldq_rw(f.w[SXX] + iv); s[1] = ldq_rw(f.w[SZZ] + iv); s[2] = ldq_rw(f.w[SXZ] + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const S2dMat m = s2d_elastic(qM.v[j], qmu.v[j], qmuipkp.v[j]);
            const float tr = __fadd_rn(d.xx.v[j], d.zz.v[j]);
            s[2].v[j] = __fmaf_rn(-m.fipkp, __fadd_rn(d.z.v[j], d.x.v[j]), s[2].v[j]);
            s[0].v[j] = __fsub_rn(s[0].v[j], s2d_normal(m.gm, tr, m.fm, d.zz.v[j]));
            s[1].v[j] = __fsub_rn(s[1].v[j], s2d_normal(m.gm, tr, m.fm, d.xx.v[j]));
        }
        int m[4];
        if (shell_quad(g, gz0, gx, m)) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (m[j] < 0) continue;
                s[0].v[j] = bnd_at<T>(g, a, SXX, m[j]);
                s[1].v[j] = bnd_at<T>(g, a, SZZ, m[j]);
                s[2].v[j] = bnd_at<T>(g, a, SXZ, m[j]);
            }
        }
        stq(f.w[SXX] + iv, s[0]);
        stq(f.w[SZZ] + iv, s[1]);
        stq(f.w[SXZ] + iv, s[2]);
    }
    Deriv d = velocity_diff<F>(a.wr, iv, sx, hc);
    if (g.abs_type == 1) cpml_velocity(g, f, gz0, gx, d);
    Q4 w[3] = {ldq_rw(a.wr[SXX] + iv), ldq_rw(a.wr[SZZ] + iv), ldq_rw(a.wr[SXZ] + iv)};
    float gM[4], gmu[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const S2dMat m = s2d_elastic(qM.v[j], qmu.v[j], qmuipkp.v[j]);
        const float tr = __fadd_rn(d.xx.v[j], d.zz.v[j]);
        const float lsxz = __fmul_rn(m.fipkp, __fadd_rn(d.z.v[j], d.x.v[j]));
        const float lsxx = s2d_normal(m.gm, tr, m.fm, d.zz.v[j]), lszz = s2d_normal(m.gm, tr, m.fm, d.xx.v[j]);
        w[0].v[j] = __fadd_rn(w[0].v[j], lsxx);
        w[1].v[j] = __fadd_rn(w[1].v[j], lszz);
        w[2].v[j] = __fadd_rn(w[2].v[j], lsxz);
        const Adj2dGrad q = adj2d_grad(g.restype, qM.v[j], qmu.v[j], s[0].v[j], s[1].v[j], s[2].v[j], lsxx, lszz, lsxz);
        gM[j] = q.M;
        gmu[j] = q.mu;
    }
    if (g.abs_type == 2) {
        Q4 *const q[3] = {&w[0], &w[1], &w[2]};
        taper2d_q<3>(g, f.taper, gz0, gx, q);
    }
    stq(a.wr[SXX] + iv, w[0]);
    stq(a.wr[SZZ] + iv, w[1]);
    stq(a.wr[SXZ] + iv, w[2]);
    if (g.bp2) return;
    grad_add4(a.grad[GM], ip, gM);
    if (g.restype == 0) grad_add4(a.grad[GMU], ip, gmu);
}

// ------------------------------------------------------------- launchers
// quads along z, columns: 16 x 8 per CTA, or 8 x 16 where that leaves fewer
// threads without a quad
static dim3 block2d(const Grid &g)
{
    const unsigned nq = (unsigned)(g.nz / 4);
    return cdiv(nq, 8) * 8 < cdiv(nq, 16) * 16 ? dim3(8, 16) : dim3(16, 8);
}
static dim3 grid2d(const Grid &g, dim3 b) { return dim3(cdiv(g.nz / 4, b.x), cdiv(g.nx, b.y), g.nb); }

bool quad2d_ok(const Grid &g)
{
    return g.nd == 2 && !g.fhalf && g.kernels == 0 && g.nz % 4 == 0 && g.L <= 3 &&
           (g.F == 4 || (g.F == 2 && g.zshift == 2));
}

void launch_quad2d_v(const Grid &g, const Fields &f, cudaStream_t st)
{
    const dim3 b = block2d(g), gr = grid2d(g, b);
    if (g.F == 4) k_v2d_q4<4><<<gr, b, 0, st>>>(g, f);
    else k_v2d_q4<2><<<gr, b, 0, st>>>(g, f);
}

template <int F, typename T>
static void launch_s_t(const Grid &g, const Fields &f, const BndSlot &bs, i64 tofs, bool surf, cudaStream_t st)
{
    const dim3 b = block2d(g), gr = grid2d(g, b);
    switch (g.L) {
    case 0: k_s2d_q4<F, 0, T><<<gr, b, 0, st>>>(g, f, bs, tofs, surf); break;
    case 1: k_s2d_q4<F, 1, T><<<gr, b, 0, st>>>(g, f, bs, tofs, surf); break;
    case 2: k_s2d_q4<F, 2, T><<<gr, b, 0, st>>>(g, f, bs, tofs, surf); break;
    default: k_s2d_q4<F, 3, T><<<gr, b, 0, st>>>(g, f, bs, tofs, surf); break;
    }
}

void launch_quad2d_s(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, bool surf, cudaStream_t st)
{
    if (g.F == 4) {
        if (prec == SFD_PREC_FP16) launch_s_t<4, __half>(g, f, b, tofs, surf, st);
        else if (prec == SFD_PREC_BF16) launch_s_t<4, __nv_bfloat16>(g, f, b, tofs, surf, st);
        else launch_s_t<4, float>(g, f, b, tofs, surf, st);
    } else {
        if (prec == SFD_PREC_FP16) launch_s_t<2, __half>(g, f, b, tofs, surf, st);
        else if (prec == SFD_PREC_BF16) launch_s_t<2, __nv_bfloat16>(g, f, b, tofs, surf, st);
        else launch_s_t<2, float>(g, f, b, tofs, surf, st);
    }
}

template <int F, typename T>
static void launch_adj_t(const Grid &g, const Fields &f, const AdjFields &a, bool stress, cudaStream_t st)
{
    const dim3 b = block2d(g), gr = grid2d(g, b);
    if (stress) k_adjs2d_q4<F, T><<<gr, b, 0, st>>>(g, f, a);
    else k_adjv2d_q4<F, T><<<gr, b, 0, st>>>(g, f, a);
}

bool launch_quad2d_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st)
{
    if (!quad2d_ok(g) || (stress && (g.L > 0 || g.hout))) return false;
    if (g.F == 4) {
        if (prec == SFD_PREC_FP16) launch_adj_t<4, __half>(g, f, a, stress, st);
        else if (prec == SFD_PREC_BF16) launch_adj_t<4, __nv_bfloat16>(g, f, a, stress, st);
        else launch_adj_t<4, float>(g, f, a, stress, st);
    } else {
        if (prec == SFD_PREC_FP16) launch_adj_t<2, __half>(g, f, a, stress, st);
        else if (prec == SFD_PREC_BF16) launch_adj_t<2, __nv_bfloat16>(g, f, a, stress, st);
        else launch_adj_t<2, float>(g, f, a, stress, st);
    }
    return true;
}

}  // namespace sfd
