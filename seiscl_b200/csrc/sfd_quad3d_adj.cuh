// sfd_quad3d_adj.cuh -- 4-cell vectorised 3D adjoint kernels and their
// launchers, templates on the kind of rows R.
#pragma once

#include "sfd_quad3d.cuh"

namespace sfd {

// ------------------------------------------- 4-cell vectorised 3D adjoint
// The adjoint kernels of k_adjv3d / k_adjs3d on quads of z cells, with the
// same per-cell arithmetic: backpropagation of the forward field (not for
// the DFT gradient, g.bp2), saved-boundary injection per cell, the adjoint
// update with CPML, and the on-the-fly gradient accumulated in FP64.
// The adjoint memory variables the stress update reads.  Nothing writes
// them in 3D but the DFT adjoint, where they are the forward arrays (the
// update stores its new values there, update_adjs3D.cl:566-583): elsewhere
// they keep the zeros the adjoint starts from, and 6 L streams a cell need
// not be read.
__device__ __forceinline__ Q4 adj_memory(const Grid &g, const float *p)
{
    return g.bp2 ? ldq_rw(p) : Q4{{0.0f, 0.0f, 0.0f, 0.0f}};
}

// L2 prefetch of one quad's cell in a per-cell stream
__device__ __forceinline__ void pf_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// PF (single-shot launches of the default selection): the thread first asks
// L2 for its quad's per-cell streams -- the forward and adjoint velocities,
// the buoyancies and the density gradient sum -- and the launch takes 4 CTAs
// per SM (an adjoint step of 100 x 200 x 200: 511 us against 519 with 3, 528
// with 5).
template <int R, typename T, bool MB = false, bool PF = false>
__global__ void __launch_bounds__(128, PF ? 4 : 1) k_adjv3d_q4(Grid g, Fields f, AdjFields a)
{
    constexpr int F = half_width(R);
    CELL3D_Q4
    if (MB) shot_adj(g, a, shot);
    if constexpr (PF) {
        const bool recon = !g.ckpt && !g.bp2;
#pragma unroll
        for (int q = VX; q <= VZ; q++) {
            pf_l2(a.wr[q] + iv);
            if (recon) pf_l2(f.w[q] + iv);
        }
        pf_l2(f.p[PRIP] + ip); pf_l2(f.p[PRJP] + ip); pf_l2(f.p[PRKP] + ip);
        if (!g.bp2) pf_l2(a.grad[GRHO] + ip);
    }
    const float *hc = g.hc;
    const Q4 rip = ldq(f.p[PRIP] + ip), rjp = ldq(f.p[PRJP] + ip), rkp = ldq(f.p[PRKP] + ip);
    Q4 vx = {{0, 0, 0, 0}}, vy = vx, vz = vx;
    if (g.ckpt) {
        vx = fwd_quad<T>(g, a, VX, iv); vy = fwd_quad<T>(g, a, VY, iv); vz = fwd_quad<T>(g, a, VZ, iv);
    } else if (!g.bp2) {  // backpropagate the forward velocities (update_adjv3D.cl:297-340)
        Q4 szz_z = dfw_z<F>(ldw(f.w[SZZ], iv), hc);
        Q4 sxx_x = dfw_q<F>(f.w[SXX], iv, sx, hc);
        Q4 sxz_x = dbw_q<F>(f.w[SXZ], iv, sx, hc);
        Q4 sxz_z = dbw_z<F>(ldw(f.w[SXZ], iv), hc);
        Q4 syz_y = dbw_q<F>(f.w[SYZ], iv, sy, hc);
        Q4 syz_z = dbw_z<F>(ldw(f.w[SYZ], iv), hc);
        Q4 syy_y = dfw_q<F>(f.w[SYY], iv, sy, hc);
        Q4 sxy_x = dbw_q<F>(f.w[SXY], iv, sx, hc);
        Q4 sxy_y = dbw_q<F>(f.w[SXY], iv, sy, hc);
        vx = ldq_rw(f.w[VX] + iv); vy = ldq_rw(f.w[VY] + iv); vz = ldq_rw(f.w[VZ] + iv);
        int mq[4] = {-1, -1, -1, -1};
        shell_quad3d(g, gz0, gy, gx, mq);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            vx.v[j] = vx.v[j] - (sxx_x.v[j] + sxy_y.v[j] + sxz_z.v[j]) * rip.v[j];
            vy.v[j] = vy.v[j] - (syy_y.v[j] + sxy_x.v[j] + syz_z.v[j]) * rjp.v[j];
            vz.v[j] = vz.v[j] - (szz_z.v[j] + sxz_x.v[j] + syz_y.v[j]) * rkp.v[j];
            const int m = mq[j];
            if (m != -1) {
                vx.v[j] = bnd_at<T>(g, a, VX, m);
                vy.v[j] = bnd_at<T>(g, a, VY, m);
                vz.v[j] = bnd_at<T>(g, a, VZ, m);
            }
        }
        stq(f.w[VX] + iv, vx); stq(f.w[VY] + iv, vy); stq(f.w[VZ] + iv, vz);
    }
    Q4 szz_zr = dfw_z<F>(ldw(a.wr[SZZ], iv), hc);
    Q4 sxx_xr = dfw_q<F>(a.wr[SXX], iv, sx, hc);
    Q4 sxz_xr = dbw_q<F>(a.wr[SXZ], iv, sx, hc);
    Q4 sxz_zr = dbw_z<F>(ldw(a.wr[SXZ], iv), hc);
    Q4 syz_yr = dbw_q<F>(a.wr[SYZ], iv, sy, hc);
    Q4 syz_zr = dbw_z<F>(ldw(a.wr[SYZ], iv), hc);
    Q4 syy_yr = dfw_q<F>(a.wr[SYY], iv, sy, hc);
    Q4 sxy_xr = dbw_q<F>(a.wr[SXY], iv, sx, hc);
    Q4 sxy_yr = dbw_q<F>(a.wr[SXY], iv, sy, hc);
    if (g.abs_type == 1)
        cpml_v3d_q4<!whole_rows(R)>(g, f, gz0, gy, gx, sxx_xr, syy_yr, szz_zr, sxy_yr, sxy_xr, syz_yr, syz_zr, sxz_xr, sxz_zr);
    Q4 wx = ldq_rw(a.wr[VX] + iv), wy = ldq_rw(a.wr[VY] + iv), wz = ldq_rw(a.wr[VZ] + iv);
    float gr[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float lvx = (sxx_xr.v[j] + sxy_yr.v[j] + sxz_zr.v[j]) * rip.v[j];
        const float lvy = (syy_yr.v[j] + sxy_xr.v[j] + syz_zr.v[j]) * rjp.v[j];
        const float lvz = (szz_zr.v[j] + sxz_xr.v[j] + syz_yr.v[j]) * rkp.v[j];
        float w3[3] = {wx.v[j] + lvx, wy.v[j] + lvy, wz.v[j] + lvz};
        if (g.abs_type == 2) taper_regs<3>(g, f.taper, gz0 + j, gy, gx, w3);
        wx.v[j] = w3[0]; wy.v[j] = w3[1]; wz.v[j] = w3[2];
        gr[j] = -vx.v[j] * lvx - vy.v[j] * lvy - vz.v[j] * lvz;
    }
    stq(a.wr[VX] + iv, wx); stq(a.wr[VY] + iv, wy); stq(a.wr[VZ] + iv, wz);
    if (!g.bp2) grad_add4(a.grad[GRHO], ip, gr);
}

// CPML of the adjoint stress update (cpml_s3d with adjoint_form): as
// cpml_s3d_q4, except that a cell in both z slabs or both y slabs takes
// only the first (else-if), as update_adjs3D.cl does
template <bool DIV>
__device__ __forceinline__ void cpml_s3d_adj_q4(const Grid &g, const Fields &f, int gz0, int gy, int gx, Q4 &vxx,
                                                Q4 &vxy, Q4 &vxz, Q4 &vyx, Q4 &vyy, Q4 &vyz, Q4 &vzx, Q4 &vzy,
                                                Q4 &vzz)
{
    const int F = g.F, NAB = g.nab, NZ = g.NZl, NY = g.NY, NX = g.NX;
    const i64 nz = g.nz, ny = g.ny;
    if (cpml_slabs_apart(g)) {   // then no cell is in two slabs of an axis
        cpml_s3d_q4<DIV>(g, f, gz0, gy, gx, vxx, vxy, vxz, vyx, vyy, vyz, vzx, vzy, vzz);
        return;
    }
    const bool zq = z_quads(g);
    const int zpad = g.zpad;
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
            const bool zb = gz > NZ - NAB - F - 1 && gz < NZ - F;
            if (zb) {
                i64 i = gx - F, jj = gy - F, k = gz - NZ + NAB + F + NAB;
                int ind = 2 * NAB - 1 - (int)k;
                i64 q = (i * ny + jj) * (2 * NAB) + k;
                cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vxz.v[j]);
                cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], ind, vyz.v[j]);
                cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], ind + 1, vzz.v[j]);
            } else if (!g.freesurf && gz - F < NAB) {
                i64 i = gx - F, jj = gy - F, k = gz - F;
                i64 q = (i * ny + jj) * (2 * NAB) + k;
                cpml(f.psi[PVX_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vxz.v[j]);
                cpml(f.psi[PVY_Z], q, ktab(f, 2, 1), f.cz[CAH], f.cz[CBH], (int)k, vyz.v[j]);
                cpml(f.psi[PVZ_Z], q, ktab(f, 2, 0), f.cz[CA], f.cz[CB], (int)k, vzz.v[j]);
            }
        }
    }
    const i64 k0 = gz0 - F;
    if (gy - F < NAB) {
        i64 i = gx - F, j = gy - F;
        i64 q = (i * (2 * NAB) + j) * nz + k0;
        cpml_q<DIV>(f.psi[PVX_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vxy);
        cpml_q<DIV>(f.psi[PVY_Y], q, ktab(f, 1, 0), f.cy[CA], f.cy[CB], (int)j, vyy);
        cpml_q<DIV>(f.psi[PVZ_Y], q, ktab(f, 1, 1), f.cy[CAH], f.cy[CBH], (int)j, vzy);
    } else if (gy > NY - NAB - F - 1) {
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

// PF: prefetch of the quad's per-cell streams (forward and adjoint stresses
// and memory variables, parameters, the M and mu gradient sums) and 3 CTAs
// per SM, as k_adjv3d_q4.  The saved-boundary index of each cell of the quad
// is found once and kept for the four phases.
template <int R, int L, typename T, bool MB = false, bool PF = false>
__global__ void __launch_bounds__(128, PF ? 3 : 4) k_adjs3d_q4(Grid g, Fields f, AdjFields a)
{
    constexpr int F = half_width(R);
    CELL3D_Q4
    if (MB) shot_adj(g, a, shot);
    const bool recon = !g.ckpt && !g.bp2;
    if constexpr (PF) {
#pragma unroll
        for (int q = SXX; q <= SXZ; q++) {
            pf_l2(a.wr[q] + iv);
            if (recon) pf_l2(f.w[q] + iv);
        }
#pragma unroll
        for (int l = 0; l < L; l++)
#pragma unroll
            for (int q = 0; q < NR; q++)
                if (recon) pf_l2(f.r[q] + l * g.nvol + iv);
        constexpr int np = L > 0 ? 10 : 5;
        constexpr int pid[10] = {PM, PMU, PMUIPJP, PMUJPKP, PMUIPKP, PTAUP, PTAUS, PTAUSIPJP, PTAUSJPKP, PTAUSIPKP};
#pragma unroll
        for (int k = 0; k < np; k++) pf_l2(f.p[pid[k]] + ip);
        if (!g.bp2) {
            pf_l2(a.grad[GM] + ip);
            if (g.restype == 0) pf_l2(a.grad[GMU] + ip);
        }
    }
    int mq[4] = {-1, -1, -1, -1};
    if (recon) shell_quad3d(g, gz0, gy, gx, mq);
    const float *hc = g.hc;
    // adjoint velocity derivatives, with CPML
    Q4 vzzr = dbw_z<F>(ldw(a.wr[VZ], iv), hc), vyzr = dfw_z<F>(ldw(a.wr[VY], iv), hc);
    Q4 vxzr = dfw_z<F>(ldw(a.wr[VX], iv), hc);
    Q4 vzxr = dfw_q<F>(a.wr[VZ], iv, sx, hc), vzyr = dfw_q<F>(a.wr[VZ], iv, sy, hc);
    Q4 vyxr = dfw_q<F>(a.wr[VY], iv, sx, hc), vyyr = dbw_q<F>(a.wr[VY], iv, sy, hc);
    Q4 vxxr = dbw_q<F>(a.wr[VX], iv, sx, hc), vxyr = dfw_q<F>(a.wr[VX], iv, sy, hc);
    if (g.abs_type == 1)
        cpml_s3d_adj_q4<!whole_rows(R)>(g, f, gz0, gy, gx, vxxr, vxyr, vxzr, vyxr, vyyr, vyzr, vzxr, vzyr, vzzr);
    Q4 rsh[3];   // adjoint shear sums vxy+vyx, vyz+vzy, vxz+vzx
#pragma unroll
    for (int j = 0; j < 4; j++) {
        rsh[0].v[j] = vxyr.v[j] + vyxr.v[j];
        rsh[1].v[j] = vyzr.v[j] + vzyr.v[j];
        rsh[2].v[j] = vxzr.v[j] + vzxr.v[j];
    }
    const Q4 qM = ldq(f.p[PM] + ip), qmu = ldq(f.p[PMU] + ip);
    float gM[4] = {0, 0, 0, 0}, gmu[4] = {0, 0, 0, 0};
    Q4 qc3 = {{0, 0, 0, 0}};

    // ---- normal stresses (sxx, syy, szz) with rxx, ryy, rzz: the forward
    // reconstruction of the quad, then its adjoint update
    {
        const int wid[3] = {SXX, SYY, SZZ}, rid[3] = {RXX, RYY, RZZ};
        Q4 qtaup = {{0, 0, 0, 0}}, qtaus = qtaup;
        if (L > 0) { qtaup = ldq(f.p[PTAUP] + ip); qtaus = ldq(f.p[PTAUS] + ip); }
        Q4 s3[3] = {{{0, 0, 0, 0}}, {{0, 0, 0, 0}}, {{0, 0, 0, 0}}};
        if (g.ckpt) {
#pragma unroll
            for (int c = 0; c < 3; c++) s3[c] = fwd_quad<T>(g, a, wid[c], iv);
        } else if (!g.bp2) {
            const Q4 vzz = dbw_z<F>(ldw(f.w[VZ], iv), hc);
            const Q4 vyy = dbw_q<F>(f.w[VY], iv, sy, hc);
            const Q4 vxx = dbw_q<F>(f.w[VX], iv, sx, hc);
#pragma unroll
            for (int c = 0; c < 3; c++) s3[c] = ldq_rw(f.w[wid[c]] + iv);
            Q4 rf[3][L > 0 ? L : 1];
            if constexpr (L > 0) {
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int l = 0; l < L; l++) rf[c][l] = ldq_rw(f.r[rid[c]] + l * g.nvol + iv);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float lM = qM.v[j], lmu = qmu.v[j];
                float gm = lM, fm = 2.0f * lmu, d = 0, e = 0;
                if (L > 0) {
                    const float ltaup = qtaup.v[j], ltaus = qtaus.v[j];
                    gm = lM * (1.0f + (float)L * ltaup);
                    fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
                    d = 2.0f * lmu * ltaus / g.dt; e = lM * ltaup / g.dt;
                }
                const float vxxyyzz = vxx.v[j] + vyy.v[j] + vzz.v[j], vyyzz = vyy.v[j] + vzz.v[j];
                const float vxxzz = vxx.v[j] + vzz.v[j], vxxyy = vxx.v[j] + vyy.v[j];
                const float fw[3] = {gm * vxxyyzz - fm * vyyzz, gm * vxxyyzz - fm * vxxzz, gm * vxxyyzz - fm * vxxyy};
                if (L == 0) {
#pragma unroll
                    for (int c = 0; c < 3; c++) s3[c].v[j] -= fw[c];
                } else {
                    const float dc[3] = {e * vxxyyzz - d * vyyzz, e * vxxyyzz - d * vxxzz, e * vxxyyzz - d * vxxyy};
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        float aa = 0;
#pragma unroll
                        for (int l = 0; l < L; l++) aa += rf[c][l].v[j];
                        const float ls = fw[c] + g.dt2 * aa;
                        aa = 0;
                        // 3D reconstruction keeps the forward-time coefficients (update_adjs3D.cl:357-359)
#pragma unroll
                        for (int l = 0; l < L; l++) {
                            const float el = g.eta[l];
                            const float b = g.eta_b[l], cc = g.eta_c[l];
                            aa += b * (rf[c][l].v[j] * cc - el * dc[c]);
                        }
                        s3[c].v[j] -= ls + g.dt2 * aa;
                    }
                }
                const int m = mq[j];
                if (m != -1) {
                    s3[0].v[j] = bnd_at<T>(g, a, SXX, m);
                    s3[1].v[j] = bnd_at<T>(g, a, SYY, m);
                    s3[2].v[j] = bnd_at<T>(g, a, SZZ, m);
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++) stq(f.w[wid[c]] + iv, s3[c]);
        }
        Q4 rr[3][L > 0 ? L : 1];
        if constexpr (L > 0) {
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int l = 0; l < L; l++) rr[c][l] = adj_memory(g, a.rr[rid[c]] + l * g.nvol + iv);
        }
        Q4 w3[3];
#pragma unroll
        for (int c = 0; c < 3; c++) w3[c] = ldq_rw(a.wr[wid[c]] + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float lM = qM.v[j], lmu = qmu.v[j];
            float gm = lM, fm = 2.0f * lmu, d = 0, e = 0;
            if (L > 0) {
                const float ltaup = qtaup.v[j], ltaus = qtaus.v[j];
                gm = lM * (1.0f + (float)L * ltaup);
                fm = 2.0f * lmu * (1.0f + (float)L * ltaus);
                d = 2.0f * lmu * ltaus / g.dt; e = lM * ltaup / g.dt;
            }
            const float vxxyyzzr = vxxr.v[j] + vyyr.v[j] + vzzr.v[j], vyyzzr = vyyr.v[j] + vzzr.v[j];
            const float vxxzzr = vxxr.v[j] + vzzr.v[j], vxxyyr = vxxr.v[j] + vyyr.v[j];
            float ls[3] = {gm * vxxyyzzr - fm * vyyzzr, gm * vxxyyzzr - fm * vxxzzr, gm * vxxyyzzr - fm * vxxyyr};
            if (L == 0) {
#pragma unroll
                for (int c = 0; c < 3; c++) w3[c].v[j] += ls[c];
            } else {
                const float dc[3] = {e * vxxyyzzr - d * vyyzzr, e * vxxyyzzr - d * vxxzzr, e * vxxyyzzr - d * vxxyyr};
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    float aa = 0;
#pragma unroll
                    for (int l = 0; l < L; l++) aa += rr[c][l].v[j];
                    ls[c] += g.dt2 * aa;
                    // stored into the forward memory variables; the sum keeps the
                    // last adjoint value (update_adjs3D.cl:566-583); in the DFT
                    // adjoint both are one buffer, so that value is the new one
#pragma unroll
                    for (int l = 0; l < L; l++) {
                        const float el = g.eta[l];
                        const float b = g.eta_b[l], cc = g.eta_c[l];
                        const float n = b * (rr[c][l].v[j] * cc - el * dc[c]);
                        aa = g.bp2 ? n : rr[c][l].v[j];
                        rr[c][l].v[j] = n;
                    }
                    w3[c].v[j] += ls[c] + g.dt2 * aa;
                }
            }
            if (!g.bp2 && g.restype == 0) {
                const float c1 = 1.0f / (3.0f * lM - 4.0f * lmu) / (3.0f * lM - 4.0f * lmu);
                const float c3 = 1.0f / lmu / lmu;   // kept for the shear stresses
                qc3.v[j] = c3;
                const float c5 = 1.0f / 6.0f * c3;
                const float sxx = s3[0].v[j], syy = s3[1].v[j], szz = s3[2].v[j];
                const float dM = c1 * (sxx + syy + szz) * (ls[0] + ls[1] + ls[2]);
                gM[j] = -dM;
                gmu[j] = 4.0f / 3.0f * dM - c5 * (ls[0] * (2.0f * sxx - syy - szz) + ls[1] * (2.0f * syy - sxx - szz) +
                                                  ls[2] * (2.0f * szz - sxx - syy));
            } else if (!g.bp2) {
                gM[j] = -((s3[0].v[j] + s3[1].v[j] + s3[2].v[j]) * (ls[0] + ls[1] + ls[2]));
            }
        }
        // the new adjoint memory values go to the forward arrays; a
        // checkpointed adjoint reloads those from a snapshot before they are
        // read again, so it skips the stores (its forward arrays may also be
        // FP16)
        if constexpr (L > 0) {
            if (!g.ckpt) {
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int l = 0; l < L; l++) stq(f.r[rid[c]] + l * g.nvol + iv, rr[c][l]);
            }
        }
        if (g.abs_type == 2) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float t3[3] = {w3[0].v[j], w3[1].v[j], w3[2].v[j]};
                taper_regs<3>(g, f.taper, gz0 + j, gy, gx, t3);
#pragma unroll
                for (int c = 0; c < 3; c++) w3[c].v[j] = t3[c];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) stq(a.wr[wid[c]] + iv, w3[c]);
    }

    // ---- shear stresses, one at a time: sxy (x,y), syz (y,z), sxz (x,z)
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const int wid = c == 0 ? SXY : (c == 1 ? SYZ : SXZ);
        const int rid = c == 0 ? RXY : (c == 1 ? RYZ : RXZ);
        const int pmu = c == 0 ? PMUIPJP : (c == 1 ? PMUJPKP : PMUIPKP);
        const int ptau = c == 0 ? PTAUSIPJP : (c == 1 ? PTAUSJPKP : PTAUSIPKP);
        const Q4 qmuc = ldq(f.p[pmu] + ip);
        Q4 qtauc = {{0, 0, 0, 0}};
        if (L > 0) qtauc = ldq(f.p[ptau] + ip);
        Q4 sc = {{0, 0, 0, 0}};
        if (g.ckpt) {
            sc = fwd_quad<T>(g, a, wid, iv);
        } else if (!g.bp2) {
            Q4 d1, d2;   // forward derivative pair (vxy+vyx, vyz+vzy, vxz+vzx)
            if (c == 0) { d1 = dfw_q<F>(f.w[VX], iv, sy, hc); d2 = dfw_q<F>(f.w[VY], iv, sx, hc); }
            else if (c == 1) { d1 = dfw_z<F>(ldw(f.w[VY], iv), hc); d2 = dfw_q<F>(f.w[VZ], iv, sy, hc); }
            else { d1 = dfw_z<F>(ldw(f.w[VX], iv), hc); d2 = dfw_q<F>(f.w[VZ], iv, sx, hc); }
            sc = ldq_rw(f.w[wid] + iv);
            Q4 rf[L > 0 ? L : 1];
            if constexpr (L > 0) {
#pragma unroll
                for (int l = 0; l < L; l++) rf[l] = ldq_rw(f.r[rid] + l * g.nvol + iv);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float fsum = d1.v[j] + d2.v[j];
                const float lmuc = qmuc.v[j];
                if (L == 0) {
                    sc.v[j] -= lmuc * fsum;
                } else {
                    const float lt = qtauc.v[j];
                    const float fc = lmuc * (1.0f + (float)L * lt), dc = lmuc * lt / g.dt;
                    float aa = 0;
#pragma unroll
                    for (int l = 0; l < L; l++) aa += rf[l].v[j];
                    const float ls = fc * fsum + g.dt2 * aa;
                    aa = 0;
#pragma unroll
                    for (int l = 0; l < L; l++) {
                        const float el = g.eta[l];
                        const float b = g.eta_b[l], cc = g.eta_c[l];
                        aa += b * (rf[l].v[j] * cc - el * (dc * fsum));
                    }
                    sc.v[j] -= ls + g.dt2 * aa;
                }
                const int m = mq[j];
                if (m != -1) sc.v[j] = bnd_at<T>(g, a, wid, m);
            }
            stq(f.w[wid] + iv, sc);
        }
        const Q4 rsum = rsh[c];
        Q4 rr[L > 0 ? L : 1];
        if constexpr (L > 0) {
#pragma unroll
            for (int l = 0; l < L; l++) rr[l] = adj_memory(g, a.rr[rid] + l * g.nvol + iv);
        }
        Q4 wc = ldq_rw(a.wr[wid] + iv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float lmuc = qmuc.v[j];
            float fc = lmuc, dc = 0;
            if (L > 0) {
                const float lt = qtauc.v[j];
                fc = lmuc * (1.0f + (float)L * lt);
                dc = lmuc * lt / g.dt;
            }
            float ls = fc * rsum.v[j];
            if (L == 0) {
                wc.v[j] += ls;
            } else {
                float aa = 0;
#pragma unroll
                for (int l = 0; l < L; l++) aa += rr[l].v[j];
                ls += g.dt2 * aa;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    const float el = g.eta[l];
                    const float b = g.eta_b[l], cc = g.eta_c[l];
                    const float n = b * (rr[l].v[j] * cc - el * (dc * rsum.v[j]));
                    aa = g.bp2 ? n : rr[l].v[j];
                    rr[l].v[j] = n;
                }
                wc.v[j] += ls + g.dt2 * aa;
            }
            if (!g.bp2 && g.restype == 0) {
                gmu[j] += -qc3.v[j] * (sc.v[j] * ls);
            }
        }
        if constexpr (L > 0) {
            if (!g.ckpt) {   // as for the normal stresses
#pragma unroll
                for (int l = 0; l < L; l++) stq(f.r[rid] + l * g.nvol + iv, rr[l]);
            }
        }
        if (g.abs_type == 2) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float t1[1] = {wc.v[j]};
                taper_regs<1>(g, f.taper, gz0 + j, gy, gx, t1);
                wc.v[j] = t1[0];
            }
        }
        stq(a.wr[wid] + iv, wc);
    }
    if (!g.bp2) {
        grad_add4(a.grad[GM], ip, gM);
        if (g.restype == 0) grad_add4(a.grad[GMU], ip, gmu);
    }
}

// ------------------------------------------------------------- launchers
template <int R, int L, typename T>
static void quad_adjs_l(const Grid &g, const Fields &f, const AdjFields &a, dim3 gr, dim3 b, cudaStream_t st)
{
    // kernels 5 keeps the kernels without the prefetch
    if (g.kernels == 0 && g.nb == 1) k_adjs3d_q4<R, L, T, false, true><<<gr, b, 0, st>>>(g, f, a);
    else MB_DISPATCH(g, k_adjs3d_q4<R, L, T, MBV><<<gr, b, 0, st>>>(g, f, a))
}

template <int R, typename T>
static void quad_adj_t(const Grid &g, const Fields &f, const AdjFields &a, bool stress, cudaStream_t st)
{
    if (stress) {
        const dim3 b = q4_block(g, 16, 8, 1), gr = q4_grid(g, b);
        switch (g.L) {
        case 0: quad_adjs_l<R, 0, T>(g, f, a, gr, b, st); break;
        case 1: quad_adjs_l<R, 1, T>(g, f, a, gr, b, st); break;
        case 2: quad_adjs_l<R, 2, T>(g, f, a, gr, b, st); break;
        default: quad_adjs_l<R, 3, T>(g, f, a, gr, b, st); break;
        }
        return;
    }
    const dim3 b = q4_block(g, 8, 4, 4), gr = q4_grid(g, b);
    if (g.kernels == 0 && g.nb == 1) k_adjv3d_q4<R, T, false, true><<<gr, b, 0, st>>>(g, f, a);
    else MB_DISPATCH(g, k_adjv3d_q4<R, T, MBV><<<gr, b, 0, st>>>(g, f, a))
}

template <int R>
void quad_update_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st)
{
    if (prec == SFD_PREC_FP16) quad_adj_t<R, __half>(g, f, a, stress, st);
    else if (prec == SFD_PREC_BF16) quad_adj_t<R, __nv_bfloat16>(g, f, a, stress, st);
    else quad_adj_t<R, float>(g, f, a, stress, st);
}

}  // namespace sfd
