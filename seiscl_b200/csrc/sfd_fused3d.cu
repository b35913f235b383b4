// sfd_fused3d.cu -- opt-in 3D modelling kernels built from the 4-cell cell
// updates: the cp.async-staged velocity update (kernels 7) and the fused
// one-launch step (kernels 6).
#include <algorithm>

#include "sfd_quad3d.cuh"

namespace sfd {

// ------------------------------------- velocity update staged by cp.async
// k_v3d_q4's arithmetic with its stress operands staged in shared memory by
// asynchronous copies (cp.async, 16 bytes each), so the bytes in flight do
// not hold registers.  A CTA owns a tile of AZ z cells x AY y rows and
// marches over AX x planes; one thread updates one quad (4 z cells) per
// plane.  Shared memory holds
//   ring   sxx, sxy, sxz (the x derivatives) over the tile's own columns, for
//          planes x-4 .. x+5 (10 slots; plane x+5 arrives while x is computed);
//   halo   syy, szz, syz, sxy, sxz over the tile plus a 4-cell y/z halo for
//          plane x (y and z derivatives), double-buffered.
// The copies of plane x+2 are issued after plane x is computed and committed
// as one group; cp.async.wait_group 1 then leaves only the newest group in
// flight.  The waits are on the thread's own copies: they always end.
constexpr int AZ = 32, AY = 16, AX = 16;
constexpr int AHZ = AZ + 8, AHY = AY + 8;
constexpr int ARING = 10;
struct VAsyncSmem {
    float ring[3][ARING][AY][AZ];
    float halo[2][5][AHY][AHZ];
};
constexpr size_t VASYNC_SMEM = sizeof(VAsyncSmem);

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ Q4 lds4(const float *p)
{
    const float4 t = *reinterpret_cast<const float4 *>(p);
    return Q4{{t.x, t.y, t.z, t.w}};
}
// forward / backward differences of a quad over shared-memory rows `st`
// floats apart (the operation order of dfw_q / dbw_q)
__device__ __forceinline__ Q4 dfw_s(const float *p, int st, const float *hc)
{
    Q4 a = lds4(p + st), b = lds4(p), r;
#pragma unroll
    for (int j = 0; j < 4; j++) r.v[j] = hc[0] * (a.v[j] - b.v[j]);
#pragma unroll
    for (int m = 2; m <= 4; m++) {
        a = lds4(p + m * st);
        b = lds4(p - (m - 1) * st);
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
    }
    return r;
}
__device__ __forceinline__ Q4 dbw_s(const float *p, int st, const float *hc)
{
    Q4 a = lds4(p), b = lds4(p - st), r;
#pragma unroll
    for (int j = 0; j < 4; j++) r.v[j] = hc[0] * (a.v[j] - b.v[j]);
#pragma unroll
    for (int m = 2; m <= 4; m++) {
        a = lds4(p + (m - 1) * st);
        b = lds4(p - m * st);
#pragma unroll
        for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
    }
    return r;
}
// the 12 values z0-4 .. z0+7 of a quad from a halo row (p at z0 - 4)
__device__ __forceinline__ W12 ldw_s(const float *p)
{
    W12 r;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const Q4 t = lds4(p + 4 * k);
        r.w[4 * k] = t.v[0]; r.w[4 * k + 1] = t.v[1]; r.w[4 * k + 2] = t.v[2]; r.w[4 * k + 3] = t.v[3];
    }
    return r;
}

// issue the copies of plane x: ring slot of plane x+5 (when inside the grid)
// and the haloed tiles of plane x into halo buffer hb
__device__ __forceinline__ void vasync_issue(const Grid &g, const Fields &f, VAsyncSmem &sm, int z0, int y0,
                                             int xr, int xh, int hb, int tid)
{
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    if (xr >= 0 && xr < g.NX) {
        const float *rf[3] = {f.w[SXX], f.w[SXY], f.w[SXZ]};
        const int slot = xr % ARING;
        for (int i = tid; i < 3 * AY * (AZ / 4); i += 128) {
            const int q = i / (AY * (AZ / 4)), r = (i / (AZ / 4)) % AY, c = i % (AZ / 4);
            const int gy = y0 + r, gz = z0 + 4 * c;
            if (gy < g.NY && gz + 3 < g.NZ)
                cp_async16(&sm.ring[q][slot][r][4 * c], rf[q] + xr * sx + (i64)gy * sy + gz);
        }
    }
    if (xh >= 0) {
        const float *hf[5] = {f.w[SYY], f.w[SZZ], f.w[SYZ], f.w[SXY], f.w[SXZ]};
        for (int i = tid; i < 5 * AHY * (AHZ / 4); i += 128) {
            const int q = i / (AHY * (AHZ / 4)), r = (i / (AHZ / 4)) % AHY, c = i % (AHZ / 4);
            const int gy = y0 - 4 + r, gz = z0 - 4 + 4 * c;
            if (gy >= 0 && gy < g.NY && gz >= 0 && gz + 3 < g.NZ)
                cp_async16(&sm.halo[hb][q][r][4 * c], hf[q] + xh * sx + (i64)gy * sy + gz);
        }
    }
}

__global__ void __launch_bounds__(128, 2) k_v3d_async(Grid g, Fields f)
{
    constexpr int F = 4;
    extern __shared__ __align__(16) unsigned char vasync_raw[];
    VAsyncSmem &sm = *reinterpret_cast<VAsyncSmem *>(vasync_raw);
    const int tid = threadIdx.x + 8 * threadIdx.y;
    const int z0 = F + blockIdx.x * AZ, y0 = F + blockIdx.y * AY;
    const int xb = F + blockIdx.z * AX, xe = min(xb + AX, g.NX - F);
    const int qz = threadIdx.x, yy = threadIdx.y;
    const int gz0 = z0 + 4 * qz, gy = y0 + yy;
    const bool ok = gz0 <= g.NZ - F - 1 && gy <= g.NY - F - 1;
    const float *hc = g.hc;
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    // prologue: ring planes xb-4 .. xb+4 and the halo of plane xb (group 0),
    // ring plane xb+5 and the halo of plane xb+1 (group 1)
    for (int xr = xb - 4; xr < xb + 4; xr++) vasync_issue(g, f, sm, z0, y0, xr, -1, 0, tid);
    vasync_issue(g, f, sm, z0, y0, xb + 4, xb, 0, tid);
    cp_async_commit();
    vasync_issue(g, f, sm, z0, y0, xb + 5, xb + 1 < xe ? xb + 1 : -1, 1, tid);
    cp_async_commit();
    for (int gx = xb; gx < xe; gx++) {
        const int hb = (gx - xb) & 1;
        Q4 vx, vy, vz, rip, rjp, rkp;
        const i64 iv = gx * sx + (i64)gy * sy + gz0;
        const i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz0 - F);
        if (ok) {
            vx = ldq_rw(f.w[VX] + iv); vy = ldq_rw(f.w[VY] + iv); vz = ldq_rw(f.w[VZ] + iv);
            rip = ldq(f.p[PRIP] + ip); rjp = ldq(f.p[PRJP] + ip); rkp = ldq(f.p[PRKP] + ip);
        }
        cp_async_wait<1>();
        __syncthreads();
        if (ok) {
            const float *H0 = &sm.halo[hb][0][0][0];
            const int HP = AHY * AHZ;                 // floats per haloed tile
            const int hrow = (yy + 4) * AHZ + 4 * qz;  // the quad's row, at z0 - 4 of its window
            const W12 wzz = ldw_s(H0 + 1 * HP + hrow), wxz = ldw_s(H0 + 4 * HP + hrow),
                      wyz = ldw_s(H0 + 2 * HP + hrow);
            const int RP = AY * AZ;                    // floats per ring slot
            const int rc = yy * AZ + 4 * qz;
            auto ring_at = [&](int q, int x) { return &sm.ring[q][x % ARING][0][0] + rc; };
            Q4 szz_z = dfw_z<F>(wzz, hc);
            Q4 sxx_x, sxz_x, sxy_x;
            {
                // x differences across ring slots (plane offsets wrap modulo ARING)
                const float *c0 = ring_at(0, gx);
                (void)RP;
                Q4 a = lds4(ring_at(0, gx + 1)), b = lds4(c0), r;
#pragma unroll
                for (int j = 0; j < 4; j++) r.v[j] = hc[0] * (a.v[j] - b.v[j]);
#pragma unroll
                for (int m = 2; m <= F; m++) {
                    a = lds4(ring_at(0, gx + m));
                    b = lds4(ring_at(0, gx - (m - 1)));
#pragma unroll
                    for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
                }
                sxx_x = r;
                for (int q = 1; q <= 2; q++) {
                    a = lds4(ring_at(q, gx));
                    b = lds4(ring_at(q, gx - 1));
#pragma unroll
                    for (int j = 0; j < 4; j++) r.v[j] = hc[0] * (a.v[j] - b.v[j]);
#pragma unroll
                    for (int m = 2; m <= F; m++) {
                        a = lds4(ring_at(q, gx + m - 1));
                        b = lds4(ring_at(q, gx - m));
#pragma unroll
                        for (int j = 0; j < 4; j++) r.v[j] = fmaf(hc[m - 1], a.v[j] - b.v[j], r.v[j]);
                    }
                    if (q == 1) sxy_x = r;
                    else sxz_x = r;
                }
            }
            Q4 sxz_z = dbw_z<F>(wxz, hc);
            Q4 syz_y = dbw_s(H0 + 2 * HP + hrow + 4, AHZ, hc);
            Q4 syz_z = dbw_z<F>(wyz, hc);
            Q4 syy_y = dfw_s(H0 + 0 * HP + hrow + 4, AHZ, hc);
            Q4 sxy_y = dbw_s(H0 + 3 * HP + hrow + 4, AHZ, hc);
            if (g.abs_type == 1)
                cpml_v3d_q4<false>(g, f, gz0, gy, gx, sxx_x, syy_y, szz_z, sxy_y, sxy_x, syz_y, syz_z, sxz_x, sxz_z);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float v3[3] = {vx.v[j] + (sxx_x.v[j] + sxy_y.v[j] + sxz_z.v[j]) * rip.v[j],
                               vy.v[j] + (syy_y.v[j] + sxy_x.v[j] + syz_z.v[j]) * rjp.v[j],
                               vz.v[j] + (szz_z.v[j] + sxz_x.v[j] + syz_y.v[j]) * rkp.v[j]};
                if (g.abs_type == 2) taper_regs<3>(g, f.taper, gz0 + j, gy, gx, v3);
                vx.v[j] = v3[0]; vy.v[j] = v3[1]; vz.v[j] = v3[2];
            }
            stq(f.w[VX] + iv, vx);
            stq(f.w[VY] + iv, vy);
            stq(f.w[VZ] + iv, vz);
        }
        __syncthreads();   // plane gx-4's ring slot and halo buffer hb are free
        vasync_issue(g, f, sm, z0, y0, gx + 6, gx + 2 < xe ? gx + 2 : -1, hb, tid);
        cp_async_commit();
    }
    cp_async_wait<0>();
}

bool launch_update_v_async(const Grid &g, const Fields &f, cudaStream_t st)
{
    if (g.nd != 3 || g.F != 4 || g.nz % 4 || g.fhalf || g.nb != 1) return false;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_v3d_async, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VASYNC_SMEM) !=
            cudaSuccess)
            return false;
        attr = true;
    }
    const dim3 b(8, AY), gr((g.nz + AZ - 1) / AZ, (g.ny + AY - 1) / AY, (g.nx + AX - 1) / AX);
    k_v3d_async<<<gr, b, VASYNC_SMEM, st>>>(g, f);
    return true;
}

// ------------------------------------------------- fused 3D forward step
// One launch advances the whole grid one time step: velocity update, stress
// and memory-variable update and (with a free surface) the free surface, so
// the stresses the velocity stencils read are read again by the stress
// updates of nearby work units, and the velocities written are read back,
// while both are still in L2.  Per cell the arithmetic is that of k_v3d_q4,
// k_s3d_q4 and k_surf3d, in that order.
//
// Work unit: a tile of FZ z cells x FY y rows in one x plane.  A CTA takes a
// ticket (atomicAdd) and works on unit number ticket - base; units are
// numbered plane by plane (x slowest).  Unit (c, t) first updates the
// velocities of plane F + c + 4 of tile t (unit 0 also planes F .. F + 3) and
// publishes its flag, then waits for the flags of the units whose velocities
// its stress stencils read -- planes F + c - 4 .. F + c + 4 of its own tile
// (units c - 8 .. c - 1) and plane F + c of the four y/z neighbour tiles
// (units c - 4) -- and updates the stresses of plane F + c.  Every wait is
// on a unit with a lower number, taken by a CTA that started earlier, so the
// waits always end however few CTAs are resident.  Everything is updated
// in place; the same waits order every stress overwrite after all velocity
// reads of the old value: the stresses of plane F + c in tile t are read by
// the velocity updates of planes F + c - 4 .. F + c + 4 in tile t (units
// c - 8 .. c) and of plane F + c in its neighbours (units c - 4), exactly
// the units (c, t) waits for.  Velocity reads of the stress phase go
// through L2 (__ldcg): other CTAs wrote them during the launch.  Waits are
// bounded (FUSED_WAIT_NS of %globaltimer); one that runs out sets
// g_fused_status, which makes every later CTA and launch skip its work and
// the host report an error.
constexpr int FZ = 32, FY = 16;
constexpr unsigned long long FUSED_WAIT_NS = 2000000000ull;
__device__ int g_fused_status;   // 0 ok, 1 a wait ran out

__device__ __forceinline__ int ld_acquire_gpu(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int *p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// wait until *flag >= want; false when the bound ran out or another CTA's did
__device__ bool fused_wait(const int *flag, int want)
{
    if (ld_acquire_gpu(flag) >= want) return true;
    const unsigned long long t0 = global_ns();
    unsigned ns = 32;
    for (;;) {
        __nanosleep(ns);
        if (ns < 512) ns *= 2;
        if (ld_acquire_gpu(flag) >= want) return true;
        if (*(volatile int *)&g_fused_status) return false;
        if (global_ns() - t0 > FUSED_WAIT_NS) return false;
    }
}

template <int L>
__global__ void __launch_bounds__(128, 4) k_fused3d_q4(Grid g, Fields f, FusedSync fs, int epoch)
{
    constexpr int F = 4;
    __shared__ int s_unit, s_go;
    const int tid = threadIdx.x + 8 * threadIdx.y;
    if (tid == 0) {
        s_unit = (int)(atomicAdd(fs.ticket, 1u) - fs.base);
        s_go = *(volatile int *)&g_fused_status == 0;
    }
    __syncthreads();
    if (!s_go) return;
    const int ntile = fs.ntz * fs.nty, unit = s_unit;
    if (unit < 0 || unit >= fs.units) {   // the counter was not reset: never index past the flags
        if (tid == 0) atomicExch(&g_fused_status, 1);
        return;
    }
    const int c = unit / ntile, tile = unit - c * ntile, ty = tile / fs.ntz, tz = tile - ty * fs.ntz;
    const int gz0 = F + tz * FZ + 4 * threadIdx.x, gy = F + ty * FY + threadIdx.y;
    const bool ok_cell = gz0 <= g.NZ - F - 1 && gy <= g.NY - F - 1;
    const int nxp = g.NX - 2 * F;   // x planes
    const i64 sx = (i64)g.NY * g.NZ, sy = g.NZ;
    // phase 1: velocities of plane F + c + 4 (unit 0: planes F .. F + 4).
    // The stress reads take the read-only path: no stress cell read here is
    // overwritten before this unit's flag is up, and nothing in this launch
    // reads a stress value written in it.
    if (ok_cell) {
        const int x0 = c == 0 ? F : F + c + 4, x1 = min(F + c + 5, g.NX - F);
        for (int gx = x0; gx < x1; gx++) {
            const i64 iv = gx * sx + (i64)gy * sy + gz0;
            const i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz0 - F);
            v3d_q4_at<4, float, 0>(g, f, gz0, gy, gx, iv, ip);
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        st_release_gpu(fs.flags + unit, epoch);
    }
    // the units this one reads velocities of: threads 0..7 the own tile's
    // planes (units c - 8 .. c - 1; unit 0 holds planes F .. F + 4), threads
    // 8..11 the neighbours' plane F + c (unit c - 4)
    bool ok = true;
    if (tid < 12) {
        int wu = -1;
        if (tid < 8) {
            const int uc = c - 8 + tid;
            if (uc >= 0 && uc <= nxp - 5) wu = uc * ntile + tile;
        } else {
            const int nt = tid == 8 ? (tz > 0 ? tile - 1 : -1)
                         : tid == 9 ? (tz < fs.ntz - 1 ? tile + 1 : -1)
                         : tid == 10 ? (ty > 0 ? tile - fs.ntz : -1)
                                     : (ty < fs.nty - 1 ? tile + fs.ntz : -1);
            if (nt >= 0) wu = max(c - 4, 0) * ntile + nt;
        }
        if (wu >= 0) ok = fused_wait(fs.flags + wu, epoch);
        __threadfence();
    }
    if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicExch(&g_fused_status, 1);
        return;
    }
    if (!ok_cell) return;
    // phase 2: stresses, memory variables, free surface of plane F + c
    // (velocity reads through L2)
    const int gx = F + c;
    const i64 iv = gx * sx + (i64)gy * sy + gz0;
    const i64 ip = ((i64)(gx - F) * g.ny + (gy - F)) * g.nz + (gz0 - F);
    s3d_q4_at<4, L, float, 2>(g, f, gz0, gy, gx, iv, ip, g.freesurf ? SURF_FOLD : SURF_NONE);
}

FusedShape fused_shape(const Grid &g)
{
    FusedShape s{0, 0, 0, 0};
    if (!g.fused || g.nd != 3 || g.F != 4 || g.nz % 4 || g.fhalf || g.L < 0 || g.L > 3 || g.kernels != 0) return s;
    const int ntz = (g.nz + FZ - 1) / FZ, nty = (g.ny + FY - 1) / FY, nch = g.nx;
    if (g.nx < 5 || (int64_t)ntz * nty * nch > (1 << 30)) return s;
    s.ntz = ntz;
    s.nty = nty;
    s.nchunk = nch;
    s.units = (int64_t)ntz * nty * nch;
    return s;
}

bool launch_fused_step(const Grid &g, const Fields &f, int *sync, int t, cudaStream_t st)
{
    const FusedShape sh = fused_shape(g);
    if (!sh.units || g.nb != 1 || !sync) return false;
    FusedSync fs{reinterpret_cast<unsigned *>(sync), sync + 1, (unsigned)((uint64_t)t * (uint64_t)sh.units),
                 sh.ntz, sh.nty, (int)sh.units};
    const dim3 b(8, FY, 1);
    const unsigned gr = (unsigned)sh.units;
    switch (g.L) {
    case 0: k_fused3d_q4<0><<<gr, b, 0, st>>>(g, f, fs, t + 1); break;
    case 1: k_fused3d_q4<1><<<gr, b, 0, st>>>(g, f, fs, t + 1); break;
    case 2: k_fused3d_q4<2><<<gr, b, 0, st>>>(g, f, fs, t + 1); break;
    default: k_fused3d_q4<3><<<gr, b, 0, st>>>(g, f, fs, t + 1); break;
    }
    return true;
}

int fused_take_status()
{
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_fused_status, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_fused_status, &zero, sizeof(int));
    return v;
}

}  // namespace sfd
