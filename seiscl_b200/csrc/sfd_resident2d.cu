// sfd_resident2d.cu -- 2D P-SV modelling with the whole state resident on
// chip: one cooperative launch advances a segment of the time loop.
//
// A time step of a 2D grid is a few microseconds of work, so the two
// launches per step of the ordinary loop (velocity; stress with the surface,
// receivers and sources) spend most of it on launch gaps, cold pipelines and
// the last-block handshake.  Here every CTA owns a tile of one shot's grid
// and every thread NC cells of it (consecutive columns of one z row) for all
// steps of the launch: the five wave fields live in shared memory, the
// cells' parameters, memory variables and CPML memory in registers.  After
// each half step a thread sends its cells within F rows or columns of a
// neighbouring tile, and the tile receives its halo.
//
// Exchange.  Every value travels as one 64-bit word, value below and step
// number above, stored and polled with single relaxed 64-bit accesses in L2:
// the word itself says when it has arrived, so no fence, flag or barrier
// across CTAs is needed.  One buffer suffices: a tile writes the words of
// step t+1 only after it has received its neighbour's later half step of t,
// which the neighbour sent after it had read the words of step t.  All CTAs
// of the launch are resident at once (cooperative launch), so every wait
// ends; each is bounded all the same, and one that runs out sets *status and
// ends the CTA, after which its neighbours' waits run out too.
//
// What bounds it: the two exchanges of a step (L2 round trips, 500-1500
// cycles each) and the latency of the cells' arithmetic (700-2800 cycles a
// half step).  us per step on a B200, two launches per step / resident (order
// 8 unless noted): 100 x 150 order 4 12.3 / 2.7; 200 x 200 14.3 / 3.3; 300 x
// 400 15.7 / 4.7; the same with L = 3 19.7 / 5.2; 400 x 577 order 4 17.7 / 8.4;
// 8 shots of 100 x 150 order 4 17.6 / 8.0.  A form that kept parameters, CPML
// and memory variables in global memory took 7.8 at 300 x 400.
//
// Arithmetic: the functions of sfd_device.cuh that k_v2d, k_s2d and k_surf2d
// use, in the same order: the same bits as the ordinary kernels.
#include <algorithm>
#include <cstring>
#include <mutex>

#include <cuda_runtime.h>

#include "sfd_device.cuh"
#include "sfd_internal.h"
#include "sfd_kernels.h"

namespace sfd {

namespace {

constexpr int R2_THREADS = 512;
constexpr int R2_CTAS = RES2D_SMS;        // one CTA per SM
constexpr int R2_SMEM = 200 * 1024;       // dynamic shared memory a CTA may take
constexpr int r2_words(int nc) { return nc == 4 ? 4 : 2; }   // most exchange words a thread receives in a half step
constexpr int R2_POINTS = 4096;           // receivers and sources of a run

enum { W_VX, W_VZ, W_XX, W_ZZ, W_XZ, R2_NF };    // fields of a tile in shared memory

typedef unsigned long long u64;

__device__ __forceinline__ u64 ld_word(const u64 *p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(u64 *p, unsigned epoch, float v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((u64)epoch << 32) | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ long long now_ns()
{
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// tile field of a wave field (also the low bits of a source's target mask)
__device__ __forceinline__ int tile_field(int w)
{
    return w == VX ? W_VX : w == VZ ? W_VZ : w == SXX ? W_XX : w == SZZ ? W_ZZ : W_XZ;
}

// CPML of one axis at one cell: 1/K, a, b at full and half nodes, and the
// slab-local index (-1 outside the slabs)
struct Slab {
    double kf, kh;
    float af, bf, ah, bh;
    int at;
};
constexpr int R2_ROWS = 64, R2_COLS = 64;   // most rows and columns (16 warps x 4) of a tile
constexpr int row_pitch(int F) { return R2_ROWS + 2 * F; }
constexpr int field_floats(int F, int nc) { return row_pitch(F) * (R2_THREADS / 32 * nc + nc + 2 * F); }
static_assert(sizeof(float) * R2_NF * field_floats(4, 4) + R2_POINTS * (sizeof(int4) + sizeof(float)) <= R2_SMEM,
              "the largest tile and point list fit whatever the run");
static_assert(sizeof(float) * 2 * R2_NF * field_floats(4, 2) + R2_POINTS * (sizeof(int4) + sizeof(float)) <= R2_SMEM,
              "and so do the adjoint's");
__device__ __forceinline__ Slab slab_of(const Grid &g, const Fields &fl, int axis, int i, int n, bool lo)
{
    Slab s = {1.0, 1.0, 0.0f, 0.0f, 0.0f, 0.0f, -1};
    if (g.abs_type != 1) return s;
    int f, h;   // profile indices of the full and half nodes
    if (i >= n) return s;   // a dummy row
    if (i >= n - g.nab) { s.at = i - n + 2 * g.nab; f = 2 * g.nab - s.at; h = f - 1; }
    else if (lo && i < g.nab) { s.at = f = h = i; }
    else return s;
    const float *const *c = axis == 0 ? fl.cx : fl.cz;
    s.kf = fl.kq[axis][0][f]; s.af = c[CA][f]; s.bf = c[CB][f];
    s.kh = fl.kq[axis][1][h]; s.ah = c[CAH][h]; s.bh = c[CBH][h];
    return s;
}
__device__ __forceinline__ void cpml_reg(float &psi, double k, float a, float b, float &d)
{
    psi = cpml_psi(psi, a, b, d);
    d = cpml_quot(d, k, psi);
}

template <typename T>
__device__ __forceinline__ void bnd_put(void *p, i64 at, float v)
{
    ((T *)p)[at] = from_f<T>(v);
}
__device__ __forceinline__ void bnd_store(const Grid &g, const BndSlot &b, int prec, int w, i64 at, float v)
{
    v *= g.bsc[w];
    if (prec == SFD_PREC_FP16) bnd_put<__half>(b.p[w], at, v);
    else if (prec == SFD_PREC_BF16) bnd_put<__nv_bfloat16>(b.p[w], at, v);
    else bnd_put<float>(b.p[w], at, v);
}

// difference over a window held in registers, the operation order of dfw /
// dbw: w[0] is the farthest cell behind
template <int F>
__device__ __forceinline__ float diff_win(const float *w, const float *hc)
{
    float acc = __fmul_rn(hc[0], w[F] - w[F - 1]);
#pragma unroll
    for (int m = 2; m <= F; m++) acc = fmaf(hc[m - 1], w[F + m - 1] - w[F - m], acc);
    return acc;
}

}  // namespace

// One segment of the time loop: steps a.t0 .. a.t1-1 of the launch's shots.
template <int F, int L, int NC>
__global__ void __launch_bounds__(R2_THREADS, 1) k_resident2d(const __grid_constant__ Grid g,
                                                              const __grid_constant__ Fields f0,
                                                              const __grid_constant__ Res2d r,
                                                              const __grid_constant__ Res2dRun a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LL = L > 0 ? L : 1, R2_WORDS = r2_words(NC);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntile = r.ntz * r.ntx;
    const int shot = a.shot0 + blockIdx.x / ntile, tl = blockIdx.x % ntile;
    const int iz = tl % r.ntz, ix = tl / r.ntz;
    const int z0 = (int)((i64)iz * g.nz / r.ntz), tz = (int)((i64)(iz + 1) * g.nz / r.ntz) - z0;
    const int x0 = (int)((i64)ix * g.nx / r.ntx), tx = (int)((i64)(ix + 1) * g.nx / r.ntx) - x0;
    constexpr int PZ = row_pitch(F), FS = field_floats(F, NC);   // compile-time: every tap is one base plus a constant
    float *const w = reinterpret_cast<float *>(smem_raw);
    // receivers and sources of the tile: {index, next entry of the same
    // thread, cell of the thread, target mask}; a source's divisor follows
    int4 *const points = reinterpret_cast<int4 *>(smem_raw + (sizeof(float) * R2_NF * FS + 15) / 16 * 16);
    float *const divs = reinterpret_cast<float *>(points + a.rec.n + a.src.n);
    __shared__ int s_np, s_rec[R2_THREADS], s_src[R2_THREADS];
    __shared__ Slab s_sx[R2_COLS];
    __shared__ Surf2d s_surf[R2_COLS];   // free surface: columns of a tile at the top
    const float hc[4] = {g.hc[0], g.hc[1], g.hc[2], g.hc[3]};
    Fields f = f0;
    if (g.nb > 1) shot_fields(g, f, shot);

    // ---- wave fields in: the tile with its halo (neighbours' cells, or the
    // pads); columns past the tile that a thread's window may touch are zero
    const int wid[R2_NF] = {VX, VZ, SXX, SZZ, SXZ};
    for (int i = tid; i < R2_NF * FS; i += R2_THREADS) w[i] = 0.0f;
    s_rec[tid] = s_src[tid] = -1;
    if (tid == 0) s_np = 0;
    for (int x = tid; x < tx; x += R2_THREADS) s_sx[x] = slab_of(g, f, 0, x0 + x, g.nx, true);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < R2_NF; q++) {
        const float *src = f.w[wid[q]];
        for (int i = tid; i < (tz + 2 * F) * (tx + 2 * F); i += R2_THREADS) {
            const int x = i / (tz + 2 * F), z = i - x * (tz + 2 * F);
            w[q * FS + x * PZ + z] = src[(i64)(x0 + x) * g.NZ + z0 + z];
        }
    }
    // ---- the thread's cells: row z, columns xb .. xb + NC - 1
    const int nzb = (tz + 31) / 32, nxg = (R2_THREADS / 32) / nzb;
    const int z = (warp % nzb) * 32 + lane, xb = (warp / nzb) * NC;
    const bool active = warp / nzb < nxg && z < tz && xb < tx;
    const int gz = z0 + z + F;
    // points: each goes to the thread that owns its cell
    for (int i = tid; i < a.rec.n + a.src.n; i += R2_THREADS) {
        const bool rec = i < a.rec.n;
        const int p = rec ? i : i - a.rec.n;
        const i64 cell = rec ? a.rec.cell[p] : a.src.cell[p];
        if (cell < 0 || cell / g.nvol != shot) continue;
        const int c = (int)(cell % g.nvol), x = c / g.NZ - F - x0, k = c % g.NZ - F - z0;
        if (x < 0 || x >= tx || k < 0 || k >= tz) continue;
        const int owner = ((x / NC) * nzb + k / 32) * 32 + k % 32, e = atomicAdd(&s_np, 1);
        int mask = 0;
        if (!rec) {
            for (int q = 0; q < a.src.ntarget[p]; q++) mask |= 1 << tile_field(a.src.field[3 * p + q]);
            divs[e] = a.src.div[3 * p];
        }
        points[e] = make_int4(p, atomicExch(rec ? s_rec + owner : s_src + owner, e), x % NC, mask);
    }
    // parameters, CPML and memory variables
    float rip[NC], rkp[NC], psi_sxx[NC], psi_sxzx[NC], psi_szz[NC], psi_sxzz[NC], psi_vxx[NC], psi_vzx[NC], psi_vzz[NC],
        psi_vxz[NC], rr[NC][3][LL];
    S2dMat mat[NC];
    int shell[NC];
    Slab sz = {};
    int sx_at[NC];
    bool on[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) {
        on[i] = active && xb + i < tx;
        const int gx = x0 + (on[i] ? xb + i : 0) + F, zz = active ? gz : F;
        const i64 ip = (i64)(gx - F) * g.nz + (zz - F);
        rip[i] = f.p[PRIP][ip];
        rkp[i] = f.p[PRKP][ip];
        if constexpr (L == 0) mat[i] = s2d_elastic(f.p[PM][ip], f.p[PMU][ip], f.p[PMUIPKP][ip]);
        else mat[i] = s2d_visco(L, g.dt, f.p[PM][ip], f.p[PMU][ip], f.p[PMUIPKP][ip], f.p[PTAUP][ip], f.p[PTAUS][ip],
                                f.p[PTAUSIPKP][ip]);
        sx_at[i] = s_sx[on[i] ? xb + i : 0].at;
        if (i == 0) sz = slab_of(g, f, 2, zz - F, g.nz - g.zpad, !g.freesurf);
        psi_sxx[i] = psi_sxzx[i] = psi_szz[i] = psi_sxzz[i] = psi_vxx[i] = psi_vzx[i] = psi_vzz[i] = psi_vxz[i] = 0.0f;
        if (sx_at[i] >= 0) {
            const i64 q = (i64)sx_at[i] * g.nz + (zz - F);
            psi_sxx[i] = f.psi[PSXX_X][q]; psi_sxzx[i] = f.psi[PSXZ_X][q];
            psi_vxx[i] = f.psi[PVX_X][q]; psi_vzx[i] = f.psi[PVZ_X][q];
        }
        if (sz.at >= 0) {
            const i64 q = (i64)(gx - F) * (2 * g.nab) + sz.at;
            psi_szz[i] = f.psi[PSZZ_Z][q]; psi_sxzz[i] = f.psi[PSXZ_Z][q];
            psi_vzz[i] = f.psi[PVZ_Z][q]; psi_vxz[i] = f.psi[PVX_Z][q];
        }
#pragma unroll
        for (int l = 0; l < L; l++) {
            const i64 ir = l * g.nvol + (i64)gx * g.NZ + zz;
            rr[i][0][l] = f.r[RXX][ir]; rr[i][1][l] = f.r[RZZ][ir]; rr[i][2][l] = f.r[RXZ][ir];
        }
        if (on[i] && z == 0) s_surf[xb + i] = surf2d_of(mat[i]);
        shell[i] = a.bnd.nfield && on[i] ? inject_ind2d(g, gz, gx) : -1;
    }
    // ---- exchange: words of a side are [field][F][along the edge] of the
    // receiving CTA; sides z-, z+, x-, x+
    const bool nbr[4] = {iz > 0, iz < r.ntz - 1, ix > 0, ix < r.ntx - 1};
    const int side = 2 * F * r.side;
    const int to[4] = {((int)blockIdx.x - 1) * 8 + 1, ((int)blockIdx.x + 1) * 8, ((int)blockIdx.x - r.ntz) * 8 + 3,
                       ((int)blockIdx.x + r.ntz) * 8 + 2};
    // words this thread receives: where from, and the cell they go to in the
    // first (A) or second (B) field of the half step
    int from[R2_WORDS];
    int cell_in[R2_WORDS];   // cell, + 1 << 28 for the second field, + 1 << 29 for a z side; -1: none
    {
        const int nz_ = F * tx, nx_ = F * tz;
        const int n[4] = {nbr[0] ? 2 * nz_ : 0, nbr[1] ? 2 * nz_ : 0, nbr[2] ? 2 * nx_ : 0, nbr[3] ? 2 * nx_ : 0};
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++) {
            int j = tid + u * R2_THREADS, s = 0;
            cell_in[u] = -1;
            from[u] = 0;
#pragma unroll
            for (int q = 0; q < 3; q++)
                if (s == q && j >= n[q]) { j -= n[q]; s = q + 1; }
            if (j >= (s == 0 ? n[0] : s == 1 ? n[1] : s == 2 ? n[2] : n[3])) continue;
            const int n1 = s < 2 ? nz_ : nx_, fld = j / n1, m = j % n1;
            int c;
            if (s < 2) {   // [column][row from the edge]
                const int k = m % F;
                c = (m / F + F) * PZ + (s == 0 ? F - 1 - k : F + tz + k);
            } else {       // [column from the edge][row]
                const int k = m / tz;
                c = (s == 2 ? F - 1 - k : F + tx + k) * PZ + F + m % tz;
            }
            from[u] = ((int)blockIdx.x * 8 + s) * side + j;
            cell_in[u] = c + (fld << 28) + ((s < 2) << 29);
        }
    }
    const int half = 4 * side;   // from a velocity word to the stress word
    // send a cell's two values of a half step to the neighbours whose halo it
    // is in; x sides take (vx0, vx1), z sides (vz0, vz1)
    auto send = [&](int x, int z, int h, unsigned epoch, float vx0, float vx1, float vz0, float vz1) {
        const int s = side;
        if (z < F && nbr[0]) {
            u64 *p = a.words + (h + to[0] * s + x * F + z);
            st_word(p, epoch, vz0);
            st_word(p + F * tx, epoch, vz1);
        }
        if (z >= tz - F && nbr[1]) {
            u64 *p = a.words + (h + to[1] * s + x * F + (tz - 1 - z));
            st_word(p, epoch, vz0);
            st_word(p + F * tx, epoch, vz1);
        }
        if (x < F && nbr[2]) {
            u64 *p = a.words + (h + to[2] * s + x * tz + z);
            st_word(p, epoch, vx0);
            st_word(p + F * tz, epoch, vx1);
        }
        if (x >= tx - F && nbr[3]) {
            u64 *p = a.words + (h + to[3] * s + (tx - 1 - x) * tz + z);
            st_word(p, epoch, vx0);
            st_word(p + F * tz, epoch, vx1);
        }
    };
    bool failed = false;
    // fx, fz: first field on x and z sides; f1: second field
    auto receive = [&](int h, unsigned epoch, int fx, int fz, int f1) {
        u64 v[R2_WORDS];
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++)
            if (cell_in[u] >= 0) v[u] = ld_word(a.words + (from[u] + h));
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++) {
            if (cell_in[u] < 0) continue;
            long long lim = 0;
            for (int spin = 1; (unsigned)(v[u] >> 32) != epoch && !failed; spin++) {
                v[u] = ld_word(a.words + (from[u] + h));
                if (spin % 1024) continue;   // now and then: has the wait run out?
                if (!lim) lim = now_ns() + a.wait_ns;
                failed = now_ns() > lim;
            }
            const int c = cell_in[u];
            w[(c & 0xfffffff) + ((c >> 28) & 1 ? f1 : (c >> 29) & 1 ? fz : fx) * FS] = __uint_as_float((unsigned)v[u]);
        }
    };
    __syncthreads();
    const int my_rec = s_rec[tid], my_src = s_src[tid];
    // a thread's sources in ascending order, the order the source kernel adds them in
    for (int e = my_src; e >= 0; e = points[e].y)
        for (int q = points[e].y; q >= 0; q = points[q].y)
            if (points[q].x < points[e].x) {
                const int4 pe = points[e], pq = points[q];
                const float de = divs[e];
                points[e] = make_int4(pq.x, pe.y, pq.z, pq.w);
                points[q] = make_int4(pe.x, pq.y, pe.z, pe.w);
                divs[e] = divs[q];
                divs[q] = de;
            }
    const int c0 = (xb + F) * PZ + z + F;   // the thread's first cell
    // amplitude of the thread's first source, one step ahead
    auto amp_of = [&](int e, int step) { return g.dt * a.stf[(i64)points[e].x * a.nt_total + step]; };
    float amp = my_src >= 0 ? amp_of(my_src, a.t0) : 0.0f;
    // sources of a step into the fields `fields` of cell i; v: their values
    auto inject = [&](int i, int step, int field, float first, float &v) {
        for (int e = my_src; e >= 0; e = points[e].y) {
            if (points[e].z != i || !((points[e].w >> field) & 1)) continue;
            const float q = e == my_src ? first : amp_of(e, step), dv = divs[e];
            v += dv == 0.0f ? q : q / dv;
        }
    };

    // the thread's first receiver {index, next, cell or -1}, and the traces
    // of a receiver in the cell
    const int4 rec0 = my_rec >= 0 ? points[my_rec] : make_int4(0, -1, -1, 0);
    auto put = [&](int rec, int step, float vx, float vz, float sxx, float szz, float sxz) {
        float *out = a.out + (i64)rec * a.nt_total + step;
        const i64 trace = (i64)a.rec.n * a.nt_total;
        if (a.outmask & (1u << SFD_OUT_VX)) { *out = vx; out += trace; }
        if (a.outmask & (1u << SFD_OUT_VZ)) { *out = vz; out += trace; }
        if (a.outmask & (1u << SFD_OUT_SXX)) { *out = sxx; out += trace; }
        if (a.outmask & (1u << SFD_OUT_SZZ)) { *out = szz; out += trace; }
        if (a.outmask & (1u << SFD_OUT_SXZ)) { *out = sxz; out += trace; }
        if (a.outmask & (1u << SFD_OUT_P)) *out = (sxx + szz) / 2.0f;
    };

    for (int step = a.t0; step < a.t1; step++) {
        const unsigned epoch = (unsigned)step + 1;
        const int next = step + 1;
        float amp_next = 0.0f;
        // the exchange's indices are formed in each step: kept across steps
        // they would take the registers the cells' state needs
        int zs = z, xs = xb;
        asm volatile("" : "+r"(zs), "+r"(xs));
        if (my_src >= 0 && next < a.tmax) amp_next = amp_of(my_src, next);
        // ---- velocities
        if (active) {
            // x windows of the thread's columns: forward for sxx, backward for sxz
            float wf[2 * F + NC - 1], wb[2 * F + NC - 1];
#pragma unroll
            for (int k = 0; k < 2 * F + NC - 1; k++) {
                wf[k] = w[W_XX * FS + c0 + (k - F + 1) * PZ];
                wb[k] = w[W_XZ * FS + c0 + (k - F) * PZ];
            }
            bool bad = false;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int c = c0 + i * PZ;
                float zf[2 * F], zb[2 * F];
#pragma unroll
                for (int k = 0; k < 2 * F; k++) {
                    zf[k] = w[W_ZZ * FS + c + k - F + 1];
                    zb[k] = w[W_XZ * FS + c + k - F];
                }
                float vx = w[W_VX * FS + c], vz = w[W_VZ * FS + c];
                float sxx_x = diff_win<F>(wf + i, hc), sxz_x = diff_win<F>(wb + i, hc);
                float szz_z = diff_win<F>(zf, hc), sxz_z = diff_win<F>(zb, hc);
                if (sz.at >= 0) {
                    cpml_reg(psi_sxzz[i], sz.kf, sz.af, sz.bf, sxz_z);
                    cpml_reg(psi_szz[i], sz.kh, sz.ah, sz.bh, szz_z);
                }
                if (sx_at[i] >= 0) {
                    const Slab &sx = s_sx[on[i] ? xb + i : 0];
                    cpml_reg(psi_sxx[i], sx.kh, sx.ah, sx.bh, sxx_x);
                    cpml_reg(psi_sxzx[i], sx.kf, sx.af, sx.bf, sxz_x);
                }
                if (my_src >= 0 && step > 0) {   // step 0 finds its sources in the fields, and so do the stresses
                    inject(i, step, W_VX, amp, vx);
                    inject(i, step, W_VZ, amp, vz);
                }
                vx = v2d_math(vx, sxx_x, sxz_z, rip[i]);
                vz = v2d_math(vz, szz_z, sxz_x, rkp[i]);
                if (on[i]) {
                    w[W_VX * FS + c] = vx;
                    w[W_VZ * FS + c] = vz;
                    send(xs + i, zs, 0, epoch, vx, vz, vx, vz);
                    bad |= !isfinite(vx);
                }
            }
            // the scan of launch_finite_check
            if ((next % FINITE_CHECK_EVERY == 0 || next == a.tmax) && bad) atomicMin(a.first_bad, step);
        }
        receive(0, epoch, W_VX, W_VX, W_VZ);
        __syncthreads();
        // ---- stresses and memory variables, surface, receivers, next sources
        if (active) {
            float wb[2 * F + NC - 1], wf[2 * F + NC - 1];
#pragma unroll
            for (int k = 0; k < 2 * F + NC - 1; k++) {
                wb[k] = w[W_VX * FS + c0 + (k - F) * PZ];
                wf[k] = w[W_VZ * FS + c0 + (k - F + 1) * PZ];
            }
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int c = c0 + i * PZ;
                float zf[2 * F], zb[2 * F];
#pragma unroll
                for (int k = 0; k < 2 * F; k++) {
                    zf[k] = w[W_VX * FS + c + k - F + 1];
                    zb[k] = w[W_VZ * FS + c + k - F];
                }
                float sxx = w[W_XX * FS + c], szz = w[W_ZZ * FS + c], sxz = w[W_XZ * FS + c];
                float vxx = diff_win<F>(wb + i, hc), vzx = diff_win<F>(wf + i, hc);
                float vxz = diff_win<F>(zf, hc), vzz = diff_win<F>(zb, hc);
                if (sz.at >= 0) {
                    cpml_reg(psi_vxz[i], sz.kh, sz.ah, sz.bh, vxz);
                    cpml_reg(psi_vzz[i], sz.kf, sz.af, sz.bf, vzz);
                }
                if (sx_at[i] >= 0) {
                    const Slab &sx = s_sx[on[i] ? xb + i : 0];
                    cpml_reg(psi_vxx[i], sx.kf, sx.af, sx.bf, vxx);
                    cpml_reg(psi_vzx[i], sx.kh, sx.ah, sx.bh, vzx);
                }
                const S2dMat &m = mat[i];
                const float tr = __fadd_rn(vxx, vzz), sh = __fadd_rn(vxz, vzx);
                const float exx = s2d_normal(m.gm, tr, m.fm, vzz), ezz = s2d_normal(m.gm, tr, m.fm, vxx);
                if constexpr (L == 0) {
                    sxz = __fmaf_rn(m.fipkp, sh, sxz);
                    sxx = __fadd_rn(sxx, exx);
                    szz = __fadd_rn(szz, ezz);
                } else {
                    float o[3] = {0, 0, 0}, n[3] = {0, 0, 0};
                    const float q[3] = {s2d_normal(m.e, tr, m.d, vzz), s2d_normal(m.e, tr, m.d, vxx), __fmul_rn(m.dipkp, sh)};
#pragma unroll
                    for (int l = 0; l < L; l++)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            o[k] += rr[i][k][l];
                            rr[i][k][l] = s2d_memory(rr[i][k][l], g.eta[l], g.eta_b[l], g.eta_c[l], q[k]);
                            n[k] += rr[i][k][l];
                        }
                    sxz = s2d_add(sxz, __fmaf_rn(m.fipkp, sh, __fmul_rn(g.dt2, o[2])), g.dt2, n[2]);
                    sxx = s2d_add(sxx, __fmaf_rn(g.dt2, o[0], exx), g.dt2, n[0]);
                    szz = s2d_add(szz, __fmaf_rn(g.dt2, o[1], ezz), g.dt2, n[1]);
                }
                if (!on[i]) continue;
                if (shell[i] >= 0) {   // boundary shells, before the free surface
                    const i64 at = (i64)shot * (g.sb_bnd / (a.prec == SFD_PREC_FP32 ? 4 : 2)) + (i64)step * g.nbnd + shell[i];
                    bnd_store(g, a.bnd, a.prec, VX, at, w[W_VX * FS + c]);
                    bnd_store(g, a.bnd, a.prec, VZ, at, w[W_VZ * FS + c]);
                    bnd_store(g, a.bnd, a.prec, SXX, at, sxx);
                    bnd_store(g, a.bnd, a.prec, SZZ, at, szz);
                    bnd_store(g, a.bnd, a.prec, SXZ, at, sxz);
                }
                if (g.freesurf && iz == 0 && z <= F) {
                    // the arithmetic of surf2d_column, forward: the row at the
                    // surface, and the images each row leaves above it
                    if (z == 0) {
                        szz = 0.0f;
                        const Surf2d su = s_surf[xb + i];
                        const float h = surf2d_h<L == 0>(su, vxx, vzz);
                        if constexpr (L == 0) {
                            sxx = __fadd_rn(h, sxx);
                        } else {
                            float sump = 0;
#pragma unroll
                            for (int l = 0; l < L; l++) {
                                rr[i][1][l] = 0.0f;
                                sump += rr[i][0][l];
                            }
                            sxx = __fadd_rn(__fmaf_rn(-g.dt2, sump, h), sxx);
                            sump = 0;
#pragma unroll
                            for (int l = 0; l < L; l++) {
                                rr[i][0][l] = __fadd_rn(__fmul_rn(surf2d_b(g.eta[l]), surf2d_hr(su, vxx, vzz)), rr[i][0][l]);
                                sump += rr[i][0][l];
                            }
                            sxx = __fadd_rn(__fmul_rn(g.dt2, sump), sxx);
                        }
                    } else {
                        w[W_ZZ * FS + c - 2 * z] = -szz;
                    }
                    if (z < F) w[W_XZ * FS + c - 2 * z - 1] = -sxz;
                }
                if (i == rec0.z) put(rec0.x, step, w[W_VX * FS + c], w[W_VZ * FS + c], sxx, szz, sxz);
                for (int e = rec0.y; e >= 0; e = points[e].y)
                    if (points[e].z == i) put(points[e].x, step, w[W_VX * FS + c], w[W_VZ * FS + c], sxx, szz, sxz);
                if (my_src >= 0 && next < a.tmax) {
                    inject(i, next, W_XX, amp_next, sxx);
                    inject(i, next, W_ZZ, amp_next, szz);
                    inject(i, next, W_XZ, amp_next, sxz);
                }
                w[W_XX * FS + c] = sxx;
                w[W_ZZ * FS + c] = szz;
                w[W_XZ * FS + c] = sxz;
                if (next < a.t1) send(xs + i, zs, half, epoch, sxx, sxz, szz, sxz);
            }
        }
        amp = amp_next;
        if (next < a.t1) receive(half, epoch, W_XX, W_ZZ, W_XZ);
        if (__syncthreads_or(failed)) break;
    }
    if (failed) atomicExch(a.status, 1);

    // ---- state out: the tile's cells and, at the top, the images above them
#pragma unroll
    for (int q = 0; q < R2_NF; q++) {
        float *dst = f.w[wid[q]];
        const int up = iz == 0 && q >= W_XX ? F : 0;
        for (int i = tid; i < (tz + up) * tx; i += R2_THREADS) {
            const int x = i / (tz + up), k = i - x * (tz + up) + F - up;
            dst[(i64)(x0 + x + F) * g.NZ + z0 + k] = w[q * FS + (x + F) * PZ + k];
        }
    }
#pragma unroll
    for (int i = 0; i < NC; i++) {
        if (!on[i]) continue;
        const int gx = x0 + xb + i + F;
        if (sx_at[i] >= 0) {
            const i64 q = (i64)sx_at[i] * g.nz + (gz - F);
            f.psi[PSXX_X][q] = psi_sxx[i]; f.psi[PSXZ_X][q] = psi_sxzx[i];
            f.psi[PVX_X][q] = psi_vxx[i]; f.psi[PVZ_X][q] = psi_vzx[i];
        }
        if (sz.at >= 0) {
            const i64 q = (i64)(gx - F) * (2 * g.nab) + sz.at;
            f.psi[PSZZ_Z][q] = psi_szz[i]; f.psi[PSXZ_Z][q] = psi_sxzz[i];
            f.psi[PVZ_Z][q] = psi_vzz[i]; f.psi[PVX_Z][q] = psi_vxz[i];
        }
#pragma unroll
        for (int l = 0; l < L; l++) {
            const i64 ir = l * g.nvol + (i64)gx * g.NZ + gz;
            f.r[RXX][ir] = rr[i][0][l]; f.r[RZZ][ir] = rr[i][1][l]; f.r[RXZ][ir] = rr[i][2][l];
        }
    }
}

// ------------------------------------------------------------------ adjoint
// what atomicAdd does in global memory: subnormal operands and sums are zero
__device__ __forceinline__ float add_ftz(float a, float b)
{
    float r;
    asm("add.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// A segment of the boundary-saving adjoint loop of elastic shots without a
// free surface (steps a.t0, a.t0-1 .. a.t1+1, the order of k_adjs2d_q4,
// k_adjv2d_q4, k_residuals): the tile's forward and adjoint wave fields are
// resident, gradient sums and CPML memory in registers, saved boundaries are
// read one step's slice at a time.  Per step: stresses (forward
// reconstruction, adjoint update, M and mu terms), exchange, velocities (the
// same, rho term), the step's sources out and the next step's residuals in,
// exchange.  Points act on the thread's own cells: on velocities at the end of
// a step, on stresses when the next step (or the end of the segment) takes
// them up.  Bound by the exchange (two round trips between CTAs of about 1 us
// each) and the serial chain of a cell's arithmetic: 16.6 us per step of
// ordinary launches at 300 x 400, order 8, 7.5 here with two cells a thread
// (twice the fields of the forward loop: four cells would not fit the
// registers).
template <int F, int NC, typename T>
__global__ void __launch_bounds__(R2_THREADS, 1) k_resident2d_adj(const __grid_constant__ Grid g,
                                                                  const __grid_constant__ Fields f0,
                                                                  const __grid_constant__ AdjFields a0,
                                                                  const __grid_constant__ Res2d r,
                                                                  const __grid_constant__ Res2dAdj a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int R2_WORDS = 4, A = R2_NF;   // A: first adjoint field of the tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntile = r.ntz * r.ntx;
    const int shot = a.shot0 + blockIdx.x / ntile, tl = blockIdx.x % ntile;
    const int iz = tl % r.ntz, ix = tl / r.ntz;
    const int z0 = (int)((i64)iz * g.nz / r.ntz), tz = (int)((i64)(iz + 1) * g.nz / r.ntz) - z0;
    const int x0 = (int)((i64)ix * g.nx / r.ntx), tx = (int)((i64)(ix + 1) * g.nx / r.ntx) - x0;
    constexpr int PZ = row_pitch(F), FS = field_floats(F, NC);
    float *const w = reinterpret_cast<float *>(smem_raw);
    int4 *const points = reinterpret_cast<int4 *>(smem_raw + (sizeof(float) * 2 * R2_NF * FS + 15) / 16 * 16);
    float *const divs = reinterpret_cast<float *>(points + a.rec.n + a.src.n);
    __shared__ int s_np, s_rec[R2_THREADS], s_src[R2_THREADS];
    __shared__ Slab s_sx[R2_COLS];
    const float hc[4] = {g.hc[0], g.hc[1], g.hc[2], g.hc[3]};
    Fields f = f0;
    AdjFields q = a0;
    if (g.nb > 1) {
        shot_fields(g, f, shot);
        shot_adj(g, q, shot);
    }

    const int wid[R2_NF] = {VX, VZ, SXX, SZZ, SXZ};
    for (int i = tid; i < 2 * R2_NF * FS; i += R2_THREADS) w[i] = 0.0f;
    s_rec[tid] = s_src[tid] = -1;
    if (tid == 0) s_np = 0;
    for (int x = tid; x < tx; x += R2_THREADS) s_sx[x] = slab_of(g, f, 0, x0 + x, g.nx, true);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2 * R2_NF; k++) {
        const float *src = k < A ? f.w[wid[k % A]] : q.wr[wid[k % A]];
        for (int i = tid; i < (tz + 2 * F) * (tx + 2 * F); i += R2_THREADS) {
            const int x = i / (tz + 2 * F), z = i - x * (tz + 2 * F);
            w[k * FS + x * PZ + z] = src[(i64)(x0 + x) * g.NZ + z0 + z];
        }
    }
    const int nzb = (tz + 31) / 32, nxg = (R2_THREADS / 32) / nzb;
    const int z = (warp % nzb) * 32 + lane, xb = (warp / nzb) * NC;
    const bool active = warp / nzb < nxg && z < tz && xb < tx;
    const int gz = z0 + z + F;
    for (int i = tid; i < a.rec.n + a.src.n; i += R2_THREADS) {
        const bool rec = i < a.rec.n;
        const int p = rec ? i : i - a.rec.n;
        const i64 cell = rec ? a.rec.cell[p] : a.src.cell[p];
        if (cell < 0 || cell / g.nvol != shot) continue;
        const int c = (int)(cell % g.nvol), x = c / g.NZ - F - x0, k = c % g.NZ - F - z0;
        if (x < 0 || x >= tx || k < 0 || k >= tz) continue;
        const int owner = ((x / NC) * nzb + k / 32) * 32 + k % 32, e = atomicAdd(&s_np, 1);
        int mask = 0;
        if (!rec) {
            for (int n = 0; n < a.src.ntarget[p]; n++) mask |= 1 << tile_field(a.src.field[3 * p + n]);
            divs[e] = a.src.div[3 * p];
        }
        points[e] = make_int4(p, atomicExch(rec ? s_rec + owner : s_src + owner, e), x % NC, mask);
    }
    // the thread's cells
    float rip[NC], rkp[NC], psi_sxx[NC], psi_sxzx[NC], psi_szz[NC], psi_sxzz[NC], psi_vxx[NC], psi_vzx[NC], psi_vzz[NC],
        psi_vxz[NC];
    S2dMat mat[NC];
    Adj2dCoef coef[NC];
    double gM[NC], gmu[NC], gr[NC];
    int shell[NC], sx_at[NC];
    Slab sz = {};
    bool on[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) {
        on[i] = active && xb + i < tx;
        const int gx = x0 + (on[i] ? xb + i : 0) + F, zz = active ? gz : F;
        const i64 ip = (i64)(gx - F) * g.nz + (zz - F);
        rip[i] = f.p[PRIP][ip];
        rkp[i] = f.p[PRKP][ip];
        mat[i] = s2d_elastic(f.p[PM][ip], f.p[PMU][ip], f.p[PMUIPKP][ip]);
        coef[i] = adj2d_coef(f.p[PM][ip], f.p[PMU][ip]);
        gM[i] = q.grad[GM][ip];
        gmu[i] = q.grad[GMU][ip];
        gr[i] = q.grad[GRHO][ip];
        sx_at[i] = s_sx[on[i] ? xb + i : 0].at;
        if (i == 0) sz = slab_of(g, f, 2, zz - F, g.nz - g.zpad, true);
        psi_sxx[i] = psi_sxzx[i] = psi_szz[i] = psi_sxzz[i] = psi_vxx[i] = psi_vzx[i] = psi_vzz[i] = psi_vxz[i] = 0.0f;
        if (sx_at[i] >= 0) {
            const i64 k = (i64)sx_at[i] * g.nz + (zz - F);
            psi_sxx[i] = f.psi[PSXX_X][k]; psi_sxzx[i] = f.psi[PSXZ_X][k];
            psi_vxx[i] = f.psi[PVX_X][k]; psi_vzx[i] = f.psi[PVZ_X][k];
        }
        if (sz.at >= 0) {
            const i64 k = (i64)(gx - F) * (2 * g.nab) + sz.at;
            psi_szz[i] = f.psi[PSZZ_Z][k]; psi_sxzz[i] = f.psi[PSXZ_Z][k];
            psi_vzz[i] = f.psi[PVZ_Z][k]; psi_vxz[i] = f.psi[PVX_Z][k];
        }
        shell[i] = on[i] ? inject_ind2d(g, gz, gx) : -1;
    }
    // exchange words of a side: [field][F][along the edge], fields 0, 1 of the
    // forward and 2, 3 of the adjoint state
    const bool nbr[4] = {iz > 0, iz < r.ntz - 1, ix > 0, ix < r.ntx - 1};
    const int side = 4 * F * r.side, half = 4 * side;
    const int to[4] = {((int)blockIdx.x - 1) * 8 + 1, ((int)blockIdx.x + 1) * 8, ((int)blockIdx.x - r.ntz) * 8 + 3,
                       ((int)blockIdx.x + r.ntz) * 8 + 2};
    int from[R2_WORDS], cell_in[R2_WORDS];   // cell + field << 26 + (z side) << 28; -1: none
    {
        const int nz_ = F * tx, nx_ = F * tz;
        const int n[4] = {nbr[0] ? 4 * nz_ : 0, nbr[1] ? 4 * nz_ : 0, nbr[2] ? 4 * nx_ : 0, nbr[3] ? 4 * nx_ : 0};
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++) {
            int j = tid + u * R2_THREADS, s = 0;
            cell_in[u] = -1;
            from[u] = 0;
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (s == k && j >= n[k]) { j -= n[k]; s = k + 1; }
            if (j >= (s == 0 ? n[0] : s == 1 ? n[1] : s == 2 ? n[2] : n[3])) continue;
            const int n1 = s < 2 ? nz_ : nx_, fld = j / n1, m = j % n1;
            int c;
            if (s < 2) {
                const int k = m % F;
                c = (m / F + F) * PZ + (s == 0 ? F - 1 - k : F + tz + k);
            } else {
                const int k = m / tz;
                c = (s == 2 ? F - 1 - k : F + tx + k) * PZ + F + m % tz;
            }
            from[u] = ((int)blockIdx.x * 8 + s) * side + j;
            cell_in[u] = c + (fld << 26) + ((s < 2) << 28);
        }
    }
    // vx0 / vz0: first fields on x / z sides, v1: second ones, of the forward
    // (0) and the adjoint (1) state
    auto send = [&](int x, int z, int h, unsigned epoch, const float (&vx0)[2], const float (&vz0)[2], const float (&v1)[2]) {
        auto put = [&](int s, int at, int step, const float (&v0)[2]) {
            u64 *p = a.words + (h + to[s] * side + at);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                st_word(p + 2 * k * step, epoch, v0[k]);
                st_word(p + (2 * k + 1) * step, epoch, v1[k]);
            }
        };
        if (z < F && nbr[0]) put(0, x * F + z, F * tx, vz0);
        if (z >= tz - F && nbr[1]) put(1, x * F + (tz - 1 - z), F * tx, vz0);
        if (x < F && nbr[2]) put(2, x * tz + z, F * tz, vx0);
        if (x >= tx - F && nbr[3]) put(3, (tx - 1 - x) * tz + z, F * tz, vx0);
    };
    bool failed = false;
    auto receive = [&](int h, unsigned epoch, int fx, int fz, int f1) {
        u64 v[R2_WORDS];
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++)
            if (cell_in[u] >= 0) v[u] = ld_word(a.words + (from[u] + h));
#pragma unroll
        for (int u = 0; u < R2_WORDS; u++) {
            const int c = cell_in[u];
            if (c < 0) continue;
            long long lim = 0;
            for (int spin = 1; (unsigned)(v[u] >> 32) != epoch && !failed; spin++) {
                v[u] = ld_word(a.words + (from[u] + h));
                if (spin % 1024) continue;
                if (!lim) lim = now_ns() + a.wait_ns;
                failed = now_ns() > lim;
            }
            const int fld = (c >> 26) & 3, k = ((fld & 1) ? f1 : (c >> 28) & 1 ? fz : fx) + (fld >= 2 ? A : 0);
            w[(c & 0x3ffffff) + k * FS] = __uint_as_float((unsigned)v[u]);
        }
    };
    __syncthreads();
    const int my_rec = s_rec[tid], my_src = s_src[tid];
    for (int e = my_src; e >= 0; e = points[e].y)   // ascending, the order the source kernel subtracts them in
        for (int n = points[e].y; n >= 0; n = points[n].y)
            if (points[n].x < points[e].x) {
                const int4 pe = points[e], pn = points[n];
                const float de = divs[e];
                points[e] = make_int4(pn.x, pe.y, pn.z, pn.w);
                points[n] = make_int4(pe.x, pn.y, pe.z, pe.w);
                divs[e] = divs[n];
                divs[n] = de;
            }
    const int c0 = (xb + F) * PZ + z + F;
    // the sources of a step out of field `field` of cell i
    auto remove = [&](int i, int step, int field, float &v) {
        for (int e = my_src; e >= 0; e = points[e].y) {
            if (points[e].z != i || !((points[e].w >> field) & 1)) continue;
            const float amp = -__fmul_rn(g.dt, a.stf[(i64)points[e].x * a.nt_total + step]), dv = divs[e];
            v = add_ftz(v, dv == 0.0f ? amp : __fdiv_rn(amp, dv));
        }
    };
    // the residuals of a step into the adjoint stresses / velocities of cell i
    auto residual = [&](int i, int step, bool stress, float &u0, float &u1, float &u2) {
        for (int e = my_rec; e >= 0; e = points[e].y) {
            if (points[e].z != i) continue;
            const float *p = a.res + (i64)points[e].x * a.nt_total + step;
            const i64 trace = (i64)a.rec.n * a.nt_total;
            for (int o = 0; o < SFD_NOUT; o++) {
                if (!(a.outmask & (1u << o))) continue;
                if (stress && o == SFD_OUT_P) {
                    const float v = *p / 2.0f;
                    u0 = add_ftz(u0, v);
                    u1 = add_ftz(u1, v);
                } else if (stress) {
                    if (o == SXX) u0 = add_ftz(u0, *p);
                    if (o == SZZ) u1 = add_ftz(u1, *p);
                    if (o == SXZ) u2 = add_ftz(u2, *p);
                } else {
                    if (o == VX) u0 = add_ftz(u0, *p);
                    if (o == VZ) u1 = add_ftz(u1, *p);
                }
                p += trace;
            }
        }
    };

    for (int t = a.t0; t > a.t1; t--) {
        const unsigned epoch = (unsigned)(a.tmax - t);
        int zs = z, xs = xb;
        asm volatile("" : "+r"(zs), "+r"(xs));
        // saved values of slice t-1, on their way while the stresses are formed
        float bs[NC][3], bv[NC][2];
#pragma unroll
        for (int i = 0; i < NC; i++) {
            if (shell[i] < 0) continue;
            const i64 at = (i64)(t - 1) * g.nbnd + shell[i];
            bs[i][0] = bnd_at<T>(g, q, SXX, at); bs[i][1] = bnd_at<T>(g, q, SZZ, at); bs[i][2] = bnd_at<T>(g, q, SXZ, at);
            bv[i][0] = bnd_at<T>(g, q, VX, at); bv[i][1] = bnd_at<T>(g, q, VZ, at);
        }
        // derivatives of the velocities (half 0) or stresses (half 1) of the
        // state whose fields start at base, for cell i
        auto strains = [&](int base, int i, float &xx, float &zz, float &xz, float &zx) {
            const int c = base * FS + c0 + i * PZ;
            float wx[2 * F], wz[2 * F], zf[2 * F], zb[2 * F];
#pragma unroll
            for (int k = 0; k < 2 * F; k++) {
                wx[k] = w[W_VX * FS + c + (k - F) * PZ];
                wz[k] = w[W_VZ * FS + c + (k - F + 1) * PZ];
                zf[k] = w[W_VX * FS + c + k - F + 1];
                zb[k] = w[W_VZ * FS + c + k - F];
            }
            xx = diff_win<F>(wx, hc); zx = diff_win<F>(wz, hc); xz = diff_win<F>(zf, hc); zz = diff_win<F>(zb, hc);
        };
        auto forces = [&](int base, int i, float &xx_x, float &xz_x, float &zz_z, float &xz_z) {
            const int c = base * FS + c0 + i * PZ;
            float wx[2 * F], wb[2 * F], zf[2 * F], zb[2 * F];
#pragma unroll
            for (int k = 0; k < 2 * F; k++) {
                wx[k] = w[W_XX * FS + c + (k - F + 1) * PZ];
                wb[k] = w[W_XZ * FS + c + (k - F) * PZ];
                zf[k] = w[W_ZZ * FS + c + k - F + 1];
                zb[k] = w[W_XZ * FS + c + k - F];
            }
            xx_x = diff_win<F>(wx, hc); xz_x = diff_win<F>(wb, hc); zz_z = diff_win<F>(zf, hc); xz_z = diff_win<F>(zb, hc);
        };
        if (active) {
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int c = c0 + i * PZ;
                const S2dMat &m = mat[i];
                float xx, zz, xz, zx;
                strains(0, i, xx, zz, xz, zx);
                float s[3] = {w[W_XX * FS + c], w[W_ZZ * FS + c], w[W_XZ * FS + c]};
                if (my_src >= 0 && t < a.t0) {
                    remove(i, t + 1, W_XX, s[0]);
                    remove(i, t + 1, W_ZZ, s[1]);
                    remove(i, t + 1, W_XZ, s[2]);
                }
                float tr = __fadd_rn(xx, zz);
                s[2] = __fmaf_rn(-m.fipkp, __fadd_rn(xz, zx), s[2]);
                s[0] = __fsub_rn(s[0], s2d_normal(m.gm, tr, m.fm, zz));
                s[1] = __fsub_rn(s[1], s2d_normal(m.gm, tr, m.fm, xx));
                if (shell[i] >= 0) {
#pragma unroll
                    for (int k = 0; k < 3; k++) s[k] = bs[i][k];
                }
                strains(A, i, xx, zz, xz, zx);
                if (sz.at >= 0) {
                    cpml_reg(psi_vxz[i], sz.kh, sz.ah, sz.bh, xz);
                    cpml_reg(psi_vzz[i], sz.kf, sz.af, sz.bf, zz);
                }
                if (sx_at[i] >= 0) {
                    const Slab &sx = s_sx[on[i] ? xb + i : 0];
                    cpml_reg(psi_vxx[i], sx.kf, sx.af, sx.bf, xx);
                    cpml_reg(psi_vzx[i], sx.kh, sx.ah, sx.bh, zx);
                }
                tr = __fadd_rn(xx, zz);
                const float lsxz = __fmul_rn(m.fipkp, __fadd_rn(xz, zx));
                const float lsxx = s2d_normal(m.gm, tr, m.fm, zz), lszz = s2d_normal(m.gm, tr, m.fm, xx);
                float u[3] = {w[(A + W_XX) * FS + c], w[(A + W_ZZ) * FS + c], w[(A + W_XZ) * FS + c]};
                if (my_rec >= 0 && t < a.t0) residual(i, t, true, u[0], u[1], u[2]);
                u[0] = __fadd_rn(u[0], lsxx);
                u[1] = __fadd_rn(u[1], lszz);
                u[2] = __fadd_rn(u[2], lsxz);
                const Adj2dGrad d = adj2d_terms(g.restype, coef[i], s[0], s[1], s[2], lsxx, lszz, lsxz);
                gM[i] += (double)d.M;
                if (g.restype == 0) gmu[i] += (double)d.mu;
                if (!on[i]) continue;
                w[W_XX * FS + c] = s[0];
                w[W_ZZ * FS + c] = s[1];
                w[W_XZ * FS + c] = s[2];
                w[(A + W_XX) * FS + c] = u[0];
                w[(A + W_ZZ) * FS + c] = u[1];
                w[(A + W_XZ) * FS + c] = u[2];
                const float x0_[2] = {s[0], u[0]}, z0_[2] = {s[1], u[1]}, v1[2] = {s[2], u[2]};
                send(xs + i, zs, 0, epoch, x0_, z0_, v1);
            }
        }
        receive(0, epoch, W_XX, W_ZZ, W_XZ);
        __syncthreads();
        if (active) {
            bool bad = false;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int c = c0 + i * PZ;
                float xx, xzx, zz, xzz;
                forces(0, i, xx, xzx, zz, xzz);
                float vx = __fmaf_rn(-__fadd_rn(xx, xzz), rip[i], w[W_VX * FS + c]);
                float vz = __fmaf_rn(-__fadd_rn(zz, xzx), rkp[i], w[W_VZ * FS + c]);
                if (shell[i] >= 0) {
                    vx = bv[i][0];
                    vz = bv[i][1];
                }
                forces(A, i, xx, xzx, zz, xzz);
                if (sz.at >= 0) {
                    cpml_reg(psi_sxzz[i], sz.kf, sz.af, sz.bf, xzz);
                    cpml_reg(psi_szz[i], sz.kh, sz.ah, sz.bh, zz);
                }
                if (sx_at[i] >= 0) {
                    const Slab &sx = s_sx[on[i] ? xb + i : 0];
                    cpml_reg(psi_sxx[i], sx.kh, sx.ah, sx.bh, xx);
                    cpml_reg(psi_sxzx[i], sx.kf, sx.af, sx.bf, xzx);
                }
                const float lvx = __fmul_rn(__fadd_rn(xx, xzz), rip[i]), lvz = __fmul_rn(__fadd_rn(zz, xzx), rkp[i]);
                float ux = __fadd_rn(w[(A + W_VX) * FS + c], lvx), uz = __fadd_rn(w[(A + W_VZ) * FS + c], lvz);
                gr[i] += (double)__fmaf_rn(-vx, lvx, -__fmul_rn(vz, lvz));
                if (!on[i]) continue;
                bad |= !isfinite(ux);
                if (my_src >= 0) {
                    remove(i, t, W_VX, vx);
                    remove(i, t, W_VZ, vz);
                }
                float none = 0.0f;
                if (my_rec >= 0 && t - 1 > a.tmin) residual(i, t - 1, false, ux, uz, none);
                w[W_VX * FS + c] = vx;
                w[W_VZ * FS + c] = vz;
                w[(A + W_VX) * FS + c] = ux;
                w[(A + W_VZ) * FS + c] = uz;
                if (t - 1 > a.t1) {
                    const float x0_[2] = {vx, ux}, v1[2] = {vz, uz};
                    send(xs + i, zs, half, epoch, x0_, x0_, v1);
                }
            }
            if ((t % FINITE_CHECK_EVERY == 0 || t == a.tmin + 1) && bad) atomicMin(a.first_bad, t);
        }
        if (t - 1 > a.t1) receive(half, epoch, W_VX, W_VX, W_VZ);
        if (__syncthreads_or(failed)) break;
    }
    if (failed) atomicExch(a.status, 1);
    // the stresses' points of the last step's end, then the state out
#pragma unroll
    for (int i = 0; i < NC; i++) {
        if (!on[i]) continue;
        const int gx = x0 + xb + i + F, c = c0 + i * PZ;
        const i64 iv = (i64)gx * g.NZ + gz, ip = (i64)(gx - F) * g.nz + (gz - F);
        float s[3] = {w[W_XX * FS + c], w[W_ZZ * FS + c], w[W_XZ * FS + c]};
        float u[3] = {w[(A + W_XX) * FS + c], w[(A + W_ZZ) * FS + c], w[(A + W_XZ) * FS + c]};
        if (my_src >= 0) {
            remove(i, a.t1 + 1, W_XX, s[0]);
            remove(i, a.t1 + 1, W_ZZ, s[1]);
            remove(i, a.t1 + 1, W_XZ, s[2]);
        }
        if (my_rec >= 0 && a.t1 > a.tmin) residual(i, a.t1, true, u[0], u[1], u[2]);
        f.w[VX][iv] = w[W_VX * FS + c]; f.w[VZ][iv] = w[W_VZ * FS + c];
        f.w[SXX][iv] = s[0]; f.w[SZZ][iv] = s[1]; f.w[SXZ][iv] = s[2];
        q.wr[VX][iv] = w[(A + W_VX) * FS + c]; q.wr[VZ][iv] = w[(A + W_VZ) * FS + c];
        q.wr[SXX][iv] = u[0]; q.wr[SZZ][iv] = u[1]; q.wr[SXZ][iv] = u[2];
        q.grad[GM][ip] = gM[i];
        if (g.restype == 0) q.grad[GMU][ip] = gmu[i];
        q.grad[GRHO][ip] = gr[i];
        if (sx_at[i] >= 0) {
            const i64 k = (i64)sx_at[i] * g.nz + (gz - F);
            f.psi[PSXX_X][k] = psi_sxx[i]; f.psi[PSXZ_X][k] = psi_sxzx[i];
            f.psi[PVX_X][k] = psi_vxx[i]; f.psi[PVZ_X][k] = psi_vzx[i];
        }
        if (sz.at >= 0) {
            const i64 k = (i64)(gx - F) * (2 * g.nab) + sz.at;
            f.psi[PSZZ_Z][k] = psi_szz[i]; f.psi[PSXZ_Z][k] = psi_sxzz[i];
            f.psi[PVZ_Z][k] = psi_vzz[i]; f.psi[PVX_Z][k] = psi_vxz[i];
        }
    }
}

// us per step of a resident launch, and of the ordinary launches
// (sfd_quad2d.cu) of a run's nb shots: fits to a B200 (resident / ordinary:
// 100 x 150 order 4 2.8 / 8.9; 300 x 400 order 8 4.7 / 11.0, L = 2 5.2 / 12.1;
// 400 x 577 order 8 9.5 / 11.5, L = 3 11.6 / 15.7; ordinary alone: 600 x 1000
// order 8 16.6, 602 x 1503 order 8 L = 2 28.8, 8 shots of 300 x 1000 order 4
// 30.4).  4 shots of 300 x 400, L = 2: 20.2 one after the other, 17.7 together.
static double resident2d_step_us(const Res2d &r, int L)
{
    return r.nc == 1 ? 3.2 : r.nc == 2 ? 4.7 + 0.25 * L : 9.3 + 0.8 * L;
}
static double ordinary2d_step_us(const Grid &g, int nb)
{
    return 9.0 + (g.F == 2 ? 0.9e-5 : 1.2e-5) * (1.0 + 0.4 * g.L) * nb * (double)g.nz * g.nx;
}

// Tiles of a resident launch of nb shots: ctas = 0 where it does not apply.
// It takes FP32 fields, order 4 or 8, up to 3 relaxation mechanisms, CPML
// slabs that do not overlap (or no absorbing layer); every tile is at least
// F + 1 cells a side (its halo is one neighbour deep, and the surface images
// of a column come from its own tile) and its halo at most r2_words words a
// thread.  With one CTA per SM and up to 4 cells per thread that is about
// 250,000 cells; larger grids fill the chip with ordinary launches.
// adjoint: twice the fields and words, elastic without a free surface, at
// most 2 cells a thread.
static Res2d resident2d_shape(const Grid &g, int nb, int npoints, int sms, bool adjoint)
{
    Res2d best;
    memset(&best, 0, sizeof best);
    const int F = g.F;
    if (g.nd != 2 || g.fhalf || g.kernels != 0 || (F != 2 && F != 4) || g.L > 3 || g.abs_type == 2) return best;
    if (adjoint && (g.freesurf || g.L > 0 || g.hout || g.bp2 || g.ckpt || g.nab < 1)) return best;
    if (g.abs_type == 1 && (g.nx < 2 * g.nab || g.nz - g.zpad < (g.freesurf ? 1 : 2) * g.nab)) return best;
    if (g.nz < F + 1 || g.nx < F + 1 || nb < 1 || npoints > R2_POINTS) return best;
    long bestc = 0;
    for (int nc = 1; nc <= (adjoint ? 2 : 4); nc *= 2) {
        for (int ntz = 1; g.nz / ntz >= F + 1 && ntz * nb <= sms; ntz++) {
            Res2d r;
            memset(&r, 0, sizeof r);
            r.F = F;
            r.nc = nc;
            r.ntz = ntz;
            r.tz = (g.nz + ntz - 1) / ntz;
            const int nzb = (r.tz + 31) / 32, cols = (R2_THREADS / 32) / nzb * nc;
            if (cols < 1 || r.tz > R2_ROWS) continue;
            r.ntx = (g.nx + cols - 1) / cols;
            if (g.nx / r.ntx < F + 1) continue;
            r.tx = (g.nx + r.ntx - 1) / r.ntx;
            r.ctas = r.ntz * r.ntx * nb;
            r.side = std::max(r.tz, r.tx);
            const int words = (adjoint ? 8 : 4) * F * (r.tz + r.tx);
            if (r.ctas > sms || words > (adjoint ? 4 : r2_words(nc)) * R2_THREADS) continue;
            const size_t field = sizeof(float) * (size_t)field_floats(F, nc) * (adjoint ? 2 : 1) * R2_NF;
            r.smem = (field + 15) / 16 * 16 + (size_t)npoints * (sizeof(int4) + sizeof(float));
            // fewest cells a thread, then words a thread, then CTAs
            const long c = 1000000L * nc + 100000L * ((words + R2_THREADS - 1) / R2_THREADS) + r.ctas;
            if (!best.ctas || c < bestc) { best = r; bestc = c; }
        }
        if (best.ctas) break;
    }
    return best;
}

// Resident launches for the nb shots of a run: how many shots a launch takes
// (r.shots; the launches follow one another) on `sms` SMs, or ctas = 0 where
// the ordinary launches take them all together in less time.
Res2d resident2d_plan(const Grid &g, int nb, int npoints, int sms)
{
    Res2d best;
    memset(&best, 0, sizeof best);
    double best_us = 0.0;
    for (int n = nb; n >= 1; n--) {
        Res2d r = resident2d_shape(g, n, npoints, std::min(sms, R2_CTAS), false);
        if (!r.ctas) continue;
        r.shots = n;
        const double us = ((nb + n - 1) / n) * resident2d_step_us(r, g.L);
        if (!best.ctas || us < best_us) { best = r; best_us = us; }
    }
    if (best.ctas && best_us > ordinary2d_step_us(g, nb)) best.ctas = 0;
    return best;
}

// the same for the adjoint loop.  us per step on a B200, resident / ordinary:
// 100 x 150 order 4 4.1 / 12.3, 300 x 450 order 4 5.5 / 13.7, 200 x 300 order 8
// 5.0 / 16.4, 300 x 400 order 8 7.5 / 16.6, 5 shots of 200 x 200 14.8 / 19.1
// (two launches), 8 shots of 100 x 150 order 4 11.8 / 13.6; ordinary alone:
// 4 shots of 240 x 480 25.8.
Res2d resident2d_adj_plan(const Grid &g, int nb, int npoints, int sms)
{
    Res2d best;
    memset(&best, 0, sizeof best);
    double best_us = (g.F == 2 ? 12.0 : 15.5) + 2.3e-5 * nb * (double)g.nz * g.nx;
    for (int n = nb; n >= 1; n--) {
        Res2d r = resident2d_shape(g, n, npoints, std::min(sms, R2_CTAS), true);
        if (!r.ctas) continue;
        r.shots = n;
        const double step = g.F == 2 ? (r.nc == 1 ? 4.1 : 5.5) : r.nc == 1 ? 5.0 : 7.5;
        const double us = ((nb + n - 1) / n) * step;
        if (us < best_us) { best = r; best_us = us; }
    }
    return best;
}

// words of a launch: two halves, four sides, 2 (4: adjoint) fields F deep
int64_t resident2d_words(const Res2d &r, bool adjoint) { return (int64_t)r.ctas * 8 * (adjoint ? 4 : 2) * r.F * r.side; }

int64_t resident2d_bytes(const Grid &g, int batch)
{
    int64_t b = 0;
    for (int nb = 1; nb <= batch; nb++)
        for (bool adjoint : {false, true})
            b = std::max(b, (int64_t)sizeof(u64) * resident2d_words(resident2d_shape(g, nb, 0, R2_CTAS, adjoint), adjoint));
    return b;
}

template <int F, int L, int NC>
static cudaError_t launch_one(const Grid &g, const Fields &f, const Res2d &r, const Res2dRun &a, cudaStream_t st)
{
    auto k = k_resident2d<F, L, NC>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, R2_SMEM);
    if (e != cudaSuccess) return e;
    void *args[4] = {(void *)&g, (void *)&f, (void *)&r, (void *)&a};
    return cudaLaunchCooperativeKernel((const void *)k, dim3(r.ctas), dim3(R2_THREADS), args, r.smem, st);
}

template <int F, int L>
static cudaError_t launch_nc(const Grid &g, const Fields &f, const Res2d &r, const Res2dRun &a, cudaStream_t st)
{
    switch (r.nc) {
    case 1: return launch_one<F, L, 1>(g, f, r, a, st);
    case 2: return launch_one<F, L, 2>(g, f, r, a, st);
    default: return launch_one<F, L, 4>(g, f, r, a, st);
    }
}

template <int F>
static cudaError_t launch_l(const Grid &g, const Fields &f, const Res2d &r, const Res2dRun &a, cudaStream_t st)
{
    switch (g.L) {
    case 0: return launch_nc<F, 0>(g, f, r, a, st);
    case 1: return launch_nc<F, 1>(g, f, r, a, st);
    case 2: return launch_nc<F, 2>(g, f, r, a, st);
    default: return launch_nc<F, 3>(g, f, r, a, st);
    }
}

// Launches of different plans (streams, threads) of a device run one after
// the other: each waits for the previous one's event, so two sets of CTAs
// that need every one of their own resident never compete for the SMs.
namespace {
struct Turn {
    std::mutex m;
    cudaEvent_t last = nullptr;
};
Turn g_turn[64];
}  // namespace

template <class Launch>
static cudaError_t in_turn(int device, cudaStream_t st, Launch launch)
{
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    Turn &turn = g_turn[device];
    std::lock_guard<std::mutex> lock(turn.m);
    cudaError_t e;
    if (!turn.last) {
        if ((e = cudaEventCreateWithFlags(&turn.last, cudaEventDisableTiming)) != cudaSuccess) return e;
    } else if ((e = cudaStreamWaitEvent(st, turn.last, 0)) != cudaSuccess) {
        return e;
    }
    if ((e = launch()) != cudaSuccess) return e;
    return cudaEventRecord(turn.last, st);
}

cudaError_t launch_resident2d(const Grid &g, const Fields &f, const Res2d &r, const Res2dRun &a, int device,
                              cudaStream_t st)
{
    return in_turn(device, st, [&] { return g.F == 2 ? launch_l<2>(g, f, r, a, st) : launch_l<4>(g, f, r, a, st); });
}

template <int F, int NC, typename T>
static cudaError_t launch_adj_one(const Grid &g, const Fields &f, const AdjFields &q, const Res2d &r, const Res2dAdj &a,
                                  cudaStream_t st)
{
    auto k = k_resident2d_adj<F, NC, T>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, R2_SMEM);
    if (e != cudaSuccess) return e;
    void *args[5] = {(void *)&g, (void *)&f, (void *)&q, (void *)&r, (void *)&a};
    return cudaLaunchCooperativeKernel((const void *)k, dim3(r.ctas), dim3(R2_THREADS), args, r.smem, st);
}

template <int F, int NC>
static cudaError_t launch_adj_t(const Grid &g, const Fields &f, const AdjFields &q, const Res2d &r, const Res2dAdj &a,
                                int prec, cudaStream_t st)
{
    if (prec == SFD_PREC_FP16) return launch_adj_one<F, NC, __half>(g, f, q, r, a, st);
    if (prec == SFD_PREC_BF16) return launch_adj_one<F, NC, __nv_bfloat16>(g, f, q, r, a, st);
    return launch_adj_one<F, NC, float>(g, f, q, r, a, st);
}

cudaError_t launch_resident2d_adj(const Grid &g, const Fields &f, const AdjFields &q, const Res2d &r, const Res2dAdj &a,
                                  int prec, int device, cudaStream_t st)
{
    return in_turn(device, st, [&] {
        if (g.F == 2) return r.nc == 1 ? launch_adj_t<2, 1>(g, f, q, r, a, prec, st) : launch_adj_t<2, 2>(g, f, q, r, a, prec, st);
        return r.nc == 1 ? launch_adj_t<4, 1>(g, f, q, r, a, prec, st) : launch_adj_t<4, 2>(g, f, q, r, a, prec, st);
    });
}

}  // namespace sfd
