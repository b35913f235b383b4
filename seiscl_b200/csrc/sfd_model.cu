// sfd_model.cu -- material parameters prepared on the device: the transforms
// and averages of transform_model (sfd_setup.cpp; assign_modeling_case.c:
// 50-535), its checks, and the few values the host needs back.
//
// One thread per cell forms every stored parameter from the raw inputs in
// FP64 and rounds once.  Each operation is written with its rounding
// (__dmul_rn, ...) in the host's order, so the results are the host's bit for
// bit.  The averages recompute their neighbours' values instead of reading
// them back: 3 to 5 input floats a cell come in and 14 go out, bound by the
// host-to-device copy of the inputs.  On the host a model of 256^3 cells with
// attenuation took 2.4 s on one core, 240 x 480 10 ms; here a whole
// set_model call takes 0.4 ms at 240 x 480 and 2.8 ms at 128^3 with attenuation.
#include <cuda_runtime.h>

#include "sfd_internal.h"
#include "sfd_kernels.h"

namespace sfd {

typedef int64_t i64;

namespace {

struct Cell {
    double M, mu, b, taup, taus;
};

__device__ __forceinline__ Cell cell_of(const ModelIn &m, i64 i)
{
    const double r = m.rho[i], a = m.a ? (double)m.a[i] : 0.0, b = m.b ? (double)m.b[i] : 0.0;
    auto modulus = [&](double v) {
        if (m.par_type == 1) return __ddiv_rn(__dmul_rn(v, m.dt), m.dh);
        const double q = m.par_type == 2 ? __ddiv_rn(v, r) : v;
        return __ddiv_rn(__dmul_rn(__dmul_rn(__dmul_rn(q, q), r), m.dt), m.dh);
    };
    Cell c = {modulus(a), modulus(b), __ddiv_rn(m.dt, __dmul_rn(m.dh, r)), 0.0, 0.0};
    if (m.L > 0) {
        c.taup = m.taup[i];
        c.taus = m.taus[i];
        double sum = 0.0;
        for (int l = 0; l < m.L; l++) sum = __dadd_rn(sum, __dmul_rn(m.wl[l], c.taup));
        c.M = __ddiv_rn(c.M, __dadd_rn(1.0, sum));
        c.mu = __ddiv_rn(c.mu, __dadd_rn(1.0, __dmul_rn(m.sumu, c.taus)));
    }
    return c;
}
__device__ __forceinline__ double mean2(double a, double b) { return __dmul_rn(0.5, __dadd_rn(a, b)); }
__device__ __forceinline__ double harmonic4(double a, double b, double c, double d)
{
    const double s = __dadd_rn(__dadd_rn(__dadd_rn(__ddiv_rn(1.0, a), __ddiv_rn(1.0, b)), __ddiv_rn(1.0, c)),
                               __ddiv_rn(1.0, d));
    return __ddiv_rn(4.0, s);
}
__device__ __forceinline__ double mean4(double a, double b, double c, double d)
{
    return __dmul_rn(0.25, __dadd_rn(__dadd_rn(__dadd_rn(a, b), c), d));
}

}  // namespace

// checks of the slab's planes x0 .. x0+xs-1: out.bad_rho set where a density
// is not positive; the largest M b and mu b (bits of non-negative doubles
// order as integers; negative and NaN products, whose roots are NaN, drop
// out as they do from a running maximum)
__global__ void __launch_bounds__(256) k_model_check(ModelIn m, ModelCheck *out)
{
    const i64 n = (i64)m.xs * m.ny * m.nz;
    double vp = 0.0, vs = 0.0;
    bool bad = false;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        if (!(m.rho[i] > 0.0f)) { bad = true; continue; }
        const Cell c = cell_of(m, i);
        const double p = __dmul_rn(c.M, c.b), s = __dmul_rn(c.mu, c.b);
        if (p > vp) vp = p;
        if (s > vs) vs = s;
    }
    if (bad) atomicOr(&out->bad_rho, 1);
    if (vp > 0.0) atomicMax(&out->mb, (unsigned long long)__double_as_longlong(vp));
    if (vs > 0.0) atomicMax(&out->mub, (unsigned long long)__double_as_longlong(vs));
}

// every stored parameter of planes x0 .. x0+xs-1 (the slab holds plane x0+xs
// too where the grid has one)
__global__ void __launch_bounds__(256) k_model_params(ModelIn m, ModelOut o, ModelCheck *check)
{
    const i64 n = (i64)m.xs * m.ny * m.nz;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(i % m.nz), j = (int)(i / m.nz % m.ny), x = (int)(i / ((i64)m.nz * m.ny));
        const bool lx = m.x0 + x == m.nx - 1, ly = j == m.ny - 1, lz = k == m.nz - 1;   // last slabs
        const i64 sx = (i64)m.ny * m.nz, sy = m.nz;
        const i64 q = (((i64)(m.x0 + x)) * m.ny + j) * m.pitch + k;
        const Cell c = cell_of(m, i);
        auto put = [&](int id, double v) { o.p[id][q] = __double2float_rn(v); };
        put(PM, c.M);
        put(PMU, c.mu);
        put(PRHO, c.b);
        put(PTAUP, c.taup);
        put(PTAUS, c.taus);
        if (k == 0 && !(__double2float_rn(c.mu) > 0.0f)) atomicOr(&check->top_mu_zero, 1);
        const bool three = m.nd == 3;
        // neighbours that some average reads
        const Cell cx = lx ? c : cell_of(m, i + sx), cz = lz ? c : cell_of(m, i + 1);
        put(PRIP, lx ? c.b : mean2(c.b, cx.b));
        put(PRKP, lz ? c.b : mean2(c.b, cz.b));
        // two-direction means: the first direction's last slab is copied, the
        // rest of the second one's stays zero
        if (lx) {
            put(PMUIPKP, c.mu);
            put(PTAUSIPKP, c.taus);
        } else if (lz) {
            put(PMUIPKP, 0.0);
            put(PTAUSIPKP, 0.0);
        } else {
            const Cell d = cell_of(m, i + sx + 1);
            put(PMUIPKP, harmonic4(c.mu, cx.mu, cz.mu, d.mu));
            put(PTAUSIPKP, mean4(c.taus, cx.taus, cz.taus, d.taus));
        }
        if (!three) {
            for (int id : {PRJP, PMUIPJP, PMUJPKP, PTAUSIPJP, PTAUSJPKP}) put(id, 0.0);
            continue;
        }
        const Cell cy = ly ? c : cell_of(m, i + sy);
        put(PRJP, ly ? c.b : mean2(c.b, cy.b));
        if (lx) {
            put(PMUIPJP, c.mu);
            put(PTAUSIPJP, c.taus);
        } else if (ly) {
            put(PMUIPJP, 0.0);
            put(PTAUSIPJP, 0.0);
        } else {
            const Cell d = cell_of(m, i + sx + sy);
            put(PMUIPJP, harmonic4(c.mu, cx.mu, cy.mu, d.mu));
            put(PTAUSIPJP, mean4(c.taus, cx.taus, cy.taus, d.taus));
        }
        if (ly) {
            put(PMUJPKP, c.mu);
            put(PTAUSJPKP, c.taus);
        } else if (lz) {
            put(PMUJPKP, 0.0);
            put(PTAUSJPKP, 0.0);
        } else {
            const Cell d = cell_of(m, i + sy + 1);
            put(PMUJPKP, harmonic4(c.mu, cy.mu, cz.mu, d.mu));
            put(PTAUSJPKP, mean4(c.taus, cy.taus, cz.taus, d.taus));
        }
    }
}

__global__ void k_scale(const float *src, float *dst, i64 n, float s)
{
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) dst[i] = src[i] * s;
}

__global__ void k_gather(const float *src, const i64 *at, float *out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = src[at[i]];
}

static unsigned blocks_of(i64 n) { return (unsigned)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8); }

void launch_model_check(const ModelIn &m, ModelCheck *out, cudaStream_t st)
{
    k_model_check<<<blocks_of((i64)m.xs * m.ny * m.nz), 256, 0, st>>>(m, out);
}
void launch_model_params(const ModelIn &m, const ModelOut &o, ModelCheck *check, cudaStream_t st)
{
    k_model_params<<<blocks_of((i64)m.xs * m.ny * m.nz), 256, 0, st>>>(m, o, check);
}
void launch_scale(const float *src, float *dst, int64_t n, float s, cudaStream_t st)
{
    if (n > 0) k_scale<<<blocks_of(n), 256, 0, st>>>(src, dst, n, s);
}
void launch_gather(const float *src, const int64_t *at, float *out, int n, cudaStream_t st)
{
    if (n > 0) k_gather<<<(n + 127) / 128, 128, 0, st>>>(src, (const i64 *)at, out, n);
}

}  // namespace sfd
