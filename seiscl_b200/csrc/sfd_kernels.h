// sfd_kernels.h -- launchers of the FDTD kernels (host side).
#pragma once

#include <cuda_runtime.h>

#include "sfd_internal.h"

namespace sfd {

struct BndSlot {            // saved-boundary stores, by value
    void *p[NW];
    int nfield;
    int fields[NW];
};

void launch_update_v(const Grid &g, const Fields &f, cudaStream_t st);
bool launch_update_v_fast(const Grid &g, const Fields &f, cudaStream_t st);
bool launch_update_v_async(const Grid &g, const Fields &f, cudaStream_t st);
bool launch_update_s_fast(const Grid &g, const Fields &f, cudaStream_t st);
int fast3d_xchunk(const Grid &g);
bool launch_update_v_tma(const Grid &g, const Fields &f, cudaStream_t st);
bool launch_update_s_tma(const Grid &g, const Fields &f, cudaStream_t st);
bool tma_ready(const Grid &g, const Fields &f);  // the TMA kernels will run for this plan
int tma_take_status();      // 1 if a TMA stage of the last launches never arrived (and clears it)
// Free surface in a stress update's launch: not at all, in the form whose
// products are added in one rounding, or with the roundings of the separate
// launch (k_surf3d: checkpoint recomputation, boundary saving, FP16 fields,
// rows that are no whole quads).  The two differ in the last bits of
// viscoelastic 3D runs only.
enum Surf { SURF_NONE = 0, SURF_FOLD, SURF_APART };
// kinds of rows of the 4-cell 3D kernels, each with its own instances: order 4;
// order 8 in whole quads; order 8 filled up with dummy cells
constexpr int ROWS_O4 = 2, ROWS_WHOLE = 4, ROWS_FILLED = 5;
__host__ __device__ constexpr int half_width(int rows) { return rows & ~1; }
__host__ __device__ constexpr bool whole_rows(int rows) { return rows == ROWS_WHOLE; }
// 4-cell vectorised 3D kernels (sfd_quad3d.cuh);
// quad_update_s returns whether the launch applied the free surface
template <int R> void quad_update_v(const Grid &g, const Fields &f, cudaStream_t st);
// the elastic single-shot update that also saves the boundary shells
template <int R>
void quad_update_s_bnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, bool surf, cudaStream_t st);
// the same where it applies (false: not launched)
bool launch_update_s_bnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, cudaStream_t st);
template <int R> bool quad_update_s(const Grid &g, const Fields &f, cudaStream_t st, Surf surf);
template <int R>
void quad_update_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st);
// 3D stress-update family of a plan: 0 not 3D, 1 general, 2 register-blocked,
// 3 TMA-pipelined, 4 streaming, 5 4-cell vectorised
int stress_family(const Grid &g, const Fields &f);
// fold: single-shot 4-cell kernels may apply the free surface in the same
// launch (true returned: the caller skips launch_surface)
bool launch_update_s(const Grid &g, const Fields &f, cudaStream_t st, Surf fold = SURF_NONE);
// Fused 3D forward step (velocity, stress, free surface in one launch; see
// sfd_kernels.cu).  Work units = ntz x nty x nchunk; units = 0 when the plan's
// grid does not take it (sfd_config.kernels 6; 3D, 8th order, nz % 4 == 0,
// FP32 fields, L <= 3, nx >= 5).  nchunk = x planes (one unit per tile and
// plane).
struct FusedShape {
    int ntz, nty, nchunk;
    int64_t units;
};
FusedShape fused_shape(const Grid &g);
// sync: 1 + units ints (a ticket counter, one flag per unit), zeroed before
// step 0 of a run; t: the step's index in the run.  False: not launched.
bool launch_fused_step(const Grid &g, const Fields &f, int *sync, int t, cudaStream_t st);
int fused_take_status();    // 1 if a fused step's wait ran out (and clears it)
void launch_surface(const Grid &g, const Fields &f, int pdir, cudaStream_t st);
// 2D P-SV and acoustic forward: stress update, free surface, receivers of
// step tl.t and sources of step tl.tsrc in one launch (false: not 2D)
bool launch_update_s_step(const Grid &g, const Fields &f, const StepTail &tl, cudaStream_t st);
// 4-cell vectorised 2D P-SV kernels (sfd_quad2d.cu).  The stress update saves
// the boundary shells in b (nfield = 0: none) at offset tofs and then, with
// surf, applies the free surface; the adjoint launcher returns false where it
// does not apply (memory variables, Hessian)
bool quad2d_ok(const Grid &g);
void launch_quad2d_v(const Grid &g, const Fields &f, cudaStream_t st);
void launch_quad2d_s(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, bool surf, cudaStream_t st);
bool launch_quad2d_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st);
// 2D P-SV modelling with the wave fields resident on chip (sfd_resident2d.cu)
struct Res2d {              // tiles of a launch: ctas = ntz x ntx x shots, 0 where it does not apply
    int ntz, ntx, tz, tx;   // tiles along z and x, the largest tile
    int side, ctas, F, nc;  // longer side of a tile, CTAs, half width, cells per thread
    int shots;              // shots of a launch
    size_t smem;
};
constexpr long long RES2D_WAIT_NS = 2000000000LL;
struct Res2dRun {           // a segment of the time loop: steps t0 .. t1-1 of tmax
    PointSet rec, src;
    const float *stf;       // [nsrc][nt_total]
    float *out;             // [nsel][nrec][nt_total]
    unsigned outmask;
    int nt_total, t0, t1, tmax;
    int shot0;              // first shot of the launch
    BndSlot bnd;            // boundary shells to save (nfield = 0: none), in storage type prec
    int prec;
    unsigned long long *words;   // exchange words, zeroed before the run's first segment
    int *first_bad, *status;
    long long wait_ns = RES2D_WAIT_NS;   // bound of one wait
};
constexpr int RES2D_SEGMENT = 256;   // steps of one launch: bounds how long it holds the SMs
constexpr int RES2D_SMS = 148;       // most CTAs of a launch, one per SM
// launches for the nb shots of a run on the `sms` SMs a process has
Res2d resident2d_plan(const Grid &g, int nb, int npoints, int sms);
Res2d resident2d_adj_plan(const Grid &g, int nb, int npoints, int sms);
int64_t resident2d_words(const Res2d &r, bool adjoint);
int64_t resident2d_bytes(const Grid &g, int batch);   // exchange words of launches of up to `batch` shots
struct Res2dAdj {           // a segment of the adjoint loop: steps t0, t0-1 .. t1+1 of tmax-1 .. tmin+1
    PointSet rec, src;
    const float *stf, *res; // [nsrc][nt_total], [nsel][nrec][nt_total]
    unsigned outmask;
    int nt_total, t0, t1, tmax, tmin, shot0;
    unsigned long long *words;
    int *first_bad, *status;
    long long wait_ns = RES2D_WAIT_NS;
};
// q.bnd: the saved boundaries from step 0
cudaError_t launch_resident2d_adj(const Grid &g, const Fields &f, const AdjFields &q, const Res2d &r, const Res2dAdj &a,
                                  int prec, int device, cudaStream_t st);
cudaError_t launch_resident2d(const Grid &g, const Fields &f, const Res2d &r, const Res2dRun &a, int device,
                              cudaStream_t st);
void launch_savebnd(const Grid &g, const Fields &f, const BndSlot &b, int prec, int64_t tofs, cudaStream_t st);
void launch_update_adj(const Grid &g, const Fields &f, const AdjFields &a, bool stress, int prec, cudaStream_t st);
void launch_surface_adj(const Grid &g, const Fields &f, const AdjFields &a, float *q, cudaStream_t st);
void launch_sources(const Grid &g, const Fields &f, const PointSet &s, const float *src, int nt_total, int t,
                    int pdir, cudaStream_t st);
void launch_record(const Grid &g, const Fields &f, const PointSet &r, float *out, int nt_total, int t,
                   unsigned outmask, cudaStream_t st);
// receivers of step t and sources of step tsrc (-1: none) in one launch, for
// shots without a receiver on a source's cell
void launch_record_sources(const Grid &g, const Fields &f, const PointSet &r, float *out, int nt_total, int t,
                           unsigned outmask, const PointSet &s, const float *src, int tsrc, cudaStream_t st);
// adjoint sources of step t into the adjoint fields and, in the same launch,
// the sources of step tsrc (-1: none) out of the forward fields
void launch_residuals(const Grid &g, const Fields &f, const AdjFields &a, const PointSet &r, const float *res,
                      int nt_total, int t, unsigned outmask, const PointSet &s, const float *src, int tsrc,
                      cudaStream_t st);

// instability detection: if any of the n values of a wave field (FP32, or
// FP16 when g.fhalf) is not finite, *first = min(*first, t)
void launch_finite_check(const Grid &g, const float *fld, int64_t n, int t, int *first, cudaStream_t st);
constexpr int FINITE_CHECK_EVERY = 64;   // time steps between checks

// movie snapshot: the physical cells of one wave field, divided by its
// storage scale, into dst [nx][ny][nz]
void launch_movie(const Grid &g, const float *fld, float inv_scale, float *dst, cudaStream_t st);

// checkpointed gradients: copies of wave fields / memory variables between
// their FP32 arrays and stores of the saved-boundary precision (FP16 stores
// scaled by powers of two)
struct PackSet {
    static constexpr int MAXARR = NW + NR;
    const void *src[MAXARR];
    void *dst[MAXARR];
    int64_t n[MAXARR];
    float scale[MAXARR];   // applied to each value on the way
    int narr;
};
void launch_pack(const PackSet &ps, int prec, bool unpack, cudaStream_t st, bool half_src = false);

// material parameters from raw inputs (sfd_model.cu)
struct ModelIn {            // a slab of x planes x0 .. x0+xs-1 (and the next, where there is one)
    const float *a, *b, *rho, *taup, *taus;   // raw inputs of the slab, [planes][ny][nz]; a or b may be null
    int nd, nz, ny, nx, pitch;   // grid; row length of the stored parameters
    int x0, xs, L, par_type;
    double dt, dh, sumu, wl[8];
};
struct ModelOut {
    float *p[NPAR];
};
struct ModelCheck {         // zeroed before use; mb, mub: bits of the largest M b, mu b
    unsigned long long mb, mub;
    int bad_rho, top_mu_zero;
};
void launch_model_check(const ModelIn &m, ModelCheck *out, cudaStream_t st);
void launch_model_params(const ModelIn &m, const ModelOut &o, ModelCheck *check, cudaStream_t st);
void launch_scale(const float *src, float *dst, int64_t n, float s, cudaStream_t st);
void launch_gather(const float *src, const int64_t *at, float *out, int n, cudaStream_t st);

// gradient sums -> gradient of the parameters (sfd_gradient.cu)
struct GradOut {
    const double *sum[3];   // M, mu, rho: ncopy copies, `copy` apart, of rows of `pitch` with nz cells each
    int ncopy, nz, pitch;
    int64_t copy;
    int64_t n, first, count;   // cells of a copy; the range of this launch
    int par_type;           // param_type of the chain rule, -1: the sums as they are
    const float *rho, *M, *mu;
    double dt, dh;
    float *out[3];          // [count] each: M, mu, rho or their param_type counterparts
};
void launch_gradient_out(const GradOut &o, cudaStream_t st);

// DFT gradient (sfd_dft.cu)
struct DftSet {             // variables transformed by one accumulation launch
    const float *v[NW + NR];
    float2 *f[NW + NR];
    int64_t n[NW + NR];     // elements of each variable (nvol, or L*nvol)
    int nvar, nf;
    float re[MAXFREQ], im[MAXFREQ];
};
void launch_savefreqs(const DftSet &d, cudaStream_t st);
struct GradDft {            // inputs of the per-cell assembly
    const float2 *fw[2][NW], *fr[2][NR];
    int nf, par_type;
    float w[MAXFREQ];       // angular frequency of each bin (FP32, as the reference forms it)
    float tausig[8];
    float al, ntnyq;
};
void launch_calc_grad(const Grid &g, const Fields &f, const AdjFields &a, const GradDft &d, cudaStream_t st);

}  // namespace sfd
