// sfd_gradient.cu -- the accumulated gradient sums turned into the gradient
// of the chosen parameters on the device (transf_grad,
// src/calc_grad.c:975-1107).
//
// One thread per cell: the FP64 sums of the batch's shots are added in shot
// order, taken through the chain rule in FP64 with the FP32 parameters the
// stencils use, and rounded once to FP32.  Reads 24 bytes per shot copy and
// 12 of parameters and writes 12 per cell, so it is bound by HBM; the three
// FP32 arrays that cross to the host are half the bytes of the sums.  With
// the sums copied and transformed by the host, a gradient pass of 120 steps
// on 100 x 200 x 200 cells took 165 ms, with this kernel 104 ms; 8 shots of
// 300 x 1000 (400 steps) 144 and 130 ms.
#include <cuda_runtime.h>

#include "sfd_internal.h"
#include "sfd_kernels.h"

namespace sfd {

typedef int64_t i64;

__global__ void __launch_bounds__(256) k_gradient_out(GradOut o)
{
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < o.count; q += (i64)gridDim.x * blockDim.x) {
        const i64 u = o.first + q, i = u / o.nz * o.pitch + u % o.nz;
        double s[3];   // M, mu, rho
#pragma unroll
        for (int k = 0; k < 3; k++) {
            s[k] = o.sum[k][i];
            for (int b = 1; b < o.ncopy; b++) s[k] += o.sum[k][b * o.copy + i];
        }
        if (o.par_type >= 0) {
            const double rho = 1.0 / o.rho[i] * o.dt / o.dh;
            const double M = o.M[i] * o.dh / o.dt, mu = o.mu[i] * o.dh / o.dt;
#pragma unroll
            for (int k = 0; k < 3; k++) s[k] /= o.dt;
            if (o.par_type != 1) {
                s[2] += M / rho * s[0];
                if (mu > 0) s[2] += mu / rho * s[1];
                s[0] *= 2.0 * sqrt(o.par_type == 0 ? rho * M : M / rho);
                s[1] *= 2.0 * sqrt(o.par_type == 0 ? rho * mu : mu / rho);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; k++) o.out[k][q] = (float)s[k];
    }
}

void launch_gradient_out(const GradOut &o, cudaStream_t st)
{
    if (o.count <= 0) return;
    i64 blocks = (o.count + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    k_gradient_out<<<(unsigned)blocks, 256, 0, st>>>(o);
}

}  // namespace sfd
