// sfd_launch.cuh -- launch helpers shared by the kernel files: grid sizes,
// batched dispatch and programmatic dependent launch.
#pragma once

#include <cstdlib>
#include <utility>

#include <cuda_runtime.h>

#include "sfd_internal.h"

namespace sfd {

static inline unsigned cdiv(long a, long b) { return (unsigned)((a + b - 1) / b); }


// batched launches (several shots) use the MB = true instantiations
#define MB_DISPATCH(g, ...)                                                     \
    if ((g).nb > 1) { constexpr bool MBV = true; __VA_ARGS__; }                  \
    else { constexpr bool MBV = false; __VA_ARGS__; }

// Programmatic dependent launch for the single-shot 3D loop: the receivers
// and the sources are launched with programmatic stream serialization, so
// they may be resident while the previous kernel drains its last wave; they
// wait (pdl_wait) before they read or write anything the previous kernels
// touch, and read those fields with plain loads (a read-only-path load may be
// hoisted above the wait).  The velocity and stress kernels are ordinary
// launches: their stencils are faster through the read-only path than any
// overlap gains (256^3, L=2: 911 against 919 us per step).  On unless the
// environment sets SEISCL_B200_PDL=0.
static bool pdl_enabled()
{
    static const bool on = [] {
        const char *e = std::getenv("SEISCL_B200_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args &&...args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = 0;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, std::forward<Args>(args)...);
}

// kernel<<<grid, block, 0, st>>>(args...), with programmatic serialization when `pdl`
template <typename... KArgs, typename... Args>
static void launch_maybe_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t st,
                             Args &&...args)
{
    if (pdl) launch_pdl(kernel, grid, block, st, std::forward<Args>(args)...);
    else kernel<<<grid, block, 0, st>>>(std::forward<Args>(args)...);
}

}  // namespace sfd
