// sfd_quad3d_adj_o4.cu -- the 4-cell 3D adjoint kernels of order 4.
#include "sfd_quad3d_adj.cuh"

namespace sfd {

template void quad_update_adj<ROWS_O4>(const Grid &, const Fields &, const AdjFields &, bool, int, cudaStream_t);

}  // namespace sfd
