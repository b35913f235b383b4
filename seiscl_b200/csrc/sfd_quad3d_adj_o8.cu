// sfd_quad3d_adj_o8.cu -- the 4-cell 3D adjoint kernels of order 8 on rows
// of whole quads.
#include "sfd_quad3d_adj.cuh"

namespace sfd {

template void quad_update_adj<ROWS_WHOLE>(const Grid &, const Fields &, const AdjFields &, bool, int, cudaStream_t);

}  // namespace sfd
