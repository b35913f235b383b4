// sfd_quad3d_o8f.cu -- the 4-cell 3D forward kernels of order 8 on rows
// filled up with dummy cells.
#include "sfd_quad3d.cuh"

namespace sfd {

template void quad_update_v<ROWS_FILLED>(const Grid &, const Fields &, cudaStream_t);
template bool quad_update_s<ROWS_FILLED>(const Grid &, const Fields &, cudaStream_t, Surf);
template void quad_update_s_bnd<ROWS_FILLED>(const Grid &, const Fields &, const BndSlot &, int, int64_t, bool, cudaStream_t);

}  // namespace sfd
