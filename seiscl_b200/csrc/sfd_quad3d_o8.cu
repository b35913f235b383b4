// sfd_quad3d_o8.cu -- the 4-cell 3D forward kernels of order 8 on rows
// of whole quads.
#include "sfd_quad3d.cuh"

namespace sfd {

template void quad_update_v<ROWS_WHOLE>(const Grid &, const Fields &, cudaStream_t);
template bool quad_update_s<ROWS_WHOLE>(const Grid &, const Fields &, cudaStream_t, Surf);
template void quad_update_s_bnd<ROWS_WHOLE>(const Grid &, const Fields &, const BndSlot &, int, int64_t, bool, cudaStream_t);

}  // namespace sfd
