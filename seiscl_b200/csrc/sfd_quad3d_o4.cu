// sfd_quad3d_o4.cu -- the 4-cell 3D forward kernels of order 4.
#include "sfd_quad3d.cuh"

namespace sfd {

template void quad_update_v<ROWS_O4>(const Grid &, const Fields &, cudaStream_t);
template bool quad_update_s<ROWS_O4>(const Grid &, const Fields &, cudaStream_t, Surf);
template void quad_update_s_bnd<ROWS_O4>(const Grid &, const Fields &, const BndSlot &, int, int64_t, bool, cudaStream_t);

}  // namespace sfd
