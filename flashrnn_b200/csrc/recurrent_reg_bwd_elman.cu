// Instantiations of recurrent_reg_bwd.cuh for one cell.
#include "recurrent_reg_bwd.cuh"

namespace frnn {
template int launch_bwd_reg_cell<kElman>(const BwdParams&, const void*, const float*, const float*, const float*, int, cudaStream_t, int, bool);
}  // namespace frnn
