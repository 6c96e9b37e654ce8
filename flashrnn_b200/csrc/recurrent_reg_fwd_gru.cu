// Instantiations of recurrent_reg_fwd.cuh for one cell.
#include "recurrent_reg_fwd.cuh"

namespace frnn {
template int launch_fwd_reg_cell<kGRU>(const FwdParams&, const void*, int, cudaStream_t, int, bool);
}  // namespace frnn
