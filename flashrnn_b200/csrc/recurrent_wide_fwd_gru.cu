// Instantiations of recurrent_wide_fwd.cuh for one cell.
#include "recurrent_wide_fwd.cuh"

namespace frnn {
template int launch_fwd_wide_cell<kGRU>(const FwdParams&, const void*, int, int, int, cudaStream_t, bool);
}  // namespace frnn
