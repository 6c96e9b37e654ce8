// Instantiations of recurrent_wide_bwd.cuh for one cell.
#include "recurrent_wide_bwd.cuh"

namespace frnn {
template int launch_bwd_wide_cell<kGRU>(const BwdParams&, const void*, const float*, const float*, const float*, int, int, int, cudaStream_t, bool);
}  // namespace frnn
