// Line-pass kernels for lines of 512 points (see line_kernels.cuh).
#include "line_kernels.cuh"

namespace mtb {
template void rows_dispatch_mode<512>(RowMode, const RowArgs&, int, cudaStream_t);
template void cols_dispatch_flags<512>(int, const ColArgs&, int, cudaStream_t);
template int cols_det_width<512>();
template bool rows_has_variant<512>(int, int, bool);
template bool cols_has_variant<512>(int);
}  // namespace mtb
