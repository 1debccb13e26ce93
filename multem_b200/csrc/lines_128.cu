// Line-pass kernels for lines of 128 points (see line_kernels.cuh).
#include "line_kernels.cuh"

namespace mtb {
template void rows_dispatch_mode<128>(RowMode, const RowArgs&, int, cudaStream_t);
template void cols_dispatch_flags<128>(int, const ColArgs&, int, cudaStream_t);
template int cols_det_width<128>();
template bool rows_has_variant<128>(int, int, bool);
template bool cols_has_variant<128>(int);
}  // namespace mtb
