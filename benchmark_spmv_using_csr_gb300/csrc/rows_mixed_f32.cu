// rows_mixed_f32.cu -- the row kernel of the mixed-precision form with FP32 storage.
#include "policies_mixed.cuh"
#include "row_kernel.cuh"

namespace spmv {

cudaError_t launch_rows_mixed_f32(const RowLaunch& l, cudaStream_t st) { return launch_rows<PolMixed<float>>(l, st); }

}  // namespace spmv
