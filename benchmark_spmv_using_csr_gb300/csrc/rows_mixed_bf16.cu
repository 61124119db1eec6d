// rows_mixed_bf16.cu -- the row kernel of the mixed-precision form with BF16 storage.
#include "policies_mixed.cuh"
#include "row_kernel.cuh"

namespace spmv {

cudaError_t launch_rows_mixed_bf16(const RowLaunch& l, cudaStream_t st) { return launch_rows<PolMixed<__nv_bfloat16>>(l, st); }

}  // namespace spmv
