// rows_f64.cu -- the plain row kernel instantiated for PolF64, one translation unit per value type.
#include "policies_plain.cuh"
#include "row_kernel.cuh"

namespace spmv {

cudaError_t launch_rows_f64(const RowLaunch& l, cudaStream_t st) { return launch_rows<PolF64>(l, st); }

}  // namespace spmv
