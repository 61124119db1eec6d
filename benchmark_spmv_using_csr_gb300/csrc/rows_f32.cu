// rows_f32.cu -- the plain row kernel instantiated for PolF32, one translation unit per value type.
#include "policies_plain.cuh"
#include "row_kernel.cuh"

namespace spmv {

cudaError_t launch_rows_f32(const RowLaunch& l, cudaStream_t st) { return launch_rows<PolF32>(l, st); }

}  // namespace spmv
