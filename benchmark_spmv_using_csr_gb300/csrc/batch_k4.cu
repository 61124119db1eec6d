// batch_k4.cu -- the batched form's work-list kernels at 4 right-hand sides.
#include "batch_kernel.cuh"

namespace spmv {

template int batch_work_grid<4>(const BatchWork&, int);
template cudaError_t launch_batch_work<4>(const BatchLaunch&, const BatchWork&, int, cudaStream_t);

}  // namespace spmv
