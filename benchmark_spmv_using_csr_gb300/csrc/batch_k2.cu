// batch_k2.cu -- the batched form's work-list kernels at 2 right-hand sides.
#include "batch_kernel.cuh"

namespace spmv {

template int batch_work_grid<2>(const BatchWork&, int);
template cudaError_t launch_batch_work<2>(const BatchLaunch&, const BatchWork&, int, cudaStream_t);

}  // namespace spmv
