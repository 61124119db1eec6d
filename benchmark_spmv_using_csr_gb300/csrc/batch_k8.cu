// batch_k8.cu -- the batched form's work-list kernels at 8 right-hand sides.
#include "batch_kernel.cuh"

namespace spmv {

template int batch_work_grid<8>(const BatchWork&, int);
template cudaError_t launch_batch_work<8>(const BatchLaunch&, const BatchWork&, int, cudaStream_t);

}  // namespace spmv
