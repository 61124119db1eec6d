// batch_k1.cu -- the batched form's kernels over work lists at one right-hand side.
//
// Tile workers as at 2 to 8 right-hand sides; the row blocks, by the lane layout that suits them, in
// one launch of the row kernel (row_kernel.cuh) per layout, each the programmatic dependent of the
// one before: it starts as that one drains, which hides the tails.  A layout known at compile time is
// what makes the difference: with a run-time one a non-zero takes about 20 instructions, as many as
// the tile kernel (64 matrices: 131 us).
//
// Bound by memory in the regular members (27-point stencils 6830 GB/s, 32 x 32 blocks 6650) and by
// latency in the tile workers'.  Measured against the tile kernel over the whole batch: 128 matrices of
// five kinds 220 -> 199 us, 64 124 -> 110, 16 58 -> 50, 2 12.6 -> 6.9; 5 (3.3 M non-zeros) 27 -> 29;
// 64 matrices of one kind: 27-point stencils 107 -> 76.5, 32 x 32 blocks 125 -> 97, 5-point stencils
// 45 -> 29, uniform density 147 -> 107.  Fewer tile workers at a time, to leave room for row workers
// beside them, were slower (3 CTAs per SM instead of 6: 128 matrices 220 us).
#include "batch_kernel.cuh"
#include "policies_mixed.cuh"

namespace spmv {

cudaError_t launch_rows_listed(const RowLaunch& l, cudaStream_t st) {
#define SPMV_LIST_FORM(T, NG)                         \
    if (l.form.lanes == T && l.form.groups == NG)     \
        return launch_row_kernel<PolMixed<float>, T, NG, true>(l, st)
    SPMV_LIST_FORM(1, 2);
    SPMV_LIST_FORM(1, 4);
    SPMV_LIST_FORM(1, 7);
    SPMV_LIST_FORM(2, 4);
    SPMV_LIST_FORM(2, 7);
    SPMV_LIST_FORM(4, 7);
#undef SPMV_LIST_FORM
    return cudaErrorInvalidValue;
}

// the tile workers' carry records, once every kernel before is done
__global__ void k_batch_calibrate(const int* rec_row, const VecD<1>* rec_val, int nrec, VecF<1>* y,
                                  int m, uint32_t* err) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int warp = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int base = warp * 32; base < nrec; base += warps * 32)
        calibrate_records<PolMixedK<1>>(rec_row, rec_val, nrec, base, y, m, err);
}

template int batch_work_grid<1>(const BatchWork&, int);

template <>
cudaError_t launch_batch_work<1>(const BatchLaunch& l, const BatchWork& b, int seg,
                                 cudaStream_t st) {
    cudaError_t e = launch_batch_tiles<1>(l, b, seg, st);
    if (e != cudaSuccess) return e;
    RowLaunch r;
    r.row_ptr = l.row_ptr;
    r.col = l.col;
    r.val = l.val;
    r.x = l.x;
    r.y = l.y;
    r.ticket = nullptr;
    r.err = l.err;
    r.m = l.m;
    r.nnz = l.nnz;
    for (int i = 0; i < b.nlists; ++i) {
        r.form = b.lists[i].form;
        r.blocks = b.blocks + b.lists[i].first;
        r.nblocks = b.lists[i].count;
        r.dependent = i > 0 || b.ntiles > 0;
        e = launch_rows_listed(r, st);
        if (e != cudaSuccess) return e;
    }
    if (b.ntiles > 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid_for(b.ntiles, 256, 8));
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_batch_calibrate, b.rec_row,
                               static_cast<const VecD<1>*>(b.rec_val), b.ntiles,
                               static_cast<VecF<1>*>(l.y), l.m, l.err);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace spmv
