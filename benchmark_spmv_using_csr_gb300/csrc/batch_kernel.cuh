// batch_kernel.cuh -- the batched form's kernels over work lists (at one right-hand side the row
// workers' is another one, batch_k1.cu).
//
// The matrices of a batch differ in structure, so no one kernel suits the concatenated matrix.
// Blocks of 256 rows whose rows are short, even and local go to row workers (lanes on whole rows, as
// row_kernel.cuh), a kernel per lane layout; the runs of blocks between them are cut into tile workers
// (consecutive non-zeros, tile_kernel.cuh) over a window of the matrix: row_ptr and y from the run's
// first row, slots outside its non-zeros padding.  The tile workers' kernel runs first; each row
// kernel, a programmatic dependent of the one before, fills the SMs as that drains, and the last one
// ends by adding the carry records.
//
// Measured on 64 matrices of five kinds (39 M non-zeros) against the tile kernel over the whole
// batch: 171 -> 120 us at 2 right-hand sides, 271 -> 149 us at 4, 395 -> 230 us at 8 (memory 71 us;
// the FP32 pipe 78 us for 10 operations per non-zero and right-hand side).  By kind at 8: 27-point
// stencils 521 -> 234 us, 32 x 32 blocks 543 -> 307, 5-point stencils 152 -> 68, uniform density 280
// -> 194, power-law rows (all tile workers) 328 -> 315.  What is saved is the tile kernel's segmented
// scan of 64-byte accumulators, about 35 instructions per non-zero.  One row kernel for all layouts,
// the lanes per row a run-time value, spends as many instructions on indexes as on arithmetic (34 per
// non-zero): 130, 163 and 250 us.  Row and tile workers in one kernel were slower than either alone
// (K = 8: 563-980 us): the code does not fit the instruction cache, and its registers leave 16 warps
// for the tile workers.
#pragma once
#include "policies_batched.cuh"
#include "row_kernel.cuh"

namespace spmv {

constexpr int BATCH_WARPS = 4;
template <int K>
struct BatchArgs {
    TileArgs<PolMixedK<K>> t;  // the whole batch; windows are cut from it
    const TileWork* __restrict__ tiles;
    int ntiles;
};

// ---- tile workers ----
// OH, XL2: the kernel variant, chosen from the tile workers' own rows and columns.  With rows of 512
// near columns between 27-point stencils, half of the non-zeros each, the per-slot form with L2-only
// gathers takes 107 us at one right-hand side and 168 at two, the variant of these rows 60 and 88.
template <int K, int S, bool OH, bool XL2>
__device__ __forceinline__ void batch_tile_workers(const BatchArgs<K>& a, uint32_t* words, int* rowof) {
    using P = PolMixedK<K>;
    const int lane = threadIdx.x & 31;
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    for (;;) {
        int w = 0;
        if (lane == 0) w = atomicAdd(a.t.ticket, 1);
        w = __shfl_sync(SPMV_FULL_MASK, w, 0);
        if (w >= a.ntiles) break;
        const TileWork d = a.tiles[w];
        TileArgs<P> t = a.t;
        t.row_ptr = a.t.row_ptr + d.row0;
        t.y = a.t.y + d.row0;
        t.m = d.row1 - d.row0;
        t.begin = __ldg(a.t.row_ptr + d.row0);
        t.nnz = __ldg(a.t.row_ptr + d.row1);
        t.row0 = d.row0;
        t.tile_ptr = a.t.tile_ptr + d.at;
        tile_worker<P, S, OH, false, XL2, true>(t, w, d.first, d.last, words, rowof);
        __syncwarp();
    }
    if (lane == 0) {
        __threadfence();  // this warp's last draw comes before its count
        if (atomicAdd(a.t.ticket + 1, 1) == warps - 1) {  // every warp has drawn for the last time
            atomicExch(a.t.ticket, 0);
            atomicExch(a.t.ticket + 1, 0);
        }
    }
}
template <int K, int S, bool OH, bool XL2>
__global__ void __launch_bounds__(BATCH_WARPS * 32) k_batch_tiles(BatchArgs<K> a) {
    __shared__ uint32_t s_words[BATCH_WARPS][32];
    __shared__ int s_rowof[BATCH_WARPS][32 * S];
    asm volatile("griddepcontrol.launch_dependents;");
    const int warp = threadIdx.x >> 5;
    batch_tile_workers<K, S, OH, XL2>(a, s_words[warp], s_rowof[warp]);
}
// as k_tiles_persistent_capped: 16 resident warps per SM for 4 and 8 right-hand sides
template <int K, int S, bool XL2>
__global__ void __launch_bounds__(BATCH_WARPS * 32, 16 / BATCH_WARPS)
    k_batch_tiles_capped(BatchArgs<K> a) {
    __shared__ uint32_t s_words[BATCH_WARPS][32];
    __shared__ int s_rowof[BATCH_WARPS][32 * S];
    asm volatile("griddepcontrol.launch_dependents;");
    const int warp = threadIdx.x >> 5;
    batch_tile_workers<K, S, false, XL2>(a, s_words[warp], s_rowof[warp]);
}
template <int K>
using BatchTilesKernel = void (*)(BatchArgs<K>);
template <int K, int S>
BatchTilesKernel<K> batch_tiles_variant(bool one_head, bool x_l2) {
    if constexpr (K >= 4)
        return x_l2 ? &k_batch_tiles_capped<K, S, true> : &k_batch_tiles_capped<K, S, false>;
    else if constexpr (K == 2)
        return x_l2 ? &k_batch_tiles<K, S, false, true> : &k_batch_tiles<K, S, false, false>;
    else if (one_head)
        return x_l2 ? &k_batch_tiles<K, S, true, true> : &k_batch_tiles<K, S, true, false>;
    else
        return x_l2 ? &k_batch_tiles<K, S, false, true> : &k_batch_tiles<K, S, false, false>;
}
template <int K>
BatchTilesKernel<K> batch_tiles_kernel(const BatchWork& b, int seg) {
    return seg == 8    ? batch_tiles_variant<K, 8>(b.one_head, b.x_l2)
           : seg == 16 ? batch_tiles_variant<K, 16>(b.one_head, b.x_l2)
                       : batch_tiles_variant<K, 32>(b.one_head, b.x_l2);
}

// ---- row workers ----
// A lane has U slots' x entries in flight while it multiplies the U before them.  U and the CTAs per
// SM trade loads in flight against warps: on the 64-matrix mix K = 2 takes 120 us at U = 8 and 5 or
// 6 CTAs, 130-140 at 4 or 7 CTAs or U of 4 or 6; K = 4 148 us at U = 4 and 5 or 6 CTAs, 160-168 at U of
// 2 or 8; K = 8 229 us at U = 2 and 5 or 6 CTAs, 236 at U = 4 and 4 (which is 6 % faster on 27-point
// stencils and 32 x 32 blocks alone; for those layouts only it makes the mix 243).  Rows of up to 12 non-zeros have two stages per warp, since their passes are too
// short to hide the next one's copies; longer ones one, since a second one of that size costs more in
// L1 and warps than it hides (K = 2: 150 against 140 us).
template <int K>
struct BatchRowArgs {
    const int* __restrict__ row_ptr;
    const int* __restrict__ col;
    const float* __restrict__ val;
    const VecF<K>* __restrict__ x;
    VecF<K>* y;
    uint32_t* err;
    int m, nnz;
    const int* __restrict__ blocks;  // first rows of the blocks of BATCH_BLOCK rows to do
    int ppw, nworkers;               // a worker is ppw consecutive passes of a block
    const int* rec_row;  // the tile workers' carry records, added by the last kernel
    const VecD<K>* rec_val;
    int nrec;
};
template <int K, int T, int NG>
struct BatchRows {
    static constexpr int U = K == 2 ? 8 : K == 4 ? 4 : 2;
    static constexpr int STAGES = NG <= 3 ? 2 : 1;
    static constexpr int NNZ = 32 * 4 * NG + 16;
    static constexpr int COL = NNZ * 4;
    static constexpr int STAGE_BYTES = (NNZ * 8 + 127) / 128 * 128;
    static constexpr int BAR = STAGES * STAGE_BYTES;
    static constexpr int WARP_BYTES = (BAR + 8 * STAGES + 127) / 128 * 128;
    static constexpr int CTAS = K == 2 ? 6 : 5;
};

// A lane's row in the stage: non-zeros j, j + T, ... of len; ROT: begun at the rot-th one (rows of
// 8, 16, 32, ... non-zeros start in the same shared-memory banks).
template <int K, int T, bool ROT>
struct BatchLane {
    using P = PolMixedK<K>;
    using XT = typename P::XT;
    const XT* __restrict__ x;
    const int* col;
    const float* val;
    int len, j, rot, low;

    __device__ __forceinline__ int at(int k) const {
        if constexpr (!ROT) return k;
        const int i = k + rot;
        return i - (i >= len ? len : 0);
    }
    // whether every row of the pass has slots u .. u + n - 1
    __device__ __forceinline__ bool whole(int u, int n) const { return (u + n) * T <= low; }
    template <int U>
    __device__ __forceinline__ void gather(int u0, XT (&xv)[U]) const {
        const int k0 = u0 * T + j;
        if (whole(u0, U)) {
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = ld_x(x + col[at(k0 + u * T)], 0);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool on = k0 + u * T < len;
                int c = 0;
                if (on) c = col[at(k0 + u * T)];
                xv[u] = ld_x_if(x + c, on);
            }
        }
    }
    template <int U>
    __device__ __forceinline__ void multiply(int u0, const XT (&xv)[U], typename P::Acc& acc) const {
        const int k0 = u0 * T + j;
        if (whole(u0, U)) {
#pragma unroll
            for (int u = 0; u < U; ++u) acc = P::fma(val[at(k0 + u * T)], xv[u], acc);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float v = 0.f;
                if (k0 + u * T < len) v = val[at(k0 + u * T)];
                acc = P::fma(v, xv[u], acc);
            }
        }
    }
};

// The blocks of one lane layout: T lanes to a row, rows of up to 4 * NG * T non-zeros.  One kernel
// of several in a row for a batch: each may start while the one before it drains, and waits for that
// one before it ends, so that the last one's end is the end of all.
template <int K, int T, int NG, bool ROT>
__global__ void __launch_bounds__(BATCH_WARPS * 32, (BatchRows<K, T, NG>::CTAS))
    k_batch_rows(BatchRowArgs<K> a) {
    using P = PolMixedK<K>;
    using L = BatchRows<K, T, NG>;
    using XT = typename P::XT;
    constexpr int R = 32 / T, BLOCK_PASSES = BATCH_BLOCK / R;
    extern __shared__ __align__(128) unsigned char batch_smem[];
    asm volatile("griddepcontrol.launch_dependents;");
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int j = lane & (T - 1);
    unsigned char* const st = batch_smem + warp * L::WARP_BYTES;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(st + L::BAR);
    if (lane < L::STAGES) {
        mbar_init(bar + lane, 1);
        fence_barrier_init();
    }
    __syncwarp();
    const int nnz8 = a.nnz & ~7;
    const uint64_t pol_s = policy_evict_first();
    const int gwarps = gridDim.x * BATCH_WARPS;
    const int gwarp = blockIdx.x * BATCH_WARPS + warp;

    // every gwarps-th worker; its block's first row is loaded a worker ahead, a pass's row bounds
    // a pass ahead
    int w = gwarp, nblock = 0;
    auto find_block = [&]() {
        if (w < a.nworkers) nblock = __ldg(a.blocks + w * a.ppw / BLOCK_PASSES);
    };
    find_block();
    int prow = 0, prow_end = 0, nrow = 0, nstart = 0, nend = 0;
    auto fetch_next = [&]() {
        prow += R;
        if (prow >= prow_end) {
            if (w >= a.nworkers) {
                nrow = -1;
                prow_end = 0;
                return;
            }
            prow = nblock + w * a.ppw % BLOCK_PASSES * R;
            prow_end = prow + a.ppw * R;
            w += gwarps;
            find_block();
        }
        nrow = prow + lane / T;
        nstart = __ldg(a.row_ptr + min(nrow, a.m));
        nend = __ldg(a.row_ptr + min(nrow + 1, a.m));
    };
    int off = 0, len = 0, row = -1;  // the lane's row of the pass filled last; -1: no pass
    auto fill_stage = [&](int s) {
        row = nrow;
        if (row < 0) return;
        float* const s_val = reinterpret_cast<float*>(st + s * L::STAGE_BYTES);
        int* const s_col = reinterpret_cast<int*>(st + s * L::STAGE_BYTES + L::COL);
        const int e0 = __shfl_sync(SPMV_FULL_MASK, nstart, 0);
        const int e1 = __shfl_sync(SPMV_FULL_MASK, nend, 31);
        const int a0 = e0 & ~7;
        const int a1 = min((e1 + 7) & ~7, nnz8);
        off = nstart - a0;
        len = nend - nstart;
        if (lane == 0) {
            const int cnt = max(a1 - a0, 0);
            mbar_arrive_expect_tx(bar + s, (uint32_t)cnt * 8u);
            if (cnt > 0) {
                bulk_g2s(s_val, a.val + a0, (uint32_t)cnt * 4u, bar + s, pol_s);
                bulk_g2s(s_col, a.col + a0, (uint32_t)cnt * 4u, bar + s, pol_s);
            }
        }
        if (e1 > nnz8) {  // the batch's last, partial group of 8 non-zeros
            const int e = nnz8 + lane;
            if (e < a.nnz) {
                s_val[e - a0] = a.val[e];
                s_col[e - a0] = a.col[e];
            }
        }
        fetch_next();
    };
    fetch_next();
    fill_stage(0);
    int stage = 0;
    uint32_t phases = 0u;  // bit s: stage s's phase
    while (row >= 0) {
        const int my_row = row;
        BatchLane<K, T, ROT> r;
        r.x = a.x;
        r.val = reinterpret_cast<const float*>(st + stage * L::STAGE_BYTES) + off;
        r.col = reinterpret_cast<const int*>(st + stage * L::STAGE_BYTES + L::COL) + off;
        r.len = len;
        r.j = j;
        const int top = __reduce_max_sync(SPMV_FULL_MASK, len);
        r.low = __reduce_min_sync(SPMV_FULL_MASK, len);
        r.rot = ROT ? ((off >> 5) * T) % max(len, 1) : 0;
        if (L::STAGES == 2) fill_stage(stage ^ 1);
        if (!mbar_wait_bounded(bar + stage, phases >> stage & 1u)) {
            if (lane == 0) raise_error(a.err, ERR_WAIT_TIMEOUT);
            // once more for the copies in flight, then give up
            mbar_wait_bounded(bar + stage, phases >> stage & 1u);
            if (L::STAGES == 2 && row >= 0) mbar_wait_bounded(bar + (stage ^ 1), phases >> (stage ^ 1) & 1u);
            break;
        }
        phases ^= 1u << stage;
        __syncwarp();  // the partial group's plain stores
        const int slots = (top + T - 1) / T;
        typename P::Acc acc = P::zero();
        // rounds of U slots, each one's x entries in flight while the one before multiplies
        constexpr int U = L::U;
        XT xa[U], xb[U];
        if (slots > 0) {
            r.template gather<U>(0, xa);
            for (int u = 0;;) {
                if (u + U < slots) r.template gather<U>(u + U, xb);
                r.template multiply<U>(u, xa, acc);
                if ((u += U) >= slots) break;
                if (u + U < slots) r.template gather<U>(u + U, xa);
                r.template multiply<U>(u, xb, acc);
                if ((u += U) >= slots) break;
            }
        }
        fence_proxy_async();  // the reads of the stage come before the copies that reuse it
        __syncwarp();
        if (L::STAGES == 1)
            fill_stage(0);
        else
            stage ^= 1;
#pragma unroll
        for (int d = 1; d < T; d <<= 1) acc = P::add(acc, sh_xor(acc, d));
        if (j == 0 && my_row < a.m) a.y[my_row] = P::out_acc(acc);
    }
    if (gwarp == 0 || gwarp * 32 < a.nrec) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int base = gwarp * 32; base < a.nrec; base += gwarps * 32)
        calibrate_records<P>(a.rec_row, a.rec_val, a.nrec, base, a.y, a.m, a.err);
}

// resident grid of the tile workers' kernel on the current device (0 on failure)
template <int K>
int batch_work_grid(const BatchWork& b, int seg) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_tiles_kernel<K>(b, seg),
                                                      BATCH_WARPS * 32, 0) != cudaSuccess)
        return 0;
    return device_sm_count() * (per_sm > 0 ? per_sm : 1);
}

template <int K>
cudaError_t launch_batch_tiles(const BatchLaunch& l, const BatchWork& b, int seg, cudaStream_t st) {
    if (b.ntiles == 0) return cudaSuccess;
    BatchArgs<K> a;
    a.t = batch_tile_args<K>(l);
    a.t.tile_ptr = b.tile_ptr;
    a.t.rec_row = b.rec_row;
    a.t.rec_val = static_cast<VecD<K>*>(b.rec_val);
    a.tiles = b.tiles;
    a.ntiles = b.ntiles;
    batch_tiles_kernel<K>(b, seg)<<<b.tiles_grid, BATCH_WARPS * 32, 0, st>>>(a);
    return cudaGetLastError();
}

template <int K, int T, int NG, bool ROT>
cudaError_t launch_batch_list(BatchRowArgs<K> a, int nblocks, bool dependent, cudaStream_t st) {
    constexpr auto kernel = &k_batch_rows<K, T, NG, ROT>;
    constexpr int bytes = BATCH_WARPS * BatchRows<K, T, NG>::WARP_BYTES;
    int per_sm = 0;
    cudaError_t e = resident_ctas<kernel>(BATCH_WARPS * 32, bytes, &per_sm);
    if (e != cudaSuccess) return e;
    const int ctas = device_sm_count() * per_sm;
    const int npasses = nblocks * (BATCH_BLOCK / 32 * T);
    a.ppw = npasses >= 12 * ctas * BATCH_WARPS ? 2 : 1;
    a.nworkers = npasses / a.ppw;
    const int need = (a.nworkers + BATCH_WARPS - 1) / BATCH_WARPS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(need < ctas ? need : ctas);
    cfg.blockDim = dim3(BATCH_WARPS * 32);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int K>
cudaError_t launch_batch_work(const BatchLaunch& l, const BatchWork& b, int seg, cudaStream_t st) {
    cudaError_t e = launch_batch_tiles<K>(l, b, seg, st);
    BatchRowArgs<K> a;
    a.row_ptr = l.row_ptr;
    a.col = l.col;
    a.val = l.val;
    a.x = static_cast<const VecF<K>*>(l.x);
    a.y = static_cast<VecF<K>*>(l.y);
    a.err = l.err;
    a.m = l.m;
    a.nnz = l.nnz;
    a.rec_row = b.rec_row;
    a.rec_val = static_cast<const VecD<K>*>(b.rec_val);
    for (int i = 0; i < b.nlists && e == cudaSuccess; ++i) {
        const RowList& r = b.lists[i];
        const bool dependent = i > 0 || b.ntiles > 0;
        a.blocks = b.blocks + r.first;
        a.nrec = i == b.nlists - 1 ? b.ntiles : 0;
        e = cudaErrorInvalidValue;
#define SPMV_BATCH_LIST(T, NG)                                                            \
    if (r.form.lanes == T && r.form.groups == NG)                                         \
        e = r.form.rotate ? launch_batch_list<K, T, NG, true>(a, r.count, dependent, st) \
                          : launch_batch_list<K, T, NG, false>(a, r.count, dependent, st)
        SPMV_BATCH_LIST(1, 3);
        SPMV_BATCH_LIST(1, 7);
        SPMV_BATCH_LIST(2, 7);
        SPMV_BATCH_LIST(4, 7);
        SPMV_BATCH_LIST(8, 7);
#undef SPMV_BATCH_LIST
    }
    return e;
}

}  // namespace spmv
