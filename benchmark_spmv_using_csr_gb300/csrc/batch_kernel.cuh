// batch_kernel.cuh -- the batched form's two kernels over work lists (at one right-hand side the
// row workers' is another one, batch_k1.cu).
//
// The matrices of a batch differ in structure, so no one kernel suits the concatenated matrix.
// Blocks of 256 rows whose rows are short, even and local are cut into row workers (lanes on whole
// rows, as row_kernel.cuh); the runs of blocks between them into tile workers (consecutive
// non-zeros, tile_kernel.cuh) over a window of the matrix: row_ptr and y from the run's first row,
// slots outside its non-zeros padding.  The tile workers' kernel runs first; the row workers'
// kernel, its programmatic dependent, fills the SMs as it drains and ends by adding the carry
// records, for which it waits.
//
// Measured on 64 matrices of five kinds (39 M non-zeros) against the tile kernel over the whole
// batch: 171 -> 134 us at 2 right-hand sides, 271 -> 165 us at 4, 395 -> 255 us at 8 (memory 71 us;
// the FP32 pipe 78 us for 10 operations per non-zero and right-hand side); 16 matrices at 8: 163 ->
// 86 us.  By kind at 8: 27-point stencils 521 -> 253 us, 32 x 32 blocks 543 -> 294, 5-point stencils
// 152 -> 95, uniform density 280 -> 216, power-law rows (all tile workers) 328.  What is saved is
// the tile kernel's segmented scan of 64-byte accumulators, about 35 instructions per non-zero.
// Both kinds of worker in one kernel were slower than either alone (K = 8: 563-980 us): the code
// does not fit the instruction cache, and its registers leave 16 warps for the tile workers.
#pragma once
#include "policies_batched.cuh"
#include "row_kernel.cuh"

namespace spmv {

constexpr int BATCH_WARPS = 4;
template <int K>
struct BatchArgs {
    TileArgs<PolMixedK<K>> t;  // the whole batch; windows are cut from it
    const TileWork* __restrict__ tiles;
    const RowWork* __restrict__ rows;
    int ntiles, nrows, nrec;
    int* row_ticket;
};

// ---- tile workers ----
template <int K, int S>
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
        tile_worker<P, S, false, false, true, true>(t, w, d.first, d.last, words, rowof);
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
template <int K, int S>
__global__ void __launch_bounds__(BATCH_WARPS * 32) k_batch_tiles(BatchArgs<K> a) {
    __shared__ uint32_t s_words[BATCH_WARPS][32];
    __shared__ int s_rowof[BATCH_WARPS][32 * S];
    asm volatile("griddepcontrol.launch_dependents;");
    const int warp = threadIdx.x >> 5;
    batch_tile_workers<K, S>(a, s_words[warp], s_rowof[warp]);
}
// as k_tiles_persistent_capped: 16 resident warps per SM for 4 and 8 right-hand sides
template <int K, int S>
__global__ void __launch_bounds__(BATCH_WARPS * 32, 16 / BATCH_WARPS)
    k_batch_tiles_capped(BatchArgs<K> a) {
    __shared__ uint32_t s_words[BATCH_WARPS][32];
    __shared__ int s_rowof[BATCH_WARPS][32 * S];
    asm volatile("griddepcontrol.launch_dependents;");
    const int warp = threadIdx.x >> 5;
    batch_tile_workers<K, S>(a, s_words[warp], s_rowof[warp]);
}
template <int K, int S>
constexpr auto batch_tiles_kernel() {
    if constexpr (K >= 4)
        return &k_batch_tiles_capped<K, S>;
    else
        return &k_batch_tiles<K, S>;
}

// ---- row workers ----
// A lane has U slots' x entries in flight while it multiplies the U before them (K = 8: 64 of its
// 128 registers; U = 2 is 5 % slower on the 27-point stencils, U = 8 at K = 4 level).  One stage
// per warp: a second one hid the copies and cost more in L1 and warps (K = 2: 150 against 140 us).
// CTAs per SM, measured at 3 to 6: 5 for K = 2 and 4, 4 for K = 8.
template <int K>
struct BatchRows {
    static constexpr int U = K == 2 ? 8 : 4;
    static constexpr int NNZ = 32 * BATCH_SLOTS + 16;
    static constexpr int COL = NNZ * 4;
    static constexpr int BAR = NNZ * 8;
    static constexpr int WARP_BYTES = (BAR + 8 + 127) / 128 * 128;
};

// A lane's row in the stage: non-zeros j, j + T, ... of len, T = 1 << tl (a run-time value: a copy
// of the code for each layout would not fit the instruction cache).
template <int K>
struct BatchLane {
    using P = PolMixedK<K>;
    using XT = typename P::XT;
    const XT* __restrict__ x;
    const int* col;
    const float* val;
    int len, j, tl, rot, low;

    __device__ __forceinline__ int at(int k) const {
        const int i = k + rot;
        return i - (i >= len ? len : 0);
    }
    // whether every row of the pass has slots u .. u + n - 1
    __device__ __forceinline__ bool whole(int u, int n) const { return (u + n) << tl <= low; }
    template <int U>
    __device__ __forceinline__ void gather(int u0, XT (&xv)[U]) const {
        if (whole(u0, U)) {
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = ld_x(x + col[at(((u0 + u) << tl) + j)], 0);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = ((u0 + u) << tl) + j;
                int c = 0;
                if (k < len) c = col[at(k)];
                xv[u] = ld_x_if(x + c, k < len);
            }
        }
    }
    template <int U>
    __device__ __forceinline__ void multiply(int u0, const XT (&xv)[U], typename P::Acc& acc) const {
        if (whole(u0, U)) {
#pragma unroll
            for (int u = 0; u < U; ++u) acc = P::fma(val[at(((u0 + u) << tl) + j)], xv[u], acc);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = ((u0 + u) << tl) + j;
                float v = 0.f;
                if (k < len) v = val[at(k)];
                acc = P::fma(v, xv[u], acc);
            }
        }
    }
};

template <int K>
__global__ void __launch_bounds__(BATCH_WARPS * 32, K == 8 ? 4 : 5) k_batch_rows(BatchArgs<K> a) {
    using P = PolMixedK<K>;
    using L = BatchRows<K>;
    using XT = typename P::XT;
    extern __shared__ __align__(128) unsigned char batch_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    unsigned char* const st = batch_smem + warp * L::WARP_BYTES;
    float* const s_val = reinterpret_cast<float*>(st);
    int* const s_col = reinterpret_cast<int*>(st + L::COL);
    uint64_t* const bar = reinterpret_cast<uint64_t*>(st + L::BAR);
    if (lane == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    __syncwarp();
    const int m = a.t.m, nnz8 = a.t.nnz & ~7;
    const int* __restrict__ const row_ptr = a.t.row_ptr;
    const uint64_t pol_s = policy_evict_first();
    const int warps = gridDim.x * BATCH_WARPS;

    // the next worker's descriptor (word l in lane l) and the number of the one after it, drawn
    // and loaded ahead of their use
    int w = blockIdx.x * BATCH_WARPS + warp;
    int nd = 0;
    bool more = true;
    auto word = [&](int l) { return __shfl_sync(SPMV_FULL_MASK, nd, l); };
    auto next_work = [&]() {
        const int i = __shfl_sync(SPMV_FULL_MASK, w, 0);
        more = i < a.nrows;
        if (!more) return;
        if (lane < 3) nd = __ldg(reinterpret_cast<const int*>(a.rows + i) + lane);
        if (lane == 0) w = warps + atomicAdd(a.row_ticket, 1);
    };
    // the pass after the one in the stage
    int prow = 0, prow_end = 0, pform = 0, nrow = 0, nstart = 0, nend = 0, nform = 0;
    auto fetch_next = [&]() {
        prow += 32 >> (pform & 7);
        if (prow >= prow_end) {
            const int f = more ? word(0) : -1;
            if (f < 0) {  // no work left, or the carry records
                nrow = -1;
                return;
            }
            pform = f;
            prow = word(1);
            prow_end = word(2);
            next_work();
        }
        nform = pform;
        nrow = prow + (lane >> (pform & 7));
        nstart = __ldg(row_ptr + min(nrow, m));
        nend = __ldg(row_ptr + min(nrow + 1, m));
    };
    int off = 0, len = 0, row = -1, form = 0;  // the lane's row of the pass in the stage
    auto fill_stage = [&]() {
        row = nrow;
        if (row < 0) return;
        form = nform;
        const int e0 = __shfl_sync(SPMV_FULL_MASK, nstart, 0);
        const int e1 = __shfl_sync(SPMV_FULL_MASK, nend, 31);
        const int a0 = e0 & ~7;
        const int a1 = min((e1 + 7) & ~7, nnz8);
        off = nstart - a0;
        len = nend - nstart;
        if (lane == 0) {
            const int cnt = max(a1 - a0, 0);
            mbar_arrive_expect_tx(bar, (uint32_t)cnt * 8u);
            if (cnt > 0) {
                bulk_g2s(s_val, a.t.val + a0, (uint32_t)cnt * 4u, bar, pol_s);
                bulk_g2s(s_col, a.t.col + a0, (uint32_t)cnt * 4u, bar, pol_s);
            }
        }
        if (e1 > nnz8) {  // the batch's last, partial group of 8 non-zeros
            const int e = nnz8 + lane;
            if (e < a.t.nnz) {
                s_val[e - a0] = a.t.val[e];
                s_col[e - a0] = a.t.col[e];
            }
        }
        fetch_next();
    };
    next_work();
    fetch_next();
    fill_stage();
    uint32_t phase = 0u;
    bool ok = true;
    while (row >= 0) {
        if (!mbar_wait_bounded(bar, phase)) {
            if (lane == 0) atomicOr(a.t.err, ERR_WAIT_TIMEOUT);
            mbar_wait_bounded(bar, phase);  // once more for the copies in flight, then give up
            ok = false;
            break;
        }
        phase ^= 1u;
        __syncwarp();  // the partial group's plain stores
        BatchLane<K> r;
        r.x = a.t.x;
        r.col = s_col + off;
        r.val = s_val + off;
        r.len = len;
        r.tl = form & 3;
        r.j = lane & ((1 << r.tl) - 1);
        const bool rotate = (form & 8) != 0;
        const int top = __reduce_max_sync(SPMV_FULL_MASK, r.len);
        r.low = __reduce_min_sync(SPMV_FULL_MASK, r.len);
        r.rot = rotate ? ((off >> 5) << r.tl) % max(r.len, 1) : 0;
        const int slots = (top + (1 << r.tl) - 1) >> r.tl;
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
        const int my_row = row;
        fence_proxy_async();  // the reads of the stage come before the copies that reuse it
        __syncwarp();
        fill_stage();
        for (int d = 1; d < 1 << r.tl; d <<= 1) acc = P::add(acc, sh_xor(acc, d));
        if (r.j == 0 && my_row < m) a.t.y[my_row] = P::out_acc(acc);
    }
    // the carry records: the tile workers' kernel, which this one may have overlapped, has to be done
    if (more && ok) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        while (more) {
            const int first = word(1), last = word(2);
            next_work();
            for (int base = first; base < last; base += 32)
                calibrate_records<P>(a.t.rec_row, a.t.rec_val, a.nrec, base, a.t.y, m, a.t.err);
        }
    }
    if (lane == 0) {
        __threadfence();  // this warp's last draw comes before its count
        if (atomicAdd(a.row_ticket + 1, 1) == warps - 1) {  // every warp has drawn for the last time
            atomicExch(a.row_ticket, 0);
            atomicExch(a.row_ticket + 1, 0);
        }
    }
}

// resident grids of the two kernels on the current device (0 on failure)
template <int K, int S>
int batch_tiles_grid() {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, batch_tiles_kernel<K, S>(), BATCH_WARPS * 32, 0) != cudaSuccess)
        return 0;
    return device_sm_count() * (per_sm > 0 ? per_sm : 1);
}
template <int K>
int batch_rows_grid() {
    constexpr int bytes = BATCH_WARPS * BatchRows<K>::WARP_BYTES;
    int per_sm = 0;
    if (cudaFuncSetAttribute(k_batch_rows<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_rows<K>, BATCH_WARPS * 32,
                                                      bytes) != cudaSuccess)
        return 0;
    return device_sm_count() * (per_sm > 0 ? per_sm : 1);
}

template <int K, int S>
cudaError_t launch_batch_work_t(const BatchLaunch& l, const BatchWork& b, cudaStream_t st) {
    BatchArgs<K> a;
    a.t = batch_tile_args<K>(l);
    a.t.tile_ptr = b.tile_ptr;
    a.t.rec_row = b.rec_row;
    a.t.rec_val = static_cast<VecD<K>*>(b.rec_val);
    a.tiles = b.tiles;
    a.rows = b.rows;
    a.ntiles = a.nrec = b.ntiles;
    a.nrows = b.nrows;
    a.row_ticket = b.row_ticket;
    if (b.ntiles > 0)
        batch_tiles_kernel<K, S>()<<<b.tiles_grid, BATCH_WARPS * 32, 0, st>>>(a);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b.rows_grid);
    cfg.blockDim = dim3(BATCH_WARPS * 32);
    cfg.dynamicSmemBytes = BATCH_WARPS * BatchRows<K>::WARP_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = b.ntiles > 0 ? 1 : 0;  // a dependent only of the tile workers' kernel
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_batch_rows<K>, a);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int K>
void batch_work_grids(int seg, int* tiles, int* rows) {
    *rows = batch_rows_grid<K>();
    *tiles = seg == 8    ? batch_tiles_grid<K, 8>()
             : seg == 16 ? batch_tiles_grid<K, 16>()
                         : batch_tiles_grid<K, 32>();
}
template <int K>
cudaError_t launch_batch_work(const BatchLaunch& l, const BatchWork& b, int seg, cudaStream_t st) {
    switch (seg) {
        case 8: return launch_batch_work_t<K, 8>(l, b, st);
        case 16: return launch_batch_work_t<K, 16>(l, b, st);
        default: return launch_batch_work_t<K, 32>(l, b, st);
    }
}

}  // namespace spmv
