// spmv_batched.cu -- the batched multi-RHS form: many CSR matrices of uneven size, k in
// {1, 2, 4, 8} right-hand sides, FP32 storage with the compensated FP32 arithmetic of the mixed
// form, replayed from a CUDA graph.  No counterpart in the reference.
//
// The batch is one block-diagonal CSR: the matrices' rows are concatenated (row_ptr carries
// global non-zero offsets) and their column indices are offset into one concatenated x.  x and
// y hold the k right-hand sides interleaved ([row][k]), so one gather brings all k values of an
// x entry (k*4 bytes, one 256-bit load at k = 8).
//
// A batch in which rows of whole-lane shape hold at least a quarter of the non-zeros runs over work
// lists: row workers for the blocks of 256 rows that suit lanes on whole rows, tile workers for the
// runs between them (batch_kernel.cuh; batch_k1.cu at one right-hand side).  Else, and where a
// variant is forced, one tile partition covers the whole batch: a persistent kernel sized to the
// GPU's resident capacity hands out workers (consecutive tile ranges) from a global atomic ticket,
// so that the uneven matrices load-balance over the SMs, and the calibration kernel adds the carry
// records.  Either way a CUDA graph of the kernels is replayed where the buffers stay the same
// (tickets are left at zero for the next launch).
#include <algorithm>
#include <cstdio>
#include <new>
#include <string>
#include <vector>

#include "../../include/spmv_gb300.h"
#include "internal.h"
#include "policies_batched.cuh"

namespace spmv {

// the persistent kernel for K right-hand sides: register-capped from 4 on.  OH (the one-head
// chunk form) exists for one right-hand side only, whose accumulator is scalar.
template <int K, int S, int WARPS, bool OH, bool XL2>
constexpr auto persistent_kernel() {
    if constexpr (K >= 4)
        return &k_tiles_persistent_capped<PolMixedK<K>, S, WARPS, false, XL2>;
    else
        return &k_tiles_persistent<PolMixedK<K>, S, WARPS, OH && K == 1, XL2>;
}

template <int K, int S, int WARPS, bool OH, bool XL2>
static cudaError_t enqueue_batched(const TileArgs<PolMixedK<K>>& a, int tpw, int nworkers,
                                   int ntiles, int grid, cudaStream_t st) {
    if (nworkers > 0)
        persistent_kernel<K, S, WARPS, OH, XL2>()<<<grid, WARPS * 32, 0, st>>>(a, tpw, nworkers,
                                                                               ntiles);
    const int cb = grid_for(nworkers, 256, 8);
    k_calibrate<PolMixedK<K>><<<cb, 256, 0, st>>>(a.rec_row, a.rec_val, nworkers, a.y, a.tile_ptr,
                                                  a.m, a.err);
    return cudaGetLastError();
}

template <int K, int S, int WARPS, bool OH, bool XL2>
static int persistent_grid() {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, persistent_kernel<K, S, WARPS, OH, XL2>(), WARPS * 32, 0) != cudaSuccess)
        return 0;
    return device_sm_count() * (per_sm > 0 ? per_sm : 1);
}

// The plan's kernel variant: the one-head chunk form (one right-hand side, few short rows) and
// L2-only x gathers (columns without locality), both chosen from counts made on the device.
struct BatchVariant {
    bool one_head = false;
    bool x_l2 = false;
};

template <int K, int S, int WARPS, bool OH, bool XL2>
static cudaError_t enqueue_k(const BatchLaunch& l, int tpw, int grid, cudaStream_t st) {
    const TileArgs<PolMixedK<K>> a = batch_tile_args<K>(l);
    const int nt = num_tiles(l.nnz, 32 * S);
    const int nw = (nt + tpw - 1) / tpw;
    return enqueue_batched<K, S, WARPS, OH, XL2>(a, tpw, nw, nt, grid, st);
}

// dispatch over the variant (one-head form for k = 1 only, L2-only gathers), then S and warps
template <int K, int S, int WARPS>
static cudaError_t enqueue_v(const BatchLaunch& l, const BatchVariant& v, int tpw, int grid,
                             cudaStream_t st) {
    if (K == 1 && v.one_head)
        return v.x_l2 ? enqueue_k<K, S, WARPS, true, true>(l, tpw, grid, st)
                      : enqueue_k<K, S, WARPS, true, false>(l, tpw, grid, st);
    return v.x_l2 ? enqueue_k<K, S, WARPS, false, true>(l, tpw, grid, st)
                  : enqueue_k<K, S, WARPS, false, false>(l, tpw, grid, st);
}
template <int K>
static cudaError_t enqueue_any(const BatchLaunch& l, const TileConfig& c, const BatchVariant& v,
                               int grid, cudaStream_t st) {
    const bool w8 = c.warps_per_cta == 8;
    const int tpw = c.tiles_per_worker;
    switch (c.seg) {
        case 8: return w8 ? enqueue_v<K, 8, 8>(l, v, tpw, grid, st) : enqueue_v<K, 8, 4>(l, v, tpw, grid, st);
        case 16: return w8 ? enqueue_v<K, 16, 8>(l, v, tpw, grid, st) : enqueue_v<K, 16, 4>(l, v, tpw, grid, st);
        case 32: return w8 ? enqueue_v<K, 32, 8>(l, v, tpw, grid, st) : enqueue_v<K, 32, 4>(l, v, tpw, grid, st);
        default: return cudaErrorInvalidValue;
    }
}
static cudaError_t enqueue_batch(const BatchLaunch& l, int k, const TileConfig& c,
                                 const BatchVariant& v, int grid, cudaStream_t st) {
    switch (k) {
        case 1: return enqueue_any<1>(l, c, v, grid, st);
        case 2: return enqueue_any<2>(l, c, v, grid, st);
        case 4: return enqueue_any<4>(l, c, v, grid, st);
        case 8: return enqueue_any<8>(l, c, v, grid, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int K, int S, int WARPS>
static int grid_v(const BatchVariant& v) {
    if (K == 1 && v.one_head)
        return v.x_l2 ? persistent_grid<K, S, WARPS, true, true>()
                      : persistent_grid<K, S, WARPS, true, false>();
    return v.x_l2 ? persistent_grid<K, S, WARPS, false, true>()
                  : persistent_grid<K, S, WARPS, false, false>();
}
template <int K>
static int grid_any(const TileConfig& c, const BatchVariant& v) {
    const bool w8 = c.warps_per_cta == 8;
    switch (c.seg) {
        case 8: return w8 ? grid_v<K, 8, 8>(v) : grid_v<K, 8, 4>(v);
        case 16: return w8 ? grid_v<K, 16, 8>(v) : grid_v<K, 16, 4>(v);
        case 32: return w8 ? grid_v<K, 32, 8>(v) : grid_v<K, 32, 4>(v);
        default: return 0;
    }
}
static int batch_grid(int k, const TileConfig& c, const BatchVariant& v) {
    switch (k) {
        case 1: return grid_any<1>(c, v);
        case 2: return grid_any<2>(c, v);
        case 4: return grid_any<4>(c, v);
        case 8: return grid_any<8>(c, v);
        default: return 0;
    }
}

}  // namespace spmv

using namespace spmv;

struct bhsp_batch {
    int count = 0, k = 1;
    int m = 0, n = 0, nnz = 0;  // totals of the concatenated block-diagonal matrix
    TileConfig cfg{};
    bool tpw_by_rule = false;  // the tiles per worker are the rule's, not the caller's
    BatchVariant var{};
    int short_rows = 0, x_sampled = 0, x_near = 0;  // the counts the variant came from
    int ntiles = 0, nworkers = 0, grid = 0;
    const int* row_ptr = nullptr;
    const int* col = nullptr;
    uint32_t* tile_ptr = nullptr;
    int* rec_row = nullptr;
    void* rec_val = nullptr;
    uint32_t* err = nullptr;
    int* ticket = nullptr;
    // the work lists of row and tile workers, taken when `mixed` is set and no variant was forced
    bool mixed = false, variant_set = false;
    BatchWork work{};
    // the graph and the buffers it was captured with
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    struct Buffers {
        const float* val = nullptr;
        const void* x = nullptr;
        void* y = nullptr;
        bool operator==(const Buffers& o) const { return val == o.val && x == o.x && y == o.y; }
    };
    Buffers captured, last;  // of the graph, and of the last execute with use_graph
    std::string last_error;
};

static void batch_work_release(bhsp_batch* b) {
    cudaFree(b->work.tiles);
    cudaFree(b->work.blocks);
    cudaFree(b->work.tile_ptr);
    cudaFree(b->work.rec_row);
    cudaFree(b->work.rec_val);
    b->work = BatchWork{};
    b->mixed = false;
}

static void batch_release(bhsp_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    cudaFree(b->tile_ptr);
    cudaFree(b->rec_row);
    cudaFree(b->rec_val);
    cudaFree(b->err);
    cudaFree(b->ticket);
    batch_work_release(b);
    b->exec = nullptr;
    b->graph = nullptr;
}

static int batch_cuda(bhsp_batch* b, cudaError_t e, const char* what) {
    b->last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? BHSPARSE_OUT_OF_MEMORY : BHSPARSE_CUDA_ERROR;
}

// The default tiles per worker.  A longer worker saves a start and a carry record per tile and
// leaves fewer workers to even out the warps' last ones, so it is worth its length only where
// every resident warp has many tiles.  Measured at one right-hand side and 16 non-zeros per lane
// with 1, 2, 3 and 4 tiles (us): 2 matrices (0.7 tiles per warp) 13.5, 16.6, 18.7, 21.8; 5 (1.8)
// 27.5, 37.1, 46.6, 57.8; 32 (12) 71, 76, 84, 98; 128 (47) 257, 229, 220, 231; 256 (90) 460, 402,
// 394, 387.  From two right-hand sides on, where a warp's tile costs more and so evens out sooner,
// a worker grows at half as many tiles: power-law matrices at 8 right-hand sides (26 tiles per warp)
// 344, 314, 311, 313; rows of 300 to 1500 random columns at 8 right-hand sides (8.6) 102, 95, 91, 98,
// at 4 (10.1) 151, 146, 147, 147; rows of 512 near columns at 8 (10.1) 117, 119, 121, 125.
// The one-head form (long rows at one right-hand side) spends its time on a worker's start, not on
// the ends of rows: rows of 300 to 1500 random columns (0.5 tiles per warp) 18.5, 24.6, 26.3, 31.1;
// (1.6) 27.3, 24.9, 31.2, 37.3; (2.6) 36.4, 35.4, 31.6, 37.4; (4.2) 48.2, 49.5, 48.4, 45.6; (5.8)
// 66.5, 65.7, 66.6, 63.0; (13.5) 144, 140, 137, 130.
static int batch_tiles_per_worker(const bhsp_batch* b) {
    const long long warps = (long long)b->grid * b->cfg.warps_per_cta;
    if (b->var.one_head) return b->ntiles >= 4 * warps ? 4 : 1;
    int tpw = 1;
    while (tpw < 4 && b->ntiles >= ((b->k == 1 ? 14LL : 7LL) << (tpw - 1)) * warps) ++tpw;
    return tpw;
}

// The batch's work lists (see batch_kernel.cuh): row workers for the blocks of 256 rows that suit
// lanes on whole rows, tile workers for the runs between them.  Leaves b->mixed false where the row
// workers would hold less than a quarter of the batch.
//  * A block suits the row workers where its longest row fits (224 non-zeros; 112 at one right-hand
//    side) and its rows fill 0.4 of the slots that their passes walk.  Random columns are no bar
//    here: an x entry is 8 to 32 bytes, its own sector or a good part of one, whichever lane reads
//    it.  64 matrices of uniform density (Poisson rows of up to 20, random columns): 147 -> 107,
//    167 -> 128, 247 -> 158 and 280 -> 216 us at 1, 2, 4 and 8 right-hand sides; thresholds of 0.2
//    to 0.5 differ by 3 %.
//  * Each lane layout is a kernel of its own, so one with fewer passes than the GPU holds warps gives
//    its blocks to the next larger one, the last one to the tile workers.  (Half and twice that
//    bound differ by up to 10 % either way on 8 and 16 matrices; two blocks of the last layout as a
//    kernel of their own took 15-25 us of a 64-matrix batch.)
//  * From two right-hand sides on the layouts of many lanes run first: their passes are the longest.
//    64 matrices 127.5, 161 and 236 -> 119.5, 149 and 230 us at 2, 4 and 8; at one right-hand side 64
//    matrices 110 -> 108, but 8 and 16 matrices 27 -> 31 and 51 -> 54, so there they run last.
static cudaError_t batch_work_build(bhsp_batch* b, cudaStream_t st) {
    const int nblocks = (int)(((long long)b->m + BATCH_BLOCK - 1) / BATCH_BLOCK);
    // (row numbers of whole passes must not pass 2^31)
    if (b->nnz == 0 || b->m > 0x7fffff00) return cudaSuccess;
    std::vector<BlockStat> stat((size_t)nblocks);
    BlockStat* d_stat = nullptr;
    cudaError_t e = cudaMalloc(&d_stat, sizeof(BlockStat) * (size_t)nblocks);
    const int cw = batch_chunk_width(b->k, b->cfg.seg);
    const int step = b->nnz > (1 << 17) ? b->nnz / (1 << 17) : 1;  // (a search per sample: 55 us for 2^20)
    if (e == cudaSuccess)
        e = launch_block_stats(b->row_ptr, b->col, b->m, b->nnz, cw, step, d_stat, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(stat.data(), d_stat, sizeof(BlockStat) * (size_t)nblocks,
                            cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_stat);
    if (e != cudaSuccess) return e;
    const int tile = 32 * b->cfg.seg;
    const long long warps = (long long)device_sm_count() * 16;
    auto nnz_to = [&](int i) { return i < nblocks ? stat[(size_t)i].first : b->nnz; };
    const ListForm* const forms = b->k == 1 ? LIST_FORMS_1 : LIST_FORMS_K;
    // the layout of a block, or -1
    auto form_of = [&](int i) -> int {
        const BlockStat& s = stat[(size_t)i];
        const int nnz = nnz_to(i + 1) - s.first;
        if (nnz == 0) return 0;
        if (s.max_len > (b->k == 1 ? 4 : 8) * BATCH_SLOTS) return -1;
        int t = 0;
        while (s.max_len > BATCH_SLOTS << t) ++t;
        if (nnz < 0.4 * 128.0 * s.groups[t]) return -1;
        int f = 0;  // the smallest layout of T lanes that holds the longest row
        while (forms[f].lanes < 1 << t || s.max_len > 4 * forms[f].groups << t) ++f;
        return f;
    };
    std::vector<int> form((size_t)nblocks);
    long long count[NLIST_FORMS] = {};  // blocks by layout
    for (int i = 0; i < nblocks; ++i)
        if ((form[(size_t)i] = form_of(i)) >= 0) ++count[form[(size_t)i]];
    // the layout that takes a layout's blocks (-1: the tile workers)
    int taken[NLIST_FORMS];
    for (int f = 0; f < NLIST_FORMS; ++f) {
        const long long passes = count[f] * (BATCH_BLOCK / 32) * forms[f].lanes;
        const int up = forms[f].into;
        const bool few = up >= 0 ? passes < warps : 4 * passes < warps;
        taken[f] = few ? up : f;
        if (few && up >= 0) count[up] += count[f];
    }
    long long row_nnz = 0, shorts = 0, sampled = 0, near = 0;
    for (int i = 0; i < nblocks; ++i) {
        int& f = form[(size_t)i];
        const BlockStat& s = stat[(size_t)i];
        while (f >= 0 && taken[f] != f) f = taken[f];
        if (f >= 0) {
            row_nnz += nnz_to(i + 1) - s.first;
        } else {
            shorts += s.shorts;
            sampled += s.sampled;
            near += s.near;
        }
    }
    if (4 * row_nnz < b->nnz) return cudaSuccess;
    b->work.one_head = b->k == 1 && one_head_pays(shorts, b->nnz - row_nnz, cw);
    // (the one-head form gathers through L1 whatever the columns: rows of 300 to 1500 random columns
    // between stencils, x of 50,000, 216,000 and 1,000,000 entries: 62, 67.5 and 70.0 us through L1,
    // 80, 68.9 and 69.9 from L2 only)
    b->work.x_l2 = !b->work.one_head && x_l2_pays(sampled, near);
    // tiles per tile worker: up to 1024 non-zeros, as many as leave every warp six workers (on the
    // 128-matrix mix at one right-hand side 199 us; 204 at three workers, 207 at 2048 non-zeros too).
    // In the one-head form, whose workers cost more to start, up to 2048 and two workers: rows of 512
    // and of 256 near columns between stencils 67.8 -> 59.7 and 62.2 -> 52.4 us.
    const bool oh = b->work.one_head;
    const int tpw = (int)std::min<long long>(
        {oh && b->tpw_by_rule ? 4 : b->cfg.tiles_per_worker, std::max((oh ? 2048 : 1024) / tile, 1),
         (int)std::max<long long>((b->nnz - row_nnz) / tile / ((oh ? 2 : 6) * warps), 1)});
    b->work.tpw = tpw;
    std::vector<TileWork> tiles;
    std::vector<TileRun> runs;
    std::vector<int> blocks[NLIST_FORMS];
    int rotate[NLIST_FORMS] = {};  // blocks of a list whose rows start in the same banks
    int nbounds = 0;
    for (int i = 0; i < nblocks;) {
        const int f = form[(size_t)i];
        int j = i + 1;
        while (j < nblocks && form[(size_t)j] == f) ++j;
        const int row0 = i * BATCH_BLOCK;
        const int row1 = (int)std::min<long long>((long long)j * BATCH_BLOCK, b->m);
        if (f >= 0) {
            for (int at = i; at < j; ++at) {
                blocks[f].push_back(at * BATCH_BLOCK);
                rotate[f] += 2 * stat[(size_t)at].eights > stat[(size_t)at].filled;
            }
        } else {
            TileRun r{row0, row1, nnz_to(i) / tile, (int)(((long long)nnz_to(j) + tile - 1) / tile),
                      nbounds};
            nbounds += r.t1 - r.t0 + 1;
            runs.push_back(r);
            for (int t = r.t0; t < r.t1; t += tpw)
                tiles.push_back(TileWork{t, std::min(t + tpw, r.t1), row0, row1, r.at - r.t0});
        }
        i = j;
    }
    BatchWork& w = b->work;
    std::vector<int> listed;
    for (int i = 0; i < NLIST_FORMS; ++i) {
        const int f = b->k == 1 ? i : NLIST_FORMS - 1 - i;
        if (blocks[f].empty()) continue;
        RowList& l = w.lists[w.nlists++];
        l.form.lanes = forms[f].lanes;
        l.form.groups = forms[f].groups;
        l.form.rotate = 2 * rotate[f] > (int)blocks[f].size();
        l.first = (int)listed.size();
        l.count = (int)blocks[f].size();
        listed.insert(listed.end(), blocks[f].begin(), blocks[f].end());
    }
    w.ntiles = (int)tiles.size();
    TileRun* d_runs = nullptr;
    e = cudaMalloc(&w.blocks, sizeof(int) * (listed.size() + 1));
    if (e == cudaSuccess) e = cudaMalloc(&w.tiles, sizeof(TileWork) * (tiles.size() + 1));
    if (e == cudaSuccess) e = cudaMalloc(&w.tile_ptr, sizeof(uint32_t) * (size_t)(nbounds + 1));
    if (e == cudaSuccess) e = cudaMalloc(&w.rec_row, sizeof(int) * (tiles.size() + 1));
    if (e == cudaSuccess) e = cudaMalloc(&w.rec_val, sizeof(double) * b->k * (tiles.size() + 1));
    if (e == cudaSuccess) e = cudaMalloc(&d_runs, sizeof(TileRun) * (runs.size() + 1));
    if (e == cudaSuccess && !listed.empty())
        e = cudaMemcpyAsync(w.blocks, listed.data(), sizeof(int) * listed.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && !tiles.empty())
        e = cudaMemcpyAsync(w.tiles, tiles.data(), sizeof(TileWork) * tiles.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && !runs.empty())
        e = cudaMemcpyAsync(d_runs, runs.data(), sizeof(TileRun) * runs.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = launch_run_tiles(b->row_ptr, d_runs, (int)runs.size(), nbounds, tile, w.tile_ptr, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_runs);
    if (e != cudaSuccess) return e;
    switch (b->k) {
        case 1: w.tiles_grid = batch_work_grid<1>(w, b->cfg.seg); break;
        case 2: w.tiles_grid = batch_work_grid<2>(w, b->cfg.seg); break;
        case 4: w.tiles_grid = batch_work_grid<4>(w, b->cfg.seg); break;
        default: w.tiles_grid = batch_work_grid<8>(w, b->cfg.seg); break;
    }
    b->mixed = w.tiles_grid > 0 && w.nlists > 0;
    return cudaSuccess;
}

// The work lists, or none where there is no memory for them: the one tile kernel needs none.
static cudaError_t batch_work_try(bhsp_batch* b, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    try {
        e = batch_work_build(b, st);
    } catch (const std::bad_alloc&) {
        e = cudaErrorMemoryAllocation;
    }
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();  // clear the allocation's error
    batch_work_release(b);
    return cudaSuccess;
}

// Whether an execute runs the work list (else the tile kernel over the whole batch).
static bool batch_takes_work(const bhsp_batch* b) { return b->mixed && !b->variant_set; }

extern "C" int bhsp_batch_create(bhsp_batch** out, int count, int m_total, int n_total,
                                 int nnz_total, const int* d_row_ptr, const int* d_col_idx, int k,
                                 int seg, int tiles_per_worker, int warps_per_cta, void* stream) {
    if (!out) return BHSPARSE_INVALID_ARGUMENT;
    *out = nullptr;
    if (count < 1 || m_total < 1 || n_total < 1 || nnz_total < 0 || nnz_total > BHSP_MAX_NNZ ||
        !d_row_ptr || (nnz_total > 0 && !d_col_idx) || (k != 1 && k != 2 && k != 4 && k != 8))
        return BHSPARSE_INVALID_ARGUMENT;
    if ((long long)m_total * k > 0x7fffffffLL || (long long)n_total * k > 0x7fffffffLL)
        return BHSPARSE_INVALID_ARGUMENT;
    TileConfig c;
    // default schedule: S = 16, except S = 32 for 4 right-hand sides (+1.7 % on the batched workload)
    c.seg = seg > 0 ? seg : (k == 4 ? 32 : 16);
    c.tiles_per_worker = tiles_per_worker > 0 ? tiles_per_worker : 1;  // 0: chosen below
    c.warps_per_cta = warps_per_cta > 0 ? warps_per_cta : 4;
    c.stages = 0;
    if ((c.seg != 8 && c.seg != 16 && c.seg != 32) || (c.warps_per_cta != 4 && c.warps_per_cta != 8))
        return BHSPARSE_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(d_col_idx) % 32 != 0) return BHSPARSE_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = bhsp_validate_csr(d_row_ptr, d_col_idx, m_total, n_total, nnz_total, stream);
    if (rc) return rc;
    bhsp_batch* b = new bhsp_batch;
    b->count = count;
    b->k = k;
    b->m = m_total;
    b->n = n_total;
    b->nnz = nnz_total;
    b->cfg = c;
    b->row_ptr = d_row_ptr;
    b->col = d_col_idx;
    b->ntiles = num_tiles(nnz_total, 32 * c.seg);
    cudaError_t e = cudaSuccess;
    {
        // the kernel variant, as for a single matrix's plan: short rows against the chunk
        // width of the batched kernel, and the locality of about 2^20 sampled columns
        const int cw = batch_chunk_width(k, c.seg);
        const int step = nnz_total > (1 << 20) ? nnz_total / (1 << 20) : 1;
        struct Counts {
            RowCounts rows;
            uint32_t locality[2];
        } h = {};
        Counts* counts = nullptr;
        e = cudaMalloc(&counts, sizeof h);
        if (e == cudaSuccess) e = launch_row_counts(d_row_ptr, m_total, cw, &counts->rows, st);
        if (e == cudaSuccess)
            e = launch_x_locality(d_row_ptr, d_col_idx, m_total, nnz_total, step, counts->locality,
                                  st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, counts, sizeof h, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaFree(counts);
        b->short_rows = (int)h.rows.short_rows;
        b->x_sampled = (int)h.locality[0];
        b->x_near = (int)h.locality[1];
        b->var.one_head = k == 1 && one_head_pays(b->short_rows, nnz_total, cw);
        b->var.x_l2 = x_l2_pays(h.locality[0], h.locality[1]);
    }
    b->grid = e == cudaSuccess ? batch_grid(k, c, b->var) : 0;
    if (e == cudaSuccess && b->grid <= 0) e = cudaErrorInvalidConfiguration;
    if (tiles_per_worker <= 0) {
        b->tpw_by_rule = true;
        b->cfg.tiles_per_worker = c.tiles_per_worker = batch_tiles_per_worker(b);
    }
    b->nworkers = (b->ntiles + c.tiles_per_worker - 1) / c.tiles_per_worker;
    const size_t nw = b->nworkers > 0 ? (size_t)b->nworkers : 1;
    if (e == cudaSuccess) e = cudaMalloc(&b->tile_ptr, sizeof(uint32_t) * ((size_t)b->ntiles + 1));
    if (e == cudaSuccess) e = cudaMalloc(&b->rec_row, sizeof(int) * nw);
    if (e == cudaSuccess) e = cudaMalloc(&b->rec_val, sizeof(double) * k * nw);
    if (e == cudaSuccess) e = cudaMalloc(&b->err, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&b->ticket, 2 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemsetAsync(b->err, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->ticket, 0, 2 * sizeof(int), st);
    if (e == cudaSuccess) e = launch_partition(d_row_ptr, m_total, nnz_total, 32 * c.seg, b->tile_ptr, st);
    if (e == cudaSuccess) e = batch_work_try(b, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        rc = batch_cuda(b, e, "batch setup");
        batch_release(b);
        delete b;
        return rc;
    }
    *out = b;
    return BHSPARSE_SUCCESS;
}

static BatchLaunch batch_launch(bhsp_batch* b, const float* val, const void* x, void* y) {
    BatchLaunch l;
    l.row_ptr = b->row_ptr;
    l.col = b->col;
    l.val = val;
    l.x = x;
    l.y = y;
    l.tile_ptr = b->tile_ptr;
    l.rec_row = b->rec_row;
    l.rec_val = b->rec_val;
    l.err = b->err;
    l.ticket = b->ticket;
    l.m = b->m;
    l.n = b->n;
    l.nnz = b->nnz;
    return l;
}

static cudaError_t enqueue(bhsp_batch* b, const BatchLaunch& l, cudaStream_t st) {
    if (!batch_takes_work(b)) return enqueue_batch(l, b->k, b->cfg, b->var, b->grid, st);
    switch (b->k) {
        case 1: return launch_batch_work<1>(l, b->work, b->cfg.seg, st);
        case 2: return launch_batch_work<2>(l, b->work, b->cfg.seg, st);
        case 4: return launch_batch_work<4>(l, b->work, b->cfg.seg, st);
        default: return launch_batch_work<8>(l, b->work, b->cfg.seg, st);
    }
}

// capture_now: a new set of buffers is captured at once (the tuner, which times replays)
static int batch_execute(bhsp_batch* b, const float* d_val, const float* d_x, float* d_y,
                         int use_graph, bool capture_now, void* stream) {
    if (!b || !d_y || (b->nnz > 0 && (!d_val || !d_x))) return BHSPARSE_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(d_val) % 32 != 0 ||
        reinterpret_cast<uintptr_t>(d_x) % (4 * b->k) != 0 || reinterpret_cast<uintptr_t>(d_y) % (4 * b->k) != 0)
        return BHSPARSE_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const BatchLaunch l = batch_launch(b, d_val, d_x, d_y);
    // A set of buffers is captured when it comes a second time in a row: the capture and
    // instantiation of one to seven kernels cost more than they save in one call.  Two x / y pairs in
    // turn, per call with a capture each and launched directly: 36 -> 7 us on 2 matrices (1 kernel),
    // 42 -> 28.5 on 5 (3 kernels), 117 -> 112 on 64 (7 kernels, one right-hand side); the first call
    // on new buffers, waited for, 50 -> 22, 98 -> 56 and 180 -> 126.
    const bhsp_batch::Buffers now{d_val, d_x, d_y};
    const bool again = capture_now || b->last == now;
    if (use_graph) b->last = now;
    const bool ready = b->exec && b->captured == now;
    if (!use_graph || (!ready && !again)) {
        cudaError_t e = enqueue(b, l, st);
        return e == cudaSuccess ? BHSPARSE_SUCCESS : batch_cuda(b, e, "batched launch");
    }
    if (!ready) {
        // (re)capture the batch's kernels
        if (b->exec) cudaGraphExecDestroy(b->exec);
        if (b->graph) cudaGraphDestroy(b->graph);
        b->exec = nullptr;
        b->graph = nullptr;
        cudaStream_t cs = nullptr;
        cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        if (e != cudaSuccess) return batch_cuda(b, e, "capture stream");
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            cudaError_t e2 = enqueue(b, l, cs);
            e = cudaStreamEndCapture(cs, &b->graph);
            if (e == cudaSuccess) e = e2;
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
        cudaStreamDestroy(cs);
        if (e != cudaSuccess) return batch_cuda(b, e, "graph capture");
        b->captured = now;
    }
    cudaError_t e = cudaGraphLaunch(b->exec, st);
    return e == cudaSuccess ? BHSPARSE_SUCCESS : batch_cuda(b, e, "graph launch");
}

extern "C" int bhsp_batch_execute(bhsp_batch* b, const float* d_val, const float* d_x, float* d_y,
                                  int use_graph, void* stream) {
    return batch_execute(b, d_val, d_x, d_y, use_graph, false, stream);
}

extern "C" int bhsp_batch_check(bhsp_batch* b, void* stream) {
    if (!b) return BHSPARSE_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, b->err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return batch_cuda(b, e, "batch check");
    if (h) {
        cudaMemsetAsync(b->err, 0, sizeof(uint32_t), st);
        cudaStreamSynchronize(st);
        char buf[96];
        snprintf(buf, sizeof buf, "device-side check failed (error word 0x%x)", h);
        b->last_error = buf;
        return BHSPARSE_DEVICE_CHECK_FAILED;
    }
    return BHSPARSE_SUCCESS;
}

extern "C" int bhsp_batch_info(const bhsp_batch* b, int* ntiles, int* nworkers, int* grid,
                               int* launches) {
    if (!b) return BHSPARSE_INVALID_ARGUMENT;
    if (ntiles) *ntiles = b->ntiles;
    if (nworkers) *nworkers = b->nworkers;
    if (grid) *grid = batch_takes_work(b) ? b->work.tiles_grid : b->grid;
    if (launches)
        *launches = !batch_takes_work(b) ? (b->nworkers > 0 ? 2 : 1)
                    // (at one right-hand side the carry records are a kernel of their own)
                    : b->work.nlists + (b->work.ntiles == 0 ? 0 : b->k == 1 ? 2 : 1);
    return BHSPARSE_SUCCESS;
}

extern "C" const char* bhsp_batch_last_error(const bhsp_batch* b) {
    return b ? b->last_error.c_str() : "null batch";
}

extern "C" void bhsp_batch_destroy(bhsp_batch* b) {
    if (!b) return;
    batch_release(b);
    delete b;
}

extern "C" int bhsp_batch_variant(const bhsp_batch* b, int* one_head, int* l2_only) {
    if (!b) return BHSPARSE_INVALID_ARGUMENT;
    if (one_head) *one_head = b->var.one_head ? 1 : 0;
    if (l2_only) *l2_only = b->var.x_l2 ? 1 : 0;
    return BHSPARSE_SUCCESS;
}

extern "C" int bhsp_batch_lists(const bhsp_batch* b, int* row_lists, int* tile_workers, int* one_head,
                                int* l2_only) {
    if (!b) return BHSPARSE_INVALID_ARGUMENT;
    const BatchWork w = batch_takes_work(b) ? b->work : BatchWork{};
    if (row_lists) *row_lists = w.nlists;
    if (tile_workers) *tile_workers = w.ntiles;
    if (one_head) *one_head = w.ntiles > 0 && w.one_head ? 1 : 0;
    if (l2_only) *l2_only = w.ntiles > 0 && w.x_l2 ? 1 : 0;
    return BHSPARSE_SUCCESS;
}

extern "C" int bhsp_batch_set_variant(bhsp_batch* b, int one_head, int l2_only) {
    if (!b || one_head < -1 || one_head > 1 || l2_only < -1 || l2_only > 1 ||
        (one_head == 1 && b->k != 1))
        return BHSPARSE_INVALID_ARGUMENT;
    BatchVariant v = b->var;
    if (one_head >= 0) v.one_head = one_head == 1;
    if (l2_only >= 0) v.x_l2 = l2_only == 1;
    const int grid = batch_grid(b->k, b->cfg, v);
    if (grid <= 0) return batch_cuda(b, cudaErrorInvalidConfiguration, "batch variant");
    b->var = v;
    b->grid = grid;
    if (one_head >= 0 || l2_only >= 0) b->variant_set = true;
    // the captured graph launches the previous kernel: capture again at the next execute
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    return BHSPARSE_SUCCESS;
}

// ---------------------------------------------------------------------------------------
// Schedule tuner of the batched form
// ---------------------------------------------------------------------------------------
namespace {
struct BatchCand {
    int seg, tpw, warps;
};
// S in {8, 16, 32} x tiles per worker in {1, 2, 4, 8} x warps per CTA in {4, 8}
const BatchCand kBatchCands[] = {
    {8, 1, 4},  {8, 1, 8},  {8, 2, 4},  {8, 2, 8},  {8, 4, 4},  {8, 4, 8},  {8, 8, 4},  {8, 8, 8},
    {16, 1, 4}, {16, 1, 8}, {16, 2, 4}, {16, 2, 8}, {16, 4, 4}, {16, 4, 8}, {16, 8, 4}, {16, 8, 8},
    {32, 1, 4}, {32, 1, 8}, {32, 2, 4}, {32, 2, 8}, {32, 4, 4}, {32, 4, 8}, {32, 8, 4}, {32, 8, 8},
};
constexpr int kNumBatchCands = sizeof(kBatchCands) / sizeof(kBatchCands[0]);
}  // namespace

extern "C" int bhsp_batch_tune_num_candidates(void) { return kNumBatchCands; }

extern "C" int bhsp_batch_tune_candidate(int index, int* seg, int* tiles_per_worker,
                                         int* warps_per_cta) {
    if (index < 0 || index >= kNumBatchCands) return BHSPARSE_INVALID_ARGUMENT;
    if (seg) *seg = kBatchCands[index].seg;
    if (tiles_per_worker) *tiles_per_worker = kBatchCands[index].tpw;
    if (warps_per_cta) *warps_per_cta = kBatchCands[index].warps;
    return BHSPARSE_SUCCESS;
}

extern "C" int bhsp_batch_autotune(int count, int m_total, int n_total, int nnz_total,
                                   const int* d_row_ptr, const int* d_col_idx, int k,
                                   const float* d_val, const float* d_x, float* d_y, int warmup,
                                   int reps, float* ms_out, int* best, void* stream) {
    if (warmup < 0 || reps < 1 || !ms_out) return BHSPARSE_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        if (e0) cudaEventDestroy(e0);
        return BHSPARSE_CUDA_ERROR;
    }
    // a write of twice the L2 size before every timed run (skipped if it cannot be allocated)
    void* flush = nullptr;
    size_t flush_bytes = 0;
    int dev = 0, l2 = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) == cudaSuccess && l2 > 0) {
        flush_bytes = 2 * (size_t)l2;
        if (cudaMalloc(&flush, flush_bytes) != cudaSuccess) {
            flush = nullptr;
            cudaGetLastError();
        }
    }
    int rc = BHSPARSE_SUCCESS, best_i = -1;
    float best_ms = 0.f;
    std::vector<float> t((size_t)reps);
    // Over work lists several candidates are one schedule (the lists' kernels have 4 warps per CTA and
    // a bound on a worker's tiles; without tile workers there is none): it is timed once, so that the
    // pick is not the luckiest of several runs of it.
    struct Lists {
        bool used;
        int seg, tpw;
    } lists[kNumBatchCands] = {};
    for (int i = 0; i < kNumBatchCands && rc == BHSPARSE_SUCCESS; ++i) {
        bhsp_batch* b = nullptr;
        rc = bhsp_batch_create(&b, count, m_total, n_total, nnz_total, d_row_ptr, d_col_idx, k,
                               kBatchCands[i].seg, kBatchCands[i].tpw, kBatchCands[i].warps,
                               stream);
        if (rc) break;
        lists[i].used = batch_takes_work(b);
        if (lists[i].used && b->work.ntiles > 0) {
            lists[i].seg = b->cfg.seg;
            lists[i].tpw = b->work.tpw;
        }
        int same = 0;
        while (same < i && !(lists[i].used && lists[same].used && lists[same].seg == lists[i].seg &&
                             lists[same].tpw == lists[i].tpw))
            ++same;
        if (same < i) {
            ms_out[i] = ms_out[same];
            bhsp_batch_destroy(b);
            continue;
        }
        for (int w = 0; w < warmup && rc == 0; ++w) rc = batch_execute(b, d_val, d_x, d_y, 1, true, stream);
        for (int r = 0; r < reps && rc == 0; ++r) {
            if (flush && cudaMemsetAsync(flush, r & 0xff, flush_bytes, st) != cudaSuccess)
                rc = BHSPARSE_CUDA_ERROR;
            if (!rc && cudaEventRecord(e0, st) != cudaSuccess) rc = BHSPARSE_CUDA_ERROR;
            if (!rc) rc = batch_execute(b, d_val, d_x, d_y, 1, true, stream);
            if (!rc && cudaEventRecord(e1, st) != cudaSuccess) rc = BHSPARSE_CUDA_ERROR;
            if (!rc && cudaEventSynchronize(e1) != cudaSuccess) rc = BHSPARSE_CUDA_ERROR;
            if (!rc && cudaEventElapsedTime(&t[(size_t)r], e0, e1) != cudaSuccess)
                rc = BHSPARSE_CUDA_ERROR;
        }
        if (!rc) rc = bhsp_batch_check(b, stream);
        bhsp_batch_destroy(b);
        if (rc) break;
        std::sort(t.begin(), t.end());
        ms_out[i] = t[(size_t)reps / 2];
        if (best_i < 0 || ms_out[i] < best_ms) {
            best_i = i;
            best_ms = ms_out[i];
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (flush) cudaFree(flush);
    if (best) *best = best_i;
    return rc;
}
