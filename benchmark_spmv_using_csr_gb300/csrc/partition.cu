// partition.cu -- tile_ptr construction (binary-search partition + dirty bits), the
// bit-flag parity kernel, and the CSR validation pass run before a matrix is accepted.
#include <atomic>

#include "internal.h"
#include "tile.cuh"

namespace spmv {

// One thread per tile boundary: tile_ptr[t] = search_right(min(t*TILE, nnz)) - 1
// (spmv_cuda/kernels_cuda.h:43-49).  The reference searches each boundary inside every
// SpMV launch (twice for boundaries shared by adjacent warps); here it is done once per
// matrix and reused by every call.
__global__ void k_tile_rows(const int* __restrict__ row_ptr, int m, int nnz, int tile,
                            int ntiles, uint32_t* __restrict__ tile_ptr) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > ntiles) return;
    long long b = (long long)t * tile;
    if (b > nnz) b = nnz;
    tile_ptr[t] = (uint32_t)(search_right(row_ptr, (int)b, m + 1) - 1);
}

// One thread per row: an empty row r with o = row_ptr[r] lies strictly inside the span of
// tile (o % TILE == 0 ? o/TILE - 1 : o/TILE) (clamped to the last tile), which is exactly
// the tile whose span the reference scans and finds it in (kernels_cuda.h:119-145).
// Leading empty rows (o == 0) belong to no tile.  Setting a bit is idempotent, so the
// result does not depend on the order of the atomics.
__global__ void k_mark_dirty(const int* __restrict__ row_ptr, int m, int tile, int ntiles,
                             uint32_t* __restrict__ tile_ptr) {
    const long long stride = (long long)gridDim.x * blockDim.x;  // 64-bit: m may be near 2^31
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < m; r += stride) {
        const int o = __ldg(row_ptr + r);
        if (o != __ldg(row_ptr + r + 1)) continue;
        int t = (o % tile == 0) ? o / tile - 1 : o / tile;
        if (t > ntiles - 1) t = ntiles - 1;
        if (t >= 0) atomicOr(tile_ptr + t, DIRTY_BIT);
    }
}

// One warp per tile: the raw bit-flag words of every tile, produced by the same tile_rows()
// the SpMV kernels use (exposed for parity against the reference's words).
template <int S>
__global__ void k_bitflags(const int* __restrict__ row_ptr, int m, int nnz, int ntiles,
                           const uint32_t* __restrict__ tile_ptr, uint32_t* __restrict__ words) {
    __shared__ uint32_t s_words[8][32];
    __shared__ int s_rowof[8][32 * S];
    const int warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 8 + warp;
    if (t >= ntiles) return;
    const uint32_t tp0 = tile_ptr[t], tp1 = tile_ptr[t + 1];
    const int lo = (int)(tp0 & ROW_MASK);
    const RowBatch rb = prefetch_rows(row_ptr, m, lo);
    const uint32_t w = tile_rows<S, double>(row_ptr, m, t * 32 * S, lo, (int)(tp1 & ROW_MASK), rb,
                                            s_words[warp], s_rowof[warp], nullptr);
    words[(size_t)t * 32 + lane_id()] = w;
    (void)nnz;
}

// CSR validation: row_ptr[0] == 0, non-decreasing, row_ptr[m] == nnz, 0 <= col < n.
// Any violation sets a bit in *bad (bit0 row_ptr, bit1 col_idx).
__global__ void k_validate(const int* __restrict__ row_ptr, const int* __restrict__ col, int m,
                           int n, int nnz, uint32_t* bad) {
    // 64-bit counters: m and nnz may be within one stride of 2^31
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tid == 0 && (row_ptr[0] != 0 || row_ptr[m] != nnz)) atomicOr(bad, 1u);
    for (long long r = tid; r < m; r += stride)
        if (__ldg(row_ptr + r) > __ldg(row_ptr + r + 1)) atomicOr(bad, 1u);
    for (long long e = tid; e < nnz; e += stride) {
        const int c = __ldg(col + e);
        if (c < 0 || c >= n) atomicOr(bad, 2u);
    }
}


int device_sm_count() {
    static std::atomic<int> cache[64];  // zero: not looked up yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 1;
    if (dev < 64) {
        const int c = cache[dev].load(std::memory_order_relaxed);
        if (c > 0) return c;
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        return 1;
    if (dev < 64) cache[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

int grid_for(long long work, int threads, int cap_per_sm) {
    long long g = (work + threads - 1) / threads;
    const long long cap = (long long)cap_per_sm * device_sm_count();
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

cudaError_t launch_partition(const int* row_ptr, int m, int nnz, int tile, uint32_t* tile_ptr,
                             cudaStream_t st) {
    const int nt = num_tiles(nnz, tile);
    k_tile_rows<<<(unsigned)(((long long)nt + 1 + 255) / 256), 256, 0, st>>>(row_ptr, m, nnz, tile, nt,
                                                                tile_ptr);
    if (m > 0 && nt > 0)
        k_mark_dirty<<<grid_for(m, 256, 16), 256, 0, st>>>(row_ptr, m, tile, nt, tile_ptr);
    return cudaGetLastError();
}

cudaError_t launch_bitflags(const int* row_ptr, int m, int nnz, int seg, const uint32_t* tile_ptr,
                            uint32_t* words, cudaStream_t st) {
    const int nt = num_tiles(nnz, 32 * seg);
    if (nt == 0) return cudaSuccess;
    const int blocks = (nt + 7) / 8;
    switch (seg) {
        case 1: k_bitflags<1><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        case 2: k_bitflags<2><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        case 4: k_bitflags<4><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        case 8: k_bitflags<8><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        case 16: k_bitflags<16><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        case 32: k_bitflags<32><<<blocks, 256, 0, st>>>(row_ptr, m, nnz, nt, tile_ptr, words); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// One thread per row (a warp: 32 consecutive rows, aligned).
//  * Non-empty rows shorter than cw non-zeros.  Only such a row puts two row heads into one lane's
//    chunk of cw slots (heads at s and s + len share an aligned chunk only if len < cw), and it
//    does so in at most one chunk.
//  * What the row kernel needs: see RowCounts.
// The warps' counts meet in shared memory first: an atomic per warp and count on the few global
// addresses took 56 us on 4.2 M rows, an atomic per CTA 19 us.
__global__ void k_row_counts(const int* __restrict__ row_ptr, int m, int cw,
                             RowCounts* __restrict__ counts) {
    const long long stride = (long long)gridDim.x * blockDim.x;  // 64-bit: m may be near 2^31
    __shared__ RowCounts s;
    if (threadIdx.x == 0) s = RowCounts{};
    __syncthreads();
    const int lane = threadIdx.x & 31;
    unsigned shorts = 0, top = 0, eights = 0;
    unsigned long long groups[4] = {0, 0, 0, 0};
    for (long long r0 = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; r0 < m;
         r0 += stride) {  // warp-uniform
        const long long r = r0 + lane;
        const int len = r < m ? __ldg(row_ptr + r + 1) - __ldg(row_ptr + r) : 0;
        shorts += (len > 0 && len < cw) ? 1u : 0u;
        eights += (len > 0 && len % 8 == 0) ? 1u : 0u;
        int most = len;  // the longest row of 4, 8, 16 and then 32 consecutive ones
#pragma unroll
        for (int t = 3, d = 1; t >= 0; --t) {
            const int rows = 32 >> t;
            for (; d < rows; d <<= 1) most = max(most, __shfl_xor_sync(SPMV_FULL_MASK, most, d));
            if ((lane & (rows - 1)) == 0) groups[t] += (unsigned)((most + (4LL << t) - 1) >> (2 + t));
        }
        top = max(top, (unsigned)most);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        shorts += __shfl_xor_sync(SPMV_FULL_MASK, shorts, d);
        eights += __shfl_xor_sync(SPMV_FULL_MASK, eights, d);
#pragma unroll
        for (int t = 0; t < 4; ++t) groups[t] += __shfl_xor_sync(SPMV_FULL_MASK, groups[t], d);
    }
    if (lane == 0) {
        atomicAdd(&s.short_rows, (unsigned long long)shorts);
        atomicAdd(&s.eights, (unsigned long long)eights);
        atomicMax(&s.max_len, (unsigned long long)top);
#pragma unroll
        for (int t = 0; t < 4; ++t) atomicAdd(&s.groups[t], groups[t]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&counts->short_rows, s.short_rows);
        atomicAdd(&counts->eights, s.eights);
        atomicMax(&counts->max_len, s.max_len);
#pragma unroll
        for (int t = 0; t < 4; ++t) atomicAdd(&counts->groups[t], s.groups[t]);
    }
}

// Locality of the columns for the x gathers, on every step-th non-zero: near when its column is
// within 4 of the previous entry of its row, or of the entry at the same position of the
// previous row (a stencil's neighbour rows reuse the same x lines).
__device__ __forceinline__ bool near_column(const int* __restrict__ row_ptr,
                                            const int* __restrict__ col, int m, int j, int* row) {
    // the row of non-zero j: the last r with row_ptr[r] <= j (rows 0..m-1)
    int lo = 0, hi = m - 1;
    while (lo < hi) {
        const int mid = (int)(((long long)lo + hi + 1) >> 1);
        if (__ldg(row_ptr + mid) <= j)
            lo = mid;
        else
            hi = mid - 1;
    }
    const int r = *row = lo;
    const int start = __ldg(row_ptr + r);
    const int c = __ldg(col + j);
    if (j > start && abs(c - __ldg(col + j - 1)) <= 4) return true;
    if (r == 0) return false;
    const int ps = __ldg(row_ptr + r - 1);
    return ps + (j - start) < start && abs(c - __ldg(col + ps + (j - start))) <= 4;
}
__global__ void k_x_locality(const int* __restrict__ row_ptr, const int* __restrict__ col, int m,
                             int nnz, int step, uint32_t* __restrict__ counts) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    uint32_t seen = 0, near = 0;
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s * step < nnz;
         s += stride) {
        int row = 0;
        ++seen;
        near += near_column(row_ptr, col, m, (int)(s * step), &row) ? 1u : 0u;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        seen += __shfl_xor_sync(SPMV_FULL_MASK, seen, d);
        near += __shfl_xor_sync(SPMV_FULL_MASK, near, d);
    }
    if ((threadIdx.x & 31) == 0 && seen) {
        atomicAdd(counts, seen);
        atomicAdd(counts + 1, near);
    }
}

cudaError_t launch_x_locality(const int* row_ptr, const int* col, int m, int nnz, int step,
                              uint32_t* counts, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    if (m > 0 && nnz > 0 && step > 0) {
        const long long samples = ((long long)nnz + step - 1) / step;
        k_x_locality<<<grid_for(samples, 256, 8), 256, 0, st>>>(row_ptr, col, m, nnz, step,
                                                                       counts);
    }
    return cudaGetLastError();
}

cudaError_t launch_row_counts(const int* row_ptr, int m, int cw, RowCounts* counts,
                              cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(RowCounts), st);
    if (e != cudaSuccess) return e;
    if (m > 0) k_row_counts<<<grid_for(m, 256, 8), 256, 0, st>>>(row_ptr, m, cw, counts);
    return cudaGetLastError();
}

// One warp per block of 256 rows.
__global__ void k_block_stats(const int* __restrict__ row_ptr, int m, int nblocks, int cw,
                              BlockStat* __restrict__ stat) {
    const int lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    for (int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += nwarps) {
        int max_len = 0, eights = 0, filled = 0, shorts = 0, groups[4] = {0, 0, 0, 0};
        for (int i = 0; i < BATCH_BLOCK; i += 32) {
            const long long r = (long long)b * BATCH_BLOCK + i + lane;
            const int lo = r < m ? __ldg(row_ptr + r) : 0;
            const int len = r < m ? __ldg(row_ptr + r + 1) - lo : 0;
            filled += __popc(__ballot_sync(SPMV_FULL_MASK, len > 0));
            eights += __popc(__ballot_sync(SPMV_FULL_MASK, len > 0 && len % 8 == 0));
            shorts += __popc(__ballot_sync(SPMV_FULL_MASK, len > 0 && len < cw));
            int most = len;
#pragma unroll
            for (int t = 3, d = 1; t >= 0; --t) {
                const int rows = 32 >> t;
                for (; d < rows; d <<= 1) most = max(most, __shfl_xor_sync(SPMV_FULL_MASK, most, d));
                groups[t] += (lane & (rows - 1)) == 0 ? min((int)((most + (4LL << t) - 1) >> (2 + t)), 0x7fff) : 0;
            }
            max_len = max(max_len, most);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) groups[t] = __reduce_add_sync(SPMV_FULL_MASK, groups[t]);
        if (lane == 0) {
            BlockStat s{};
            s.first = __ldg(row_ptr + b * BATCH_BLOCK);
            s.max_len = (uint16_t)min(max_len, 0xffff);
            for (int t = 0; t < 4; ++t) s.groups[t] = (uint16_t)min(groups[t], 0xffff);
            s.eights = (uint16_t)eights;
            s.filled = (uint16_t)filled;
            s.shorts = (uint16_t)shorts;
            stat[b] = s;
        }
    }
}

// The locality counts of k_x_locality, per block of 256 rows.
__global__ void k_block_locality(const int* __restrict__ row_ptr, const int* __restrict__ col,
                                 int m, int nnz, int step, BlockStat* __restrict__ stat) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (long long s0 = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; s0 * step < nnz;
         s0 += stride) {  // warp-uniform
        const long long j = (s0 + lane) * step;
        int row = 0;
        const bool near = j < nnz && near_column(row_ptr, col, m, (int)j, &row);
        // one pair of atomics for the lanes of a block, which are neighbours
        const unsigned lanes =
            __match_any_sync(SPMV_FULL_MASK, j < nnz ? row / BATCH_BLOCK : -1);
        const unsigned hits = __ballot_sync(SPMV_FULL_MASK, near) & lanes;
        if (j < nnz && lane == __ffs(lanes) - 1) {
            atomicAdd(&stat[row / BATCH_BLOCK].sampled, (uint32_t)__popc(lanes));
            if (hits) atomicAdd(&stat[row / BATCH_BLOCK].near, (uint32_t)__popc(hits));
        }
    }
}

// One thread per tile boundary of every run (as k_tile_rows, on the run's rows; the first
// boundary is the run's first row, so that its leading empty rows lie in a span).
__global__ void k_run_tiles(const int* __restrict__ row_ptr, const TileRun* __restrict__ runs,
                            int nruns, int nbounds, int tile, uint32_t* __restrict__ tile_ptr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nbounds) return;
    int lo = 0, hi = nruns - 1;  // the run of boundary i: the last one with at <= i
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (runs[mid].at <= i)
            lo = mid;
        else
            hi = mid - 1;
    }
    const TileRun r = runs[lo];
    const int t = r.t0 + i - r.at;
    const int m = r.row1 - r.row0;
    if (t == r.t0) {
        tile_ptr[i] = 0u;
        return;
    }
    const int end = __ldg(row_ptr + r.row1);
    const long long key = min((long long)t * tile, (long long)end);
    tile_ptr[i] = (uint32_t)(search_right(row_ptr + r.row0, (int)key, m + 1) - 1);
}

cudaError_t launch_block_stats(const int* row_ptr, const int* col, int m, int nnz, int cw, int step,
                               BlockStat* stat, cudaStream_t st) {
    const int nblocks = (int)(((long long)m + BATCH_BLOCK - 1) / BATCH_BLOCK);
    if (nblocks > 0)
        k_block_stats<<<grid_for((long long)nblocks * 32, 256, 8), 256, 0, st>>>(
            row_ptr, m, nblocks, cw, stat);
    if (m > 0 && nnz > 0)
        k_block_locality<<<grid_for(((long long)nnz + step - 1) / step, 256, 8), 256, 0, st>>>(
            row_ptr, col, m, nnz, step, stat);
    return cudaGetLastError();
}

cudaError_t launch_run_tiles(const int* row_ptr, const TileRun* runs, int nruns, int nbounds,
                             int tile, uint32_t* tile_ptr, cudaStream_t st) {
    if (nbounds > 0)
        k_run_tiles<<<(nbounds + 255) / 256, 256, 0, st>>>(row_ptr, runs, nruns, nbounds, tile,
                                                           tile_ptr);
    return cudaGetLastError();
}

// Whether a matrix takes the row kernel, and with which lane layout.
//  * The longest row fits in T = 8 lanes of 28 slots (224 non-zeros), FP64 in 32 non-zeros: its
//    slots beyond the row's end cost as much of the narrow FP64 pipe as real ones, and with 2 or
//    more lanes to a row it was 0.86-1.1x the tile kernel.
//  * The rows fill a share of the slots that their passes walk.  Measured against the tile kernel at
//    the best of six schedules (time tile / time rows), by value type and columns:
//    - 4- and 2-byte values, near columns (banded matrices of 1e6-4e7 non-zeros): from a share of
//      0.6 on 0.97-2.0x, at 0.5 and below 0.87-1.2x;
//    - 4- and 2-byte values, random columns (Poisson and constant rows, 2e6-6e7 non-zeros): from
//      0.35 on 1.01-2.4x (1.2x at 8e6), at 0.2-0.3 0.88-1.5x.  The threshold is lower because the
//      tile kernel's gathers wait in turn where a pass has all of its own in flight;
//    - FP64, rows of up to 12 non-zeros, near columns: 1.1-1.9x from 0.6 on;
//    - FP64 else: 1.0-1.5x from 0.84 on, 0.58-0.98x below (Poisson rows: the longest of 32 rows is
//      twice the mean, and so is the FP64 pipe's time).
RowForm choose_row_form(const RowCounts& c, int m, int nnz, bool x_l2, bool f64) {
    RowForm f;
    // the kernel counts rows in whole passes of 32: their numbers must not pass 2^31
    if (nnz == 0 || m > 0x7fffff00 || c.max_len > (f64 ? 32u : 224u)) return f;
    int t = 0;  // log2 of the lanes per row
    while (c.max_len > (28ull << t)) ++t;
    const double slots = 128.0 * (double)c.groups[t];
    const double share = f64 ? (x_l2 || c.max_len > 12 ? 0.84 : 0.6) : x_l2 ? 0.33 : 0.6;
    if ((double)nnz < share * slots) return f;
    f.lanes = 1 << t;
    f.groups = (int)((c.max_len + (4u << t) - 1) >> (2 + t));
    f.rotate = 2 * c.eights > (unsigned long long)m;
    return f;
}

cudaError_t launch_validate(const int* row_ptr, const int* col, int m, int n, int nnz,
                            uint32_t* bad, cudaStream_t st) {
    long long work = (long long)(m > nnz ? m : nnz);
    k_validate<<<grid_for(work, 256, 8), 256, 0, st>>>(row_ptr, col, m, n, nnz, bad);
    return cudaGetLastError();
}

}  // namespace spmv
