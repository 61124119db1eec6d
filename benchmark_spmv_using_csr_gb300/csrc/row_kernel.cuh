// row_kernel.cuh -- y = A.x for matrices whose rows are short and fill their lanes' slots, with
// lanes assigned to whole rows; generic over the arithmetic policies of tile_kernel.cuh.
//
// A pass is 32 / T consecutive rows, T lanes to a row (T = 1, 2, 4 or 8).  The pass's stretch of
// col and val arrives in shared memory by one bulk copy each; lane j of a row then takes the
// row's non-zeros j, j + T, ... (at most 4 * NG of them): columns and values from shared memory
// into registers, all its x entries in flight at once, one multiply-add each, a butterfly over
// the row's T lanes, and the row's lane 0 stores y.  No row crosses a pass, so there are no carry
// records and no calibration launch.
//
// Why lanes take rows here and consecutive non-zeros in tile_kernel.cuh: in a stencil or block
// matrix neighbouring rows reference neighbouring columns, so that at slot k the 32 lanes read
// a few consecutive runs of x (2-3 lines instead of about 10), and there are no bit flags, row
// maps and segmented scans to pay for: about 12 instructions per non-zero and lane instead of 32
// in the plain forms.
//
// Measured on the 27-point stencil on 160^3 (109 M non-zeros), tile kernel at its best schedule
// -> this one: mixed FP32 176 -> 136 us (6800 GB/s: memory-bound), FP64 262 -> 229 us (6090 GB/s;
// the FP64 pipe needs 195 us for its 28 slots a row, memory 208 us); BF16 storage on 121 x 97 x
// 143 86 -> 49.5 us (5800 GB/s); the 5-point stencil on 256^2, FP64, 8.6-8.9 -> 6.5-7.4 us (the
// host's launch path).
//
// Random columns: Poisson rows of 8, 8 M non-zeros, mixed FP32 46 -> 38 us (a gather's sector per
// slot: 227 G/s, the L2-to-SM rate for random sectors being 290-320); read from L2 only they are
// 1-2 % faster above 5e7 non-zeros and up to 20 % slower below, so they allocate in L1.
//
// What bounds it: bytes in flight.  The stage is free once it has been read into registers, so
// the next pass's copies run during this pass's gathers and multiply-adds, and 16-40 warps per SM
// keep 60-140 KB under way.  Loops of 8-slot rounds over the stage, two stages per warp (fewer
// warps: the 27-point FP64 stencil 373-420 us) and passes of 512 non-zeros with a lane layout per
// 32 rows (152-166 us mixed FP32) were slower.
#pragma once
#include <atomic>

#include "internal.h"
#include "tile_kernel.cuh"

namespace spmv {

template <class P>
struct RowArgs {
    const int* __restrict__ row_ptr;
    const int* __restrict__ col;
    const typename P::VS* __restrict__ val;
    const typename P::XT* __restrict__ x;
    typename P::YT* __restrict__ y;
    int* ticket;  // [0] the next worker beyond the grid's own, [1] warps done; zero between launches
    uint32_t* err;
    int m, nnz;
    int npasses, ppw, nworkers;  // a worker is ppw consecutive passes
    bool rotate, by_ticket;
    const int* __restrict__ blocks;  // the first rows of the blocks of 256 rows to do (LIST)
};

// one x entry where `on`, 0 elsewhere (the load is predicated: an absent slot reads nothing)
__device__ __forceinline__ double ld_x_if(const double* p, bool on) {
    double v = 0.0;
    asm volatile("{.reg .pred q; setp.ne.b32 q, %2, 0; @q ld.global.nc.f64 %0, [%1];}"
                 : "+d"(v)
                 : "l"(p), "r"((int)on));
    return v;
}
__device__ __forceinline__ float ld_x_if(const float* p, bool on) {
    float v = 0.f;
    asm volatile("{.reg .pred q; setp.ne.b32 q, %2, 0; @q ld.global.nc.f32 %0, [%1];}"
                 : "+f"(v)
                 : "l"(p), "r"((int)on));
    return v;
}

// Shared memory of one warp: the col / val stream of one pass, widened to whole groups of 8
// non-zeros (the bulk copies' 16-byte alignment for 2-byte values).
template <class P, int NG>
struct RowStage {
    static constexpr int NNZ = 32 * 4 * NG + 16;
    static constexpr int COL = NNZ * (int)sizeof(typename P::VS);
    static constexpr int BAR = COL + NNZ * 4;
    static constexpr int WARP_BYTES = (BAR + 8 + 127) / 128 * 128;
};

constexpr int ROW_WARPS = 4;  // warps per CTA
// CTAs per SM asked of the register allocator.  FP64 from 24 slots on: 4 (128 registers, 16 warps);
// at 5 it spills and its 220 KB of stages leave the x lines no L1 (hit rate 34 % instead of 63 %:
// 272 against 229 us on the 27-point stencil), at 3 there are too few warps (236 us).
template <class P, int NG>
constexpr int row_min_ctas() {
    if (sizeof(typename P::VS) == 8) return NG >= 6 ? 4 : NG >= 4 ? 5 : NG == 3 ? 6 : 8;
    return NG >= 6 ? 5 : NG >= 4 ? 6 : 8;
}

// How the warps take workers beyond their first.  Every gwarps-th one suits equal passes: no
// atomics, and the warps stay close together in the matrix (2-6 % faster than the ticket for
// every 4- and 2-byte value type).  The long FP64 passes, which queue for the FP64 pipe, differ
// in cost enough for the ticket to gain 4 % where a warp draws at least twice; its one address
// takes a draw per 1.5 ns, which short passes would exceed.
template <class P, int NG>
constexpr bool row_ticket_pays() {
    return sizeof(typename P::VS) == 8 && NG >= 3;
}

// LIST: the rows are those of a list of blocks, one kernel of several in a row for a batch.  Each
// may start while the one before it drains and waits for that one before it ends, so that the last
// one's end is the end of all.
template <class P, int T, int NG, bool LIST>
__global__ void __launch_bounds__(ROW_WARPS * 32, (row_min_ctas<P, NG>())) k_rows(RowArgs<P> a) {
    if constexpr (LIST) asm volatile("griddepcontrol.launch_dependents;");
    using L = RowStage<P, NG>;
    using VS = typename P::VS;
    using VC = typename P::VC;
    using XT = typename P::XT;
    using Acc = typename P::Acc;
    constexpr int R = 32 / T, U = 4 * NG;
    extern __shared__ __align__(128) unsigned char row_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int j = lane & (T - 1);
    unsigned char* const st = row_smem + warp * L::WARP_BYTES;
    VS* const s_val = reinterpret_cast<VS*>(st);
    int* const s_col = reinterpret_cast<int*>(st + L::COL);
    uint64_t* const bar = reinterpret_cast<uint64_t*>(st + L::BAR);
    if (lane == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    __syncwarp();
    const int gwarps = gridDim.x * ROW_WARPS;
    const int nnz8 = a.nnz & ~7;
    const uint64_t pol_s = policy_evict_first();

    // A warp's first worker is its own number.  Later ones: every gwarps-th, or from the ticket,
    // drawn one worker ahead of its use (lane 0 holds the number).
    const bool queue = row_ticket_pays<P, NG>() && a.by_ticket;
    int w = blockIdx.x * ROW_WARPS + warp;
    constexpr int BLOCK_PASSES = BATCH_BLOCK / R;
    int nblock = 0, base = 0;  // LIST: the first row of worker w's block; of pass 0 were it there
    auto find_block = [&]() {
        if (LIST && w < a.nworkers) nblock = __ldg(a.blocks + w * a.ppw / BLOCK_PASSES);
    };
    auto draw = [&]() {
        if (!queue)
            w += gwarps;
        else if (lane == 0)
            w = gwarps + atomicAdd(a.ticket, 1);
        find_block();
    };
    find_block();
    // the pass after the one in the stage: the lane's row and its bounds, loaded one pass ahead
    int pass = 0, pass_end = 0, nrow = 0, nstart = 0, nend = 0;
    auto fetch_next = [&]() {
        if (++pass >= pass_end) {
            const int t = queue ? __shfl_sync(SPMV_FULL_MASK, w, 0) : w;
            if (t >= a.nworkers) {
                nrow = -1;
                pass_end = 0;
                return;
            }
            pass = t * a.ppw;
            pass_end = min(pass + a.ppw, a.npasses);
            if constexpr (LIST) base = nblock - pass / BLOCK_PASSES * BATCH_BLOCK;
            draw();
        }
        nrow = base + pass * R + lane / T;
        nstart = __ldg(a.row_ptr + min(nrow, a.m));
        nend = __ldg(a.row_ptr + min(nrow + 1, a.m));
    };
    int off = 0, len = 0, row = -1;  // the lane's row of the pass in the stage; -1: no pass
    auto fill_stage = [&]() {
        row = nrow;
        if (row < 0) return;
        const int e0 = __shfl_sync(SPMV_FULL_MASK, nstart, 0);
        const int e1 = __shfl_sync(SPMV_FULL_MASK, nend, 31);
        const int a0 = e0 & ~7;
        const int a1 = min((e1 + 7) & ~7, nnz8);
        off = nstart - a0;
        len = nend - nstart;
        if (lane == 0) {
            const int cnt = max(a1 - a0, 0);
            mbar_arrive_expect_tx(bar, (uint32_t)(cnt * (4 + (int)sizeof(VS))));
            if (cnt > 0) {
                bulk_g2s(s_val, a.val + a0, (uint32_t)(cnt * sizeof(VS)), bar, pol_s);
                bulk_g2s(s_col, a.col + a0, (uint32_t)(cnt * 4), bar, pol_s);
            }
        }
        if (e1 > nnz8) {  // the matrix's last, partial group of 8 non-zeros
            const int e = nnz8 + lane;
            if (e < a.nnz) {
                s_val[e - a0] = a.val[e];
                s_col[e - a0] = a.col[e];
            }
        }
        fetch_next();
    };
    fetch_next();
    fill_stage();
    uint32_t phase = 0u;
    while (row >= 0) {
        const int top = __reduce_max_sync(SPMV_FULL_MASK, len);
        const int low = __reduce_min_sync(SPMV_FULL_MASK, len);
        if (!mbar_wait_bounded(bar, phase)) {
            if (lane == 0) raise_error(a.err, ERR_WAIT_TIMEOUT);
            mbar_wait_bounded(bar, phase);  // once more for the copies in flight, then give up
            break;
        }
        phase ^= 1u;
        __syncwarp();  // the partial group's plain stores
        const int my_row = row, my_len = len;
        const int* const col = s_col + off;
        const VS* const val = s_val + off;
        // groups of 4 slots: every row has them / some rows do / none does.  Absent slots are
        // zeros, set on every path: an array left undefined on one of them stays live across the
        // loop and costs 100 registers.
        int c[U];
        VC v[U];
        XT x[U];
        auto read_stage = [&](auto at) {
#pragma unroll
            for (int g = 0; g < U; g += 4) {
                if ((g + 4) * T <= low) {
#pragma unroll
                    for (int u = g; u < g + 4; ++u) {
                        c[u] = col[at(u * T + j)];
                        v[u] = to_compute(val[at(u * T + j)]);
                    }
                } else if (g * T < top) {
#pragma unroll
                    for (int u = g; u < g + 4; ++u) {
                        c[u] = 0;
                        v[u] = VC(0);
                        if (u * T + j < my_len) {
                            c[u] = col[at(u * T + j)];
                            v[u] = to_compute(val[at(u * T + j)]);
                        }
                    }
                } else {
#pragma unroll
                    for (int u = g; u < g + 4; ++u) {
                        c[u] = 0;
                        v[u] = VC(0);
                    }
                }
            }
        };
        if (a.rotate) {
            // rows of 8, 16, 32, ... non-zeros start in the same shared-memory banks: each row
            // starts at another of its non-zeros, T * (its offset / 32) on
            const int rot = ((off >> 5) * T) % max(len, 1);
            read_stage([&](int k) { return k + rot - (k + rot >= my_len ? my_len : 0); });
        } else {
            read_stage([](int k) { return k; });
        }
        // the stage has been read: the next pass's copies run during this pass's gathers and
        // multiply-adds (the fence orders the reads before the copies' writes)
        fence_proxy_async();
        __syncwarp();
#pragma unroll
        for (int g = 0; g < U; g += 4) {
            if ((g + 4) * T <= low) {
#pragma unroll
                for (int u = g; u < g + 4; ++u) x[u] = ld_x(a.x + c[u], 0);
            } else if (g * T < top) {
#pragma unroll
                for (int u = g; u < g + 4; ++u) x[u] = ld_x_if(a.x + c[u], u * T + j < my_len);
            } else {
#pragma unroll
                for (int u = g; u < g + 4; ++u) x[u] = XT(0);
            }
        }
        fill_stage();
        // plain FP32 sums in 4 parts, so that the chains of roundings are no longer than the tile
        // kernel's (one part: 1.16x its error on Poisson rows of 20; 4 parts: 0.85x)
        constexpr int NP = std::is_same<Acc, float>::value ? 4 : 1;
        Acc part[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) part[i] = P::zero();
#pragma unroll
        for (int g = 0; g < U; g += 4) {
            if (g * T < top) {
#pragma unroll
                for (int u = g; u < g + 4; ++u) part[u % NP] = P::fma(v[u], x[u], part[u % NP]);
            }
        }
#pragma unroll
        for (int d = 1; d < NP; d <<= 1) {
#pragma unroll
            for (int i = 0; i < NP; i += 2 * d) part[i] = P::add(part[i], part[i + d]);
        }
        Acc acc = part[0];
#pragma unroll
        for (int d = 1; d < T; d <<= 1) acc = P::add(acc, sh_xor(acc, d));
        if (j == 0 && my_row < a.m) a.y[my_row] = P::out_acc(acc);
    }
    if (LIST && blockIdx.x == 0 && threadIdx.x == 0)
        asm volatile("griddepcontrol.wait;" ::: "memory");
    if (queue && lane == 0) {
        __threadfence();  // this warp's last draw comes before its count
        if (atomicAdd(a.ticket + 1, 1) == gwarps - 1) {  // every warp has drawn for the last time
            atomicExch(a.ticket, 0);
            atomicExch(a.ticket + 1, 0);
        }
    }
}

// A kernel's resident CTAs per SM on the current device, looked up once per device, with its
// shared-memory opt-in (setting it twice from racing host threads is harmless).
template <auto KERNEL>
cudaError_t resident_ctas(int threads, int bytes, int* per_sm) {
    static std::atomic<int> ctas_of[64];  // 0: not looked up
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    *per_sm = dev < 64 ? ctas_of[dev].load(std::memory_order_acquire) : 0;
    if (*per_sm > 0) return cudaSuccess;
    e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, KERNEL, threads, bytes);
    if (e != cudaSuccess) return e;
    if (*per_sm < 1) return cudaErrorInvalidConfiguration;
    if (dev < 64) ctas_of[dev].store(*per_sm, std::memory_order_release);
    return cudaSuccess;
}

template <class P, int T, int NG, bool LIST = false>
cudaError_t launch_row_kernel(const RowLaunch& l, cudaStream_t st) {
    constexpr int bytes = ROW_WARPS * RowStage<P, NG>::WARP_BYTES;
    constexpr auto kernel = &k_rows<P, T, NG, LIST>;
    int per_sm = 0;
    cudaError_t e = resident_ctas<kernel>(ROW_WARPS * 32, bytes, &per_sm);
    if (e != cudaSuccess) return e;
    RowArgs<P> a;
    a.row_ptr = l.row_ptr;
    a.col = l.col;
    a.val = static_cast<const typename P::VS*>(l.val);
    a.x = static_cast<const typename P::XT*>(l.x);
    a.y = static_cast<typename P::YT*>(l.y);
    a.ticket = l.ticket;
    a.err = l.err;
    a.m = l.m;
    a.nnz = l.nnz;
    a.rotate = l.form.rotate;
    a.blocks = l.blocks;
    a.npasses = LIST ? l.nblocks * (BATCH_BLOCK * T / 32) : (int)(((long long)l.m * T + 31) / 32);
    const long long ctas = (long long)device_sm_count() * per_sm;
    const long long warps = ctas * ROW_WARPS;
    a.by_ticket = row_ticket_pays<P, NG>() && a.npasses >= 8 * warps;
    a.ppw = a.by_ticket ? 4 : a.npasses >= 4 * warps ? 2 : 1;
    a.nworkers = (a.npasses + a.ppw - 1) / a.ppw;
    const long long need = ((long long)a.nworkers + ROW_WARPS - 1) / ROW_WARPS;
    const int grid = (int)(need < ctas ? need : ctas);
    if constexpr (LIST) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(ROW_WARPS * 32);
        cfg.dynamicSmemBytes = bytes;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = l.dependent ? 1 : 0;
        e = cudaLaunchKernelEx(&cfg, kernel, a);
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    kernel<<<grid, ROW_WARPS * 32, bytes, st>>>(a);
    return cudaGetLastError();
}

template <class P>
cudaError_t launch_rows(const RowLaunch& l, cudaStream_t st) {
    const RowForm& f = l.form;
#define SPMV_ROW_FORM(T, NG) \
    if (f.lanes == T && f.groups == NG) return launch_row_kernel<P, T, NG>(l, st)
    SPMV_ROW_FORM(1, 1);
    SPMV_ROW_FORM(1, 2);
    SPMV_ROW_FORM(1, 3);
#define SPMV_ROW_FORMS(T)  \
    SPMV_ROW_FORM(T, 4);   \
    SPMV_ROW_FORM(T, 5);   \
    SPMV_ROW_FORM(T, 6);   \
    SPMV_ROW_FORM(T, 7)
    SPMV_ROW_FORMS(1);
    if constexpr (sizeof(typename P::VS) == 8) {
        SPMV_ROW_FORM(2, 4);  // FP64 rows have at most 32 non-zeros (choose_row_form)
    } else {
        SPMV_ROW_FORMS(2);
        SPMV_ROW_FORMS(4);
        SPMV_ROW_FORMS(8);
    }
#undef SPMV_ROW_FORMS
#undef SPMV_ROW_FORM
    return cudaErrorInvalidValue;
}

}  // namespace spmv
