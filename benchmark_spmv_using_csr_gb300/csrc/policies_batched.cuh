// policies_batched.cuh -- arithmetic policy of the batched form: the mixed-FP32 arithmetic of
// policies_mixed.cuh on k interleaved right-hand sides.
#pragma once
#include "internal.h"
#include "tile_kernel.cuh"

namespace spmv {

// ---- k interleaved FP32 values, accumulators and FP64 records ----
template <int K>
struct alignas(4 * K) VecF {
    float v[K];
    __device__ VecF() {}
    __device__ explicit VecF(int z) {
#pragma unroll
        for (int j = 0; j < K; ++j) v[j] = (float)z;
    }
};
template <int K>
struct VecD {
    double v[K];
};
// The float-float accumulators of K right-hand sides.  From two on they are held as pairs of
// right-hand sides, (s0, s1) and (e0, e1), for the packed FP32 instructions.
template <int K>
struct AccK {
    unsigned long long s[K / 2], e[K / 2];
};
template <>
struct AccK<1> {
    float2 v;
};

__device__ __forceinline__ VecF<1> ld_x(const VecF<1>* p, uint64_t) {
    VecF<1> r;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(r.v[0]) : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<2> ld_x(const VecF<2>* p, uint64_t) {
    VecF<2> r;
    asm volatile("ld.global.nc.v2.f32 {%0,%1}, [%2];" : "=f"(r.v[0]), "=f"(r.v[1]) : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<4> ld_x(const VecF<4>* p, uint64_t) {
    VecF<4> r;
    asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3])
                 : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<8> ld_x(const VecF<8>* p, uint64_t) {
    VecF<8> r;
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]),
                   "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
                 : "l"(p));
    return r;
}

// the same gathers where `on`, zeros elsewhere
__device__ __forceinline__ VecF<1> ld_x_if(const VecF<1>* p, bool on) {
    VecF<1> r(0);
    asm volatile("{.reg .pred q; setp.ne.b32 q, %2, 0; @q ld.global.nc.f32 %0, [%1];}"
                 : "+f"(r.v[0])
                 : "l"(p), "r"((int)on));
    return r;
}
__device__ __forceinline__ VecF<2> ld_x_if(const VecF<2>* p, bool on) {
    VecF<2> r(0);
    asm volatile("{.reg .pred q; setp.ne.b32 q, %3, 0; @q ld.global.nc.v2.f32 {%0,%1}, [%2];}"
                 : "+f"(r.v[0]), "+f"(r.v[1])
                 : "l"(p), "r"((int)on));
    return r;
}
__device__ __forceinline__ VecF<4> ld_x_if(const VecF<4>* p, bool on) {
    VecF<4> r(0);
    asm volatile("{.reg .pred q; setp.ne.b32 q, %5, 0; @q ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];}"
                 : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3])
                 : "l"(p), "r"((int)on));
    return r;
}
__device__ __forceinline__ VecF<8> ld_x_if(const VecF<8>* p, bool on) {
    VecF<8> r(0);
    asm volatile("{.reg .pred q; setp.ne.b32 q, %9, 0;"
                 " @q ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];}"
                 : "+f"(r.v[0]), "+f"(r.v[1]), "+f"(r.v[2]), "+f"(r.v[3]), "+f"(r.v[4]),
                   "+f"(r.v[5]), "+f"(r.v[6]), "+f"(r.v[7])
                 : "l"(p), "r"((int)on));
    return r;
}

// the same gathers from L2 only (ld.global.cg), the batch's plan choice when its columns have no
// locality
__device__ __forceinline__ VecF<1> ld_x_l2(const VecF<1>* p) {
    VecF<1> r;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(r.v[0]) : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<2> ld_x_l2(const VecF<2>* p) {
    VecF<2> r;
    asm volatile("ld.global.cg.v2.f32 {%0,%1}, [%2];" : "=f"(r.v[0]), "=f"(r.v[1]) : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<4> ld_x_l2(const VecF<4>* p) {
    VecF<4> r;
    asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3])
                 : "l"(p));
    return r;
}
__device__ __forceinline__ VecF<8> ld_x_l2(const VecF<8>* p) {
    VecF<8> r;
    asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]),
                   "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
                 : "l"(p));
    return r;
}

template <int K, class F>
__device__ __forceinline__ AccK<K> acc_each(const AccK<K>& a, F&& f) {
    AccK<K> r;
    if constexpr (K == 1) {
        r.v = f(a.v);
    } else {
#pragma unroll
        for (int j = 0; j < K / 2; ++j) {
            r.s[j] = f(a.s[j]);
            r.e[j] = f(a.e[j]);
        }
    }
    return r;
}
__device__ __forceinline__ unsigned long long sh_down(unsigned long long v, int d) { return __shfl_down_sync(SPMV_FULL_MASK, v, d); }
__device__ __forceinline__ unsigned long long sh_idx(unsigned long long v, int s) { return __shfl_sync(SPMV_FULL_MASK, v, s); }
__device__ __forceinline__ unsigned long long sh_xor(unsigned long long v, int d) { return __shfl_xor_sync(SPMV_FULL_MASK, v, d); }
template <int K>
__device__ __forceinline__ AccK<K> sh_down(const AccK<K>& a, int d) {
    return acc_each(a, [d](auto v) { return sh_down(v, d); });
}
template <int K>
__device__ __forceinline__ AccK<K> sh_idx(const AccK<K>& a, int s) {
    return acc_each(a, [s](auto v) { return sh_idx(v, s); });
}
template <int K>
__device__ __forceinline__ AccK<K> sh_xor(const AccK<K>& a, int d) {
    return acc_each(a, [d](auto v) { return sh_xor(v, d); });
}

// Two FP32 values in one 64-bit register and the packed instructions on them (add, sub, mul, fma
// .rn.f32x2): each half is rounded as the scalar instruction rounds it, at half the issue slots.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// compensated float-float steps (TwoProduct by FMA + Knuth TwoSum), rounded explicitly
__device__ __forceinline__ float2 ffk_add_product(float v, float x, float2 a) {
    const float p = __fmul_rn(v, x);
    const float ep = __fmaf_rn(v, x, -p);
    const float s = __fadd_rn(a.x, p);
    const float bb = __fsub_rn(s, a.x);
    const float es = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    return make_float2(s, __fadd_rn(a.y, __fadd_rn(es, ep)));
}
__device__ __forceinline__ float2 ffk_add(float2 a, float2 b) {
    const float s = __fadd_rn(a.x, b.x);
    const float bb = __fsub_rn(s, a.x);
    const float es = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
    return make_float2(s, __fadd_rn(__fadd_rn(a.y, b.y), es));
}
// The same steps on two right-hand sides at once.  np is the product negated (exact), which the
// product's FMA residual needs: a - np is the sum a + p and np + bb is -(p - bb), rounded alike.
__device__ __forceinline__ void ffk2_add_product(unsigned long long v, unsigned long long nv,
                                                 unsigned long long x, unsigned long long& s,
                                                 unsigned long long& e) {
    const unsigned long long np = mul2(nv, x);
    const unsigned long long ep = fma2(v, x, np);
    const unsigned long long t = sub2(s, np);
    const unsigned long long bb = sub2(t, s);
    const unsigned long long es = sub2(sub2(s, sub2(t, bb)), add2(np, bb));
    s = t;
    e = add2(e, add2(es, ep));
}
__device__ __forceinline__ void ffk2_add(unsigned long long& s, unsigned long long& e,
                                         unsigned long long bs, unsigned long long be) {
    const unsigned long long t = add2(s, bs);
    const unsigned long long bb = sub2(t, s);
    const unsigned long long es = add2(sub2(s, sub2(t, bb)), sub2(bs, bb));
    s = t;
    e = add2(add2(e, be), es);
}

// The mixed-FP32 arithmetic of spmv_mixed.cu applied to k right-hand sides at once.
template <int K>
struct PolMixedK {
    using VS = float;
    using VC = float;
    using XT = VecF<K>;
    using YT = VecF<K>;
    using Acc = AccK<K>;
    using Carry = AccK<K>;
    using Rec = VecD<K>;
    __device__ static Acc zero() {
        Acc r;
        if constexpr (K == 1) {
            r.v = make_float2(0.f, 0.f);
        } else {
#pragma unroll
            for (int j = 0; j < K / 2; ++j) r.s[j] = r.e[j] = 0ull;
        }
        return r;
    }
    __device__ static Carry carry_zero() { return zero(); }
    __device__ static Acc fma(float v, const XT& x, const Acc& a) {
        Acc r = a;
        if constexpr (K == 1) {
            r.v = ffk_add_product(v, x.v[0], a.v);
        } else {
            const unsigned long long vv = pack2(v, v), nv = pack2(-v, -v);
#pragma unroll
            for (int j = 0; j < K / 2; ++j)
                ffk2_add_product(vv, nv, pack2(x.v[2 * j], x.v[2 * j + 1]), r.s[j], r.e[j]);
        }
        return r;
    }
    __device__ static Acc add(const Acc& a, const Acc& b) {
        Acc r = a;
        if constexpr (K == 1) {
            r.v = ffk_add(a.v, b.v);
        } else {
#pragma unroll
            for (int j = 0; j < K / 2; ++j) ffk2_add(r.s[j], r.e[j], b.s[j], b.e[j]);
        }
        return r;
    }
    __device__ static Carry carry_from(const Acc& a) { return a; }
    __device__ static Acc carry_to_acc(const Carry& c) { return c; }
    __device__ static Carry carry_add(const Carry& c, const Acc& a) { return add(c, a); }
    __device__ static YT out_acc(const Acc& a) {
        YT r;
        if constexpr (K == 1) {
            r.v[0] = __fadd_rn(a.v.x, a.v.y);
        } else {
#pragma unroll
            for (int j = 0; j < K / 2; ++j) {
                const float2 t = unpack2(add2(a.s[j], a.e[j]));
                r.v[2 * j] = t.x;
                r.v[2 * j + 1] = t.y;
            }
        }
        return r;
    }
    __device__ static YT out_carry(const Carry& c) { return out_acc(c); }
    __device__ static Rec rec_from(const Carry& c) {
        Rec r;
        if constexpr (K == 1) {
            r.v[0] = (double)c.v.x + (double)c.v.y;
        } else {
#pragma unroll
            for (int j = 0; j < K / 2; ++j) {
                const float2 s = unpack2(c.s[j]), e = unpack2(c.e[j]);
                r.v[2 * j] = (double)s.x + (double)e.x;
                r.v[2 * j + 1] = (double)s.y + (double)e.y;
            }
        }
        return r;
    }
    __device__ static Rec rec_add(const Rec& a, const Rec& b) {
        Rec r;
#pragma unroll
        for (int j = 0; j < K; ++j) r.v[j] = a.v[j] + b.v[j];
        return r;
    }
    __device__ static Rec rec_of_y(const YT& y) {
        Rec r;
#pragma unroll
        for (int j = 0; j < K; ++j) r.v[j] = (double)y.v[j];
        return r;
    }
    __device__ static YT out_rec(const Rec& r) {
        YT y;
#pragma unroll
        for (int j = 0; j < K; ++j) y.v[j] = __double2float_rn(r.v[j]);
        return y;
    }
};

template <int K>
TileArgs<PolMixedK<K>> batch_tile_args(const BatchLaunch& l) {
    TileArgs<PolMixedK<K>> a;
    a.row_ptr = l.row_ptr;
    a.col = l.col;
    a.val = l.val;
    a.x = static_cast<const VecF<K>*>(l.x);
    a.y = static_cast<VecF<K>*>(l.y);
    a.tile_ptr = l.tile_ptr;
    a.rec_row = l.rec_row;
    a.rec_val = static_cast<VecD<K>*>(l.rec_val);
    a.err = l.err;
    a.m = l.m;
    a.n = l.n;
    a.nnz = l.nnz;
    a.phase = 3;
    a.ticket = l.ticket;
    return a;
}

// batch_k<K>.cu
template <int K>
int batch_work_grid(const BatchWork& b, int seg);
template <int K>
cudaError_t launch_batch_work(const BatchLaunch& l, const BatchWork& b, int seg, cudaStream_t st);
template <>
cudaError_t launch_batch_work<1>(const BatchLaunch& l, const BatchWork& b, int seg, cudaStream_t st);

}  // namespace spmv
