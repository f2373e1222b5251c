// nt2g_accum.cuh -- compensated FP32 accumulation shared by the fold and
// scan kernels: a running sum carried as s + c, c collecting the exact
// rounding error of every addition (TwoSum).
#pragma once
#if !defined(__CUDACC_RTC__)  // the run-time compiler (folds of expressions) embeds this header
#include <cuda_runtime.h>
#endif

namespace nt2g {

// Compensated sum: value = s + c, c collecting the exact rounding errors.
struct CSum {
    float s, c;
};
__device__ __forceinline__ void csum_add(CSum &a, float v)
{
    const float s = __fadd_rn(a.s, v);
    const float bb = __fsub_rn(s, a.s);
    const float e = __fadd_rn(__fsub_rn(a.s, __fsub_rn(s, bb)), __fsub_rn(v, bb));
    a.s = s;
    a.c = __fadd_rn(a.c, e);
}
__device__ __forceinline__ void csum_merge(CSum &a, const CSum &b)
{
    csum_add(a, b.s);
    a.c = __fadd_rn(a.c, b.c);
}

// Three floats, each carrying the rounding errors of the one before: 72 bits, so
// what is combined so holds no less than FP64.  (An FP64 instruction takes a warp
// sixteen cycles, however few of its lanes need it: the eight warps of a fold's 128
// outputs in FP64 would take 28 of them where this takes five.)
struct Sum3 {
    float s, c, d;
    static __device__ __forceinline__ Sum3 of(const CSum &x) { return Sum3{x.s, x.c, 0.0f}; }
    static __device__ __forceinline__ float two_sum(float &a, float b)
    {
        const float t = __fadd_rn(a, b), bb = __fsub_rn(t, a);
        const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(t, bb)), __fsub_rn(b, bb));
        a = t;
        return e;
    }
    __device__ __forceinline__ void add(const CSum &x)
    {
        const float e1 = two_sum(s, x.s), e2 = two_sum(c, x.c), e3 = two_sum(c, e1);
        d = __fadd_rn(d, __fadd_rn(e2, e3));
    }
    __device__ __forceinline__ void add(const Sum3 &x)
    {
        add(CSum{x.s, x.c});
        d = __fadd_rn(d, x.d);
    }
    __device__ __forceinline__ bool in_range() const { return s - s == 0.0f; }
    __device__ __forceinline__ double wide() const { return (double)s + ((double)c + (double)d); }
};

// Warp reduction of compensated sums (lane 0 receives the total).
__device__ __forceinline__ CSum warp_csum(CSum a)
{
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        CSum b{__shfl_down_sync(0xffffffffu, a.s, off), __shfl_down_sync(0xffffffffu, a.c, off)};
        csum_merge(a, b);
    }
    return a;
}
}  // namespace nt2g
