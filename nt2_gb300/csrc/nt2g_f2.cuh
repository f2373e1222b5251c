// nt2g_f2.cuh -- two FP32 lanes per instruction (the sm_100 family's packed
// add/sub/mul/fma.rn.f32x2).  Each half rounds exactly as the scalar operation
// does.  One caution: a packed product whose only use is a packed sum may be
// contracted into an FMA by the code generator, rounding mode or not, so where
// the two roundings matter the sum is taken per lane (__fadd_rn).
// Also compiled by NVRTC (nothing is included).
#pragma once

namespace nt2g {

struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pk(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk(f2 a, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f2 dup(float x) { return pk(x, x); }
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
// -a by flipping both sign bits (integer pipe, exact, no FP32 slot)
__device__ __forceinline__ f2 negx2(f2 a)
{
    f2 r;
    r.v = a.v ^ 0x8000000080000000ull;
    return r;
}
__device__ __forceinline__ f2 neg2(f2 a) { return negx2(a); }
template <class F> __device__ __forceinline__ f2 lanes(f2 a, F f)
{
    float x, y;
    upk(a, x, y);
    return pk(f(x), f(y));
}
template <class F> __device__ __forceinline__ f2 lanes(f2 a, f2 b, F f)
{
    float x0, x1, y0, y1;
    upk(a, x0, x1);
    upk(b, y0, y1);
    return pk(f(x0, y0), f(x1, y1));
}

// Horner in NT2's coefficient order, as horner<Fast>.
__device__ __forceinline__ f2 horner2(f2, f2 acc) { return acc; }
template <class... R> __device__ __forceinline__ f2 horner2(f2 x, f2 acc, float c, R... rest)
{
    return horner2(x, fma2(x, acc, dup(c)), rest...);
}

}  // namespace nt2g
