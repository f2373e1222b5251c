// nt2g_fold_kernels.cuh -- device side of the reductions along one dimension
// (sum, prod, max, min, mean, asum1, asum2, norm2, var, stdev, nbtrue,
// all/any/none, nansum, nanmean) of values viewed as [lo, inner, hi]
// (column-major), folding over `inner`: out[l + lo*h] = fold_k x(l + lo*(k + inner*h)).
//
// The element values come from a source type Src with
//   float at(int64_t pos)      the element at linear position pos
//   Raw fetch(int64_t pos)     what it is made of, loaded; fetch4: of the four
//                              elements pos .. pos+3 (pos a multiple of 4; only
//                              called when the source is 16-byte addressable)
//   float value(Raw, pos), value4(Raw, pos, float (&)[4])  the elements
//   kBatch                     fetches a thread has in flight
// The library instantiates the bodies over a table (nt2g_fold.cu); the
// run-time compiler instantiates them over a compiled expression, so a fold of
// an expression (sum(exp(x)*y), sum(abs(x - y), 1), ...) evaluates every
// element in registers inside the fold: one pass, no temporary table.  This
// header is also compiled by NVRTC, so it includes nothing under
// __CUDACC_RTC__ (the run-time source puts nt2g_math.cuh and nt2g_accum.cuh
// ahead of it).
//
// NT2 reshapes every reduction this way before folding
// (core/reduction/include/nt2/dsl/functions/reduction/run.hpp:51-89): a fold
// over the first non-singleton dimension is an inner_fold over contiguous
// segments (lo = 1), a fold over a later dimension an outer_fold over strided
// ones (lo > 1).  The global forms (globalsum, globalmax, ...) fold the
// flattened table: lo = hi = 1.
//
// NT2 policy: one thread per output folds its elements in index order from
// the neutral element with NT2's unfused float operations, the order of NT2's
// per-segment fold (shared_memory/worker/inner_fold.hpp:47-80,
// worker/outer_fold.hpp, details/fold_step.hpp:31-43): bit-identical to NT2
// wherever NT2 spreads the outputs over threads.  mean = rec(float(n)) * sum
// (core/functions/expr/mean.hpp:22-33), asum1 = sum(abs), asum2 = sum(sqr_abs),
// norm2 = sqrt(asum2) (expr/asum1.hpp, expr/asum2.hpp, expr/norm2.hpp),
// var = f * asum2(a - mean(a)) with f = rec(n - 1) (rec(n) for var(a, 1); 1
// when n <= 1) and stdev = sqrt(var) (expr/var.hpp, expr/stdev.hpp): a mean
// pass, then the centred sum of squares.
//
// Fast policy: sums are compensated FP32 (TwoSum; squares carry their FMA
// product error) per thread and over a warp's lanes, warps and chunks combined
// with the bits and the range of FP64; var/stdev take one pass: the deviations
// from the mean of the chunk's first few elements, and their squares, are summed
// compensated, and again about the chunk's own mean where that is far away;
// meanad centres on the mean of a first pass; prod in FP64; max/min are exact.
// Contiguous segments are folded by 8, 32 or 256 threads each (inner_body),
// strided ones by warps over 32 columns (four each with 128-bit loads), rows
// split over a block's warps (outer_body), so that a block hands on one
// partial per output.  With more than one chunk per output, partials go to
// the caller's workspace and a second kernel combines them in a fixed order,
// so results are deterministic for a given shape.
#pragma once
#if !defined(__CUDACC_RTC__)
#include <stdint.h>
#include "nt2g_accum.cuh"
#include "nt2g_f2.cuh"
#define NT2G_FOLD_INF __builtin_huge_valf()
#define NT2G_FOLD_NAN __builtin_nanf("")
#define NT2G_FOLD_SELDOM __forceinline__
#else
#define NT2G_FOLD_INF __int_as_float(0x7f800000)
#define NT2G_FOLD_NAN __int_as_float(0x7fffffff)
#define NT2G_FOLD_SELDOM __noinline__
#endif

namespace nt2g {
namespace fold {

// fold operations (the values of nt2g_fold_op, repeated here because the
// run-time compiled source cannot include the C header)
enum : int {
    SUM = 0, PROD = 1, MAX = 2, MIN = 3, MEAN = 4, ASUM1 = 5, ASUM2 = 6, NORM2 = 7, VAR = 8, STDEV = 9,
    VAR1 = 10, STDEV1 = 11, NBTRUE = 12, ALL = 13, ANY = 14, NONE = 15, NANSUM = 16, NANMEAN = 17, MEANAD = 18,
    // internal: the mean of each output written with the rounding error of its
    // float value (the centre of a fast-policy variance); the count of non-NaN
    // elements (the divisor of nanmean)
    MEAN_C = 100, NOT_NAN = 101
};

constexpr int kThreads = 256;
constexpr int kItems = 64;  // work items of a block of inner_body, at most

__host__ __device__ constexpr bool is_var(int op) { return op == VAR || op == STDEV || op == VAR1 || op == STDEV1; }
// counts of elements: nbtrue and the logical folds all/any/none over x != 0
__host__ __device__ constexpr bool is_count(int op) { return op == NBTRUE || op == ALL || op == ANY || op == NONE; }
// folds of the deviations from each output's mean
__host__ __device__ constexpr bool is_centred(int op) { return is_var(op) || op == MEANAD; }
// folds that need a per-output value from a first pass (the centre, the count);
// the fast policy takes variances in one
__host__ __device__ constexpr bool is_two_pass(int op) { return is_centred(op) || op == NANMEAN; }
__host__ __device__ constexpr bool is_two_pass_fast(int op) { return op == MEANAD || op == NANMEAN; }
__host__ __device__ constexpr bool is_sum(int op)
{
    return op == SUM || op == MEAN || op == ASUM1 || op == ASUM2 || op == NORM2 || op == MEAN_C || is_var(op) ||
           is_count(op) || op == NANSUM || op == NANMEAN || op == NOT_NAN || op == MEANAD;
}

// max/min in NT2's order: the fold keeps acc unless x is strictly better, so
// among equal values (== : +0 and -0 included) the LAST wins; the index
// reported is the FIRST element equal to the result (NT2's globalmax(a, i)
// = globalfind(a == max), common/globalmax.hpp:36-48).  NaN: the fast
// policy propagates it (the first NaN wins).
struct Best {
    float v;
    int64_t ilast, ifirst;
};
template <bool MX> __device__ __forceinline__ bool better(float a, float b) { return MX ? a > b : a < b; }
// Symmetric merge of two partial results (ilast < 0: empty).  Strictly
// better wins; among equal values the bits of the later element and the
// index of the earlier one; a NaN beats numbers, the earlier NaN another NaN.
template <bool MX> __device__ __forceinline__ Best best_merge(const Best &a, const Best &b)
{
    if (a.ilast < 0) return b;
    if (b.ilast < 0) return a;
    const bool an = a.v != a.v, bn = b.v != b.v;
    if (an || bn) {
        if (an && bn) return a.ifirst <= b.ifirst ? a : b;
        return an ? a : b;
    }
    if (better<MX>(a.v, b.v)) return a;
    if (better<MX>(b.v, a.v)) return b;
    Best r = a.ilast > b.ilast ? a : b;
    r.ifirst = a.ifirst < b.ifirst ? a.ifirst : b.ifirst;
    return r;
}

// Per-thread running max/min over elements visited in increasing position,
// positions relative to the thread's chunk start (32-bit), branch-free:
// x replaces v unless v is strictly better (NT2's rule), the first position
// of the current value and the first NaN are kept.  to_best() rebases.
template <bool MX, bool FIRST = true> struct Run {
    float v = MX ? -NT2G_FOLD_INF : NT2G_FOLD_INF;
    int32_t ifirst = -1, ilast = -1, inan = -1;
    __device__ __forceinline__ void add(float x, int32_t k)
    {
        const bool isn = x != x;
        const bool gt = MX ? x > v : x < v;
        const bool eq = x == v;
        inan = (isn && inan < 0) ? k : inan;
        if (FIRST) ifirst = (gt || (eq && ifirst < 0)) ? k : ifirst;  // only for a requested index
        ilast = (gt || eq) ? k : ilast;
        v = (gt || eq) ? x : v;
    }
    __device__ __forceinline__ Best to_best(int64_t base) const
    {
        if (inan >= 0) return Best{__int_as_float(0x7fffffff), base + inan, base + inan};
        if (ilast < 0) return Best{0.0f, -1, -1};
        return Best{v, base + ilast, base + ifirst};
    }
};

// per-op element contribution to a compensated sum
template <int OP> __device__ __forceinline__ void sum_elem(CSum &a, float x)
{
    if (OP == ASUM1) {
        csum_add(a, fabsf(x));
    } else if (OP == ASUM2 || OP == NORM2) {
        const float p = __fmul_rn(x, x);
        csum_add(a, p);
        a.c = __fadd_rn(a.c, __fmaf_rn(x, x, -p));  // exact product error
    } else if (is_count(OP)) {
        csum_add(a, x != 0.0f ? 1.0f : 0.0f);  // NaN counts: NT2's is_nez(NaN) is true
    } else if (OP == NOT_NAN) {
        csum_add(a, x == x ? 1.0f : 0.0f);
    } else if (OP == NANSUM || OP == NANMEAN) {
        csum_add(a, x == x ? x : 0.0f);
    } else {
        csum_add(a, x);
    }
}

// Mean absolute deviation terms: |x - mu| with mu = m + md (the float mean and
// its rounding error), the difference kept exactly as dh + dl (TwoSum), as
// |dh| plus the low part dl - md with the sign of dh (|lo| where dh is 0).
template <int OP> __device__ __forceinline__ void sum_elem_c(CSum &a, float x, float m, float md = 0.0f)
{
    if constexpr (OP == MEANAD) {
        const float dh = __fsub_rn(x, m);
        const float bb = __fsub_rn(dh, x);
        const float dl = __fadd_rn(__fsub_rn(x, __fsub_rn(dh, bb)), __fsub_rn(-m, bb));
        const float lo = __fsub_rn(dl, md);
        csum_add(a, fabsf(dh));
        a.c = __fadd_rn(a.c, dh > 0.0f ? lo : dh < 0.0f ? -lo : fabsf(lo));
    } else {
        sum_elem<OP>(a, x);
    }
}

// ---------------------------------------------------------------- partials --
// What a thread or a warp hands on: a compensated sum (variances: of the
// deviations from the pivot, and of their squares), times `up`, which is one but
// where lanes within the float range are not together (lanes_sums); a product; a
// Best.
struct Sums {
    CSum s1, s2;
    float piv, up;
};
struct Share {
    union {
        Sums v;
        double d;
        Best b;
    };
};
__device__ __forceinline__ double wide(const CSum &a) { return (double)a.s + (double)a.c; }
// times `up`, by the exponent's bits (a multiplication not needed costs as much of
// the FP64 pipe as one that is)
__device__ __forceinline__ double wide(const CSum &a, float up)
{
    const double t = wide(a);
    const int hi = __double2hiint(t), e = hi & 0x7ff00000;
    return __hiloint2double(hi + (up != 1.0f && e != 0 && e != 0x7ff00000 ? 64 << 20 : 0), __double2loint(t));
}
// What a block hands on per (chunk, output), chunk-major: its warps together, in
// FP64.
struct Partial {
    union {
        struct { double s1, s2; float piv; } v;
        double d;
        Best b;
    };
};

// Chunks of one output combined in order.  A variance's sums are shifted to
// the first chunk's pivot in FP64: what cancels when they are brought to the
// mean is at most the number of elements times the result, 2^-53 of that.
template <int OP> struct Total {
    double t = OP == PROD ? 1.0 : 0.0, t2 = 0.0, p0 = 0.0;
    Best b{0.0f, -1, -1};
    bool any = false;
    __device__ __forceinline__ void add(const Partial &p, double n)
    {
        if constexpr (is_var(OP)) {
            if (!any) p0 = (double)p.v.piv;
            const double d = (double)p.v.piv - p0, nd = n * d;
            t += p.v.s1 + nd;
            t2 += p.v.s2 + d * (2.0 * p.v.s1 + nd);
            any = true;
        } else if constexpr (is_sum(OP)) {
            t += p.v.s1;
        } else if constexpr (OP == PROD) {
            t *= p.d;
        } else {
            b = best_merge<OP == MAX>(b, p.b);
        }
    }
    // the one share, or partial, of an output
    __device__ __forceinline__ void set(const Share &r)
    {
        if constexpr (is_sum(OP)) t = wide(r.v.s1, r.v.up);
        if constexpr (is_var(OP)) t2 = wide(r.v.s2, r.v.up);
        if constexpr (OP == PROD) t = r.d;
        if constexpr (!is_sum(OP) && OP != PROD) b = r.b;
    }
    __device__ __forceinline__ void set(const Partial &p)
    {
        if constexpr (is_sum(OP)) t = p.v.s1;
        if constexpr (is_var(OP)) t2 = p.v.s2;
        if constexpr (OP == PROD) t = p.d;
        if constexpr (!is_sum(OP) && OP != PROD) b = p.b;
    }
    __device__ __forceinline__ void add(const Total &o, double n)  // n: the elements of o
    {
        if constexpr (is_var(OP)) {
            if (!o.any) return;
            if (!any) { *this = o; return; }
            const double d = o.p0 - p0, nd = n * d;
            t += o.t + nd;
            t2 += o.t2 + d * (2.0 * o.t + nd);
        } else if constexpr (is_sum(OP)) {
            t += o.t;
        } else if constexpr (OP == PROD) {
            t *= o.t;
        } else {
            b = best_merge<OP == MAX>(b, o.b);
        }
    }
    __device__ __forceinline__ void put(float *out, int64_t *index, double *out64, int64_t o, int64_t n_out, int64_t inner,
                                        const float *cen) const;
};

// The FP64 value of a sum-type (or product) fold before it is rounded to the
// float output: mean = t/n, norm2 = sqrt(t), a count or a sum as is.
template <int OP> __device__ __forceinline__ double finish_double(double t, int64_t inner)
{
    if (OP == MEAN || OP == MEANAD) return t / (double)inner;
    if (OP == NORM2) return sqrt(t);
    return t;
}

// Writes output o of a sum-type (or product) fold from its FP64 total (and,
// when out64 is given, that total's FP64 result: the mean, the norm, the
// variance, ... before rounding to float).
// Variance: t is the sum of squares about the mean, divided by n - 1 (by n for
// VAR1/STDEV1; 1 when n <= 1); not a number (an infinity or a NaN among the
// elements, or their squares past the float range) gives 0.
template <int OP>
__device__ __forceinline__ void fold_put(float *out, double *out64, int64_t o, int64_t n_out, double t, int64_t inner,
                                         const float *cen)
{
    double r = 0.0;
    if constexpr (OP == MEAN_C) {
        const double mu = t / (double)inner;
        const float m = (float)mu;
        out[o] = m;
        out[n_out + o] = (float)(mu - (double)m);
        return;
    } else if constexpr (is_count(OP)) {
        const bool all = t == (double)inner, none = t == 0.0;
        r = OP == NBTRUE ? t : OP == ALL ? (all ? 1.0 : 0.0) : OP == ANY ? (none ? 0.0 : 1.0) : (none ? 1.0 : 0.0);
    } else if constexpr (OP == NANMEAN) {  // nansum / max(count, 1)
        const double c = (double)cen[o];
        r = t / (c > 1.0 ? c : 1.0);
    } else if constexpr (is_var(OP)) {
        const double n = (double)inner;
        double v = t > 0.0 ? t : 0.0;
        const bool by_n = OP == VAR1 || OP == STDEV1;
        if (inner > 1) v /= by_n ? n : n - 1.0;
        r = (OP == STDEV || OP == STDEV1) ? sqrt(v) : v;
    } else {
        r = finish_double<OP>(t, inner);
    }
    out[o] = (float)r;
    if (out64) out64[o] = r;
}

template <int OP>
__device__ __forceinline__ void Total<OP>::put(float *out, int64_t *index, double *out64, int64_t o, int64_t n_out,
                                               int64_t inner, const float *cen) const
{
    if constexpr (is_var(OP)) {
        fold_put<OP>(out, out64, o, n_out, t2 - t * (t / (double)inner), inner, cen);
    } else if constexpr (is_sum(OP) || OP == PROD) {
        fold_put<OP>(out, out64, o, n_out, t, inner, cen);
    } else {
        out[o] = b.v;
        if (index) index[o] = b.ifirst;
    }
}

// ------------------------------------------------- per-thread accumulators --
// One-pass variance: the sums of the deviations d = x - p from a pivot p and of
// their squares, both compensated, d exact as dh + dl (TwoSum) and the square's
// rounding error carried; two elements per packed f32x2 instruction (each half
// rounds as the scalar operation does), which halves the issue slots of its 28
// operations an element pair.
struct VarAcc {
    f2 s1, c1, s2, c2, p;
    static __device__ __forceinline__ float half(f2 v, int i)
    {
        float a, b;
        upk(v, a, b);
        return i ? b : a;
    }
    static __device__ __forceinline__ void csum2(f2 &s, f2 &c, f2 v)
    {
        const f2 t = add2(s, v), bb = sub2(t, s);
        c = add2(c, add2(sub2(s, sub2(t, bb)), sub2(v, bb)));
        s = t;
    }
    __device__ __forceinline__ void start(float pivot, float pivot1)
    {
        s1 = c1 = s2 = c2 = dup(0.0f);
        p = pk(pivot, pivot1);
    }
    __device__ __forceinline__ void take2(f2 x)
    {
        const f2 d = sub2(x, p), nd = negx2(d);
        const f2 bb = sub2(d, x);  // TwoSum of x and -p: bb is -p's share
        const f2 dl = sub2(sub2(x, sub2(d, bb)), add2(p, bb));
        const f2 q = mul2(d, d);
        csum2(s1, c1, d);
        c1 = add2(c1, dl);
        csum2(s2, c2, q);
        c2 = sub2(c2, fma2(add2(nd, nd), dl, fma2(nd, d, q)));  // less q - d^2 - 2 d dl
    }
    // one element: the other half adds zero
    __device__ __forceinline__ void take(float x) { take2(pk(x, half(p, 1))); }
    __device__ __forceinline__ Sums sums() const
    {
        Sums r{CSum{half(s1, 0), half(c1, 0)}, CSum{half(s2, 0), half(c2, 0)}, half(p, 0), 1.0f};
        csum_merge(r.s1, CSum{half(s1, 1), half(c1, 1)});
        csum_merge(r.s2, CSum{half(s2, 1), half(c2, 1)});
        return r;
    }
    // of one half alone
    __device__ __forceinline__ Sums sums(int i, float piv) const
    {
        return Sums{CSum{half(s1, i), half(c1, i)}, CSum{half(s2, i), half(c2, i)}, piv, 1.0f};
    }
    // Whether the n deviations, summing to a and their squares to b, are worth
    // summing again about their mean: squares past the float range though no
    // element is infinite or not a number, or a pivot so far off (more than 2.8
    // times the deviation; a trend's start is 1.7) that bringing the squares to the
    // mean cancels more than three of their bits.
    static __device__ __forceinline__ bool off(float a, float b, float n)
    {
        if (!(b - b == 0.0f)) return a - a == 0.0f;
        return 1.125f * a * __fdividef(a, n) > b;
    }
    static __device__ __forceinline__ bool off(const Sums &r, int64_t n)
    {
        const float a = r.s1.s + r.s1.c, b = r.s2.s + r.s2.c;
        return off(r.up == 1.0f ? a : a * 0x1p32f, b, (float)n);  // (squares scaled by 2^-64)
    }
    // of FP64 sums that may be out of the float range
    static __device__ __forceinline__ bool off(double a, double b, int64_t n)
    {
        const float fb = (float)b;
        if (fb - fb == 0.0f) return off((float)a, fb, (float)n);
        return b - b == 0.0 ? 1.125 * a * (a / (double)n) > b : a - a == 0.0;
    }
    static __device__ __forceinline__ float mean(const Sums &r, int64_t n)
    {
        return r.piv + r.up * __fdividef(r.s1.s + r.s1.c, (float)n);
    }
};

// max/min over batches of up to 32 elements: the batch's extreme over the W
// lanes that work together first (an instruction an element), and only when
// it reaches the running one are the positions looked for -- about the
// logarithm of the number of batches for data in no order.  W lanes of `mask`
// call it together.
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b)
{
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <bool MX, bool FIRST, int W> struct BatchRun {
    // not a number: nothing yet, so the first batch's extreme is a new one whatever
    // it is, the neutral infinity too (masked elements, logarithms of zeros)
    float cur = NT2G_FOLD_NAN, v = 0.0f;
    int32_t ifirst = -1, ilast = -1, inan = -1;
    // elements e[u][c], u < n, at positions pos + u * step + c
    template <int U, int V>
    __device__ __forceinline__ void batch(const float (&e)[U][V], int n, int32_t pos, int32_t step, unsigned mask)
    {
        float m = MX ? -NT2G_FOLD_INF : NT2G_FOLD_INF;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < V; ++c)
                if (u < n) m = MX ? max_nan(m, e[u][c]) : min_nan(m, e[u][c]);
        if constexpr (W > 1) {
#pragma unroll
            for (int off = W / 2; off; off >>= 1) {
                const float o = __shfl_xor_sync(mask, m, off);
                m = MX ? max_nan(m, o) : min_nan(m, o);
            }
        }
        if (better<MX>(cur, m)) return;
        // Equal numbers have equal bits but for zeros, so only there does the last
        // one matter; otherwise the first position of a new extreme is all.
        if (m == m && m != cur) {
            cur = v = m;
            ifirst = ilast = -1;
            if (!FIRST && m != 0.0f) {
                ilast = pos;
            } else if (m != 0.0f) {
#pragma unroll
                for (int u = U - 1; u >= 0; --u)
#pragma unroll
                    for (int c = V - 1; c >= 0; --c)
                        if (u < n && e[u][c] == m) ifirst = pos + u * step + c;
                ilast = ifirst;
            }
        } else if (U * V == 1 && n && e[0][0] == m && m != 0.0f) {  // the ends of a segment come last
            ifirst = (unsigned)pos < (unsigned)ifirst ? pos : ifirst;
            ilast = ifirst;
        }
        if (m != m) rare<true>(e, n, pos, step);  // elements beside a NaN count for nothing: the result is the NaN
        else if (m == 0.0f) rare<false>(e, n, pos, step);
    }
    // The first NaN, or the first and the last zero.
    template <bool NANS, int U, int V>
    __device__ __forceinline__ void rare(const float (&e)[U][V], int n, int32_t pos, int32_t step)
    {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < V; ++c)
                if (u < n && (NANS ? e[u][c] != e[u][c] : e[u][c] == 0.0f)) {
                    const int32_t at = pos + u * step + c;
                    if (NANS) {
                        inan = (unsigned)at < (unsigned)inan ? at : inan;
                    } else {
                        ifirst = (unsigned)at < (unsigned)ifirst ? at : ifirst;
                        if (at > ilast) { ilast = at; v = e[u][c]; }
                    }
                }
    }
    // The result of the W lanes together (they share `cur`).
    __device__ __forceinline__ Best best(int64_t base, unsigned mask) const
    {
        const unsigned nan = lanes_min((unsigned)inan, mask), first = lanes_min((unsigned)ifirst, mask);
        const unsigned last = ~lanes_min(~(unsigned)(ilast + 1), mask);  // the largest ilast + 1
        const int owner = __ffs(__ballot_sync(mask, ilast >= 0 && (unsigned)(ilast + 1) == last) & mask) - 1;
        const float val = __shfl_sync(mask, v, owner < 0 ? (int)(threadIdx.x & 31) : owner);
        if (nan != ~0u) return Best{__int_as_float(0x7fffffff), base + nan, base + nan};
        if (last == 0) return Best{0.0f, -1, -1};
        return Best{val, base + last - 1, FIRST ? base + first : base + last - 1};
    }
    static __device__ __forceinline__ unsigned lanes_min(unsigned x, unsigned mask)
    {
        if constexpr (W == 32) {
            return __reduce_min_sync(mask, x);
        } else {
#pragma unroll
            for (int off = W / 2; off; off >>= 1) {
                const unsigned o = __shfl_xor_sync(mask, x, off);
                x = o < x ? o : x;
            }
            return x;
        }
    }
    __device__ __forceinline__ Best to_best(int64_t base) const
    {
        if (inan >= 0) return Best{__int_as_float(0x7fffffff), base + inan, base + inan};
        if (ilast < 0) return Best{0.0f, -1, -1};
        return Best{v, base + ilast, base + ifirst};
    }
};

// ------------------------------------------- merges over W lanes (fast) --
template <int W> __device__ __forceinline__ CSum lanes_csum(CSum a, unsigned mask)
{
#pragma unroll
    for (int off = W / 2; off; off >>= 1) {
        const CSum b{__shfl_down_sync(mask, a.s, off), __shfl_down_sync(mask, a.c, off)};
        csum_merge(a, b);
    }
    return a;
}
// The sums of W lanes, TWO or the first alone.  `check`: where lanes within the
// float range are not together, again with every lane's share scaled -- in folds of
// expressions by a call, seldom made: inline it took registers from their loads
// (sum(abs(x - y), 1) of 16384 squared 7.5e11 elements/s, 8.6e11 so; a table's, sum(A,
// 1) of the same size, 1.76e12 inline and 1.71e12 by a call).
template <int W, bool TWO> __device__ NT2G_FOLD_SELDOM void lanes_scaled(Sums &r, CSum a1, CSum a2, unsigned mask)
{
    constexpr float down = 0x1p-64f;
    r.up = 0x1p64f;
    r.s1 = lanes_csum<W>(CSum{a1.s * down, a1.c * down}, mask);
    if constexpr (TWO) r.s2 = lanes_csum<W>(CSum{a2.s * down, a2.c * down}, mask);
}
template <int W, bool TWO> __device__ __forceinline__ void lanes_sums(Sums &r, unsigned mask, bool check)
{
    const CSum a1 = r.s1, a2 = r.s2;
    r.s1 = lanes_csum<W>(a1, mask);
    if constexpr (TWO) r.s2 = lanes_csum<W>(a2, mask);
    r.up = 1.0f;
    if (!check) return;
    bool out = !(r.s1.s - r.s1.s == 0.0f);
    if constexpr (TWO) out |= !(r.s2.s - r.s2.s == 0.0f);
    if (__shfl_sync(mask, (int)out, (int)(threadIdx.x & 31 & ~(W - 1)))) lanes_scaled<W, TWO>(r, a1, a2, mask);
}
template <int W> __device__ __forceinline__ double lanes_sum64(double a, unsigned mask)
{
#pragma unroll
    for (int off = W / 2; off; off >>= 1) a += __shfl_down_sync(mask, a, off);
    return a;
}
template <int W> __device__ __forceinline__ double lanes_prod(double a, unsigned mask)
{
#pragma unroll
    for (int off = W / 2; off; off >>= 1) a *= __shfl_down_sync(mask, a, off);
    return a;
}
template <bool MX, int W> __device__ __forceinline__ Best lanes_best(Best a, unsigned mask)
{
#pragma unroll
    for (int off = W / 2; off; off >>= 1) {
        const Best b{__shfl_down_sync(mask, a.v, off), __shfl_down_sync(mask, a.ilast, off),
                     __shfl_down_sync(mask, a.ifirst, off)};
        a = best_merge<MX>(a, b);  // symmetric: lanes hold interleaved elements
    }
    return a;
}

// ---------------------------------------------------- a thread's own ring --
// A table's vectors go through shared memory, where a thread's next kRing of
// them wait without holding registers: S at a time, each thread its own slots,
// so there is nothing to synchronise.  (Loads into registers were in flight
// only between one batch's arithmetic and the next.  6000 x 8192, along either
// dimension: variances 56 us then, 55 and 52 now, which leaves their two dozen
// operations a pair; means 35, now 33; maxima along rows 45, now 40.)
constexpr int kRing = 8;
__device__ __forceinline__ void ring_copy(float4 *to, const float *from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
// take(e, n, r): the thread's rows r .. r + n of `rows`, `stride` floats apart
// from `at` on, as e[u][0..4)
template <int S, class Take>
__device__ __forceinline__ void ring_rows(float4 *ring, const float *at, int64_t stride, int rows, Take take)
{
    constexpr int R = kRing / S;
    float4 *const mine = ring + threadIdx.x;
    auto fill = [&](int s) {
#pragma unroll
        for (int u = 0; u < S; ++u) {
            if (s * S + u < rows) ring_copy(mine + ((s & (R - 1)) * S + u) * kThreads, at);
            at += stride;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < R; ++s) fill(s);
    for (int s = 0; s * S < rows; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(R - 1) : "memory");
        float e[S][4];
#pragma unroll
        for (int u = 0; u < S; ++u) {
            const float4 v = mine[((s & (R - 1)) * S + u) * kThreads];
            e[u][0] = v.x; e[u][1] = v.y; e[u][2] = v.z; e[u][3] = v.w;
        }
        if (rows - s * S >= S) take(e, S, s * S);
        else take(e, rows - s * S, s * S);
        fill(s + R);  // (the slot just read)
    }
}

// ----------------------------------------- contiguous segments (lo == 1) --
// G threads (8, 32 or the block's 256) per (segment, chunk) work item, a few
// items a block one after the other: a segment's loads are in flight at once
// and blocks are short (a warp per segment of 6000 left the last wave of
// blocks alone on the GPU for a quarter of the time: 39 us for 8192 of them,
// 33 now).  Whole vectors wherever the segment starts: the ends before the
// first and after the last multiple of 4 go element by element.  FINAL: one
// chunk per segment; a block turns all its items into outputs at its end, a
// thread each (FP64).  vec: the source is 16-byte addressable at multiples of 4.
template <bool FIRST, class A, class B> struct Pick { typedef A type; };
template <class A, class B> struct Pick<false, A, B> { typedef B type; };
template <class Src, int OP, bool FINAL, bool IDX, int G>
__device__ __forceinline__ void inner_body(const Src &src, int64_t inner, int64_t hi, int64_t chunk, int64_t q,
                                           int vec, Partial *__restrict__ part, float *__restrict__ out,
                                           int64_t *__restrict__ index, const float *__restrict__ cen,
                                           double *__restrict__ out64)
{
    constexpr bool MX = OP == MAX, EXT = OP == MAX || OP == MIN;
    constexpr int W = G < 32 ? G : 32, kGroups = kThreads / G, kWarps = kThreads / 32;
    constexpr int kBatch = Src::kBatch;
    constexpr bool kAsync = Src::kAsync && !EXT;  // (extremes look at a batch of all lanes)
    __shared__ float4 s_ring[kAsync ? kRing * kThreads : 1];
    static_assert(FINAL || G > 32, "chunks are a block's");
    typedef typename Pick<(G > 32), Partial, Share>::type Item;
    __shared__ Item s_item[FINAL ? kItems : 1];
    __shared__ typename Pick<is_sum(OP), Share, Item>::type s_warp[2][kWarps];
    __shared__ float s_mean;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tid = threadIdx.x % G;
    const unsigned mask = W == 32 ? 0xffffffffu : 0xffu << (lane & 24);
    const int64_t items = hi * q;
    const int per = (int)(((items + gridDim.x - 1) / gridDim.x + kGroups - 1) / kGroups) * kGroups;  // <= kItems
    const int64_t item0 = (int64_t)blockIdx.x * per;
    const bool long_segment = G > 8 && chunk > 1024;  // (shorter ones are a warp's whole range anyhow)
    int turn = 0;
    for (int i = threadIdx.x / G; i < per && item0 + i < items; i += kGroups) {
        const int64_t item = item0 + i, seg = item / q, c = item - seg * q;
        const int64_t k0 = c * chunk, k1 = (k0 + chunk < inner) ? k0 + chunk : inner;
        const int64_t p0 = seg * inner + k0, p1 = seg * inner + k1;  // positions in the table
        CSum acc{0.0f, 0.0f};
        double prod = 1.0;
        VarAcc var;
        BatchRun<MX, IDX, W> run;
        const float m = OP == MEANAD ? cen[seg] : 0.0f;
        const float md = OP == MEANAD ? cen[hi + seg] : 0.0f;
        // n batch rows e[u][0..V) at position pos + u * step (relative to p0)
        auto take = [&](const auto &e, int n, int32_t pos, int32_t step) {
            [[maybe_unused]] constexpr int U = sizeof(e) / sizeof(e[0]), V = sizeof(e[0]) / sizeof(float);
            if constexpr (EXT) {
                run.batch(e, n, pos, step, mask);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (u >= n) break;
                    if constexpr (is_var(OP) && V == 4) {
                        var.take2(pk(e[u][0], e[u][1]));
                        var.take2(pk(e[u][2], e[u][3]));
                    } else {
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            if constexpr (is_var(OP)) var.take(e[u][v]);
                            else if constexpr (OP == PROD) prod *= (double)e[u][v];
                            else sum_elem_c<OP>(acc, e[u][v], m, md);
                        }
                    }
                }
            }
        };
        auto sweep = [&]() {
            if (vec) {
                const int64_t a = (p0 + 3) >> 2, b = p1 >> 2;  // whole vectors [a, b)
                if constexpr (kAsync) {
                    const int64_t left = b - a - tid;
                    ring_rows<2>(s_ring, src.x + 4 * (a + tid), 4 * G, left > 0 ? (int)((left + G - 1) / G) : 0,
                                 [&](const float(&e)[2][4], int n, int) { take(e, n, 0, 0); });
                } else {
                    for (int64_t j = a; j < b; j += kBatch * G) {
                        const int64_t left = b - j - tid;
                        float e[kBatch][4];
                        typename Src::Raw raw[kBatch];
                        const int n = left <= 0 ? 0 : left > (kBatch - 1) * G ? kBatch : (int)((left + G - 1) / G);
    #pragma unroll
                        for (int u = 0; u < kBatch; ++u) {  // (past the end: the last one again, so that no load waits for a branch)
                            const int64_t at = j + tid + u * G;
                            raw[u] = src.fetch4(4 * (at < b ? at : b - 1));
                        }
    #pragma unroll
                        for (int u = 0; u < kBatch; ++u) {
                            const int64_t at = j + tid + u * G;
                            src.value4(raw[u], 4 * (at < b ? at : b - 1), e[u]);
                        }
                        const int32_t pos = (int32_t)(4 * (j + tid) - p0);
                        if (j + kBatch * G <= b) take(e, kBatch, pos, 4 * G);
                        else take(e, n, pos, 4 * G);
                    }
                }
                // up to three elements on either side
                const int64_t first = 4 * a < p1 ? 4 * a : p1, last = 4 * b > first ? 4 * b : first;
                if (p0 < first || last < p1) {
                    const int64_t at = tid < 4 ? p0 + tid : last + tid - 4;
                    const int n = tid < 4 ? at < first : tid < 8 && at < p1;
                    float e[1][1];
                    if (n) e[0][0] = src.at(at);
                    take(e, n, (int32_t)(at - p0), 0);
                }
            } else {
                for (int64_t j = p0; j < p1; j += kBatch * G) {
                    const int64_t left = p1 - j - tid;
                    float e[kBatch][1];
                    typename Src::Raw raw[kBatch];
                    const int n = left <= 0 ? 0 : left > (kBatch - 1) * G ? kBatch : (int)((left + G - 1) / G);
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const int64_t at = j + tid + u * G;
                        raw[u] = src.fetch(at < p1 ? at : p1 - 1);
                    }
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const int64_t at = j + tid + u * G;
                        e[u][0] = src.value(raw[u], at < p1 ? at : p1 - 1);
                    }
                    take(e, n, (int32_t)(j + tid - p0), G);
                }
            }
        };
        // the item's threads together; thread 0 of the item has the result.
        // (Two sets of shared slots in turn: a barrier an item is enough.)
        Item r;
        bool off = false;   // a variance: to be summed again, about
        float mean = 0.0f;  // its mean
        auto together = [&]() {
            if constexpr (is_sum(OP)) {
                Share w;
                if constexpr (is_var(OP)) w.v = var.sums();
                else w.v.s1 = acc;
                lanes_sums<W, is_var(OP)>(w.v, mask, long_segment);
                if constexpr (G > 32) {
                    if (lane == 0) s_warp[turn][wid] = w;
                    __syncthreads();
                    if (threadIdx.x < kWarps) {
                        w = s_warp[turn][lane];
                        constexpr unsigned few = (1u << kWarps) - 1;
                        r.v.s1 = lanes_sum64<kWarps>(wide(w.v.s1, w.v.up), few);
                        if constexpr (is_var(OP)) {
                            r.v.s2 = lanes_sum64<kWarps>(wide(w.v.s2, w.v.up), few);
                            r.v.piv = w.v.piv;
                            off = VarAcc::off(r.v.s1, r.v.s2, k1 - k0);
                            if (off) mean = (float)((double)w.v.piv + r.v.s1 / (double)(k1 - k0));
                        }
                    }
                    turn ^= 1;
                } else {
                    r = w;
                    if constexpr (is_var(OP)) {
                        off = VarAcc::off(w.v, k1 - k0);
                        mean = VarAcc::mean(w.v, k1 - k0);
                    }
                }
            } else {
                if constexpr (EXT) r.b = run.best(k0, mask);
                else r.d = lanes_prod<W>(prod, mask);
                if constexpr (G > 32) {
                    if (lane == 0) s_warp[turn][wid] = r;
                    __syncthreads();
                    if (threadIdx.x < kWarps) {
                        r = s_warp[turn][lane];
                        constexpr unsigned few = (1u << kWarps) - 1;
                        if constexpr (EXT) r.b = lanes_best<MX, kWarps>(r.b, few);
                        else r.d = lanes_prod<kWarps>(r.d, few);
                    }
                    turn ^= 1;
                }
            }
        };
        float piv = 0.0f;  // the mean of the first W elements, in every warp
        if constexpr (is_var(OP)) {
            const int few = k1 - k0 < W ? (int)(k1 - k0) : W, at = lane & (W - 1);
            if (at < few) piv = __fdividef(src.at(p0 + at), (float)few);
#pragma unroll
            for (int off = W / 2; off; off >>= 1) piv += __shfl_xor_sync(mask, piv, off);
            var.start(piv, piv);
        }
        sweep();
        together();
        if constexpr (is_var(OP)) {
            if (!off) mean = piv;
            if constexpr (G > 32) {
                if (threadIdx.x == 0) s_mean = mean;
                __syncthreads();
                mean = s_mean;
            } else {
                mean = __shfl_sync(mask, mean, lane & ~(W - 1));
            }
            if (mean != piv && mean - mean == 0.0f) {
                var.start(mean, mean);
                sweep();
                together();
            }
        }
        if (tid == 0) {
            if constexpr (FINAL) s_item[i] = r;
            else part[c * hi + seg] = r;
        }
    }
    if constexpr (FINAL) {
        __syncthreads();
        for (int i = threadIdx.x; i < per && item0 + i < items; i += kThreads) {
            Total<OP> t;
            t.set(s_item[i]);
            t.put(out, index, out64, item0 + i, hi, inner, cen);
        }
    }
}

// Short contiguous segments: one thread per segment, in order.
template <class Src, int OP>
__device__ __forceinline__ void short_body(const Src &src, int64_t inner, int64_t hi, float *__restrict__ out,
                                           int64_t *__restrict__ index, const float *__restrict__ cen,
                                           double *__restrict__ out64)
{
    for (int64_t seg = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; seg < hi;
         seg += (int64_t)gridDim.x * blockDim.x) {
        const int64_t base = seg * inner;
        CSum acc{0.0f, 0.0f};
        double prod = 1.0;
        Run<OP == MAX> run;
        VarAcc var;
        if constexpr (is_var(OP)) {
            // the first elements stay in registers: their mean is the pivot
            constexpr int F = 8;
            const int few = inner < F ? (int)inner : F;
            float e[F], piv = 0.0f;
#pragma unroll
            for (int u = 0; u < F; ++u) e[u] = u < few ? src.at(base + u) : 0.0f;
#pragma unroll
            for (int u = 0; u < F; ++u) piv += __fdividef(e[u], (float)few);
            auto sweep = [&](float piv) {
                var.start(piv, piv);
#pragma unroll
                for (int u = 0; u < F; u += 2) {
                    if (u + 2 <= few) var.take2(pk(e[u], e[u + 1]));
                    else if (u < few) var.take(e[u]);
                }
                int64_t k = F;
                for (; k + 2 <= inner; k += 2) var.take2(pk(src.at(base + k), src.at(base + k + 1)));
                if (k < inner) var.take(src.at(base + k));
            };
            sweep(piv);
            Share r;
            r.v = var.sums();
            const float mean = VarAcc::mean(r.v, inner);
            if (VarAcc::off(r.v, inner) && mean - mean == 0.0f) {
                sweep(mean);
                r.v = var.sums();
            }
            Total<OP> t;
            t.set(r);
            t.put(out, index, out64, seg, hi, inner, cen);
            continue;
        }
        const float m = OP == MEANAD ? cen[seg] : 0.0f;
        const float md = OP == MEANAD ? cen[hi + seg] : 0.0f;
        for (int64_t k = 0; k < inner; ++k) {
            const float v = src.at(base + k);
            if (is_sum(OP)) sum_elem_c<OP>(acc, v, m, md);
            else if (OP == PROD) prod *= (double)v;
            else run.add(v, (int32_t)k);
        }
        if (is_sum(OP)) fold_put<OP>(out, out64, seg, hi, (double)acc.s + (double)acc.c, inner, cen);
        else if (OP == PROD) { out[seg] = (float)prod; if (out64) out64[seg] = prod; }
        else {
            const Best b = run.to_best(0);
            out[seg] = b.v;
            if (index) index[seg] = b.ifirst;
        }
    }
}

// ---------------------------------------------- strided folds (lo > 1) --
// A block takes 32 threads' worth of outputs (VEC: four neighbouring ones each,
// via float4) over the chunk [c*ck, min((c+1)*ck, inner)) of the fold range,
// grid.y = chunk; its warps take every eighth row, a batch of rows in
// flight each, and their accumulators combine in shared memory: one partial
// per output and block.  (A thread per output and chunk wrote eight times the
// partials -- 20 MB for 6000 rows of 8192, 16 to 49 us to combine -- and had
// one or two loads in flight.)
template <class Src, int OP, int VEC, bool FINAL>
__device__ __forceinline__ void outer_body(const Src &src, int64_t lo, int64_t inner, int64_t hi, int64_t ck,
                                           int64_t q, Partial *__restrict__ part, float *__restrict__ out,
                                           int64_t *__restrict__ index, const float *__restrict__ cen,
                                           double *__restrict__ out64)
{
    constexpr bool MX = OP == MAX, EXT = OP == MAX || OP == MIN;
    constexpr int kWarps = kThreads / 32, kRows = Src::kBatch;
    constexpr bool kAsync = Src::kAsync && VEC == 4;
    // the rings, and then in their place the warps' partials
    constexpr int kPartBytes = kWarps * 32 * VEC * (int)sizeof(Share), kRingBytes = kAsync ? kRing * kThreads * 16 : 0;
    __shared__ __align__(16) char s_mem[kPartBytes > kRingBytes ? kPartBytes : kRingBytes];
    float4 *const s_ring = (float4 *)s_mem;
    Share(*const s_part)[32 * VEC] = (Share(*)[32 * VEC])s_mem;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t lv = lo / VEC;  // thread columns per h
    const int64_t c = blockIdx.y;
    const int64_t k0 = c * ck, k1 = (k0 + ck < inner) ? k0 + ck : inner;
    for (int64_t t0 = (int64_t)blockIdx.x * 32; t0 < lv * hi; t0 += (int64_t)gridDim.x * 32) {
        const int64_t t = t0 + lane;
        const bool live = t < lv * hi;
        const int64_t h = t / lv, l = (t - h * lv) * VEC;
        const int64_t base = l + lo * inner * h;
        CSum acc[VEC];
        double prod[VEC];
        BatchRun<MX, true, 1> run[VEC];
        // a variance's two sums of each output, one half of VarAcc's pairs each
        VarAcc var[(VEC + 1) / 2];
        float m[VEC], md[VEC], piv[VEC];
        auto start = [&]() {
#pragma unroll
            for (int v = 0; v < VEC; v += 2) var[v / 2].start(piv[v], piv[v + (VEC > 1)]);
        };
        auto fetch = [&](int64_t k) {
            if constexpr (VEC == 4) return src.fetch4(base + lo * k);
            else return src.fetch(base + lo * k);
        };
        auto value = [&](const typename Src::Raw &r, int64_t k, float (&e)[VEC]) {
            if constexpr (VEC == 4) src.value4(r, base + lo * k, e);
            else e[0] = src.value(r, base + lo * k);
        };
        // n rows k, k + kWarps, ...
        auto take = [&](const auto &e, int n, int64_t k) {
            constexpr int U = sizeof(e) / sizeof(e[0]);
            if constexpr (EXT) {
#pragma unroll
                for (int v = 0; v < VEC; ++v) {
                    float col[U][1];
#pragma unroll
                    for (int u = 0; u < U; ++u) col[u][0] = e[u][v];
                    run[v].batch(col, n, (int32_t)(k - k0), kWarps, 0);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (u >= n) break;
#pragma unroll
                    for (int v = 0; v < VEC; ++v) {
                        if constexpr (is_var(OP)) {  // (VEC == 1: both halves the same)
                            if (v % 2 == 0) var[v / 2].take2(pk(e[u][v], e[u][v + (VEC > 1)]));
                        } else if constexpr (OP == PROD) {
                            prod[v] *= (double)e[u][v];
                        } else {
                            sum_elem_c<OP>(acc[v], e[u][v], m[v], md[v]);
                        }
                    }
                }
            }
        };
        auto sweep = [&]() {
            if constexpr (kAsync) {
                const int64_t left = k1 - k0 - wid;
                ring_rows<EXT ? 4 : 2>(s_ring, src.x + base + lo * (k0 + wid), lo * kWarps,
                                       left > 0 ? (int)((left + kWarps - 1) / kWarps) : 0,
                                       [&](const auto &e, int n, int r) { take(e, n, k0 + wid + r * kWarps); });
                return;
            }
            int64_t k = k0 + wid;
            for (; k + (kRows - 1) * kWarps < k1; k += kRows * kWarps) {
                float e[kRows][VEC];
                typename Src::Raw raw[kRows];
#pragma unroll
                for (int u = 0; u < kRows; ++u) raw[u] = fetch(k + u * kWarps);
#pragma unroll
                for (int u = 0; u < kRows; ++u) value(raw[u], k + u * kWarps, e[u]);
                take(e, kRows, k);
            }
            for (; k < k1; k += kWarps) {
                float e[1][VEC];
                value(fetch(k), k, e[0]);
                take(e, 1, k);
            }
        };
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            acc[v] = CSum{0.0f, 0.0f};
            prod[v] = 1.0;
            m[v] = OP == MEANAD && live ? cen[l + v + lo * h] : 0.0f;
            md[v] = OP == MEANAD && live ? cen[lo * hi + l + v + lo * h] : 0.0f;
        }
        if constexpr (is_var(OP)) {  // the pivots: the mean of the warps' first rows
            __shared__ float s_first[kWarps][32 * VEC];
            const int few = k1 - k0 < kWarps ? (int)(k1 - k0) : kWarps;
#pragma unroll
            for (int v = 0; v < VEC; ++v) piv[v] = 0.0f;
            if (live && wid < few) value(fetch(k0 + wid), k0 + wid, piv);
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
                s_first[wid][lane * VEC + v] = __fdividef(piv[v], (float)few);
                piv[v] = 0.0f;
            }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < kWarps; ++w)
#pragma unroll
                for (int v = 0; v < VEC; ++v) piv[v] += s_first[w][lane * VEC + v];
            start();
        }
        if (live) sweep();
        // warps combine: thread i finishes output i of the block's
        auto give = [&]() {
            if constexpr (kAsync) __syncthreads();  // (the partials take the rings' place)
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
                Share &r = s_part[wid][lane * VEC + v];
                if constexpr (is_var(OP)) {
                    r.v = var[v / 2].sums(v & 1, piv[v]);
                } else if constexpr (EXT) {
                    r.b = run[v].to_best(k0);
                } else if constexpr (OP == PROD) {
                    r.d = prod[v];
                } else {
                    r.v.s1 = acc[v];
                }
            }
            __syncthreads();
        };
        bool off = false;   // a variance: to be summed again, about
        float mean = 0.0f;  // its mean
        auto together = [&](int i) {
            Partial r;
            if constexpr (is_sum(OP)) {
                Sum3 t1 = Sum3::of(s_part[0][i].v.s1), t2 = Sum3::of(s_part[0][i].v.s2);
#pragma unroll
                for (int w = 1; w < kWarps; ++w) {
                    t1.add(s_part[w][i].v.s1);
                    if constexpr (is_var(OP)) t2.add(s_part[w][i].v.s2);
                }
                r.v.s1 = t1.wide();
                if constexpr (is_var(OP)) {
                    r.v.s2 = t2.wide();
                    r.v.piv = s_part[0][i].v.piv;
                    const float n = (float)(k1 - k0), a = t1.s + t1.c, b = t2.s + t2.c;
                    off = VarAcc::off(a, b, n);
                    mean = r.v.piv + __fdividef(a, n);
                }
                if (!t1.in_range() || (is_var(OP) && !t2.in_range())) {  // warps within the float range are not together
                    double s1 = 0.0, s2 = 0.0;
                    for (int w = 0; w < kWarps; ++w) {
                        s1 += wide(s_part[w][i].v.s1);
                        if constexpr (is_var(OP)) s2 += wide(s_part[w][i].v.s2);
                    }
                    r.v.s1 = s1;
                    if constexpr (is_var(OP)) {
                        r.v.s2 = s2;
                        off = VarAcc::off(s1, s2, k1 - k0);
                        mean = (float)((double)r.v.piv + s1 / (double)(k1 - k0));
                    }
                }
                return r;
            } else {
                const Share &o = s_part[0][i];
                if constexpr (OP == PROD) r.d = o.d;
                else r.b = o.b;
#pragma unroll
                for (int w = 1; w < kWarps; ++w) {
                    const Share &o = s_part[w][i];
                    if constexpr (OP == PROD) r.d *= o.d;
                    else r.b = best_merge<MX>(r.b, o.b);
                }
                return r;
            }
        };
        give();
        const int i = threadIdx.x;
        Partial r;
        if (i < 32 * VEC) r = together(i);
        if constexpr (is_var(OP)) {
            __shared__ float s_mean[32 * VEC];
            const bool again = i < 32 * VEC && off && mean - mean == 0.0f;
            if (i < 32 * VEC) s_mean[i] = again ? mean : r.v.piv;
            if (__syncthreads_or(again)) {
#pragma unroll
                for (int v = 0; v < VEC; ++v) piv[v] = s_mean[lane * VEC + v];
                start();
                if (live) sweep();
                give();
                if (i < 32 * VEC) r = together(i);
            }
        }
        const int64_t ti = t0 + i / VEC;
        if (i < 32 * VEC && ti < lv * hi) {
            const int64_t hh = ti / lv, o = (ti - hh * lv) * VEC + i % VEC + lo * hh;
            if (FINAL) {
                Total<OP> t;
                t.set(r);
                t.put(out, index, out64, o, lo * hi, inner, cen);
            } else {
                part[c * (lo * hi) + o] = r;
            }
        }
        __syncthreads();
    }
}

// Strided folds of a few rows: a thread per output (VEC: four neighbouring ones),
// all its rows, a batch of them in flight.  (Rows shared out over a block's warps
// leave most of those idle, and the block's steps cost more than the rows: ten
// rows of 2^20 outputs, a sum and a maximum, 29 and 48 us so, 7.2 and 11 this way.)
template <class Src, int OP, int VEC>
__device__ __forceinline__ void columns_body(const Src &src, int64_t lo, int64_t inner, int64_t hi,
                                             float *__restrict__ out, int64_t *__restrict__ index,
                                             const float *__restrict__ cen, double *__restrict__ out64)
{
    constexpr bool MX = OP == MAX, EXT = OP == MAX || OP == MIN;
    const int64_t lv = lo / VEC, n_out = lo * hi;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < lv * hi; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t h = t / lv, l = (t - h * lv) * VEC, o = l + lo * h;
        const int64_t base = l + lo * inner * h;
        CSum acc[VEC];
        double prod[VEC];
        Run<MX> run[VEC];
        VarAcc var[(VEC + 1) / 2];
        float m[VEC], md[VEC], piv[VEC];
        bool again = false;
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            acc[v] = CSum{0.0f, 0.0f};
            prod[v] = 1.0;
            m[v] = OP == MEANAD ? cen[o + v] : 0.0f;
            md[v] = OP == MEANAD ? cen[n_out + o + v] : 0.0f;
        }
        // rows k .. k + U
        auto rows = [&](auto &e, int64_t k) {
            constexpr int U = sizeof(e) / sizeof(e[0]);
            typename Src::Raw raw[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (VEC == 4) raw[u] = src.fetch4(base + lo * (k + u));
                else raw[u] = src.fetch(base + lo * (k + u));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (VEC == 4) src.value4(raw[u], base + lo * (k + u), e[u]);
                else e[u][0] = src.value(raw[u], base + lo * (k + u));
            }
            if constexpr (is_var(OP)) {
                if (k == 0) {
                    if (!again) {  // the pivots: the mean of the first rows
#pragma unroll
                        for (int v = 0; v < VEC; ++v) {
                            piv[v] = 0.0f;
#pragma unroll
                            for (int u = 0; u < U; ++u) piv[v] += e[u][v] * (1.0f / U);
                        }
                    }
#pragma unroll
                    for (int v = 0; v < VEC; v += 2) var[v / 2].start(piv[v], piv[v + (VEC > 1)]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < VEC; ++v) {
                    if constexpr (is_var(OP)) {  // (VEC == 1: both halves the same)
                        if (v % 2 == 0) var[v / 2].take2(pk(e[u][v], e[u][v + (VEC > 1)]));
                    } else if constexpr (OP == PROD) {
                        prod[v] *= (double)e[u][v];
                    } else if constexpr (EXT) {
                        run[v].add(e[u][v], (int32_t)(k + u));
                    } else {
                        sum_elem_c<OP>(acc[v], e[u][v], m[v], md[v]);
                    }
                }
        };
        do {
            int64_t k = 0;
            for (; k + Src::kBatch <= inner; k += Src::kBatch) {
                float e[Src::kBatch][VEC];
                rows(e, k);
            }
            for (; k < inner; ++k) {
                float e[1][VEC];
                rows(e, k);
            }
            if constexpr (is_var(OP)) {
                if (again) break;
#pragma unroll
                for (int v = 0; v < VEC; ++v) {
                    const Sums r = var[v / 2].sums(v & 1, piv[v]);
                    const float mean = VarAcc::mean(r, inner);
                    if (VarAcc::off(r, inner) && mean - mean == 0.0f) {
                        piv[v] = mean;
                        again = true;
                    }
                }
            }
        } while (again);
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            if constexpr (OP == SUM || OP == ASUM1 || OP == ASUM2 || OP == NBTRUE || OP == NANSUM || OP == NOT_NAN) {
                if (!out64) {  // rounded once, without an FP64 instruction
                    out[o + v] = __fadd_rn(acc[v].s, acc[v].c);
                    continue;
                }
            }
            Share r;
            if constexpr (is_var(OP)) r.v = var[v / 2].sums(v & 1, piv[v]);
            else if constexpr (EXT) r.b = run[v].to_best(0);
            else if constexpr (OP == PROD) r.d = prod[v];
            else r.v = Sums{acc[v], acc[v], 0.0f, 1.0f};
            Total<OP> total;
            total.set(r);
            total.put(out, index, out64, o + v, n_out, inner, cen);
        }
    }
}

// ------------------------------------------------ NT2 policy: in order --
template <class Src, int OP>
__device__ __forceinline__ void nt2_body(const Src &src, int64_t lo, int64_t inner, int64_t hi,
                                         float *__restrict__ out, int64_t *__restrict__ index,
                                         const float *__restrict__ cen)
{
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < lo * hi; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t h = o / lo, l = o - h * lo;
        const int64_t base = l + lo * inner * h;
        float acc = OP == PROD ? 1.0f
                  : OP == MAX  ? -__int_as_float(0x7f800000)
                  : OP == MIN  ? __int_as_float(0x7f800000)
                               : 0.0f;
        const float m = is_two_pass(OP) ? cen[o] : 0.0f;
        for (int64_t k = 0; k < inner; ++k) {
            const float v = src.at(base + lo * k);
            if constexpr (is_var(OP)) {  // asum2(center(a)): (x - mean(a))^2 in order
                const float d = __fsub_rn(v, m);
                acc = __fadd_rn(acc, __fmul_rn(d, d));
                continue;
            }
            if constexpr (OP == MEANAD) {  // sum(abs(center(a))) in order
                acc = __fadd_rn(acc, fabsf(__fsub_rn(v, m)));
                continue;
            }
            if constexpr (is_count(OP)) {  // nbtrue: the sum of is_nez(x)
                acc = __fadd_rn(acc, v != 0.0f ? 1.0f : 0.0f);
                continue;
            }
            if constexpr (OP == NOT_NAN) {
                acc = __fadd_rn(acc, v == v ? 1.0f : 0.0f);
                continue;
            }
            if constexpr (OP == NANSUM || OP == NANMEAN) {  // sum(if_zero_else(is_nan(x), x))
                acc = __fadd_rn(acc, v == v ? v : 0.0f);
                continue;
            }
            switch (OP) {
            case PROD: acc = __fmul_rn(acc, v); break;
            case MAX: acc = (acc > v) ? acc : v; break;
            case MIN: acc = (acc < v) ? acc : v; break;
            case ASUM1: acc = __fadd_rn(acc, fabsf(v)); break;
            case ASUM2: case NORM2: acc = __fadd_rn(acc, __fmul_rn(v, v)); break;
            default: acc = __fadd_rn(acc, v); break;
            }
        }
        if (OP == MEAN || OP == MEANAD) acc = __fmul_rn(__fdiv_rn(1.0f, (float)inner), acc);  // mean: rec(n) * sum
        if (OP == NORM2) acc = __fsqrt_rn(acc);
        if constexpr (is_count(OP)) {
            const float n = (float)inner;
            acc = OP == NBTRUE ? acc
                : OP == ALL    ? (acc == n ? 1.0f : 0.0f)
                : OP == ANY    ? (acc != 0.0f ? 1.0f : 0.0f)
                               : (acc == 0.0f ? 1.0f : 0.0f);
        }
        if constexpr (OP == NANMEAN)  // rec(max(nbtrue(is_not_nan(a)), 1)) * nansum(a)
            acc = __fmul_rn(__fdiv_rn(1.0f, m > 1.0f ? m : 1.0f), acc);
        if constexpr (is_var(OP)) {  // var = f * asum2, f = n <= 1 ? 1 : rec(n - 1) (rec(n) for w = 1)
            const float n = (float)inner;
            const bool by_n = OP == VAR1 || OP == STDEV1;
            const float f = (n <= 1.0f) ? 1.0f : __fdiv_rn(1.0f, by_n ? n : __fsub_rn(n, 1.0f));
            acc = __fmul_rn(f, acc);
            if (OP == STDEV || OP == STDEV1) acc = __fsqrt_rn(acc);
        }
        out[o] = acc;
        if ((OP == MAX || OP == MIN) && index) {
            int64_t f = -1;
            for (int64_t k = 0; k < inner && f < 0; ++k)
                if (src.at(base + lo * k) == acc) f = k;
            index[o] = f;
        }
    }
}

}  // namespace fold
}  // namespace nt2g
