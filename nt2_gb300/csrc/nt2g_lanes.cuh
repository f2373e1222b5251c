// nt2g_lanes.cuh -- the fast policy's functions over the lanes a thread holds
// (in the run-time compiled kernels 4 consecutive elements of a transform, 4 or
// 8 of a batch item, 1 or 4 of a fold, 2 of reverse mode), two lanes per packed
// instruction, the special values handled once for all lanes: a thread
// first asks whether any of its lanes is outside the common range of the
// function, and if one is, all its lanes take the scalar function.  Within the
// common range each lane performs exactly the operations of the scalar
// function of nt2g_math.cuh, so both give the same bits, and the interpreter,
// which evaluates one lane at a time, agrees with the compiled kernels.
// What bounds these kernels is instruction issue: compares and selects per
// special value and lane were a third of it, packed arithmetic halves another
// (2^24 elements of sin(x) cos(y), pow(x, y) and erf(y) + gammaln(x) in one tie:
// 220 us one lane at a time, 142 so).
// Also compiled by NVRTC (the run-time source puts nt2g_math.cuh and
// nt2g_f2.cuh ahead of it).
#pragma once
#if !defined(__CUDACC_RTC__)
#include "nt2g_f2.cuh"
#include "nt2g_math.cuh"
#endif

namespace nt2g {

// log<Fast> of positive normal numbers, lane for lane.
__device__ __forceinline__ f2 log_pos_fast2(f2 z)
{
    float z0, z1;
    upk(z, z0, z1);
    const uint32_t u0 = f_bits(z0), u1 = f_bits(z1);
    const float m0 = bits_f((u0 & 0x007fffffu) | 0x3f000000u), m1 = bits_f((u1 & 0x007fffffu) | 0x3f000000u);
    const bool l0 = m0 < bits_f(NT2G_SQRT_2O_2), l1 = m1 < bits_f(NT2G_SQRT_2O_2);
    f2 fe = sub2(pk(bits_f(0x4B000000u | (uint32_t)((int32_t)u0 >> 23)),
                    bits_f(0x4B000000u | (uint32_t)((int32_t)u1 >> 23))),
                 pk(l0 ? 8388735.0f : 8388734.0f, l1 ? 8388735.0f : 8388734.0f));
    f2 m = pk(m0, m1);
    f2 mm = add2(m, m);
    float mm0, mm1;
    upk(mm, mm0, mm1);
    f2 x = sub2(pk(l0 ? mm0 : m0, l1 ? mm1 : m1), dup(1.0f));
    f2 x2 = mul2(x, x);
    f2 y = horner2(x, dup(bits_f(0xbda5dff0u)), bits_f(0x3e0229f9u), bits_f(0xbe04d6b7u), bits_f(0x3e116e80u),
                   bits_f(0xbe2a6aa0u), bits_f(0x3e4cd0a3u), bits_f(0xbe800064u), bits_f(0x3eaaaaa9u));
    y = mul2(mul2(y, x), x2);
    y = fma2(fe, dup(bits_f(NT2G_LOG_2LO)), y);
    y = fma2(dup(-0.5f), x2, y);
    return fma2(dup(bits_f(NT2G_LOG_2HI)), fe, add2(x, y));
}

__device__ __forceinline__ f2 erfc_tail_poly2(f2 w)
{
    f2 d = sub2(w, dup(0.5f));
    return horner2(d, dup(0x1.5af3d4p-5f), -0x1.38d8fcp-6f, -0x1.382c16p-4f, 0x1.c51560p-5f, 0x1.908f48p-4f,
                   -0x1.a94032p-4f, -0x1.604ccep-3f, 0x1.2a8c2ep-3f, 0x1.1e2dc2p-1f, 0x1.5fd384p-1f, 0x1.058672p-1f);
}

// 1/b correctly rounded for normal b whose reciprocal is normal (what
// Fast::div(1, b) gives): one Newton step on the SFU's reciprocal rounds
// correctly for every significand (tested over all 2^23, through gammaln, log1p
// and pow).
__device__ __forceinline__ f2 recip_rn2(f2 b)
{
    const f2 nb = negx2(b), y = lanes(b, [](float v) { return Fast::rcp(v); });
    return fma2(y, fma2(nb, y, dup(1.0f)), y);
}

// one lane of the pair (the array form below has the scalar's name)
template <class P> __device__ __forceinline__ void one_normcdf_pair(float x, float &pos, float &neg)
{
    normcdf_pair<P>(x, pos, neg);
}

namespace lane {

// A thread's lanes as an argument: the first L of an array of A.
template <int L, int A> struct Of {
    float (&v)[A];
};

__device__ __forceinline__ bool positive_normal(float x) { return f_bits(x) - 0x00800000u < 0x7f000000u; }

// e^a = (1 + s) 2^k, exp_fast_parts lane for lane.
__device__ __forceinline__ f2 exp_parts2(f2 a, f2 &scale)
{
    const f2 shifter = dup(12582912.0f);
    const f2 kf = fma2(a, dup(bits_f(NT2G_INVLOG_2)), shifter), nk = sub2(shifter, kf);
    f2 x = fma2(nk, dup(bits_f(NT2G_LOG_2HI)), a);
    x = fma2(nk, dup(bits_f(NT2G_LOG_2LO)), x);
    const f2 q = horner2(x, dup(0x1.a157b2p-13f), 0x1.6d4926p-10f, 0x1.1110c4p-7f, 0x1.5554e4p-5f, 0x1.555556p-3f, 0.5f);
    float k0, k1;
    upk(kf, k0, k1);  // 1.5 * 2^23 has no bits below the 23rd to be shifted out
    scale = pk(bits_f((f_bits(k0) << 23) + 0x3f800000u), bits_f((f_bits(k1) << 23) + 0x3f800000u));
    return fma2(q, mul2(x, x), x);
}
// exp<Fast> below Maxlog
__device__ __forceinline__ f2 exp2l(f2 a)
{
    f2 scale;
    const f2 s = exp_parts2(a, scale);
    float r0, r1, a0, a1;
    upk(mul2(add2(s, dup(1.0f)), scale), r0, r1);
    upk(a, a0, a1);
    return pk(a0 <= bits_f(NT2G_MINLOG) ? 0.0f : r0, a1 <= bits_f(NT2G_MINLOG) ? 0.0f : r1);
}
// erfc_tail_fast for a >= 0
template <bool HALF_SQ> __device__ __forceinline__ f2 erfc_tail2(f2 a)
{
    const float q = HALF_SQ ? 0.353553390593273762f : 0.5f, s2 = HALF_SQ ? -0.5f : -1.0f, amax = HALF_SQ ? 13.2f : 9.3f;
    const f2 one = dup(1.0f);
    const f2 nden = fma2(dup(-q), a, dup(-1.0f));
    const f2 ndlo = fma2(dup(-q), a, sub2(dup(-1.0f), nden));
    f2 w = lanes(nden, [](float v) { return Fast::rcp(-v); });
    w = fma2(w, fma2(nden, w, one), w);
    const f2 r = fma2(ndlo, w, fma2(nden, w, one));
    const f2 hi = mul2(a, a), lo = fma2(a, a, negx2(hi));
    f2 scale;
    f2 e = exp_parts2(mul2(dup(s2), hi), scale);
    const f2 c = fma2(dup(s2), lo, r);
    e = add2(e, fma2(c, e, c));
    const f2 wr = mul2(w, erfc_tail_poly2(w));
    float t0, t1, a0, a1;
    upk(mul2(fma2(e, wr, wr), scale), t0, t1);
    upk(a, a0, a1);
    return pk(a0 < amax ? t0 : 0.0f, a1 < amax ? t1 : 0.0f);
}

// The frame of every function: L lanes of arrays of A; scalar for NT2's policy
// or single lanes, or when any lane is odd(x).
#define NT2G_LANES_HEAD(scalar_stmt, odd_expr)                      \
    if constexpr (P::exact || L == 1) {                             \
        _Pragma("unroll") for (int j = 0; j < L; ++j) scalar_stmt;  \
        return;                                                     \
    }                                                               \
    bool odd = false;                                               \
    _Pragma("unroll") for (int j = 0; j < L; ++j) odd |= odd_expr;  \
    if (odd) {                                                      \
        _Pragma("unroll") for (int j = 0; j < L; ++j) scalar_stmt;  \
        return;                                                     \
    }

template <class P, int L, int A> __device__ __forceinline__ void exp(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::exp<P>(a[j]), !(a[j] < bits_f(NT2G_MAXLOG)))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) upk(exp2l(pk(a[j], a[j + 1])), r[j], r[j + 1]);
}

template <class P, int L, int A> __device__ __forceinline__ void log(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::log<P>(a[j]), !positive_normal(a[j]))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) upk(log_pos_fast2(pk(a[j], a[j + 1])), r[j], r[j + 1]);
}

// log1p where u = 1 + a is a positive normal number; the quotient of u's
// rounding error by u correctly rounded (Markstein: q + (c - q u) y with y the
// correctly rounded 1/u; c is 0 or at least 2^-49 where u != 1, so no step
// underflows; u = 1 divides exactly, and above 2^25 c is 0)
__device__ __forceinline__ f2 log1p2(f2 a, f2 u)
{
    const f2 c = sub2(a, sub2(u, dup(1.0f))), y = recip_rn2(u), nu = negx2(u);
    const f2 q = mul2(c, y);
    return add2(log_pos_fast2(u), fma2(fma2(nu, q, c), y, q));
}
template <class P, int L, int A> __device__ __forceinline__ void log1p(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::log1p<P>(a[j]), !positive_normal(Fast::add(1.0f, a[j])))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        const f2 x = pk(a[j], a[j + 1]);
        upk(log1p2(x, add2(dup(1.0f), x)), r[j], r[j + 1]);
    }
}

// exp(-x^2): exp_neg_sqr lane for lane
template <class P, int L, int A> __device__ __forceinline__ void exp_neg_sqr(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::exp_neg_sqr<P>(a[j]), is_nan(a[j]))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        const f2 x = pk(a[j], a[j + 1]), hi = mul2(x, x), nhi = negx2(hi), nlo = negx2(fma2(x, x, nhi));
        f2 scale;
        f2 s = exp_parts2(nhi, scale);
        s = add2(s, fma2(nlo, s, nlo));
        float r0, r1, h0, h1;
        upk(mul2(add2(s, dup(1.0f)), scale), r0, r1);
        upk(nhi, h0, h1);
        r[j] = h0 <= bits_f(NT2G_MINLOG) ? 0.0f : r0;
        r[j + 1] = h1 <= bits_f(NT2G_MINLOG) ? 0.0f : r1;
    }
}

template <class P, int L, int A>
__device__ __forceinline__ void normcdf_pair(const float (&a)[A], float (&pos)[A], float (&neg)[A])
{
    NT2G_LANES_HEAD(one_normcdf_pair<P>(a[j], pos[j], neg[j]), is_nan(a[j]))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        float t[2];
        upk(erfc_tail2<true>(pk(fabsf(a[j]), fabsf(a[j + 1]))), t[0], t[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float h = Fast::mul(0.5f, t[i]), o = Fast::sub(1.0f, h);
            const bool n = a[j + i] < 0.0f;
            pos[j + i] = n ? h : o;
            neg[j + i] = n ? o : h;
        }
    }
}
template <class P, int L, int A> __device__ __forceinline__ void normcdf(const float (&a)[A], float (&r)[A])
{
    float other[A];
    normcdf_pair<P, L>(a, r, other);
}

template <class P, int L, int A> __device__ __forceinline__ void fastnormcdf(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::fastnormcdf<P>(a[j]), is_nan(a[j]))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        const f2 l = pk(fminf(fabsf(a[j]), 100.0f), fminf(fabsf(a[j + 1]), 100.0f));
        const f2 nden = fma2(dup(-0.2316419f), l, dup(-1.0f));
        f2 k = lanes(nden, [](float v) { return Fast::rcp(-v); });
        k = fma2(fma2(nden, k, dup(1.0f)), k, k);
        f2 w = horner2(k, dup(bits_f(0x3faa466fu)), bits_f(0xbfe91eeau), bits_f(0x3fe40778u), bits_f(0xbeb68f87u),
                       bits_f(0x3ea385fau));
        w = mul2(w, mul2(mul2(k, dup(bits_f(NT2G_INVSQRT_2PI))), exp2l(mul2(mul2(l, l), dup(-0.5f)))));
        float w0, w1;
        upk(w, w0, w1);
        r[j] = a[j] > 0.0f ? Fast::sub(1.0f, w0) : w0;
        r[j + 1] = a[j + 1] > 0.0f ? Fast::sub(1.0f, w1) : w1;
    }
}

// sin and cos in radians up to NT2G_TRIG_FAST_MAX
template <class P, int L, int A, bool COS> __device__ __forceinline__ void sincos(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = COS ? nt2g::cos<P>(a[j]) : nt2g::sin<P>(a[j]), !(fabsf(a[j]) <= NT2G_TRIG_FAST_MAX))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        const f2 x = pk(fabsf(a[j]), fabsf(a[j + 1]));
        float t[2], kf[2];
        upk(mul2(x, dup(0x1.45f306p-1f)), t[0], t[1]);
        kf[0] = Fast::add(t[0], 12582912.0f);  // to the nearest integer, in the low bits
        kf[1] = Fast::add(t[1], 12582912.0f);
        const f2 nk = sub2(dup(12582912.0f), pk(kf[0], kf[1]));
        f2 xr = fma2(nk, dup(0x1.921fb6p+0f), x);
        xr = fma2(nk, dup(-0x1.777a5cp-25f), xr);
        xr = fma2(nk, dup(-0x1.ee59dap-50f), xr);
        const f2 z = mul2(xr, xr);
        const f2 yc = horner2(z, dup(bits_f(0x37ccf5ceu)), bits_f(0xbab60619u), bits_f(0x3d2aaaa5u));
        const f2 cv = add2(dup(1.0f), fma2(z, dup(-0.5f), mul2(yc, mul2(z, z))));
        const f2 ys = horner2(z, dup(bits_f(0xb94ca1f9u)), bits_f(0x3c08839du), bits_f(0xbe2aaaa2u));
        const f2 sv = fma2(mul2(ys, z), xr, xr);
        float c[2], s[2];
        upk(cv, c[0], c[1]);
        upk(sv, s[0], s[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t n = f_bits(kf[i]);
            const bool swap = n & 1u;
            const float v = COS ? (swap ? s[i] : c[i]) : (swap ? c[i] : s[i]);
            // cos: negative in quadrants 1 and 2; sin: in 2 and 3, times the argument's sign
            const uint32_t sign = COS ? (n + 1u) << 30 : f_bits(a[j + i]) ^ (n << 30);
            r[j + i] = bits_f(f_bits(v) ^ (sign & 0x80000000u));
        }
    }
}
template <class P, int L, int A> __device__ __forceinline__ void sin(const float (&a)[A], float (&r)[A])
{
    sincos<P, L, A, false>(a, r);
}
template <class P, int L, int A> __device__ __forceinline__ void cos(const float (&a)[A], float (&r)[A])
{
    sincos<P, L, A, true>(a, r);
}

// pow for positive normal a != 1 and finite b: pow_core_fast lane for lane
template <class P, int L, int A>
__device__ __forceinline__ void pow(const float (&a)[A], const float (&b)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::pow<P>(a[j], b[j]),
                    !positive_normal(a[j]) || a[j] == 1.0f || !(fabsf(b[j]) < f_inf()))
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        float m_[2], o_[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t u = f_bits(a[j + i]);
            const float m = bits_f((u & 0x007fffffu) | 0x3f800000u);
            const bool big = m > 1.41421354f;
            m_[i] = big ? Fast::mul(m, 0.5f) : m;
            o_[i] = big ? 8388734.0f : 8388735.0f;  // 2^23 + the bias (less one)
        }
        const f2 fe = sub2(pk(bits_f(0x4B000000u | f_bits(a[j]) >> 23), bits_f(0x4B000000u | f_bits(a[j + 1]) >> 23)),
                           pk(o_[0], o_[1]));
        const f2 m = pk(m_[0], m_[1]), y = pk(b[j], b[j + 1]), one = dup(1.0f);
        const f2 num = sub2(m, one), den = add2(m, one), den_lo = sub2(m, sub2(den, one));
        const f2 rc = recip_rn2(den);
        const f2 s_hi = mul2(num, rc), ns = negx2(s_hi);
        const f2 s_lo = mul2(fma2(ns, den_lo, fma2(ns, den, num)), rc);
        const f2 q_hi = mul2(s_hi, s_hi), q_lo = fma2(s_hi, s_hi, negx2(q_hi));
        const f2 c3_hi = mul2(s_hi, q_hi), c3_lo = fma2(s_hi, q_lo, fma2(s_hi, q_hi, negx2(c3_hi)));
        const f2 TT_hi = dup(0x1.555556p-1f), TT_lo = dup(-0x1.555556p-26f);
        const f2 t3_hi = mul2(c3_hi, TT_hi);
        const f2 t3_lo = fma2(c3_lo, TT_hi, fma2(c3_hi, TT_lo, fma2(c3_hi, TT_hi, negx2(t3_hi))));
        const f2 rest = mul2(mul2(c3_hi, q_hi), horner2(q_hi, dup(0x1.3b13b2p-3f), 0x1.745d18p-3f, 0x1.c71c72p-3f,
                                                        0x1.24924ap-2f, 0x1.99999ap-2f));
        const f2 s2 = mul2(dup(2.0f), s_lo);
        // (a product and its only sum: per lane, two roundings)
        const f2 tail = lanes(t3_lo, rest, [](float u, float v) { return Fast::add(u, v); });
        const f2 lo_sum = add2(fma2(s2, q_hi, s2), tail);
        const f2 h0 = add2(s_hi, s_hi), h = add2(h0, t3_hi);
        const f2 l = add2(add2(sub2(h0, h), t3_hi), lo_sum);
        const f2 l_hi = add2(h, l), l_lo = add2(sub2(h, l_hi), l);
        const f2 C_hi = dup(0x1.715476p+0f), C_lo = dup(0x1.4ae0c0p-26f);
        const f2 g_hi = mul2(l_hi, C_hi);
        const f2 g_lo = add2(fma2(l_hi, C_hi, negx2(g_hi)), fma2(l_lo, C_hi, mul2(l_hi, C_lo)));
        const f2 t_hi = add2(fe, g_hi), t_lo = add2(add2(sub2(fe, t_hi), g_hi), g_lo);
        const f2 p_hi = mul2(y, t_hi), p_lo = fma2(y, t_lo, fma2(y, t_hi, negx2(p_hi)));
        const f2 kf = lanes(p_hi, [](float v) { return Fast::add(v, 12582912.0f); });
        const f2 k = sub2(kf, dup(12582912.0f));
        const f2 f = add2(sub2(p_hi, k), p_lo);
        const f2 c = horner2(f, dup(0x1.ffcbfcp-17f), 0x1.430912p-13f, 0x1.5d87fep-10f, 0x1.3b2ab6p-7f, 0x1.c6b08ep-5f,
                             0x1.ebfbe0p-3f, 0x1.62e430p-1f);
        float v[2], k_[2], ph[2];
        upk(fma2(c, f, one), v[0], v[1]);
        upk(kf, k_[0], k_[1]);
        upk(p_hi, ph[0], ph[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int ki = (int)(f_bits(k_[i]) - 0x4B400000u), k1 = ki >> 1, k2 = ki - k1;
            float t = Fast::mul(Fast::mul(v[i], bits_f((uint32_t)(k1 + 127) << 23)), bits_f((uint32_t)(k2 + 127) << 23));
            t = ph[i] > -152.0f ? t : 0.0f;
            r[j + i] = ph[i] < 129.0f ? t : f_inf();
        }
    }
}

template <class P, int L, int A> __device__ __forceinline__ void erf(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::erf<P>(a[j]), is_nan(a[j]))
    bool large = false;
#pragma unroll
    for (int j = 0; j < L; ++j) large |= !(fabsf(a[j]) < bits_f(NT2G_TWOTHIRD));
    float tail[A];
    if (large)
#pragma unroll
        for (int j = 0; j + 1 < L; j += 2) upk(erfc_tail2<false>(pk(fabsf(a[j]), fabsf(a[j + 1]))), tail[j], tail[j + 1]);
#pragma unroll
    for (int j = 0; j + 1 < L; j += 2) {
        const f2 x = pk(a[j], a[j + 1]);
        float s[2];
        upk(mul2(x, horner2(mul2(x, x), dup(bits_f(0xba1fc83bu)), bits_f(0x3ba4468du), bits_f(0xbcdb61f4u),
                            bits_f(0x3de70f22u), bits_f(0xbec0937eu), bits_f(0x3f906ebau))),
            s[0], s[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float v = a[j + i], t = Fast::sub(1.0f, tail[j + i]);
            r[j + i] = fabsf(v) < bits_f(NT2G_TWOTHIRD) ? s[i] : v < 0.0f ? -t : t;
        }
    }
}

// gammaln for 2^-20 <= a <= Maxgammaln: gammaln_pos, its two ranges each taken
// where any lane needs it
template <class P, int L, int A> __device__ __forceinline__ void gammaln(const float (&a)[A], float (&r)[A])
{
    NT2G_LANES_HEAD(r[j] = nt2g::gammaln<P>(a[j]), !(a[j] >= 0x1p-20f && a[j] <= bits_f(0x7bc3f8eau)))
    bool small = false, large = false;
#pragma unroll
    for (int j = 0; j < L; ++j) {
        small |= a[j] < 6.5f;
        large |= !(a[j] < 6.5f);
    }
    if (small)
#pragma unroll
        for (int j = 0; j + 1 < L; j += 2) {
            // The steps towards (1.5, 2.5]: down by 1 to 4 from above 2.5 (exact
            // subtractions), up by 1 or 2 from below 1.5.  The products of all the
            // steps are at hand after four multiplications, and each comparison
            // picks the product and the shift of one more step.
            const f2 x = pk(a[j], a[j + 1]), one = dup(1.0f);
            const f2 d1 = sub2(x, one), d2 = mul2(d1, sub2(x, dup(2.0f))), d3 = mul2(d2, sub2(x, dup(3.0f))),
                     d4 = mul2(d3, sub2(x, dup(4.0f))), u1 = add2(x, one), u2 = mul2(x, u1);
            float z[2], nx[2], d1_[2], d2_[2], d3_[2], d4_[2], u1_[2], u2_[2];
            upk(d1, d1_[0], d1_[1]);
            upk(d2, d2_[0], d2_[1]);
            upk(d3, d3_[0], d3_[1]);
            upk(d4, d4_[0], d4_[1]);
            upk(u1, u1_[0], u1_[1]);
            upk(u2, u2_[0], u2_[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float v = a[j + i];
                z[i] = 1.0f, nx[i] = -2.0f;
                if (v < 1.5f) z[i] = v, nx[i] = -1.0f;
                if (u1_[i] < 1.5f) z[i] = u2_[i], nx[i] = 0.0f;
                if (v > 2.5f) z[i] = d1_[i], nx[i] = -3.0f;
                if (v > 3.5f) z[i] = d2_[i], nx[i] = -4.0f;
                if (v > 4.5f) z[i] = d3_[i], nx[i] = -5.0f;
                if (v > 5.5f) z[i] = d4_[i], nx[i] = -6.0f;
            }
            const f2 xb = add2(x, pk(nx[0], nx[1]));
            float lz[2];
            upk(log_pos_fast2(pk(z[0], z[1])), lz[0], lz[1]);
            const f2 gb = horner2(xb, dup(bits_f(0x3a1ebb94u)), bits_f(0xbaabeab1u), bits_f(0x3b3ba883u), bits_f(0xbbf164fdu),
                                  bits_f(0x3ca89ed8u), bits_f(0xbd89f07eu), bits_f(0x3ea51a64u), bits_f(0x3ed87730u));
            const f2 rb = fma2(xb, gb, pk(a[j] < 1.5f ? -lz[0] : lz[0], a[j + 1] < 1.5f ? -lz[1] : lz[1]));
            const f2 xc = sub2(x, one);
            const f2 rc = mul2(xc, horner2(xc, dup(bits_f(0x3e0c3c4fu)), bits_f(0xbe22d329u), bits_f(0x3e2d4dabu),
                                           bits_f(0xbe53c04fu), bits_f(0x3e8a898bu), bits_f(0xbecd27a8u), bits_f(0x3f528d34u),
                                           bits_f(0xbf13c468u)));
            float b_[2], c_[2];
            upk(rb, b_[0], b_[1]);
            upk(rc, c_[0], c_[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) r[j + i] = a[j + i] >= 0.75f && a[j + i] < 1.25f ? c_[i] : b_[i];
        }
    if (large)
#pragma unroll
        for (int j = 0; j + 1 < L; j += 2) {
            const f2 x = pk(a[j], a[j + 1]);
            const f2 g = fma2(sub2(x, dup(0.5f)), log_pos_fast2(x), sub2(dup(bits_f(0x3f6b3f8eu)), x));
            const f2 z = recip_rn2(x), p = mul2(z, z);
            const f2 gc = fma2(z, horner2(p, dup(bits_f(0x3a31fd69u)), bits_f(0xbb358701u), bits_f(0x3daaaa94u)), g);
            float g_[2], c_[2];
            upk(g, g_[0], g_[1]);
            upk(gc, c_[0], c_[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (!(a[j + i] < 6.5f)) r[j + i] = a[j + i] <= 1.0e4f ? c_[i] : g_[i];
        }
}

#undef NT2G_LANES_HEAD
}  // namespace lane

template <class P, int L, int A>
__device__ __forceinline__ void normcdf_pair(lane::Of<L, A> x, lane::Of<L, A> pos, lane::Of<L, A> neg)
{
    lane::normcdf_pair<P, L>(x.v, pos.v, neg.v);
}
}  // namespace nt2g
