// nt2g_fold.cu -- reductions along one dimension of a table or of an
// expression: the host side (plans, workspace, launches) and the kernels over
// a table.  The folding itself is nt2g_fold_kernels.cuh, shared with the
// run-time compiled kernels that fold an expression (nt2g_jit.cu).
#include "nt2g_fold_kernels.cuh"
#include "nt2g_common.cuh"
#include "nt2g_internal.h"

namespace nt2g {

using namespace fold;
static_assert((int)SUM == (int)NT2G_FOLD_SUM &&
              (int)PROD == (int)NT2G_FOLD_PROD &&
              (int)MAX == (int)NT2G_FOLD_MAX &&
              (int)MIN == (int)NT2G_FOLD_MIN &&
              (int)MEAN == (int)NT2G_FOLD_MEAN &&
              (int)ASUM1 == (int)NT2G_FOLD_ASUM1 &&
              (int)ASUM2 == (int)NT2G_FOLD_ASUM2 &&
              (int)NORM2 == (int)NT2G_FOLD_NORM2 &&
              (int)VAR == (int)NT2G_FOLD_VAR &&
              (int)STDEV == (int)NT2G_FOLD_STDEV &&
              (int)VAR1 == (int)NT2G_FOLD_VAR1 &&
              (int)STDEV1 == (int)NT2G_FOLD_STDEV1 &&
              (int)NBTRUE == (int)NT2G_FOLD_NBTRUE &&
              (int)ALL == (int)NT2G_FOLD_ALL &&
              (int)ANY == (int)NT2G_FOLD_ANY &&
              (int)NONE == (int)NT2G_FOLD_NONE &&
              (int)NANSUM == (int)NT2G_FOLD_NANSUM &&
              (int)NANMEAN == (int)NT2G_FOLD_NANMEAN &&
              (int)MEANAD == (int)NT2G_FOLD_MEANAD,
              "fold op numbering");

constexpr int kFoldThreads = kThreads;
constexpr int64_t kChunk = 16384;        // elements per chunk a contiguous fold asks workspace for
constexpr int64_t kWave = 152 * 4;       // blocks the GPU holds at once
constexpr int64_t kBlocks = 152 * 12;    // blocks a fold is cut into at least: a few waves, so that none is nearly empty
constexpr int64_t kSmallSeg = 64;        // (many) segments up to this length: one thread each
constexpr int64_t kMostPerThread = 512;  // elements of a contiguous segment that one thread sums

// A table as a fold source: streaming loads.
struct RawSrc {
    static constexpr int kBatch = 4;  // vectors a thread has in flight
    static constexpr bool kAsync = true;
    const float *x;
    typedef float4 Raw;
    __device__ __forceinline__ float at(int64_t pos) const { return ld_stream(x + pos); }
    __device__ __forceinline__ Raw fetch(int64_t pos) const { return make_float4(ld_stream(x + pos), 0.0f, 0.0f, 0.0f); }
    __device__ __forceinline__ Raw fetch4(int64_t pos) const { return ld_stream((const float4 *)(x + pos)); }
    __device__ __forceinline__ float value(const Raw &r, int64_t) const { return r.x; }
    __device__ __forceinline__ void value4(const Raw &r, int64_t, float (&e)[4]) const
    {
        e[0] = r.x; e[1] = r.y; e[2] = r.z; e[3] = r.w;
    }
};

template <int OP, bool FINAL, bool IDX, int G>
__global__ void __launch_bounds__(kFoldThreads, is_var(OP) ? 3 : 4) k_fold_inner(RawSrc src, int64_t inner, int64_t hi, int64_t chunk,
                                                             int64_t q, int vec, Partial *__restrict__ part,
                                                             float *__restrict__ out, int64_t *__restrict__ index,
                                                             const float *__restrict__ cen, double *__restrict__ out64)
{
    pdl_trigger();  // the kernel that combines the partials lines up
    pdl_wait_for(src.x, part, out, index, cen, out64);
    inner_body<RawSrc, OP, FINAL, IDX, G>(src, inner, hi, chunk, q, vec, part, out, index, cen, out64);
}

template <int OP>
__global__ void __launch_bounds__(kFoldThreads) k_fold_short(RawSrc src, int64_t inner, int64_t hi,
                                                             float *__restrict__ out, int64_t *__restrict__ index,
                                                             const float *__restrict__ cen, double *__restrict__ out64)
{
    short_body<RawSrc, OP>(src, inner, hi, out, index, cen, out64);
}

template <int OP, int VEC, bool FINAL>
__global__ void __launch_bounds__(kFoldThreads, is_var(OP) ? 3 : 4) k_fold_outer(RawSrc src, int64_t lo, int64_t inner, int64_t hi,
                                                             int64_t ck, int64_t q, Partial *__restrict__ part,
                                                             float *__restrict__ out, int64_t *__restrict__ index,
                                                             const float *__restrict__ cen, double *__restrict__ out64)
{
    pdl_trigger();
    pdl_wait_for(src.x, part, out, index, cen, out64);
    outer_body<RawSrc, OP, VEC, FINAL>(src, lo, inner, hi, ck, q, part, out, index, cen, out64);
}

template <int OP, int VEC>
__global__ void __launch_bounds__(kFoldThreads, VEC == 4 || is_var(OP) || OP == MEANAD ? 4 : 8)
k_fold_columns(RawSrc src, int64_t lo, int64_t inner, int64_t hi, float *__restrict__ out, int64_t *__restrict__ index,
               const float *__restrict__ cen, double *__restrict__ out64)
{
    pdl_trigger();
    pdl_wait_for(src.x, out, index, cen, out64);
    columns_body<RawSrc, OP, VEC>(src, lo, inner, hi, out, index, cen, out64);
}

template <int OP>
__global__ void __launch_bounds__(kFoldThreads) k_fold_nt2(RawSrc src, int64_t lo, int64_t inner, int64_t hi,
                                                           float *__restrict__ out, int64_t *__restrict__ index,
                                                           const float *__restrict__ cen)
{
    nt2_body<RawSrc, OP>(src, lo, inner, hi, out, index, cen);
}

// Combine the q partials of each output: 32 outputs a block, the partials of
// neighbouring outputs next to each other, in eight consecutive ranges of
// chunks (a thread each), whose totals then combine in order.
constexpr int kRanges = kFoldThreads / 32;
template <int OP>
__global__ void __launch_bounds__(kFoldThreads) k_fold_finish(const Partial *__restrict__ part, int64_t n_out,
                                                              int64_t q, int64_t chunk, int64_t inner,
                                                              float *__restrict__ out, int64_t *__restrict__ index,
                                                              const float *__restrict__ cen, double *__restrict__ out64)
{
    __shared__ Total<OP> st[kRanges][32];
    pdl_trigger();
    pdl_wait_for(part, out, index, cen, out64);
    const int lane = threadIdx.x & 31, range = threadIdx.x >> 5;
    const int64_t per = (q + kRanges - 1) / kRanges, c0 = range * per, c1 = c0 + per < q ? c0 + per : q;
    for (int64_t o0 = (int64_t)blockIdx.x * 32; o0 < n_out; o0 += (int64_t)gridDim.x * 32) {
        const int64_t o = o0 + lane;
        Total<OP> t;
        if (o < n_out)
#pragma unroll 4
            for (int64_t c = c0; c < c1; ++c)
                t.add(part[c * n_out + o], (double)(inner - c * chunk < chunk ? inner - c * chunk : chunk));
        st[range][lane] = t;
        __syncthreads();
        if (range == 0 && o < n_out) {
            for (int r = 1; r < kRanges; ++r) {
                const int64_t k0 = r * per * chunk, k1 = (r + 1) * per * chunk < inner ? (r + 1) * per * chunk : inner;
                t.add(st[r][lane], k1 > k0 ? (double)(k1 - k0) : 0.0);
            }
            t.put(out, index, out64, o, n_out, inner, cen);
        }
        __syncthreads();
    }
}

// Few outputs of many partials (global folds): one block per output, thread t
// combining its consecutive partials, then a shared-memory tree over the
// threads' totals in order.
template <int OP>
__global__ void __launch_bounds__(kFoldThreads) k_fold_finish_block(const Partial *__restrict__ part, int64_t n_out,
                                                                    int64_t q, int64_t chunk, int64_t inner,
                                                                    float *__restrict__ out,
                                                                    int64_t *__restrict__ index,
                                                                    const float *__restrict__ cen,
                                                                    double *__restrict__ out64)
{
    __shared__ Total<OP> st[kFoldThreads];
    pdl_trigger();
    pdl_wait_for(part, out, index, cen, out64);
    const int64_t per = (q + kFoldThreads - 1) / kFoldThreads, c0 = threadIdx.x * per,
                  c1 = c0 + per < q ? c0 + per : q;
    for (int64_t o = blockIdx.x; o < n_out; o += gridDim.x) {
        Total<OP> t;
#pragma unroll 8
        for (int64_t c = c0; c < c1; ++c)
            t.add(part[c * n_out + o], (double)(inner - c * chunk < chunk ? inner - c * chunk : chunk));
        st[threadIdx.x] = t;
        __syncthreads();
        for (int w = 1; w < kFoldThreads; w <<= 1) {
            if ((threadIdx.x & (2 * w - 1)) == 0) {
                const int64_t k0 = (threadIdx.x + w) * per * chunk, k = k0 + w * per * chunk, k1 = k < inner ? k : inner;
                st[threadIdx.x].add(st[threadIdx.x + w], k1 > k0 ? (double)(k1 - k0) : 0.0);
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) st[0].put(out, index, out64, o, n_out, inner, cen);
        __syncthreads();
    }
}

// --------------------------------------------------------------- plans --
struct FoldPlan {
    int kind = 0;       // 0 short segments, 1 contiguous (lo == 1), 2 strided, 3 strided with few rows
    int group = 0;      // contiguous: log2 of the threads per segment, as the index 0: 8, 1: 32, 2: 256
    int64_t chunk = 0;  // elements per chunk along the fold
    int64_t q = 1;      // chunks per output
    int vec = 0;
};

// Whether a strided fold goes a thread per output, its rows one after the other
// (columns_body), rather than shared out over a block's warps: few rows always,
// more of them the more outputs there are to keep the GPU's loads in flight; more
// than 31 rows only where a thread each fills the GPU, and not where the FP64 result
// is asked for (a thread's sum is a pair of floats, what blocks hand on FP64).  Aligned rows (four outputs a thread; times
// in us, warps and columns): 10^5 sums of 8 rows 4.4 and 2.2, of 24 5.2 and 3.6;
// 4096 of 8 2.1 and 1.9, of 24 2.2 and 2.9; 2^20 of 64 53 and 40.  Others (one
// output a thread, a warp's rows 128 bytes): 62000 sums of 24 rows 6.7 and 3.0,
// maxima of 48 10.5 and 6.3; 301000 sums of 200 62.9 and 44.2.
static bool by_columns(int64_t threads, int64_t inner, bool aligned, int op, bool want64)
{
    if (inner <= 8) return true;
    if ((op == MAX || op == MIN) && !aligned && threads >= 49152 && inner <= 64) return true;
    const bool many = threads >= 152 * 1024 && !want64;
    if (aligned) return inner <= (many ? 64 : threads >= 16384 ? 31 : threads >= 4096 ? 20 : 8);
    return inner <= (many ? 256 : threads >= 16384 ? 31 : 8);
}

static FoldPlan plan_fold(int64_t lo, int64_t inner, int64_t hi, bool aligned, int op, bool want64)
{
    FoldPlan p;
    if (lo == 1) {
        if (inner <= kSmallSeg && hi >= 1024) { p.kind = 0; return p; }
        p.kind = 1;
        p.vec = aligned;
        // at least 32 elements (eight float4 loads) a thread, with more threads a
        // segment where there are too few segments to fill the GPU, and at most 512 of
        // a sum's: a thread holds a pair of floats, what it hands on FP64 within a warp
        // (us, sums: 4000 of 65 elements 3.8 by 32 threads, 2.4 by 8; 16000 of 257 8.7
        // and 5.2; 838 of 600 4.1 by 256, 3.1 by 32; 3000 of 2049 12.9 by 256, 5.7 by 32)
        p.group = inner <= (hi < 152 * 8 ? 64 : hi < 152 * 32 ? 128 : hi < 152 * 64 ? 256 : 640) ? 0 : 1;
        if (p.group == 1 && inner > 512 &&
            hi < (inner <= 1024 ? 152 * 4 : inner < 4096 ? 152 * 8 : inner < 8192 ? 152 * 12 : 152 * 16))
            p.group = 2;
        const int64_t most = is_sum(op) ? kMostPerThread : (int64_t)1 << 20;
        if (inner > most * 32) p.group = 2;
        p.chunk = inner > 0 ? inner : 1;
        if (p.group == 2 && (hi < kBlocks || inner > most * kFoldThreads)) {
            // one wave of four blocks an SM for a few long segments (2^24 elements:
            // a sum of exponentials and a maximum 26.0 and 16.9 us in 1824 blocks,
            // 22.3 and 13.2 in 608, 27.1 and 15.8 in 912; their partials 12.2 us to
            // combine, now 7.3); more, and shorter, blocks for more segments and for
            // tables far larger than the L2 cache, where the wave's last blocks cost
            // more than that (10^8 elements: 120 and 118 us)
            int64_t per = hi <= kWave / 2 && inner * hi <= 1 << 25 ? kWave / hi : (kBlocks + hi - 1) / hi;
            // (waves more where chunks would be too long, not part of one: 2^28 elements,
            // a sum of exponentials 8.5e11 elements/s in four waves, 8.2e11 in 3.4)
            while (per * most * kFoldThreads < inner) per += (kWave + hi - 1) / hi;
            int64_t chunk = (inner + per - 1) / per;
            if (chunk < 4096) chunk = 4096;
            // one chunk, and no kernel to combine its partials, for short segments, and
            // for longer ones the more of them there are (us: 838 sums of 5000 9.1 in two
            // chunks each, 5.4 in one; 10 of them 4.4 and 2.4; 838 of 17000 14.1 and 8.6)
            if (inner < 8192 || (hi >= kWave / 2 && inner < 32768)) chunk = inner;
            p.chunk = (chunk + 1023) / 1024 * 1024;
            p.q = (inner + p.chunk - 1) / p.chunk;
            if (p.q < 1) p.q = 1;
        }
        return p;
    }
    p.kind = 2;
    p.vec = aligned && (lo % 4 == 0) ? 4 : 1;
    if (by_columns(lo * hi / p.vec, inner, p.vec == 4, op, want64)) {
        p.kind = 3;
        if (is_var(op)) p.vec = 1;  // (its FP64 ends keep a thread busy: more threads)
        return p;
    }
    const int64_t columns = (lo * hi / p.vec + 31) / 32;  // blocks side by side
    // (a variance's partials cost some ten FP64 instructions each to combine)
    int64_t q = ((is_var(op) ? kBlocks / 2 : kBlocks) + columns - 1) / columns;
    const int64_t qmax = inner / 64 > 0 ? inner / 64 : 1;  // eight rows a warp at least
    if (q > qmax) q = qmax;
    if (q > 65535) q = 65535;  // grid.y
    if ((inner + q - 1) / q > (1 << 30)) q = (inner + (1 << 30) - 1) >> 30;  // 32-bit positions in a chunk
    p.chunk = (inner + q - 1) / q;
    p.q = (inner + p.chunk - 1) / p.chunk;
    return p;
}

// Workspace: the partials of the chunked plans, then (for two-pass folds) each
// output's centre and its rounding error, 16-byte aligned.  A fold asks for
// room for a partial of every warp (contiguous) or every 1024 threads an SM
// (strided); the plans above, a partial per block, need less.
static int64_t fold_chunks_asked(int64_t lo, int64_t inner, int64_t hi, bool aligned)
{
    if (lo == 1) {
        if (inner <= 64 && hi >= 1024) return 1;
        const int64_t want = 152 * 8 * 4;
        int64_t chunk = kChunk;
        if (hi * ((inner + chunk - 1) / chunk) < want) {
            const int64_t per = hi > 0 ? (want + hi - 1) / hi : 1;
            chunk = (inner + per - 1) / per;
            if (chunk < 1024) chunk = 1024;
        }
        chunk = (chunk + 127) / 128 * 128;
        return (inner + chunk - 1) / chunk;
    }
    const int64_t threads = lo * hi / (aligned && (lo % 4 == 0) ? 4 : 1);
    int64_t q = 1;
    if (threads > 0 && threads < 152 * 1024) {
        q = (152 * 1024 + threads - 1) / threads;
        const int64_t qmax = inner / 16 > 0 ? inner / 16 : 1;
        if (q > qmax) q = qmax;
        if (q > 65535) q = 65535;
    }
    if ((inner + q - 1) / q > (1 << 30)) q = (inner + (1 << 30) - 1) >> 30;
    const int64_t chunk = (inner + q - 1) / q;
    return chunk > 0 ? (inner + chunk - 1) / chunk : 1;
}
static size_t fold_partial_bytes(int64_t lo, int64_t inner, int64_t hi)
{
    const int64_t a = fold_chunks_asked(lo, inner, hi, true), b = fold_chunks_asked(lo, inner, hi, false);
    const int64_t q = a > b ? a : b;
    return q > 1 ? (size_t)(lo * hi) * (size_t)q * sizeof(Partial) : 0;
}
static size_t fold_centre_offset(int64_t lo, int64_t inner, int64_t hi)
{
    return (fold_partial_bytes(lo, inner, hi) + 15) / 16 * 16;
}

nt2g_status fold_partials_bytes(int64_t lo, int64_t inner, int64_t hi, size_t *bytes)
{
    *bytes = fold_partial_bytes(lo, inner, hi);
    return NT2G_OK;
}

nt2g_status fold_workspace_bytes(int64_t lo, int64_t inner, int64_t hi, size_t *bytes)
{
    *bytes = fold_centre_offset(lo, inner, hi) + (size_t)(lo * hi) * 2 * sizeof(float);
    return NT2G_OK;
}

// Where a fold's elements come from: a table, or the FOLD value of a program
// whose element function is compiled at run time.
struct FoldInput {
    bool expr = false;  // the elements are an expression's (else the table x)
    const float *x = nullptr;
    const std::vector<nt2g_op> *ops = nullptr;
    const std::vector<uint8_t> *logical = nullptr;
    const DArgs *args = nullptr;
    int precision = 0;       // the fold: NT2's index order or the compensated one
    int elem_precision = 0;  // an expression's arithmetic (nt2g_precision, NT2_ELEMENTS included)
    bool aligned = false;    // 128-bit reads allowed at multiples of 4
};

static cudaError_t launch_by_handle(cudaKernel_t k, dim3 grid, void **params, cudaStream_t st)
{
    return cudaLaunchKernel((const void *)k, grid, dim3(kFoldThreads), params, 0, st);
}

template <int OP>
static nt2g_status launch_fold_op(const FoldInput &in, int64_t lo, int64_t inner, int64_t hi, void *ws,
                                  size_t ws_bytes, float *out, int64_t *index, double *out64, cudaStream_t st,
                                  const float *cen = nullptr)
{
    const int precision = in.precision;
    const int64_t n_out = lo * hi;
    if constexpr (is_two_pass(OP)) {
        // (a variance asks for the centres' room under either policy)
        if (!cen && (!ws || fold_centre_offset(lo, inner, hi) + (size_t)n_out * 2 * sizeof(float) > ws_bytes)) {
            set_error("fold: workspace of %zu bytes, %zu needed", ws_bytes,
                      fold_centre_offset(lo, inner, hi) + (size_t)n_out * 2 * sizeof(float));
            return NT2G_ERR_INVALID;
        }
        // first the centre of every output: NT2's float mean, or (fast, meanad) the mean and its rounding
        // error; for nanmean the count of non-NaN elements
        if (!cen && (is_two_pass_fast(OP) || precision == NT2G_PREC_NT2 || inner == 0)) {
            const size_t off = fold_centre_offset(lo, inner, hi);
            float *c = (float *)((char *)ws + off);
            nt2g_status s;
            if constexpr (OP == NANMEAN)
                s = launch_fold_op<NOT_NAN>(in, lo, inner, hi, ws, off, c, nullptr, nullptr, st);
            else if (precision == NT2G_PREC_NT2 || inner == 0)
                s = launch_fold_op<MEAN>(in, lo, inner, hi, ws, off, c, nullptr, nullptr, st);
            else
                s = launch_fold_op<MEAN_C>(in, lo, inner, hi, ws, off, c, nullptr, nullptr, st);
            if (s != NT2G_OK) return s;
            return launch_fold_op<OP>(in, lo, inner, hi, ws, ws_bytes, out, index, out64, st, c);
        }
    }
    const JitFoldKernels *jk = nullptr;
    if (in.expr) {
        std::string why;
        jk = jit_fold_kernels(*in.ops, *in.logical, in.elem_precision, OP, &why);
        if (!jk) {
            set_error("fold of an expression: no run-time compiled kernel (%s)", why.c_str());
            return NT2G_ERR_UNSUPPORTED;
        }
    }
    const RawSrc src{in.x};
    const DArgs *jargs = in.args;
    auto cap = [](int64_t g) { return (int)(g < 152 * 32 ? (g > 0 ? g : 1) : 152 * 32); };
    cudaError_t ce = cudaSuccess;
    if (precision == NT2G_PREC_NT2 || inner == 0) {  // (an empty fold yields the neutral element)
        const dim3 g(cap((n_out + kFoldThreads - 1) / kFoldThreads));
        if (!in.expr) {
            k_fold_nt2<OP><<<g, kFoldThreads, 0, st>>>(src, lo, inner, hi, out, index, cen);
            ce = cudaGetLastError();
        } else {
            void *pr[] = {(void *)jargs, &lo, &inner, &hi, &out, &index, &cen};
            ce = launch_by_handle(jk->nt2, g, pr, st);
        }
        if (ce != cudaSuccess) return cuda_status(ce, "fold launch");
        return NT2G_OK;
    }
    FoldPlan p = plan_fold(lo, inner, hi, in.aligned, OP, out64 != nullptr);
    if (p.q > 1 && (size_t)(n_out * p.q) * sizeof(Partial) > ws_bytes) {
        set_error("fold: workspace of %zu bytes, %zu needed", ws_bytes, (size_t)(n_out * p.q) * sizeof(Partial));
        return NT2G_ERR_INVALID;
    }
    Partial *part = (Partial *)ws;
    if (p.kind == 0) {
        const dim3 g(cap((hi + kFoldThreads - 1) / kFoldThreads));
        if (!in.expr) {
            k_fold_short<OP><<<g, kFoldThreads, 0, st>>>(src, inner, hi, out, index, cen, out64);
            ce = cudaGetLastError();
        } else {
            void *pr[] = {(void *)jargs, &inner, &hi, &out, &index, &cen, &out64};
            ce = launch_by_handle(jk->shrt, g, pr, st);
        }
    } else if (p.kind == 1) {
        const int64_t items = hi * p.q;
        static const int kItemsPerBlock[3] = {kFoldThreads / 8, kFoldThreads / 32, 1};
        // several items a block, which shares the FP64 of their results, while
        // that leaves enough blocks for a few waves
        int64_t per = kItemsPerBlock[p.group];
        while (p.q == 1 && per < kItems && (items + 2 * per - 1) / (2 * per) >= kBlocks) per *= 2;
        const dim3 g((unsigned)((items + per - 1) / per));
        const bool idx = index != nullptr && (OP == MAX || OP == MIN);
        const bool fin = p.q == 1;
        int64_t chunk = p.chunk, q = p.q;
        int vec = p.vec;
        if (!in.expr) {
#define NT2G_INNER(F, I, G) ce = launch_dependent(k_fold_inner<OP, F, I, G>, g, kFoldThreads, st, src, inner, hi, chunk, q, vec,  \
                                                  part, out, index, cen, out64)
#define NT2G_INNER_I(F, G) do { if (EXT && idx) NT2G_INNER(F, EXT, G); else NT2G_INNER(F, false, G); } while (0)
            constexpr bool EXT = OP == MAX || OP == MIN;  // only these have positions
            if (!fin) NT2G_INNER_I(false, 256);
            else if (p.group == 0) NT2G_INNER_I(true, 8);
            else if (p.group == 1) NT2G_INNER_I(true, 32);
            else NT2G_INNER_I(true, 256);
#undef NT2G_INNER_I
#undef NT2G_INNER
        } else {
            void *pr[] = {(void *)jargs, &inner, &hi, &chunk, &q, &vec, &part, &out, &index, &cen, &out64};
            ce = launch_by_handle(jk->inner[fin ? p.group : 3][idx], g, pr, st);
        }
    } else if (p.kind == 3) {
        const dim3 g(cap((n_out / p.vec + kFoldThreads - 1) / kFoldThreads));
        if (!in.expr) {
            if (!is_var(OP) && p.vec == 4)
                ce = launch_dependent(k_fold_columns<OP, is_var(OP) ? 1 : 4>, g, kFoldThreads, st, src, lo, inner, hi, out,
                                      index, cen, out64);
            else
                ce = launch_dependent(k_fold_columns<OP, 1>, g, kFoldThreads, st, src, lo, inner, hi, out, index, cen, out64);
        } else {
            void *pr[] = {(void *)jargs, &lo, &inner, &hi, &out, &index, &cen, &out64};
            ce = launch_by_handle(jk->columns[p.vec == 4], g, pr, st);
        }
    } else {
        const int64_t threads = n_out / p.vec;
        const dim3 g(cap((threads + 31) / 32), (unsigned)p.q);
        const bool fin = p.q == 1;
        int64_t chunk = p.chunk, q = p.q;
        if (!in.expr) {
#define NT2G_OUTER(V, F) ce = launch_dependent(k_fold_outer<OP, V, F>, g, kFoldThreads, st, src, lo, inner, hi, chunk, q, part, out, \
                                               index, cen, out64)
            if (p.vec == 4) { if (fin) NT2G_OUTER(4, true); else NT2G_OUTER(4, false); }
            else { if (fin) NT2G_OUTER(1, true); else NT2G_OUTER(1, false); }
#undef NT2G_OUTER
        } else {
            void *pr[] = {(void *)jargs, &lo, &inner, &hi, &chunk, &q, &part, &out, &index, &cen, &out64};
            ce = launch_by_handle(jk->outer[p.vec == 4][fin], g, pr, st);
        }
    }
    if (ce != cudaSuccess) return cuda_status(ce, "fold launch");
    if (p.q > 1 && p.kind != 0) {
        // a block per output where eight threads each would walk long ranges
        if (n_out < 32 || (n_out <= 2048 && p.q > 128))
            ce = launch_dependent(k_fold_finish_block<OP>, dim3(cap(n_out)), kFoldThreads, st, part, n_out, p.q, p.chunk, inner, out,
                                  index, cen, out64);
        else
            ce = launch_dependent(k_fold_finish<OP>, dim3(cap((n_out + 31) / 32)), kFoldThreads, st, part, n_out, p.q, p.chunk,
                                  inner, out, index, cen, out64);
        if (ce != cudaSuccess) return cuda_status(ce, "fold combine launch");
        NT2G_LAUNCH_CHECK("fold combine launch");
    }
    return NT2G_OK;
}

static nt2g_status fold_dispatch(const FoldInput &in, int64_t lo, int64_t inner, int64_t hi, int op, void *ws,
                                 size_t ws_bytes, float *out, int64_t *index, double *out64, cudaStream_t st)
{
    if (lo * hi == 0) return NT2G_OK;
#define NT2G_OP_CASE(O) \
    case O: return launch_fold_op<O>(in, lo, inner, hi, ws, ws_bytes, out, index, out64, st);
    switch (op) {
    NT2G_OP_CASE(SUM) NT2G_OP_CASE(PROD) NT2G_OP_CASE(MAX) NT2G_OP_CASE(MIN) NT2G_OP_CASE(MEAN)
    NT2G_OP_CASE(ASUM1) NT2G_OP_CASE(ASUM2) NT2G_OP_CASE(NORM2) NT2G_OP_CASE(VAR) NT2G_OP_CASE(STDEV)
    NT2G_OP_CASE(VAR1) NT2G_OP_CASE(STDEV1) NT2G_OP_CASE(NBTRUE) NT2G_OP_CASE(ALL) NT2G_OP_CASE(ANY)
    NT2G_OP_CASE(NONE) NT2G_OP_CASE(NANSUM) NT2G_OP_CASE(MEANAD)
    default: return launch_fold_op<NANMEAN>(in, lo, inner, hi, ws, ws_bytes, out, index, out64, st);
    }
#undef NT2G_OP_CASE
}

nt2g_status launch_fold(const float *x, int64_t lo, int64_t inner, int64_t hi, int op, int precision, void *ws,
                        size_t ws_bytes, float *out, int64_t *index, cudaStream_t st)
{
    FoldInput in;
    in.x = x;
    in.precision = precision;
    in.aligned = aligned16(x);
    return fold_dispatch(in, lo, inner, hi, op, ws, ws_bytes, out, index, nullptr, st);
}

// trapz(y, dim) (core/functions/expr/trapz.hpp:24-50): NT2 folds adjfun(plus,
// y, dim) -- the n - 1 float sums y_k + y_(k+1) of neighbours along the
// dimension -- and halves the sum.  NT2 policy: one thread per output, those
// sums folded in index order from 0, times 1/2.  Fast policy: the
// compensated fold of y (FP64 combine) less half of the two ends,
// sum(y) - (y_0 + y_(n-1))/2, NT2's value in exact arithmetic, rounded once;
// a non-finite sum is kept as it is (an infinity at an end is NT2's result).
__global__ void __launch_bounds__(kFoldThreads) k_trapz_nt2(const float *__restrict__ x, int64_t lo, int64_t n,
                                                             int64_t hi, float *__restrict__ out)
{
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < lo * hi;
         o += (int64_t)gridDim.x * blockDim.x) {
        const float *b = x + o % lo + lo * n * (o / lo);
        float s = 0.0f;
        for (int64_t k = 0; k + 1 < n; ++k) s = __fadd_rn(s, __fadd_rn(b[lo * k], b[lo * (k + 1)]));
        out[o] = __fmul_rn(0.5f, s);
    }
}

__global__ void __launch_bounds__(kFoldThreads) k_trapz_finish(const float *__restrict__ x, int64_t lo, int64_t n,
                                                                int64_t hi, const double *__restrict__ s64,
                                                                float *__restrict__ out)
{
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < lo * hi;
         o += (int64_t)gridDim.x * blockDim.x) {
        const float *b = x + o % lo + lo * n * (o / lo);
        const double s = s64[o];
        out[o] = n < 2 ? 0.0f
                       : (s - s == 0.0 ? (float)(s - 0.5 * ((double)b[0] + (double)b[lo * (n - 1)])) : (float)s);
    }
}

nt2g_status trapz_workspace_bytes(int64_t lo, int64_t inner, int64_t hi, size_t *bytes)
{
    *bytes = (fold_partial_bytes(lo, inner, hi) + 15) / 16 * 16 + (size_t)(lo * hi) * sizeof(double);
    return NT2G_OK;
}

nt2g_status launch_trapz(const float *x, int64_t lo, int64_t inner, int64_t hi, int precision, void *ws,
                         size_t ws_bytes, float *out, cudaStream_t st)
{
    const int64_t n_out = lo * hi;
    if (n_out == 0) return NT2G_OK;
    const int g = (int)((n_out + kFoldThreads - 1) / kFoldThreads < 152 * 32 ? (n_out + kFoldThreads - 1) / kFoldThreads
                                                                              : 152 * 32);
    if (precision == NT2G_PREC_NT2 || inner < 2) {
        k_trapz_nt2<<<g, kFoldThreads, 0, st>>>(x, lo, inner, hi, out);
        NT2G_LAUNCH_CHECK("trapz launch");
        return NT2G_OK;
    }
    const size_t off = (fold_partial_bytes(lo, inner, hi) + 15) / 16 * 16;
    double *s64 = (double *)((char *)ws + off);
    FoldInput in;
    in.x = x;
    in.precision = NT2G_PREC_FAST;
    in.aligned = aligned16(x);
    nt2g_status s = fold_dispatch(in, lo, inner, hi, SUM, ws, off, out, nullptr, s64, st);
    if (s != NT2G_OK) return s;
    k_trapz_finish<<<g, kFoldThreads, 0, st>>>(x, lo, inner, hi, s64, out);
    NT2G_LAUNCH_CHECK("trapz launch");
    return NT2G_OK;
}

nt2g_status launch_fold_expr(const std::vector<nt2g_op> &ops, const std::vector<uint8_t> &logical, const DArgs &args,
                             int64_t lo, int64_t inner, int64_t hi, int op, int precision, void *ws, size_t ws_bytes,
                             float *out, int64_t *index, double *out64, cudaStream_t st)
{
    FoldInput in;
    in.expr = true;
    in.ops = &ops;
    in.logical = &logical;
    in.args = &args;
    in.precision = precision == NT2G_PREC_NT2 ? NT2G_PREC_NT2 : NT2G_PREC_FAST;  // the fold's order
    in.elem_precision = precision;
    // whole-vector element reads need every float table 16-byte and every uint8 table 4-byte aligned
    bool al = true;
    for (int s = 0; s < kMaxSlots; ++s)
        if (args.ptr[s]) al &= ((uintptr_t)args.ptr[s] & (args.dtype[s] == NT2G_F32 ? 15u : 3u)) == 0;
    in.aligned = al;
    return fold_dispatch(in, lo, inner, hi, op, ws, ws_bytes, out, index, out64, st);
}

}  // namespace nt2g
