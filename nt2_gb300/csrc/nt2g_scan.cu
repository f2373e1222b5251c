// nt2g_scan.cu -- cumulative sums, products, maxima and minima along one
// dimension (cumsum, cumprod, cummax, cummin) of a table viewed as
// [lo, inner, hi] (column-major): out[l + lo*(k + inner*h)] = the scan over
// k' <= k of x[l + lo*(k' + inner*h)].
//
// NT2 reshapes a cumulative function like a reduction and scans each segment
// in order from the neutral element: summary = bop(summary, x); out = summary
// (core/swar/include/nt2/dsl/functions/cumulative/run.hpp:26-67,
// core/swar/include/nt2/core/functions/details/scan_step.hpp:27-43; the
// functors cumsum = (plus, Zero), cumprod = (multiplies, One), cummax =
// (max, Minf), cummin = (min, Inf) in boost/simd/swar/functions/cum*.hpp).
//
// NT2 policy: one thread per segment in that order with NT2's unfused float
// operations: bit-identical wherever NT2 spreads segments over threads.
//
// Fast policy, with no block waiting on another:
//  * enough segments to fill the GPU with one worker each: one pass, a worker
//    walking its segment with a carry (contiguous segments: a block, short
//    ones sharing it; strided ones: a thread);
//  * else segments are cut into chunks: a first kernel folds each chunk to an
//    aggregate, a second one scans each chunk from the in-order sum of the
//    aggregates before it.  The first walks its chunks backwards, so that the
//    second, walking forwards, finds what was read last in L2.
// cumsum carries compensated sums (s + c; chunk prefixes in FP64), so each
// output is within about an ulp of the exact prefix; cumprod carries FP64
// products; cummax/cummin are exact: NT2's (s > x) ? s : x is not associative
// once a NaN appears (a NaN summary is replaced by the next element), so each
// element is a pair (value, starts-a-segment) with NaN elements starting
// segments, which makes the in-order combine associative and reproduces NT2's
// sequential result, NaNs included.
#include "nt2g_accum.cuh"
#include "nt2g_common.cuh"
#include "nt2g_internal.h"

namespace nt2g {

constexpr int kScanThreads = 256;
constexpr int kLineThreads = 128, kRun = 33;       // contiguous tiles: 128 threads of up to 33 elements
constexpr int kTileMax = kLineThreads * kRun;      // 17 KB of shared memory, 13 blocks an SM
constexpr int64_t kPackBelow = 1024;               // segments shorter than this share tiles
constexpr int64_t kLineChunks = 152 * 12;          // chunks (blocks) a contiguous scan is cut into at least
// strided chunks whose prefix the scan itself adds up: every thread reads the records
// above it, which with four segments a thread costs more than one more kernel from
// eight chunks on (running maxima of 4096 columns of 100, 128, 256 and 1024 rows, us:
// 9.0, 11.1, 16.6, 49.0 so; 11.7, 9.4, 10.8, 20.0 with the kernel), with one segment
// a thread not (4099 columns of 250, 1000 and 8190: 7.3, 14.7, 79.6; 10.6, 18.4,
// 86.6), but for the maxima of too few segments to hide a chain of compares (31 of
// 512 and 1024: 9.2, 14.7; 7.2, 10.2)
constexpr int64_t kInlineFew = 7, kInlinePrefix = 64;
constexpr int64_t kScanTarget = 152 * 1024;

// ------------------------------------------------------------- elements --
// MAX/MIN (the primary template): (value, flags) pairs.  flags bit 0: the
// stretch starts at a NaN element (a segment head); bit 1: the stretch is
// empty (the identity: the neutral value folded with nothing).
template <int OP> struct SE {
    float v;
    int h;
    __device__ static SE id() { return SE{OP == NT2G_SCAN_MAX ? -INFINITY : INFINITY, 2}; }
    __device__ static float op(float s, float x)
    {
        return OP == NT2G_SCAN_MAX ? ((s > x) ? s : x) : ((s < x) ? s : x);
    }
    __device__ static SE combine(const SE &a, const SE &b)  // a precedes b
    {
        if (b.h & 2) return a;
        if (a.h & 2) return SE{op(a.v, b.v), b.h};  // the neutral value meets the first element
        return (b.h & 1) ? b : SE{op(a.v, b.v), a.h};
    }
    // combine(*this, of(x)): whatever the flags, the value is NT2's step
    __device__ void push(float x)
    {
        v = op(v, x);
        h = (x != x) | (h & 1);
    }
    __device__ float out() const { return v; }
    __device__ SE shfl_up(int off) const
    {
        return SE{__shfl_up_sync(0xffffffffu, v, off), __shfl_up_sync(0xffffffffu, h, off)};
    }
};
// SUM: compensated pair
template <> struct SE<NT2G_SCAN_SUM> {
    CSum v;
    __device__ static SE id() { return SE{CSum{0.0f, 0.0f}}; }
    __device__ void push(float x) { csum_add(v, x); }
    __device__ static SE combine(const SE &a, const SE &b)  // a precedes b
    {
        SE r = a;
        csum_merge(r.v, b.v);
        return r;
    }
    __device__ float out() const { return __fadd_rn(v.s, v.c); }
    __device__ double agg() const { return (double)v.s + (double)v.c; }
    __device__ static SE from(double p)
    {
        const float hi = (float)p;
        return SE{CSum{hi, (float)(p - (double)hi)}};
    }
    __device__ SE shfl_up(int off) const
    {
        return SE{CSum{__shfl_up_sync(0xffffffffu, v.s, off), __shfl_up_sync(0xffffffffu, v.c, off)}};
    }
};
// A float as a double by its bits: the conversion is an FP64 instruction, which
// holds that pipe as long as the product it feeds does (and where a select or a
// predicate switches it off, too), so every float goes this way: both passes over
// a tile convert.  (33.5M elements in columns of 1000: 354 us, FP64 pipe 86% busy,
// with conversions; 220 so.)
__device__ __forceinline__ double widen(float x)
{
    const uint32_t u = __float_as_uint(x), a = u & 0x7fffffffu;
    const bool small = a < 0x00800000u;  // zero or subnormal: times 2^24, exactly
    const uint32_t m = small ? __float_as_uint(__fmul_rn(__uint_as_float(a), 0x1p24f)) : a;
    uint32_t hi = (m >> 3) + (small ? 0x38000000u - (24u << 20) : a < 0x7f800000u ? 0x38000000u : 0x70000000u);
    if (m == 0) hi = 0;
    return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)(m << 29));
}
// PROD: double
template <> struct SE<NT2G_SCAN_PROD> {
    double v;
    __device__ static SE id() { return SE{1.0}; }
    __device__ void push(float x) { v *= widen(x); }
    __device__ static SE combine(const SE &a, const SE &b) { return SE{a.v * b.v}; }
    __device__ float out() const { return (float)v; }
    __device__ double agg() const { return v; }
    __device__ static SE from(double p) { return SE{p}; }
    __device__ SE shfl_up(int off) const { return SE{__shfl_up_sync(0xffffffffu, v, off)}; }
};

// 16-byte chunk record in the workspace: an aggregate, later (k_scan_prefix*) its prefix
struct ScanRec {
    double d;  // SUM, PROD
    float v;   // MAX, MIN
    int h;
};
template <int OP> __device__ __forceinline__ ScanRec to_rec(const SE<OP> &e)
{
    ScanRec r{0.0, 0.0f, 0};
    if constexpr (OP == NT2G_SCAN_SUM || OP == NT2G_SCAN_PROD) r.d = e.agg();
    else { r.v = e.v; r.h = e.h; }
    return r;
}
template <int OP> __device__ __forceinline__ SE<OP> from_rec(const ScanRec &r)
{
    if constexpr (OP == NT2G_SCAN_SUM || OP == NT2G_SCAN_PROD) return SE<OP>::from(r.d);
    else return SE<OP>{r.v, r.h};
}

// Aggregates combine in FP64 (sum, prod) or by the pair rule (max, min).
template <int OP> __device__ __forceinline__ ScanRec rec_id()
{
    if constexpr (OP == NT2G_SCAN_SUM) return ScanRec{0.0, 0.0f, 0};
    else if constexpr (OP == NT2G_SCAN_PROD) return ScanRec{1.0, 0.0f, 0};
    else return to_rec<OP>(SE<OP>::id());
}
template <int OP> __device__ __forceinline__ ScanRec rec_combine(const ScanRec &a, const ScanRec &b)
{
    if constexpr (OP == NT2G_SCAN_SUM) return ScanRec{a.d + b.d, 0.0f, 0};
    else if constexpr (OP == NT2G_SCAN_PROD) return ScanRec{a.d * b.d, 0.0f, 0};
    else return to_rec<OP>(SE<OP>::combine(from_rec<OP>(a), from_rec<OP>(b)));
}

// ----------------------------------------- contiguous segments (lo == 1) --
// Tiles of up to 128 x RUN elements staged in shared memory: whatever the
// segment's length and alignment, global memory sees whole aligned 16-byte
// accesses in warp order.  (One-warp tiles, each lane reading 16 consecutive
// elements straight from global memory, took 156 us for cumsum of 8190 columns
// of 4099, where every access is 4 bytes and a warp's are 64 bytes apart; this
// takes 43.)  A thread owns RUN consecutive elements: odd, so the threads read
// conflict-free from shared memory at any alignment, and many, so that the
// scan across threads is shared by them (at 17 a thread and 256 threads it was
// a third of the instructions, 55 us).
// What bounds it: HBM (6.2 TB/s of the 6.8 a copy reaches), with the issue
// slots of two compensated adds an element close behind.
// One pass over long segments, tiles adding up the aggregates that the tiles
// before them publish, was slower: a tile spends 14 of its 20 us on chip
// waiting for round trips queued behind the loads of its own SM (93 us for
// 33.5M elements; fold 30 + scan 44 here).

// Element e (0 <= e < len) of a tile sits at buf[mis + e], mis the tile's
// offset from a 16-byte boundary, so whole vectors copy without a shift.
__device__ __forceinline__ int misalign(const float *p) { return (int)(((uintptr_t)p >> 2) & 3); }

__device__ __forceinline__ void tile_fetch(const float *g, int len, float *buf)
{
    const int mis = misalign(g), first = (4 - mis) & 3;  // elements before the first whole vector
    const int nv = len > first ? (len - first) >> 2 : 0, tail = first + 4 * nv;
    uint32_t to = (uint32_t)__cvta_generic_to_shared(buf + mis + first) + 16 * threadIdx.x;
    const float *from = g + first + 4 * threadIdx.x;
#pragma unroll 3
    for (int v = threadIdx.x; v < nv; v += kLineThreads, to += 16 * kLineThreads, from += 4 * kLineThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
    if (threadIdx.x < 4) {  // the ends
        const int e = tail + (int)threadIdx.x;
        if ((int)threadIdx.x < first && (int)threadIdx.x < len) buf[mis + threadIdx.x] = g[threadIdx.x];
        if (e < len) buf[mis + e] = g[e];
    }
}
__device__ __forceinline__ void tile_arrived()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

__device__ __forceinline__ void tile_store(float *g, int len, const float *buf, int mis)
{
    if (misalign(g) == mis) {
        const int first = (4 - mis) & 3, nv = len > first ? (len - first) >> 2 : 0, tail = first + 4 * nv;
        const float4 *from = (const float4 *)(buf + mis + first) + threadIdx.x;
        float4 *to = (float4 *)(g + first) + threadIdx.x;
#pragma unroll 3
        for (int v = threadIdx.x; v < nv; v += kLineThreads, from += kLineThreads, to += kLineThreads) st_stream(to, *from);
        if (threadIdx.x < 4) {
            const int e = tail + (int)threadIdx.x;
            if ((int)threadIdx.x < first && (int)threadIdx.x < len) g[threadIdx.x] = buf[mis + threadIdx.x];
            if (e < len) g[e] = buf[mis + e];
        }
    } else {  // out sits differently from x: coalesced single elements
        for (int e = threadIdx.x; e < len; e += kLineThreads) g[e] = buf[mis + e];
    }
}

// In-order combine over the block's threads; every thread of warp 0 has the
// result.  s: one record per warp.
template <int OP> __device__ __forceinline__ ScanRec block_rec(ScanRec r, ScanRec *s)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const ScanRec o{__shfl_down_sync(0xffffffffu, r.d, off), __shfl_down_sync(0xffffffffu, r.v, off),
                        __shfl_down_sync(0xffffffffu, r.h, off)};
        if ((lane & (2 * off - 1)) == 0) r = rec_combine<OP>(r, o);
    }
    if (lane == 0) s[wid] = r;
    __syncthreads();
    if (wid == 0) {
        r = s[0];
        for (int w = 1; w < kLineThreads / 32; ++w) r = rec_combine<OP>(r, s[w]);
    }
    return r;
}

// WALK: block b scans chunk b % q of segment b / q, tile after tile, from the
// aggregates of the chunks before it (q = 1: a whole segment).
// PACK: block b scans `pack` whole short segments, one tile (heads restart).
template <int OP, bool PACK, int RUN>
__global__ void __launch_bounds__(kLineThreads) k_scan_line(const float *x, int64_t inner, int64_t hi, int pack,
                                                            int64_t chunk, int64_t q, const ScanRec *__restrict__ rec,
                                                            float *out)
{
    constexpr int kWarps = kLineThreads / 32, kTile = kLineThreads * RUN;
    __shared__ __align__(16) float buf[kTile + 4];
    __shared__ SE<OP> wtot[kWarps], wpre[kWarps];
    __shared__ ScanRec s_rec[kWarps];
    __shared__ int whead[kWarps];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int64_t begin, end, seg = 0, c = 0;
    if constexpr (PACK) {
        const int64_t s0 = (int64_t)blockIdx.x * pack, s1 = s0 + pack < hi ? s0 + pack : hi;
        begin = s0 * inner;
        end = s1 * inner;
    } else {
        seg = blockIdx.x / q;
        c = blockIdx.x - seg * q;
        begin = seg * inner + c * chunk;
        end = (c + 1) * chunk < inner ? begin + chunk : (seg + 1) * inner;
    }
    // warp 0's: the elements before the tile, a sum's in FP64 (a pair of floats from
    // the first tile to the last of a long segment would hold fewer bits)
    ScanRec carry = rec_id<OP>();
    for (int64_t t0 = begin; t0 < end; t0 += kTile) {
        const int len = (int)(end - t0 < kTile ? end - t0 : kTile);
        const int mis = misalign(x + t0);
        tile_fetch(x + t0, len, buf);
        if (!PACK && c > 0 && t0 == begin) {  // the chunks before this one, consecutive ones to a thread
            const ScanRec *r = rec + seg * q;
            const int64_t per = (c + kLineThreads - 1) / kLineThreads, i1 = (tid + 1) * per < c ? (tid + 1) * per : c;
            ScanRec p = rec_id<OP>();
            for (int64_t i = tid * per; i < i1; ++i) p = rec_combine<OP>(p, r[i]);
            carry = block_rec<OP>(p, s_rec);
        }
        tile_arrived();
        // PACK: a short tile still occupies every thread.  WALK: a thread runs past
        // the segment's end into whatever the buffer holds (nothing before the end
        // depends on it), but threads that start past it do nothing: a product's
        // FP64 steps would cost as much as those before the end.
        const int per = PACK ? (len + kLineThreads - 1) / kLineThreads | 1 : RUN, i0 = tid * per;
        const int cnt = len - i0 < per ? (len > i0 ? len - i0 : 0) : per;
        float *p = buf + mis + i0;
        const int n32 = (int)inner, r0 = PACK ? i0 % n32 : 1;  // PACK: position in the segment
        SE<OP> inc = SE<OP>::id();
        int head = 0;
        if constexpr (!PACK) {
            if (i0 < len)
#pragma unroll
                for (int j = 0; j < RUN; ++j) inc.push(p[j]);
        } else {
            for (int j = 0, r = r0; j < cnt; ++j) {
                if (r == 0) { inc = SE<OP>::id(); head = 1; }
                inc.push(p[j]);
                if (++r == n32) r = 0;
            }
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const SE<OP> o = inc.shfl_up(off);
            const int oh = PACK ? __shfl_up_sync(0xffffffffu, head, off) : 0;
            if (lane >= off) {
                if (!PACK || !head) inc = SE<OP>::combine(o, inc);
                head |= oh;
            }
        }
        if (lane == 31) {
            wtot[wid] = inc;
            whead[wid] = head;
        }
        SE<OP> ex = inc.shfl_up(1);
        int exh = PACK ? __shfl_up_sync(0xffffffffu, head, 1) : 0;
        if (lane == 0) { ex = SE<OP>::id(); exh = 0; }
        __syncthreads();
        if (wid == 0) {  // every warp's prefix, and the next tile's carry
            SE<OP> pre = SE<OP>::id(), upto = PACK ? SE<OP>::id() : from_rec<OP>(carry);
            for (int w = 0; w < kWarps; ++w) {
                if (w == lane) pre = upto;
                upto = PACK && whead[w] ? wtot[w] : SE<OP>::combine(upto, wtot[w]);
            }
            if (lane < kWarps) wpre[lane] = pre;
            if (!PACK && t0 + kTile < end) {
                if constexpr (OP == NT2G_SCAN_SUM) {
                    upto = wtot[0];
                    for (int w = 1; w < kWarps; ++w) upto = SE<OP>::combine(upto, wtot[w]);
                    carry = rec_combine<OP>(carry, to_rec<OP>(upto));
                } else {
                    carry = to_rec<OP>(upto);
                }
            }
        }
        __syncthreads();
        SE<OP> run = PACK && exh ? ex : SE<OP>::combine(wpre[wid], ex);
        if constexpr (!PACK) {
            if (i0 < len)
#pragma unroll
                for (int j = 0; j < RUN; ++j) {
                    run.push(p[j]);
                    p[j] = run.out();
                }
        } else {
            for (int j = 0, r = r0; j < cnt; ++j) {
                if (r == 0) run = SE<OP>::id();
                run.push(p[j]);
                if (++r == n32) r = 0;
                p[j] = run.out();
            }
        }
        __syncthreads();
        tile_store(out + t0, len, buf, mis);
        if (PACK) break;
        __syncthreads();  // the next tile reuses the buffer
    }
}

// The aggregate of chunk b % q of segment b / q.
template <int OP>
__global__ void __launch_bounds__(kLineThreads) k_scan_fold(const float *__restrict__ x, int64_t inner, int64_t chunk,
                                                            int64_t q, ScanRec *__restrict__ rec)
{
    __shared__ ScanRec s_rec[kLineThreads / 32];
    const int64_t seg = blockIdx.x / q, c = blockIdx.x - seg * q;
    const int64_t begin = seg * inner + c * chunk, end = (c + 1) * chunk < inner ? begin + chunk : (seg + 1) * inner;
    const int tid = threadIdx.x;
    SE<OP> acc = SE<OP>::id();
    if constexpr (OP == NT2G_SCAN_SUM || OP == NT2G_SCAN_PROD) {
        // the order does not matter to the aggregate: whole vectors, eight loads
        // in flight a thread, from the chunk's end to its start
        const int64_t first = begin + ((4 - misalign(x + begin)) & 3), nv = end > first ? (end - first) >> 2 : 0;
        const float4 *v = (const float4 *)(x + first) + (nv - 1 - tid);
        int64_t left = nv - tid;
        constexpr int kBatch = 8 * kLineThreads;
        if (left > kBatch - kLineThreads) {
            float4 f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = __ldg(v - u * kLineThreads);
            while (true) {
                left -= kBatch;
                v -= kBatch;
                const bool more = left > kBatch - kLineThreads;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float4 e = f[u];
                    if (more) f[u] = __ldg(v - u * kLineThreads);
                    acc.push(e.x); acc.push(e.y); acc.push(e.z); acc.push(e.w);
                }
                if (!more) break;
            }
        }
        for (; left > 0; left -= kLineThreads, v -= kLineThreads) {
            const float4 f = __ldg(v);
            acc.push(f.x); acc.push(f.y); acc.push(f.z); acc.push(f.w);
        }
        const int64_t e = tid < 4 ? begin + tid : first + 4 * nv + tid - 4;  // the ends
        if (tid < 4 ? e < first && e < end : tid < 8 && e >= first && e < end) acc.push(x[e]);
    } else {
        __shared__ __align__(16) float buf[kTileMax + 4];
        const int64_t tiles = (end - begin + kTileMax - 1) / kTileMax;
        for (int64_t t = tiles - 1; t >= 0; --t) {
            const int64_t t0 = begin + t * kTileMax;
            const int len = (int)(end - t0 < kTileMax ? end - t0 : kTileMax), mis = misalign(x + t0);
            tile_fetch(x + t0, len, buf);
            tile_arrived();
            const int i0 = tid * kRun, cnt = len - i0 < kRun ? (len > i0 ? len - i0 : 0) : kRun;
            SE<OP> r = SE<OP>::id();
#pragma unroll
            for (int j = 0; j < kRun; ++j)
                if (j < cnt) r.push(buf[mis + i0 + j]);
            // thread by thread across tiles would not be in order: the tile first
            const ScanRec tot = block_rec<OP>(to_rec<OP>(r), s_rec);
            if (tid == 0) acc = SE<OP>::combine(from_rec<OP>(tot), acc);
            __syncthreads();
        }
        if (tid == 0) rec[blockIdx.x] = to_rec<OP>(acc);
        return;
    }
    const ScanRec tot = block_rec<OP>(to_rec<OP>(acc), s_rec);
    if (tid == 0) rec[blockIdx.x] = tot;
}

// ---------------------------------------------- strided scans (lo > 1) --
// Thread per segment (VEC: four neighbouring segments via float4) over the
// chunk [c*ck, min((c+1)*ck, inner)) of the scan range; grid.y = chunk.
// FOLD: the chunk's aggregate (KEEP: leaving the table in L2).  Else the scan, from the aggregates of the chunks above
// (`prefixes`: k_scan_prefix* has replaced them by their sums).
// k rows in groups, the last ones in smaller ones (running sums of ten rows of 3.3
// million segments: 126 us with the last ones one at a time, 57 so)
#define NT2G_GROUPS                                                 \
    while (k >= kGroup) { float e[kGroup][VEC]; group(e); }         \
    if (kGroup > 8 && k >= 8) { float e[8][VEC]; group(e); }        \
    if (kGroup > 4 && k >= 4) { float e[4][VEC]; group(e); }        \
    while (k > 0) { float e[1][VEC]; group(e); }
template <int OP, int VEC, bool FOLD, bool KEEP = true>
__global__ void __launch_bounds__(kScanThreads, VEC == 4 ? 4 : 0) k_scan_outer(const float *x, int64_t lo, int64_t inner, int64_t hi,
                                                             int64_t ck, int64_t q, bool prefixes,
                                                             ScanRec *__restrict__ rec, float *out)
{
    const int64_t lv = lo / VEC, n_seg = lo * hi;
    const int64_t c = blockIdx.y;
    const int64_t k0 = c * ck, k1 = (k0 + ck < inner) ? k0 + ck : inner;
    // groups of kGroup rows: all loads of a group are issued before its scan
    constexpr int kGroup = (OP == NT2G_SCAN_PROD && VEC == 4) ? 4 : VEC == 4 ? 8 : 16;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < lv * hi; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t h = t / lv, l = (t - h * lv) * VEC;
        const int64_t base = l + lo * inner * h;
        SE<OP> carry[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            const int64_t seg = l + v + lo * h;
            if (FOLD || q == 1 || c == 0) {
                carry[v] = SE<OP>::id();
            } else if (prefixes) {
                carry[v] = from_rec<OP>(rec[c * n_seg + seg]);
            } else {
                ScanRec p = rec[seg];
                for (int64_t i = 1; i < c; ++i) p = rec_combine<OP>(p, rec[i * n_seg + seg]);
                carry[v] = from_rec<OP>(p);
            }
        }
        auto fetch = [&](const float *p, float (&e)[VEC]) {
            if constexpr (VEC == 4) {
                const float4 f = FOLD && KEEP ? __ldg((const float4 *)p) : ld_stream((const float4 *)p);
                e[0] = f.x; e[1] = f.y; e[2] = f.z; e[3] = f.w;
            } else {
                e[0] = FOLD ? __ldg(p) : ld_stream(p);
            }
        };
        if constexpr (FOLD) {
            const float *p = x + base + lo * k0;
            int64_t k = k1 - k0;
            auto group = [&](auto &e) {
                constexpr int G = sizeof(e) / sizeof(e[0]);
#pragma unroll
                for (int g = 0; g < G; ++g, p += lo) fetch(p, e[g]);
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int v = 0; v < VEC; ++v) carry[v].push(e[g][v]);
                k -= G;
            };
            NT2G_GROUPS
#pragma unroll
            for (int v = 0; v < VEC; ++v) rec[c * n_seg + (l + v + lo * h)] = to_rec<OP>(carry[v]);
        } else {
            const float *p = x + base + lo * k0;
            float *o = out + base + lo * k0;
            auto step = [&](const float (&e)[VEC]) {
                float r[VEC];
#pragma unroll
                for (int v = 0; v < VEC; ++v) {
                    carry[v].push(e[v]);
                    r[v] = carry[v].out();
                }
                if constexpr (VEC == 4) st_stream((float4 *)o, make_float4(r[0], r[1], r[2], r[3]));
                else st_stream(o, r[0]);
                o += lo;
            };
            int64_t k = k1 - k0;
            auto group = [&](auto &e) {
                constexpr int G = sizeof(e) / sizeof(e[0]);
#pragma unroll
                for (int g = 0; g < G; ++g, p += lo) fetch(p, e[g]);
#pragma unroll
                for (int g = 0; g < G; ++g) step(e[g]);
                k -= G;
            };
            NT2G_GROUPS
        }
    }
}

// Strided scans of many chunks: per segment, the chunk aggregates replaced by
// their exclusive prefixes in order (one thread per segment).
template <int OP>
__global__ void __launch_bounds__(kScanThreads) k_scan_prefix(ScanRec *__restrict__ rec, int64_t n_seg, int64_t q)
{
    // record c of segment s at rec[s + c * n_seg]: coalesced over segments
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n_seg; s += (int64_t)gridDim.x * blockDim.x) {
        ScanRec *r = rec + s;
        ScanRec acc = rec_id<OP>();
        int64_t c = 0;
        for (; c + 8 <= q; c += 8) {  // eight independent loads in flight
            ScanRec a[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) a[u] = r[(c + u) * n_seg];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                r[(c + u) * n_seg] = acc;
                acc = rec_combine<OP>(acc, a[u]);
            }
        }
        for (; c < q; ++c) {
            const ScanRec a = r[c * n_seg];
            r[c * n_seg] = acc;
            acc = rec_combine<OP>(acc, a);
        }
    }
}

// For more chunks still: one block per segment.  The combine order
// is fixed for a given q.
template <int OP> __device__ __forceinline__ ScanRec rec_shfl_up(const ScanRec &a, int off)
{
    return ScanRec{__shfl_up_sync(0xffffffffu, a.d, off), __shfl_up_sync(0xffffffffu, a.v, off),
                    __shfl_up_sync(0xffffffffu, a.h, off)};
}

template <int OP>
__global__ void __launch_bounds__(kScanThreads) k_scan_prefix_block(ScanRec *__restrict__ rec, int64_t n_seg,
                                                                    int64_t q)
{
    // tiles of kScanThreads x 8 consecutive records: each thread loads its 8
    // (independent loads), the thread totals are scanned in order across the
    // block (warp shuffles, then the warp totals), and a carry runs over the tiles
    constexpr int kPer = 8, kWarps = kScanThreads / 32;
    __shared__ ScanRec wtot[kWarps];
    __shared__ ScanRec carry_s;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int64_t s = blockIdx.x; s < n_seg; s += gridDim.x) {
        ScanRec *r = rec + s;
        ScanRec carry = rec_id<OP>();
        for (int64_t t0 = 0; t0 < q; t0 += (int64_t)kScanThreads * kPer) {
            const int64_t c0 = t0 + (int64_t)tid * kPer;
            ScanRec a[kPer];
#pragma unroll
            for (int u = 0; u < kPer; ++u) a[u] = c0 + u < q ? r[(c0 + u) * n_seg] : rec_id<OP>();
            ScanRec tot = rec_id<OP>();
#pragma unroll
            for (int u = 0; u < kPer; ++u) tot = rec_combine<OP>(tot, a[u]);
            ScanRec inc = tot;  // in-order inclusive scan of the thread totals in the warp
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const ScanRec o = rec_shfl_up<OP>(inc, off);
                if (lane >= off) inc = rec_combine<OP>(o, inc);
            }
            if (lane == 31) wtot[wid] = inc;
            __syncthreads();
            if (tid == 0) {  // the warp totals in order, and the next tile's carry
                ScanRec run = carry;
                for (int w = 0; w < kWarps; ++w) {
                    const ScanRec x = wtot[w];
                    wtot[w] = run;
                    run = rec_combine<OP>(run, x);
                }
                carry_s = run;
            }
            __syncthreads();
            ScanRec ex = rec_shfl_up<OP>(inc, 1);
            if (lane == 0) ex = rec_id<OP>();
            ScanRec pre = rec_combine<OP>(wtot[wid], ex);
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                if (c0 + u < q) r[(c0 + u) * n_seg] = pre;
                pre = rec_combine<OP>(pre, a[u]);
            }
            carry = carry_s;
            __syncthreads();
        }
    }
}

// NT2 policy: the segment in order, NT2's operations.
template <int OP>
__global__ void __launch_bounds__(kScanThreads) k_scan_nt2(const float *x, int64_t lo, int64_t inner,
                                                           int64_t hi, float *out)
{
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < lo * hi; s += (int64_t)gridDim.x * blockDim.x) {
        const int64_t h = s / lo, l = s - h * lo;
        const int64_t base = l + lo * inner * h;
        float acc = OP == NT2G_SCAN_PROD ? 1.0f : OP == NT2G_SCAN_MAX ? -INFINITY : OP == NT2G_SCAN_MIN ? INFINITY : 0.0f;
        for (int64_t k = 0; k < inner; ++k) {
            const float v = x[base + lo * k];
            if (OP == NT2G_SCAN_SUM) acc = __fadd_rn(acc, v);
            else if (OP == NT2G_SCAN_PROD) acc = __fmul_rn(acc, v);
            else if (OP == NT2G_SCAN_MAX) acc = (acc > v) ? acc : v;
            else acc = (acc < v) ? acc : v;
            out[base + lo * k] = acc;
        }
    }
}

// ---------------------------------------------------------------- plans --
struct ScanPlan {
    bool lines = false;        // contiguous segments
    int pack = 1;              // lines: short segments per block
    int vec = 1;               // strided: segments per thread
    int64_t chunk = 0, q = 1;  // elements per chunk, chunks per segment
};

// Contiguous: segments shorter than kPackBelow share a block's tile, as many
// as still leave 13 blocks to each SM; longer ones get a block each, which is
// one pass, when they are one tile or fill the GPU; else chunks of whole
// tiles, 12 blocks to each SM (one wave: 13 fit).  Strided: a thread per
// segment (four with float4) if that gives 1024 threads to each SM, else
// chunks of at least 16 rows.
static ScanPlan plan_scan(int64_t lo, int64_t inner, int64_t hi, bool aligned)
{
    ScanPlan p;
    if (lo == 1) {
        p.lines = true;
        p.chunk = inner;
        if (inner < kPackBelow) {
            const int64_t most = kTileMax / (inner > 0 ? inner : 1), spread = (hi + 152 * 13 - 1) / (152 * 13);
            p.pack = (int)(most < spread ? most : spread);
        } else if (inner > kTileMax && hi < kLineChunks) {
            const int64_t tiles = (inner + kTileMax - 1) / kTileMax;
            const int64_t per = (hi * tiles + kLineChunks - 1) / kLineChunks;  // tiles per chunk
            p.q = (tiles + per - 1) / per;
            p.chunk = (tiles + p.q - 1) / p.q * kTileMax;
            p.q = (inner + p.chunk - 1) / p.chunk;
        }
        return p;
    }
    p.vec = aligned && lo % 4 == 0 ? 4 : 1;
    const int64_t threads = lo * hi / p.vec;
    int64_t q = 1;
    if (threads < kScanTarget) {
        q = (kScanTarget + threads - 1) / threads;
        const int64_t qmax = inner / 16 > 0 ? inner / 16 : 1;
        if (q > qmax) q = qmax;
        if (q > 65535) q = 65535;
    }
    p.chunk = inner > 0 ? (inner + q - 1) / q : 1;
    p.q = inner > 0 ? (inner + p.chunk - 1) / p.chunk : 1;
    return p;
}

// Contiguous scans need less than they ask for: 16 bytes for each of the
// 4864 chunks of at most 16384 elements that one warp each once took.
nt2g_status scan_workspace_bytes(int64_t lo, int64_t inner, int64_t hi, size_t *bytes)
{
    int64_t q;
    if (lo == 1) {
        const int64_t want = 152 * 8 * 4;
        int64_t chunk = 16384;
        if (hi * ((inner + chunk - 1) / chunk) < want) {
            const int64_t per = hi > 0 ? (want + hi - 1) / hi : 1;
            chunk = (inner + per - 1) / per;
            if (chunk < 1024) chunk = 1024;
        }
        chunk = (chunk + 511) / 512 * 512;
        q = inner > 0 ? (inner + chunk - 1) / chunk : 1;
    } else {
        const ScanPlan a = plan_scan(lo, inner, hi, true), b = plan_scan(lo, inner, hi, false);
        q = a.q > b.q ? a.q : b.q;
    }
    *bytes = q > 1 ? (size_t)(lo * hi) * (size_t)q * sizeof(ScanRec) : 0;
    return NT2G_OK;
}

template <int OP> static void launch_prefix(ScanRec *rec, int64_t n_seg, int64_t q, cudaStream_t st)
{
    auto cap = [](int64_t g) { return (int)(g < 152 * 32 ? (g > 0 ? g : 1) : 152 * 32); };
    if (q >= 512) k_scan_prefix_block<OP><<<cap(n_seg), kScanThreads, 0, st>>>(rec, n_seg, q);
    else k_scan_prefix<OP><<<cap((n_seg + kScanThreads - 1) / kScanThreads), kScanThreads, 0, st>>>(rec, n_seg, q);
}

template <int OP>
static nt2g_status launch_scan_op(const float *x, int64_t lo, int64_t inner, int64_t hi, int precision, void *ws,
                                  size_t ws_bytes, float *out, cudaStream_t st)
{
    const int64_t n_seg = lo * hi;
    auto cap = [](int64_t g) { return (int)(g < 152 * 32 ? (g > 0 ? g : 1) : 152 * 32); };
    if (precision == NT2G_PREC_NT2) {
        k_scan_nt2<OP><<<cap((n_seg + kScanThreads - 1) / kScanThreads), kScanThreads, 0, st>>>(x, lo, inner, hi, out);
        NT2G_LAUNCH_CHECK("scan launch");
        return NT2G_OK;
    }
    const ScanPlan p = plan_scan(lo, inner, hi, aligned16(x) && aligned16(out));
    if (p.q > 1 && (size_t)(n_seg * p.q) * sizeof(ScanRec) > ws_bytes) {
        set_error("nt2g_scan_f32: workspace of %zu bytes, %zu needed", ws_bytes, (size_t)(n_seg * p.q) * sizeof(ScanRec));
        return NT2G_ERR_INVALID;
    }
    ScanRec *rec = (ScanRec *)ws;
    if (p.lines) {
        // a launch takes up to 2^30 blocks
        const int64_t most = ((int64_t)1 << 30) / p.q * p.pack;
        for (int64_t s0 = 0; s0 < hi; s0 += most) {
            const int64_t n = hi - s0 < most ? hi - s0 : most;
            const unsigned g = (unsigned)((n + p.pack - 1) / p.pack * p.q);
            const float *xs = x + s0 * inner;
            float *os = out + s0 * inner;
            if (p.q > 1) k_scan_fold<OP><<<g, kLineThreads, 0, st>>>(xs, inner, p.chunk, p.q, rec);
#define NT2G_LINE(PACK, RUN) k_scan_line<OP, PACK, RUN><<<g, kLineThreads, 0, st>>>(xs, inner, n, p.pack, p.chunk, p.q, \
                                                                                    rec, os)
            if (p.pack > 1) NT2G_LINE(true, kRun);
            else if (p.chunk <= kLineThreads * 9) NT2G_LINE(false, 9);
            else if (p.chunk <= kLineThreads * 17) NT2G_LINE(false, 17);
            else NT2G_LINE(false, kRun);
#undef NT2G_LINE
        }
    } else {
        // blocks no wider than the segments are many (an SM holds eight of 256 threads,
        // whatever few of them have a segment)
        const int64_t threads = n_seg / p.vec;
        const int block = threads < kScanThreads ? (int)((threads + 31) / 32 * 32) : kScanThreads;
        const dim3 grid(cap((threads + kScanThreads - 1) / kScanThreads), (unsigned)p.q);
        // the fold leaves in L2 what the scan reads again where that fits (running maxima
        // of 4096 x 4096 51 us, 56 with streaming loads; of 16384 x 16384 515 and 501;
        // single columns, whose warps share sectors, always: 4099 x 8190 80 and 165)
        const bool keep = n_seg * inner <= (int64_t)24 << 20;
        const bool few = p.vec == 4 || ((OP == NT2G_SCAN_MAX || OP == NT2G_SCAN_MIN) && n_seg < 1024);
        const bool prefixes = p.q > (few ? kInlineFew : kInlinePrefix);
#define NT2G_OUTER(VEC, ...) k_scan_outer<OP, VEC, __VA_ARGS__><<<grid, block, 0, st>>>(x, lo, inner, hi, p.chunk, p.q, \
                                                                                         prefixes, rec, out)
        if (p.q > 1) {
            if (p.vec != 4) NT2G_OUTER(1, true);
            else if (keep) NT2G_OUTER(4, true);
            else NT2G_OUTER(4, true, false);
            if (prefixes) launch_prefix<OP>(rec, n_seg, p.q, st);
        }
        if (p.vec == 4) NT2G_OUTER(4, false);
        else NT2G_OUTER(1, false);
#undef NT2G_OUTER
    }
    NT2G_LAUNCH_CHECK("scan launch");
    return NT2G_OK;
}

nt2g_status launch_scan(const float *x, int64_t lo, int64_t inner, int64_t hi, int op, int precision, void *ws,
                        size_t ws_bytes, float *out, cudaStream_t st)
{
    if (lo * inner * hi == 0) return NT2G_OK;
    switch (op) {
    case NT2G_SCAN_SUM: return launch_scan_op<NT2G_SCAN_SUM>(x, lo, inner, hi, precision, ws, ws_bytes, out, st);
    case NT2G_SCAN_PROD: return launch_scan_op<NT2G_SCAN_PROD>(x, lo, inner, hi, precision, ws, ws_bytes, out, st);
    case NT2G_SCAN_MAX: return launch_scan_op<NT2G_SCAN_MAX>(x, lo, inner, hi, precision, ws, ws_bytes, out, st);
    default: return launch_scan_op<NT2G_SCAN_MIN>(x, lo, inner, hi, precision, ws, ws_bytes, out, st);
    }
}

}  // namespace nt2g
