// nt2g_median.cu -- median(a, dim) and medianad(a, dim) along one dimension.
//
// NT2 (core/reduction/include/nt2/core/functions/expr/median.hpp:37-50) sorts
// each slice ascending along dim and takes the middle element for an odd
// length n, or meanof of the two middle ones for an even n; medianad
// (expr/medianad.hpp:38-54) is median(abs(a - expand_to(median(a, dim)))).
// Both results are order statistics, so here nothing is sorted: each slice's
// rank-(n-1)/2 element is found by radix selection on order-preserving
// 32-bit keys (four 8-bit digits, most significant first: a 256-bin
// histogram of the keys that share the digits found so far picks the next
// digit), and for an even n the next order statistic is either an equal key
// or the smallest key above it.
//
//  * slices of up to kRegKeys elements: one block per slice (eight or four
//    neighbouring slices where elements are strided and they fit, so that whole
//    or half sectors are read), its keys in registers from one pass over global memory.  The first digit
//    is 10 or 11 bits wide; the few keys that share it are then gathered and ranked
//    by one warp (more digits only where they are many).
//  * short slices: one block per slice, its keys in shared memory, four 8-bit
//    digits.
//  * longer slices: 8-bit digits over global memory, many blocks per slice,
//    each adding its block histogram into the slice's histogram in the
//    workspace, the last block picking the digit; once at most kGather keys
//    share the digits found, a pass gathers them and the last block ranks them.
//
// A slice holding a NaN gives NaN (NT2 sorts with operator<, which orders no
// NaN, so its result there is unspecified).  -0 and +0 are distinct keys
// (-0 first); NT2's sort leaves their order unspecified, so where both sit
// at the middle the sign of a zero result may differ from NT2's.
#include "nt2g_common.cuh"
#include "nt2g_internal.h"

namespace nt2g {

constexpr int64_t kRegKeys = 40960;   // 1024 threads of 40 keys
constexpr int64_t kShortKeys = 1024;  // up to this length: the shared-memory kernel
constexpr int kList = 256;            // keys a warp ranks
constexpr int kGather = kList;         // keys gathered in a long slice's histogram space
constexpr int kLoadBatch = 8;         // loads a thread issues before it uses them

// Order-preserving key: all bits of a negative float flipped, the sign bit
// of a positive one set; unsigned comparison of keys is the float order.
__device__ __forceinline__ uint32_t med_key(float f)
{
    const uint32_t u = __float_as_uint(f);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float med_val(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// boost.simd's float meanof (arithmetic/functions/generic/meanof.hpp:21-33):
// m + (max - m) * 1/2 for finite arguments, else average = fma(a0, 1/2,
// a1 * 1/2), NT2's fma unfused.  a0 is the lower middle element.
__device__ __forceinline__ float nt2_meanof(float a0, float a1)
{
    const float m = a0 < a1 ? a0 : a1, M = a0 > a1 ? a0 : a1;
    const bool fin = __fsub_rn(a0, a0) == 0.0f && __fsub_rn(a1, a1) == 0.0f;
    return fin ? __fadd_rn(m, __fmul_rn(__fsub_rn(M, m), 0.5f))
               : __fadd_rn(__fmul_rn(a0, 0.5f), __fmul_rn(a1, 0.5f));
}

// Element k of slice s: x[l + lo*(k + n*h)], s = l + lo*h; medianad's
// elements are |x - centre(s)| (NT2: abs(a0 - expand_to(t0))).
template <bool AD>
__device__ __forceinline__ float med_elem(const float *__restrict__ base, int64_t lo, int64_t k, float c)
{
    const float v = base[lo * k];
    return AD ? fabsf(__fsub_rn(v, c)) : v;
}

// One warp: the bin of hist (256 counts) holding rank r, the rank left
// inside that bin and the bin's count.
template <class C>
__device__ __forceinline__ void med_find_bin(const volatile C *hist, C r, int lane, uint32_t &bin, C &rest, C &cnt, bool &mine)
{
    C b[8], t = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        b[j] = hist[lane * 8 + j];
        t += b[j];
    }
    C inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const C v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    const C exc = inc - t;
    mine = r >= exc && r < inc;
    if (mine) {
        C acc = exc;
        int j = 0;
        while (j < 7 && acc + b[j] <= r) acc += b[j++];
        bin = (uint32_t)(lane * 8 + j);
        rest = r - acc;
        cnt = b[j];
    }
}

// ------------------------------------------- short slices in shared memory --
template <bool AD>
__global__ void k_median_smem(const float *__restrict__ x, int64_t lo, int64_t n, const float *centre,
                              float *out)
{
    extern __shared__ uint32_t keys[];  // [n] keys, then 256 bins
    uint32_t *hist = keys + n;
    __shared__ uint32_t sh_bin, sh_rest, sh_cnt, sh_min;
    const int64_t s = blockIdx.x, l = s % lo, h = s / lo;
    const float *base = x + l + lo * n * h;
    const float c = AD ? centre[s] : 0.0f;
    int nan = 0;
    // kLoadBatch loads in flight per thread before any is used: one at a time,
    // the loop would wait a memory latency per element
    for (int64_t k0 = threadIdx.x; k0 < n; k0 += kLoadBatch * (int64_t)blockDim.x) {
        float v[kLoadBatch];
#pragma unroll
        for (int j = 0; j < kLoadBatch; ++j) {
            const int64_t k = k0 + j * (int64_t)blockDim.x;
            v[j] = k < n ? med_elem<AD>(base, lo, k, c) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < kLoadBatch; ++j) {
            const int64_t k = k0 + j * (int64_t)blockDim.x;
            if (k < n) {
                nan |= v[j] != v[j];
                keys[k] = med_key(v[j]);
            }
        }
    }
    if (__syncthreads_or(nan)) {
        if (threadIdx.x == 0) out[s] = __uint_as_float(0x7fc00000u);
        return;
    }
    const bool even = (n & 1) == 0;
    uint32_t r = (uint32_t)((n - (even ? 1 : 0)) >> 1), prefix = 0, mask = 0, cnt = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
            const uint32_t key = keys[k];
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            uint32_t bin = 0, rest = 0, bc = 0;
            bool mine;
            med_find_bin<uint32_t>((const volatile uint32_t *)hist, r, threadIdx.x, bin, rest, bc, mine);
            if (mine) {
                sh_bin = bin;
                sh_rest = rest;
                sh_cnt = bc;
            }
        }
        __syncthreads();
        prefix |= sh_bin << shift;
        mask |= 255u << shift;
        r = sh_rest;
        cnt = sh_cnt;
    }
    uint32_t key2 = prefix;
    if (even && r + 1 >= cnt) {  // no second copy of the lower middle key: the next key up
        if (threadIdx.x == 0) sh_min = 0xffffffffu;
        __syncthreads();
        uint32_t m = 0xffffffffu;
        for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
            const uint32_t key = keys[k];
            if (key > prefix && key < m) m = key;
        }
        m = __reduce_min_sync(0xffffffffu, m);
        if ((threadIdx.x & 31) == 0) atomicMin(&sh_min, m);
        __syncthreads();
        key2 = sh_min;
    }
    if (threadIdx.x == 0) out[s] = even ? nt2_meanof(med_val(prefix), med_val(key2)) : med_val(prefix);
}

// ------------------------------------------------- slices in registers --
// One warp: the bin of hist (BINS counts) holding rank r, the rank left inside
// it and its count (every lane has the result).
template <int BINS>
__device__ __forceinline__ void wide_find_bin(const uint32_t *hist, uint32_t r, int lane, uint32_t &bin, uint32_t &rest,
                                              uint32_t &cnt)
{
    // rows of 128 bins, four a lane: the row, the lane, the bin
    uint32_t row = 0;
    bool found = false;
#pragma unroll
    for (int j = 0; j < BINS / 128; ++j) {
        const uint4 v = ((const uint4 *)hist)[j * 32 + lane];
        const uint32_t t = __reduce_add_sync(0xffffffffu, v.x + v.y + v.z + v.w);
        if (!found) {
            if (r < t) { row = j; found = true; }
            else r -= t;
        }
    }
    const uint4 v = ((const uint4 *)hist)[row * 32 + lane];
    uint32_t inc = v.x + v.y + v.z + v.w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    const int at = __ffs((int)__ballot_sync(0xffffffffu, r < inc)) - 1;
    uint32_t left = r - (inc - (v.x + v.y + v.z + v.w)), c = v.x, i = 0;
    if (left >= c) { left -= c; c = v.y; i = 1; }
    if (i == 1 && left >= c) { left -= c; c = v.z; i = 2; }
    if (i == 2 && left >= c) { left -= c; c = v.w; i = 3; }
    bin = __shfl_sync(0xffffffffu, row * 128 + 4 * lane + i, at);
    rest = __shfl_sync(0xffffffffu, left, at);
    cnt = __shfl_sync(0xffffffffu, c, at);
}

// One warp: the keys of rank r and r + 1 among list[0..m) (r + 1 < m for the
// second one; m <= kList), all of them equal above bit `bits`.
__device__ __forceinline__ void rank_list(const uint32_t *list, int m, uint32_t r, int bits, int lane, uint32_t &key1,
                                          uint32_t &key2)
{
    if (m <= 32) {  // each lane its key's rank
        const uint32_t k = lane < m ? list[lane] : 0xffffffffu;
        uint32_t rank = lane < m ? 0u : 64u;
        for (int j = 0; j < m; ++j) {
            const uint32_t o = __shfl_sync(0xffffffffu, k, j);
            rank += o < k || (o == k && j < lane);
        }
        const int a = __ffs((int)__ballot_sync(0xffffffffu, rank == r)) - 1;
        const int b = __ffs((int)__ballot_sync(0xffffffffu, rank == r + 1)) - 1;
        key1 = __shfl_sync(0xffffffffu, k, a);
        key2 = __shfl_sync(0xffffffffu, k, b < 0 ? a : b);
        return;
    }
    uint32_t k[kList / 32];
#pragma unroll
    for (int j = 0; j < kList / 32; ++j) k[j] = lane + 32 * j < m ? list[lane + 32 * j] : 0xffffffffu;
    // bit by bit: the keys below prefix | bit among those that share the prefix
    uint32_t prefix = __shfl_sync(0xffffffffu, k[0], 0) >> bits << bits;
    uint32_t equal = (uint32_t)m;
    for (int bit = bits - 1; bit >= 0; --bit) {
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < kList / 32; ++j)
            if (32 * j < m) c += (k[j] ^ prefix) >> bit == 0 && lane + 32 * j < m;
        c = __reduce_add_sync(0xffffffffu, c);
        if (r >= c) {
            r -= c;
            prefix |= 1u << bit;
            equal -= c;
        } else {
            equal = c;
        }
    }
    key1 = key2 = prefix;
    if (r + 1 >= equal) {
        uint32_t up = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < kList / 32; ++j) up = k[j] > prefix && k[j] < up ? k[j] : up;
        key2 = __reduce_min_sync(0xffffffffu, up);
    }
}

// S slices a block (neighbouring ones, a thread taking every blockDim / S-th
// element of slice tid % S), KPT keys a thread, +inf where a thread has fewer:
// above every rank looked for, so nothing has to be checked again.  What bounds
// it: a dozen instructions a key and the serial phases of a block, hidden by
// the other blocks of the SM.  (Keys in shared memory and four 8-bit digits
// over them took 48 us for 3001 slices of 4000, and, one strided slice a
// block, 75 for 4000 slices of 3001; this takes 23 and 43.)
template <bool AD, int S, int KPT, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT < 1024 ? 1536 / MAXT : 1) k_median_regs(const float *__restrict__ x, int64_t lo,
                                                                                  int64_t n, const float *centre,
                                                                                  float *out)
{
    // the first digit's width: eight slices' histograms fit 48 KB at ten bits each
    constexpr int kDigit = S == 8 ? 10 : 11, kBins = 1 << kDigit, kFirst = 32 - kDigit;
    __shared__ __align__(16) uint32_t hist[S][kBins];
    __shared__ uint32_t list[S][kList];
    __shared__ uint32_t s_prefix[S], s_r[S], s_cnt[S], s_m[S], s_up[S];
    __shared__ int s_bits[S], s_nan[S];
    pdl_trigger();
    pdl_wait_for(x, centre, out);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, slot = tid % S;
    const int per = blockDim.x / S;  // threads a slice
    const int64_t groups = (lo + S - 1) / S, h = blockIdx.x / groups, l0 = (blockIdx.x - h * groups) * S;
    const int64_t l = l0 + slot;
    const bool live = S == 1 || l < lo, live_w = S == 1 || l0 + wid < lo;  // this thread's slice, the one this warp serves
    const float c = AD && live ? centre[l + lo * h] : 0.0f;
    uint32_t key[KPT];
    {
        const int first = tid / S;
        const int cnt = live && first < n ? (int)((n - first + per - 1) / per) : 0;  // <= KPT
        const float *p = x + l + lo * n * h + lo * first;
        const int64_t step = lo * per;
        float v[KPT];
#pragma unroll
        for (int j = 0; j < KPT; ++j, p += step) v[j] = j < cnt ? __ldcs(p) : __uint_as_float(0x7f800000u);
        for (int i = tid; i < S * kBins / 4; i += blockDim.x) ((uint4 *)hist)[i] = make_uint4(0, 0, 0, 0);
        if (tid < S) { s_nan[tid] = 0; s_m[tid] = 0; s_up[tid] = 0xffffffffu; s_prefix[tid] = s_r[tid] = s_cnt[tid] = 0; s_bits[tid] = 0; }
        __syncthreads();
        bool nan = false;
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const float e = AD ? fabsf(__fsub_rn(v[j], c)) : v[j];
            nan |= e != e;
            key[j] = med_key(e);
            atomicAdd(&hist[slot][key[j] >> kFirst], 1u);
        }
        if (nan) s_nan[slot] = 1;
    }
    __syncthreads();
    const bool even = (n & 1) == 0;
    if (wid < S && live_w) {
        uint32_t bin, rest, bc;
        wide_find_bin<kBins>(hist[wid], (uint32_t)((n - 1) >> 1), lane, bin, rest, bc);
        if (lane == 0) { s_prefix[wid] = bin << kFirst; s_r[wid] = rest; s_cnt[wid] = bc; s_bits[wid] = kFirst; }
    }
    __syncthreads();
    // more digits where too many keys share the ones found
    for (int bits = kFirst > kDigit ? kFirst - kDigit : 0;; bits = bits > kDigit ? bits - kDigit : 0) {
        bool more = false;
#pragma unroll
        for (int i = 0; i < S; ++i) more |= s_cnt[i] > kList && s_bits[i] > 0;
        if (!more) break;
        const bool mine = s_cnt[slot] > kList && s_bits[slot] > 0;
        const uint32_t prefix = s_prefix[slot], width = 1u << s_bits[slot];
        for (int i = tid; i < S * kBins / 4; i += blockDim.x) ((uint4 *)hist)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        if (mine)
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const uint32_t d = key[j] - prefix;
                if (d < width) atomicAdd(&hist[slot][d >> bits], 1u);
            }
        __syncthreads();
        if (wid < S && s_cnt[wid] > kList && s_bits[wid] > 0) {
            uint32_t bin, rest, bc;
            wide_find_bin<kBins>(hist[wid], s_r[wid], lane, bin, rest, bc);
            __syncwarp();
            if (lane == 0) { s_prefix[wid] |= bin << bits; s_r[wid] = rest; s_cnt[wid] = bc; s_bits[wid] = bits; }
        }
        __syncthreads();
    }
    // gather the keys that share the digits found; where an even length's lower
    // middle key is the last of them, look for the smallest key above
    {
        const uint32_t prefix = s_prefix[slot], width = 1u << s_bits[slot];
        if (live && s_bits[slot] > 0) {
            unsigned long long hits = 0;
#pragma unroll
            for (int j = 0; j < KPT; ++j) hits |= (unsigned long long)(key[j] - prefix < width) << j;
            if (hits) {
                uint32_t *to = list[slot] + atomicAdd(&s_m[slot], (uint32_t)__popcll(hits));
#pragma unroll
                for (int j = 0; j < KPT; ++j)
                    if (hits >> j & 1) *to++ = key[j];
            }
        }
        if (even && live && s_r[slot] + 1 >= s_cnt[slot]) {
            const uint32_t top = prefix + (width - 1);
            uint32_t up = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < KPT; ++j)
                if (key[j] > top && key[j] < up) up = key[j];
            if (up != 0xffffffffu) atomicMin(&s_up[slot], up);
        }
    }
    __syncthreads();
    if (wid < S && live_w) {
        uint32_t key1 = s_prefix[wid], key2 = key1;
        const uint32_t r = s_r[wid], m = s_cnt[wid];
        if (s_bits[wid] > 0) rank_list(list[wid], (int)m, r, s_bits[wid], lane, key1, key2);
        if (even && r + 1 >= m) key2 = s_up[wid];
        if (lane == 0)
            out[l0 + wid + lo * h] = s_nan[wid] ? __uint_as_float(0x7fc00000u)
                                     : even     ? nt2_meanof(med_val(key1), med_val(key2))
                                                : med_val(key1);
    }
}

// ------------------------------------------------ long slices, global passes --
// A slice's state; its 256 64-bit counters precede all states in the workspace
// and hold the gathered keys in the end.
struct MedState {
    unsigned long long r, cnt;  // rank left inside the keys matching prefix; their count
    uint32_t prefix, nan, key2, ticket;
};
constexpr uint32_t kDone = 0x80000000u;  // in nan: the slice's result is written

__global__ void k_median_init(MedState *st, unsigned long long *ghist, int64_t S, int64_t n)
{
    pdl_trigger();
    pdl_wait_for(st, ghist);
    const int64_t s = blockIdx.x;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) ghist[s * 256 + i] = 0;
    if (threadIdx.x == 0) st[s] = MedState{(unsigned long long)((n - 1) >> 1), (unsigned long long)n, 0, 0, 0xffffffffu, 0};
}

// What bounds it: latency of a short kernel on a table that sits in L2 (five
// launches, 15 us each for 12M elements; an earlier form of 184 blocks, with the
// digits picked and the result written by launches of their own, took 25 each
// and a sixth read).
// Pass over chunk blockIdx.x of slice blockIdx.y, by the digits found so far
// (those above bit `above`): a histogram of the next one, its bins added to the
// slice's; or, once at most kGather keys share them, those keys gathered and,
// for an even length, the smallest key above them found.  The slice's last
// block (by ticket) picks the digit, or ranks the keys and writes the result;
// the last pass has the whole key and no digit left.
template <bool AD, bool LINE>
__global__ void __launch_bounds__(256, 6) k_median_pass(const float *__restrict__ x, int64_t lo, int64_t n, int64_t chunk,
                                                     const float *centre, MedState *st, unsigned long long *ghist,
                                                     int above, int64_t s0, float *out)
{
    __shared__ uint32_t hist[256];
    __shared__ uint32_t list[kList];
    __shared__ uint32_t s_last;
    pdl_trigger();  // the next pass lines up while this one runs
    pdl_wait_for(x, centre, st, ghist, out);
    const int64_t s = s0 + blockIdx.y, l = s % lo, h = s / lo;
    MedState *ms = st + s;
    unsigned long long *gh = ghist + s * 256;
    if (ms->nan & kDone) return;
    const bool even = (n & 1) == 0;
    const float *base = x + l + lo * n * h;
    const float c = AD ? centre[s] : 0.0f;
    const uint32_t prefix = ms->prefix;
    const unsigned long long cnt = ms->cnt;
    const bool gather = above == 0 || cnt <= kGather;
    hist[threadIdx.x] = 0;
    __syncthreads();
    const int64_t k0 = blockIdx.x * chunk;
    int64_t k1 = k0 + chunk < n ? k0 + chunk : n;
    if (above == 0 && !(even && ms->r + 1 >= cnt)) k1 = k0;  // nothing left to look for
    bool nan = false;
    uint32_t up = 0xffffffffu;
    // the keys that share the digits found: those within `width` of prefix (all, at first)
    const uint32_t width = above == 32 ? 0xffffffffu : (1u << above) - 1, top = prefix + width;
    const int shift = above - 8;
    auto take = [&](float e) {
        if (AD) e = fabsf(__fsub_rn(e, c));
        nan |= e != e;
        const uint32_t key = med_key(e), d = key - prefix;
        if (gather) {
            if (d <= width && above > 0) {
                // the first word of the slice's counters counts; the keys follow, from the 17th
                const uint32_t at = atomicAdd((uint32_t *)gh, 1u);
                if (at < kGather) ((uint32_t *)gh)[16 + at] = key;
            }
            if (key > top && key < up) up = key;
        } else if (d <= width) {
            atomicAdd(&hist[d >> shift], 1u);
        }
    };
    const int64_t step = LINE ? 1 : lo;
    const float *p = base + step * (k0 + threadIdx.x);
    int64_t k = k0;
    for (; k + kLoadBatch * 256 <= k1; k += kLoadBatch * 256) {
        float v[kLoadBatch];
#pragma unroll
        for (int j = 0; j < kLoadBatch; ++j, p += step * 256) v[j] = *p;
#pragma unroll
        for (int j = 0; j < kLoadBatch; ++j) take(v[j]);
    }
    for (k += threadIdx.x; k < k1; k += 256, p += step * 256) take(*p);
    if (above == 32 && __syncthreads_or(nan) && threadIdx.x == 0) atomicOr(&ms->nan, 1u);
    if (gather) {
        if (even) {
            up = __reduce_min_sync(0xffffffffu, up);
            if ((threadIdx.x & 31) == 0 && up != 0xffffffffu) atomicMin(&ms->key2, up);
        }
    } else {
        __syncthreads();
        const uint32_t v = hist[threadIdx.x];
        if (v) atomicAdd(&gh[threadIdx.x], (unsigned long long)v);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();  // the block's additions before its ticket
        s_last = atomicAdd(&ms->ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last || threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const volatile MedState *vs = ms;
    if (!gather) {
        uint32_t bin = 0;
        unsigned long long rest = 0, bc = 0;
        bool mine;
        med_find_bin<unsigned long long>((const volatile unsigned long long *)gh, (unsigned long long)vs->r, lane, bin, rest, bc,
                                         mine);
        __syncwarp();
        if (mine) {
            ms->prefix = prefix | bin << (above - 8);
            ms->r = rest;
            ms->cnt = bc;
        }
        for (int j = 0; j < 8; ++j) gh[lane * 8 + j] = 0;
        if (lane == 0) ms->ticket = 0;
        return;
    }
    uint32_t key1 = prefix, key2 = prefix;
    const unsigned long long r = vs->r;
    if (above > 0) {
        for (int j = lane; j < (int)cnt; j += 32) list[j] = ((const volatile uint32_t *)gh)[16 + j];
        __syncwarp();
        rank_list(list, (int)cnt, (uint32_t)r, above, lane, key1, key2);
    }
    if (even && r + 1 >= cnt) key2 = vs->key2;
    if (lane == 0) {
        out[s] = (vs->nan & 1u) ? __uint_as_float(0x7fc00000u)
                 : even         ? nt2_meanof(med_val(key1), med_val(key2))
                                : med_val(key1);
        ms->nan = kDone;
    }
}

__global__ void k_median_fill_nan(float *out, int64_t S)
{
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s < S) out[s] = __uint_as_float(0x7fc00000u);
}

size_t median_workspace_bytes(int64_t lo, int64_t n, int64_t hi)
{
    if (n <= kRegKeys) return 0;
    const int64_t S = lo * hi;
    return (size_t)S * (256 * sizeof(unsigned long long) + sizeof(MedState));
}

// The fewest keys a thread whose block stays within 1024 threads: more threads
// a slice hide more of its phases.
template <bool AD, int S>
static cudaError_t launch_regs(const float *x, int64_t lo, int64_t n, int64_t hi, const float *centre, float *out, cudaStream_t st)
{
    const unsigned grid = (unsigned)((lo + S - 1) / S * hi);
    const int64_t keys = n * S;
    auto threads = [&](int kpt) {  // each slice gets the same number of threads, of kpt keys
        const int64_t per = (n + kpt - 1) / kpt;
        return (int)((per * S + 31) / 32 * 32);
    };
#define NT2G_REGS(KPT, MAXT) return launch_dependent(k_median_regs<AD, S, KPT, MAXT>, dim3(grid), threads(KPT), st, x, lo, n, centre, out)
    if (keys <= 16 * 256) NT2G_REGS(16, 256);
    else if (keys <= 16 * 768) NT2G_REGS(16, 768);
    else if (keys <= 16 * 1024) NT2G_REGS(16, 1024);
    else if (keys <= 32 * 1024) NT2G_REGS(32, 1024);
    else NT2G_REGS(40, 1024);
#undef NT2G_REGS
}

template <bool AD>
static nt2g_status median_pass(const float *x, int64_t lo, int64_t n, int64_t hi, const float *centre,
                               void *ws, float *out, cudaStream_t st)
{
    const int64_t S = lo * hi;
    if (n <= kShortKeys) {
        const size_t smem = (size_t)n * 4 + 256 * 4;
        const int threads = n >= 256 ? 256 : (int)((n + 31) / 32 * 32);
        k_median_smem<AD><<<(unsigned)S, threads, smem, st>>>(x, lo, n, centre, out);
        NT2G_LAUNCH_CHECK("median (shared memory)");
        return NT2G_OK;
    }
    if (n <= kRegKeys) {
        cudaError_t ce;
        // several slices a block, unless that leaves most SMs without one (us, medians
        // of 2621 strided elements: 64 slices 9.6 by eights, 6.3 one by one; 100 of
        // 7000 11.5 by fours and 13.5; 1000 of 2621 9.8 by eights, 10.6 by fours)
        if (lo >= 8 && n * 8 <= kRegKeys && (lo + 7) / 8 * hi >= 76) ce = launch_regs<AD, 8>(x, lo, n, hi, centre, out, st);
        else if (lo >= 4 && n * 4 <= kRegKeys && (lo + 3) / 4 * hi >= 25) ce = launch_regs<AD, 4>(x, lo, n, hi, centre, out, st);
        else ce = launch_regs<AD, 1>(x, lo, n, hi, centre, out, st);
        if (ce != cudaSuccess) return cuda_status(ce, "median (registers)");
        NT2G_LAUNCH_CHECK("median (registers)");
        return NT2G_OK;
    }
    unsigned long long *ghist = (unsigned long long *)ws;
    MedState *state = (MedState *)(ghist + S * 256);
    cudaError_t ce = launch_dependent(k_median_init, dim3((unsigned)S), 256, st, state, ghist, S, n);
    // one wave of blocks (six an SM), of at least 4096 elements each
    int64_t chunk = (n * S + 152 * 6 - 1) / (152 * 6);
    chunk = chunk < 4096 ? 4096 : chunk > 65536 ? 65536 : (chunk + 255) / 256 * 256;
    const unsigned chunks = (unsigned)((n + chunk - 1) / chunk);
    for (int above = 32; above >= 0; above -= 8) {
        for (int64_t s0 = 0; s0 < S; s0 += 65535) {  // grid.y: at most 65535 slices per launch
            const dim3 grid(chunks, (unsigned)(S - s0 < 65535 ? S - s0 : 65535));
            if (ce != cudaSuccess) return cuda_status(ce, "median (global passes)");
            ce = launch_dependent(lo == 1 ? k_median_pass<AD, true> : k_median_pass<AD, false>, grid, 256, st, x, lo, n, chunk, centre,
                                  state, ghist, above, s0, out);
        }
    }
    if (ce != cudaSuccess) return cuda_status(ce, "median (global passes)");
    NT2G_LAUNCH_CHECK("median (global passes)");
    return NT2G_OK;
}

nt2g_status launch_median(const float *x, int64_t lo, int64_t n, int64_t hi, int32_t op, void *ws, float *out,
                          cudaStream_t st)
{
    const int64_t S = lo * hi;
    if (n == 0) {  // no middle element
        k_median_fill_nan<<<(unsigned)((S + 255) / 256), 256, 0, st>>>(out, S);
        NT2G_LAUNCH_CHECK("median (empty slices)");
        return NT2G_OK;
    }
    nt2g_status r = median_pass<false>(x, lo, n, hi, nullptr, ws, out, st);
    if (r != NT2G_OK || op == NT2G_MEDIAN) return r;
    return median_pass<true>(x, lo, n, hi, out, ws, out, st);
}

}  // namespace nt2g
