// Cross-sectional kernels: one thread block per time step (row of the [T][S]
// layout).
//  - Rank (cpp/Kun/Rank.hpp:13-57): every stock's equal range in the row's
//    sorted non-NaN values, found by counting in value-range buckets;
//    out = T(sum) / T(cnt) / T(n) with the integer rank sum of the range.
//  - Scale (cpp/Kun/Scale.hpp:14-46): the sum of |x| over non-NaN stocks in
//    stock order (sequential, as the reference adds), then x / sum.
//  - DiffWithWeightedSum (KunQuant/ops/MiscOp.py:220-240).
#pragma once
#include <algorithm>
#include <type_traits>

#include "kun_device.cuh"

namespace kun {

// Order-preserving integer keys: a < b of values is a < b of keys, equal values
// (-0 and +0 too) have one key, NaN is the greatest.
template <typename T> struct SortKey;
template <> struct SortKey<float> {
    using K = uint32_t;
    static constexpr K kMax = 0xffffffffu;
    static constexpr K kNegInf = 0x007fffffu, kPosInf = 0xff800000u;
    static __device__ __forceinline__ K enc(float x) {
        const uint32_t u = __float_as_uint(kadd(x, 0.f));  // -0 + 0 is +0
        return x == x ? u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u) : kMax;
    }
    static __device__ __forceinline__ float dec(K k) {
        return __uint_as_float(k ^ ((uint32_t)((int32_t)~k >> 31) | 0x80000000u));
    }
    static __device__ __forceinline__ int bits(K k) { return 32 - __clz((int)k); }
};
template <> struct SortKey<double> {
    using K = unsigned long long;
    static constexpr K kMax = ~0ull;
    static constexpr K kNegInf = 0x000fffffffffffffull, kPosInf = 0xfff0000000000000ull;
    static __device__ __forceinline__ K enc(double x) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(x);
        if ((u & 0x7fffffffffffffffull) > 0x7ff0000000000000ull) return kMax;
        const K k = u ^ ((K)((long long)u >> 63) | 0x8000000000000000ull);
        return k == 0x7fffffffffffffffull ? 0x8000000000000000ull : k;  // -0
    }
    static __device__ __forceinline__ double dec(K k) {
        return __longlong_as_double((long long)(k ^ ((K)((long long)~k >> 63) | 0x8000000000000000ull)));
    }
    static __device__ __forceinline__ int bits(K k) { return 64 - __clzll((long long)k); }
};

// dynamic shared memory above which a launch first raises the kernel's
// limit: 48 KB less room for the kernels' static arrays
constexpr size_t kSmemOptIn = 40 * 1024;

// Rank of one row by one block, without sorting it.  A value's rank start is
// the number of smaller values in its row and its end adds the equal ones:
// exactly the equal range that the reference searches for in the sorted row
// (cpp/Kun/Rank.hpp:40-53), so the result is the sort's bit for bit.
//
//  1. Every thread holds ITEMS values of the row in registers; the block finds
//     the row's least and greatest finite value and the number of non-NaN ones.
//  2. Each value goes to one of B = threads x ITEMS buckets by a monotone map:
//     linear in the value, or linear in its order-preserving integer key
//     (logarithmic in the value) for rows of one sign crowded towards zero.
//     The first value of a bucket is its representative.
//  3. The counters are scanned; a value that differs from its bucket's
//     representative takes a place among those below or above it.  The others'
//     ranks are then known, so ties cost nothing, however many.
//  4. Those values are scattered by bucket and side, and each counts the
//     smaller and equal ones on its side.
//
// When more than kRankPoor values of a bucket lie on one side (sides are
// counted in 8 bits, which kRankWorst stays below), the map is refined
// (rank_refine), at most twice (correlations of ranks a few units in the last
// place around zero need it), then the other map is; a row that none of them
// spreads is sorted in shared memory (rank_row_sorted).  Bound by the issue rate: about 220
// instructions a value with 75% of the issue slots taken at 8192 stocks, so the
// block is as small as the row allows and several rows share an SM: 8 values a
// thread up to 4096 stocks and 16 above.  Shared memory: B keys
// (representatives, then the scattered keys over them), B counters and B
// scanned counts, 10 bytes a value in fp32.  Normal values, against a bitonic
// network in 1024-thread blocks up to 1024 stocks and, above, buckets with a
// radix sort behind them in one 1024-thread block an SM: 997 stocks x 1251
// rows 16 us (132), 3000 x 1500 37 us (88), 8192 x 2500 156 us (336), the same
// with 10 tied values 125 us (530); fp64 801 x 1000 23 us (244).
constexpr int kRankMaxStocks = 16384;
constexpr int kRankPad = 4;  // keys behind a row's, for the counting loop's step
constexpr int kRankPoor = 20;   // counting up to this many neighbours costs less than another map
constexpr int kRankWorst = 96;  // counting 96 neighbours costs about as much as sorting the row

__host__ __device__ inline int rank_threads(int S, int items) {
    const int w = (S + items * 32 - 1) / (items * 32);
    return (w < 1 ? 1 : w) * 32;
}
template <typename T> __host__ __device__ inline size_t rank_smem_bytes(int nt, int items) {
    return (size_t)nt * items * (sizeof(T) + sizeof(uint32_t) + sizeof(uint16_t)) + kRankPad * sizeof(T);
}

// register budget (launch bounds): 40 a thread for 8 values in fp32, so that
// three 512-thread blocks or their like share an SM, else 64
template <typename T> constexpr int rank_min_blocks(int items, int maxt) {
    return maxt == 1024 ? 1 : (items <= 8 && sizeof(T) == 4 ? 3 : 2);
}

// block barriers over the first nt threads (warps past them have left)
__device__ __forceinline__ void rank_sync(int nt) {
    if (nt == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
}
__device__ __forceinline__ bool rank_sync_or(int nt, bool p) {
    if (nt == 32) {
        const bool any = __any_sync(0xffffffffu, p);
        __syncwarp();
        return any;
    }
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((int)p), "r"(nt)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ uint32_t warp_min_key(uint32_t k) { return __reduce_min_sync(0xffffffffu, k); }
__device__ __forceinline__ uint32_t warp_max_key(uint32_t k) { return __reduce_max_sync(0xffffffffu, k); }
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, k, o);
        k = x < k ? x : k;
    }
    return k;
}
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, k, o);
        k = x > k ? x : k;
    }
    return k;
}
// T(sum) / T(cnt) / T(n) of the equal range [less, less + eq) with the integer
// rank sum (2 less + eq + 1) eq / 2, below 2^31: less + eq <= n <= 16384.  A
// sum that T holds exactly leaves the mean rank (2 less + eq + 1) / 2 exact, so
// only larger ones (thousands of ties, in float) need the first division.  The
// division by the row's n is Markstein's (IBM J. Res. Dev. 34, 1990): with
// r = 1/n rounded to nearest and a residual by FMA, q + (s - q n) r is the
// correctly rounded quotient.
template <typename T> struct RankDivisor;
template <> struct RankDivisor<float> {
    float n, r;
    __device__ __forceinline__ explicit RankDivisor(int cnt) {
        n = (float)cnt;
        r = __frcp_rn(n);
    }
    __device__ __forceinline__ float operator()(float s) const {
        const float q = __fmul_rn(s, r);
        return __fmaf_rn(__fmaf_rn(-q, n, s), r, q);
    }
};
template <> struct RankDivisor<double> {
    double n, r;
    __device__ __forceinline__ explicit RankDivisor(int cnt) {
        n = (double)cnt;
        r = __drcp_rn(n);
    }
    __device__ __forceinline__ double operator()(double s) const {
        const double q = __dmul_rn(s, r);
        return __fma_rn(__fma_rn(-q, n, s), r, q);
    }
};
template <typename T> __device__ __noinline__ T rank_mean_of_large(uint32_t sum, uint32_t eq) {
    return kdiv((T)(int)sum, (T)(int)eq);
}
template <typename T> __device__ __forceinline__ T rank_value(uint32_t less, uint32_t eq, const RankDivisor<T> &n) {
    const uint32_t twice = 2 * less + eq + 1, sum2 = twice * eq;
    T s = kmul((T)(int)twice, T(0.5));
    if (sizeof(T) == 4 && sum2 > (2u << 24)) s = rank_mean_of_large<T>(sum2 / 2, eq);
    return n(s);
}

// The row's keys sorted in shared memory (a bitonic network whose every
// exchange puts the smaller key first, so that it needs no padding), then two
// binary searches a value.  For rows that neither bucket map spreads.
template <typename T, typename Out>
__device__ __forceinline__ void rank_row_sorted(const T *__restrict__ row, int S, int n, int nt,
                                                typename SortKey<T>::K *keys, Out out) {
    using SK = SortKey<T>;
    using K = typename SK::K;
    const int tid = threadIdx.x;
    const RankDivisor<T> over_n(n);
    for (int i = tid; i < S; i += nt) keys[i] = SK::enc(row[i]);
    rank_sync(nt);
    int P = 1;
    while (P < S) P <<= 1;
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int q = tid; q < P / 2; q += nt) {
                const int i = (q & -j) * 2 + (q & (j - 1));
                const int o = j == (k >> 1) ? i ^ (k - 1) : i + j;  // mirrored in the first step of a merge
                if (o < S) {
                    const K a = keys[i], b = keys[o];
                    if (b < a) {
                        keys[i] = b;
                        keys[o] = a;
                    }
                }
            }
            rank_sync(nt);
        }
    }
    for (int i = tid; i < S; i += nt) {
        const K x = SK::enc(row[i]);
        T res = knan<T>();
        if (x != SK::kMax) {
            int lo = 0, hi = n;
            while (lo < hi) { const int m = (lo + hi) >> 1; if (keys[m] < x) lo = m + 1; else hi = m; }
            const int start = lo;
            hi = n;
            while (lo < hi) { const int m = (lo + hi) >> 1; if (x < keys[m]) hi = m; else lo = m + 1; }
            res = rank_value<T>((uint32_t)start, (uint32_t)(lo - start), over_n);
        }
        out(i, res);
    }
}

// counters in 16-byte groups, swizzled so that the scan's wide reads of
// consecutive groups meet no bank twice
__device__ __forceinline__ int rank_swizzle(int b) { return b ^ ((b >> 3) & 0x1c); }

// Splits every bucket of c values into up to c by the distance of their keys
// from its least key, in steps of a power of two: pk's buckets become the
// finer ones.  Exact in integers, so that values a few units in the last
// place apart (correlations of ranks) part as well as a bucket that an
// outlier made wide.  kmin: B keys over the representatives.
template <typename T, int ITEMS>
__device__ __forceinline__ void rank_refine(const typename SortKey<T>::K (&k)[ITEMS], uint32_t (&pk)[ITEMS], int nt,
                                            uint32_t *hist, const uint16_t *base, typename SortKey<T>::K *kmin) {
    using SK = SortKey<T>;
    using K = typename SK::K;
#pragma unroll
    for (int e = 0; e < ITEMS; e++) {
        kmin[e * nt + threadIdx.x] = SK::kMax;
        hist[e * nt + threadIdx.x] &= 0xffff;
    }
    rank_sync(nt);
#pragma unroll
    for (int e = 0; e < ITEMS; e++) {
        pk[e] &= 0x3fff;
        if (k[e] != SK::kMax) atomicMin(&kmin[pk[e]], k[e]);
    }
    rank_sync(nt);
#pragma unroll
    for (int e = 0; e < ITEMS; e++)
        if (k[e] != SK::kMax)  // the count is below the bits
            atomicMax(&hist[pk[e]], (hist[pk[e]] & 0xffff) | (uint32_t)SK::bits(k[e] - kmin[pk[e]]) << 16);
    rank_sync(nt);
#pragma unroll
    for (int e = 0; e < ITEMS; e++) {
        if (k[e] != SK::kMax) {
            const uint32_t w = hist[pk[e]];
            const int shift = (int)(w >> 16) - (31 - __clz((int)(w & 0xffff)));
            const K d = k[e] - kmin[pk[e]];
            pk[e] = (uint32_t)rank_swizzle(base[pk[e]] + (int)(d >> (shift > 0 ? shift : 0)));
        }
    }
}

// The bucket maps of a row, 1 .. B - 2 for finite values, monotone over all:
// -inf is 0, +inf the last or beside the greatest.  In float for both types
// (rounding to float is monotone, and FP64 arithmetic is slow here).  The shift
// brings the finite values' key distances to 32 bits; that of a double's +inf
// may have more, and counts as the greatest.
template <typename T> struct RankMap {
    using SK = SortKey<T>;
    using K = typename SK::K;
    bool by_key;
    int shift;  // key distances to 32 bits
    float scale, top;
    K lo;
    T vlo;
    static __device__ __forceinline__ uint32_t saturate(uint32_t d) { return d; }
    static __device__ __forceinline__ uint32_t saturate(unsigned long long d) {
        return d >> 32 ? 0xffffffffu : (uint32_t)d;
    }
    __device__ __forceinline__ RankMap(bool by_key_, K lo_, K hi, int B) : by_key(by_key_), lo(lo_), vlo(SK::dec(lo_)) {
        shift = SK::bits(hi - lo) > 32 ? SK::bits(hi - lo) - 32 : 0;
        const float range = by_key ? __uint2float_rn((uint32_t)((hi - lo) >> shift)) : (float)ksub(SK::dec(hi), vlo);
        top = (float)(B - 2);
        scale = fminf(__fdiv_rn((float)(B - 3), range), 3e38f);  // finite: 0 * scale is 0
    }
    __device__ __forceinline__ int operator()(K k) const {
        const float d = by_key ? (k < lo ? -1.f : __uint2float_rn(saturate((k - lo) >> shift)))
                               : (float)ksub(SK::dec(k), vlo);
        return (int)fminf(fmaxf(__fmul_rn(d, scale), -1.f), top) + 1;
    }
};

// Ranks the S <= nt * ITEMS values of a row with the block's first nt threads
// (a multiple of 32; the others must have left) and hands each stock's rank
// to out(i, rank).  smem: rank_smem_bytes<T>(nt, ITEMS), 16-byte aligned.
template <typename T, int ITEMS, typename Out>
__device__ __forceinline__ void rank_row(const T *__restrict__ row, int S, int nt, unsigned char *smem, Out out) {
    using SK = SortKey<T>;
    using K = typename SK::K;
    __shared__ K red_lo[32], red_hi[32];
    __shared__ uint32_t red_n[32], scan_w[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int B = nt * ITEMS;
    K *rep = reinterpret_cast<K *>(smem), *vals = rep;
    // count | below the representative << 16 | above << 24
    uint32_t *hist = reinterpret_cast<uint32_t *>(smem + (size_t)(B + kRankPad) * sizeof(K));
    uint16_t *base = reinterpret_cast<uint16_t *>(hist + B);
    K k[ITEMS];
#pragma unroll
    for (int e = 0; e < ITEMS; e++) {
        const int i = e * nt + tid;
        k[e] = i < S ? SK::enc(row[i]) : SK::kMax;
    }
    const T sample = row[(unsigned)(lane * S) >> 5];  // the same 32 in every warp
    auto clear = [&]() {
#pragma unroll
        for (int e = 0; e < ITEMS / 4; e++) reinterpret_cast<uint4 *>(hist)[e * nt + tid] = make_uint4(0, 0, 0, 0);
    };
    clear();
    // least and greatest value and the number of them; again over the finite
    // ones for a row that has infinities
    K lo, hi;
    int n;
    bool infinite = false;
    for (;;) {
        lo = SK::kMax, hi = 0;
        uint32_t cnt = 0;
#pragma unroll
        for (int e = 0; e < ITEMS; e++) {
            if (k[e] != SK::kMax) cnt++;
            if (infinite ? k[e] > SK::kNegInf && k[e] < SK::kPosInf : k[e] != SK::kMax) {
                lo = k[e] < lo ? k[e] : lo;
                hi = k[e] > hi ? k[e] : hi;
            }
        }
        lo = warp_min_key(lo);
        hi = warp_max_key(hi);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (nw > 1) {
            if (lane == 0) {
                red_lo[warp] = lo;
                red_hi[warp] = hi;
                red_n[warp] = cnt;
            }
            rank_sync(nt);
            lo = warp_min_key(lane < nw ? red_lo[lane] : SK::kMax);
            hi = warp_max_key(lane < nw ? red_hi[lane] : K(0));
            cnt = __reduce_add_sync(0xffffffffu, lane < nw ? red_n[lane] : 0u);
        } else {
            __syncwarp();
        }
        n = (int)cnt;
        if (infinite || n == 0 || (lo > SK::kNegInf && hi < SK::kPosInf)) break;
        infinite = true;
        rank_sync(nt);
    }
    const RankDivisor<T> over_n(n);
    if (n == 0 || (lo == hi && !infinite)) {  // no values, or one value throughout
        const T res = n ? rank_value<T>(0u, (uint32_t)n, over_n) : knan<T>();
#pragma unroll
        for (int e = 0; e < ITEMS; e++) {
            const int i = e * nt + tid;
            if (i < S) out(i, k[e] != SK::kMax ? res : knan<T>());
        }
        return;
    }
    if (lo > hi) lo = hi = SK::enc(T(0));  // infinities alone
    // by key: values of one sign most of which (20 of the 32 looked at) lie in
    // the range's sixteenth nearest zero, and a spread that float does not hold
    // (then by key only)
    const float vlo = (float)SK::dec(lo), spread = (float)ksub(SK::dec(hi), SK::dec(lo));
    const bool wide = !(spread < kinf<float>());
    const float from = sample >= T(0) ? (float)sample - vlo : (float)SK::dec(hi) - (float)sample;
    const bool key_first = wide || (((hi ^ lo) >> (sizeof(K) * 8 - 1)) == 0 &&
                                    __popc(__ballot_sync(0xffffffffu, from < spread * 0.0625f)) >= 20);
    uint32_t pk[ITEMS];  // bucket | place << 14 | relation to the representative << 30 (1 below, 2 above)
    bool sorted = false;
    for (int attempt = 0;; attempt++) {  // a map, refined, refined again; then the other
        if (attempt % 3) {
            rank_refine<T, ITEMS>(k, pk, nt, hist, base, rep);
        } else {
            const RankMap<T> map(wide || key_first != (attempt == 3), lo, hi, B);
#pragma unroll
            for (int e = 0; e < ITEMS; e++) pk[e] = (uint32_t)rank_swizzle(map(k[e]));
        }
        if (attempt) {
            rank_sync(nt);
            clear();
            rank_sync(nt);
        }
#pragma unroll
        for (int e = 0; e < ITEMS; e++)
            if (k[e] != SK::kMax && atomicAdd(&hist[pk[e]], 1u) == 0) rep[pk[e]] = k[e];
        rank_sync(nt);
        uint32_t deep = 0;
#pragma unroll
        for (int e = 0; e < ITEMS; e++) {
            const K r = rep[pk[e]];
            if (k[e] != SK::kMax && r != k[e]) {
                const bool below = k[e] < r;
                const uint32_t old = atomicAdd(&hist[pk[e]], below ? 1u << 16 : 1u << 24);
                const uint32_t place = below ? (old >> 16) & 0xff : old >> 24;
                deep = max(deep, place);
                pk[e] |= place << 14 | (below ? 1u << 30 : 2u << 30);
            }
        }
        // exclusive scan of the counts, ITEMS consecutive ones a thread
        uint32_t sum = 0;
#pragma unroll
        for (int g = 0; g < ITEMS / 4; g++) {
            const int at = tid * (ITEMS / 4) + g;
            const uint4 q = reinterpret_cast<const uint4 *>(hist)[at ^ ((at >> 3) & 7)];
            sum += (q.x & 0xffff) + (q.y & 0xffff) + (q.z & 0xffff) + (q.w & 0xffff);
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) scan_w[warp] = incl;
        rank_sync(nt);
        uint32_t run = __reduce_add_sync(0xffffffffu, lane < warp ? scan_w[lane] : 0u) + incl - sum;
#pragma unroll
        for (int g = 0; g < ITEMS / 4; g++) {
            const int at = tid * (ITEMS / 4) + g, sw = at ^ ((at >> 3) & 7);
            const uint4 q = reinterpret_cast<const uint4 *>(hist)[sw];
            const uint32_t b0 = run, b1 = b0 + (q.x & 0xffff), b2 = b1 + (q.y & 0xffff), b3 = b2 + (q.z & 0xffff);
            run = b3 + (q.w & 0xffff);
            reinterpret_cast<uint2 *>(base)[sw] = make_uint2(b0 | b1 << 16, b2 | b3 << 16);
        }
        if (!rank_sync_or(nt, deep >= (uint32_t)(attempt < 5 ? kRankPoor : kRankWorst))) break;
        if (attempt == 5) {
            sorted = true;
            break;
        }
        // a bucket that most of the row is in asks for the other map at once
        if (attempt == 0) {
            uint32_t crowd = 0;
#pragma unroll
            for (int e = 0; e < ITEMS; e++) crowd = max(crowd, hist[pk[e] & 0x3fff] & 0xffff);
            if (rank_sync_or(nt, crowd >= (uint32_t)n / 4 * 3)) attempt = 2;
        }
    }
    if (sorted) {
        rank_row_sorted<T>(row, S, n, nt, reinterpret_cast<K *>(smem), out);
        return;
    }
    // The representatives are no longer needed: the values unlike them take
    // their place, in each bucket's part those below from its start on and those
    // above towards its end.  The rest is the greatest key, and later buckets
    // hold greater values, so a count may run past its list: four values a step
    // without a test (a warp's lanes have lists of unlike length).
    constexpr int WIDE = 16 / sizeof(K);
    struct alignas(16) Keys {
        K k[WIDE];
    };
    Keys none;
#pragma unroll
    for (int q = 0; q < WIDE; q++) none.k[q] = SK::kMax;
#pragma unroll
    for (int e = 0; e < ITEMS / WIDE; e++) reinterpret_cast<Keys *>(vals)[e * nt + tid] = none;
    if (tid < kRankPad) vals[B + tid] = SK::kMax;
    rank_sync(nt);
#pragma unroll
    for (int e = 0; e < ITEMS; e++)
        if (pk[e] >> 30) {
            const int at = pk[e] & 0x3fff, place = (pk[e] >> 14) & 0xff;
            vals[base[at] + ((pk[e] >> 31) ? (int)(hist[at] & 0xffff) - 1 - place : place)] = k[e];
        }
    rank_sync(nt);
#pragma unroll
    for (int e = 0; e < ITEMS; e++) {
        const int i = e * nt + tid;
        if (i < S) {
            const int at = pk[e] & 0x3fff;
            const uint32_t w = hist[at], cnt = w & 0xffff, below = (w >> 16) & 0xff, above = w >> 24;
            // a value like the representative has all below and none above
            uint32_t less = base[at] + below, eq = cnt - below - above;
            if (pk[e] >> 30) {
                const bool up = pk[e] >> 31;
                less = up ? less + eq : less - below;  // where its list starts
                eq = 0;
                const K *v = vals + less, *end = v + (up ? above : below);
#pragma unroll 1
                for (; v < end; v += 4) {
                    const K y0 = v[0], y1 = v[1], y2 = v[2], y3 = v[3];
                    less += (y0 < k[e]);
                    eq += (y0 == k[e]);
                    less += (y1 < k[e]);
                    eq += (y1 == k[e]);
                    less += (y2 < k[e]);
                    eq += (y2 == k[e]);
                    less += (y3 < k[e]);
                    eq += (y3 == k[e]);
                }
            }
            out(i, k[e] != SK::kMax ? rank_value<T>(less, eq, over_n) : knan<T>());
        }
    }
}

template <typename T> struct RankStore {
    T *__restrict__ o;
    __device__ __forceinline__ void operator()(int i, T r) const { o[i] = r; }
};

// rows of one [length][S] plane, a block each; blockDim.x = rank_threads(S, ITEMS)
template <typename T, int ITEMS, int MAXT>
__global__ void __launch_bounds__(MAXT, rank_min_blocks<T>(ITEMS, MAXT)) rank_rows(const T *__restrict__ in, T *__restrict__ out, int S) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long t = blockIdx.x;
    rank_row<T, ITEMS>(in + t * S, S, (int)blockDim.x, smem_raw, RankStore<T>{out + t * S});
}

// Stream mode, several Rank stages at once: block (k, j) ranks segment k
// for stage j of the job table (the stages of one level of the stage graph,
// which do not depend on each other).  Each job names the stage's input and
// output rings; the segment table is the step's.
struct RankJob {
    const void *in;
    void *out;
    int32_t w_in, w_out;
};

template <typename T, int ITEMS, int MAXT>
__device__ __forceinline__ void rank_segment(const T *in, int w_in, T *out, int w_out, long long cap, long long len,
                                             long long s0, long long n, unsigned char *smem) {
    if (len <= 0 || len > (long long)blockDim.x * ITEMS) return;
    const int nt = rank_threads((int)len, ITEMS);
    if ((int)threadIdx.x >= nt) return;
    rank_row<T, ITEMS>(in + (n % w_in) * cap + s0, (int)len, nt, smem, RankStore<T>{out + (n % w_out) * cap + s0});
}

// one stage, one block per segment, each at its own ring row
template <typename T, int ITEMS, int MAXT>
__global__ void __launch_bounds__(MAXT, rank_min_blocks<T>(ITEMS, MAXT)) rank_segments(const T *in, int w_in, T *out, int w_out, long long cap,
                                                      const int32_t *seg_off, const int32_t *seg_stock0,
                                                      const long long *seg_tick, const int32_t *cnt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int k = blockIdx.x;
    if (cnt && k >= cnt[0]) return;
    rank_segment<T, ITEMS, MAXT>(in, w_in, out, w_out, cap, seg_off[k + 1] - seg_off[k], seg_stock0[k], seg_tick[k],
                                 smem_raw);
}

// A step's table lists its segments of more than kRankShort stocks first and
// holds their number in cnt[3]; a launch takes those, the others, or all.
constexpr int kRankShort = 1024;
enum RankPart { kRankAll, kRankLongOnes, kRankShortOnes };

template <typename T, int ITEMS, int MAXT>
__global__ void __launch_bounds__(MAXT, rank_min_blocks<T>(ITEMS, MAXT)) rank_multi_segments(const RankJob *__restrict__ jobs, long long cap,
                                                            const int32_t *seg_off, const int32_t *seg_stock0,
                                                            const long long *seg_tick, const int32_t *cnt,
                                                            RankPart part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int k = blockIdx.x;
    if (cnt && (k >= cnt[0] || (part != kRankAll && (k < cnt[3]) != (part == kRankLongOnes)))) return;
    const RankJob jb = jobs[blockIdx.y];
    rank_segment<T, ITEMS, MAXT>((const T *)jb.in, jb.w_in, (T *)jb.out, jb.w_out, cap, seg_off[k + 1] - seg_off[k],
                                 seg_stock0[k], seg_tick[k], smem_raw);
}

// Scale of one row by one block.  The reference adds |x| in stock order, one
// dependent addition a stock, so a row takes at least that chain (4 cycles a
// stock).  The block puts the addends in shared memory, 0 for NaN (a sum of
// magnitudes is unchanged by +0), and one thread adds them from wide loads ahead
// of the chain.  With the test for NaN and one load a stock inside the chain a
// row of 4096 took 29 us in a stream's tick (15 now), 1251 rows of 997 24 us
// (13 now).  a: scale_slots(S) values, 16-byte aligned.
template <typename T> __host__ __device__ inline long long scale_slots(long long S) { return (S + 63) / 64 * 64 + 32; }
template <typename T>
__device__ __forceinline__ void scale_row(const T *__restrict__ row, T *__restrict__ out, long long S, T *a) {
    __shared__ T total;
    struct alignas(16) Wide {
        T v[16 / sizeof(T)];
    };
    constexpr int N = 16 / sizeof(T), WIDE = 32 / N;  // loads of 32 values
    const long long slots = scale_slots<T>(S);  // the last look-ahead's values are not added
#pragma unroll 8
    for (long long i = threadIdx.x; i < slots; i += blockDim.x) {
        const T x = i < S ? row[i] : T(0);
        a[i] = kisnan(x) ? T(0) : kabs(x);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const Wide *w = reinterpret_cast<const Wide *>(a);
        Wide even[WIDE], odd[WIDE];
        T sum = 0;
        auto load = [&](Wide(&to)[WIDE]) {
#pragma unroll
            for (int k = 0; k < WIDE; k++) to[k] = *w++;
        };
        auto add = [&](const Wide(&from)[WIDE]) {
#pragma unroll
            for (int k = 0; k < WIDE; k++)
#pragma unroll
                for (int q = 0; q < N; q++) sum = kadd(sum, from[k].v[q]);
        };
        load(even);
        for (long long i = 0; i < S; i += 64) {
            load(odd);
            add(even);
            load(even);
            add(odd);
        }
        total = sum;
    }
    __syncthreads();
    const T sum = total;
#pragma unroll 8
    for (long long i = threadIdx.x; i < S; i += blockDim.x) {
        const T x = row[i];
        out[i] = (x == T(0) && sum == T(0)) ? knan<T>() : kdiv(x, sum);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) scale_rows(const T *__restrict__ in, T *__restrict__ out, long long S) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long t = blockIdx.x;
    scale_row(in + t * S, out + t * S, S, reinterpret_cast<T *>(smem_raw));
}

template <typename T>
__global__ void __launch_bounds__(256) diffwsum_rows(const T *__restrict__ in0, const T *__restrict__ in1,
                                                    T *__restrict__ out, long long S, long long length) {
    __shared__ T total;
    for (long long t = blockIdx.x; t < length; t += gridDim.x) {
        if (threadIdx.x == 0) {
            T sum = 0;
            for (long long i = 0; i < S; i++) sum = kadd(sum, kmul(in0[t * S + i], in1[t * S + i]));
            total = sum;
        }
        __syncthreads();
        T sum = total;
        for (long long i = threadIdx.x; i < S; i += blockDim.x) out[t * S + i] = ksub(in0[t * S + i], sum);
        __syncthreads();
    }
}

template <typename T>
__global__ void __launch_bounds__(512) scale_segments(const T *__restrict__ in, int w_in, T *__restrict__ out,
                                                      int w_out, long long cap, const int32_t *seg_off,
                                                      const int32_t *seg_stock0, const long long *seg_tick,
                                                      const int32_t *cnt, int max_len) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int k = blockIdx.x;
    if (cnt && k >= cnt[0]) return;
    const long long len = seg_off[k + 1] - seg_off[k], s0 = seg_stock0[k], n = seg_tick[k];
    if (len > max_len) return;
    scale_row(in + (n % w_in) * cap + s0, out + (n % w_out) * cap + s0, len, reinterpret_cast<T *>(smem_raw));
}

template <typename T>
__global__ void __launch_bounds__(256) diffwsum_segments(const T *__restrict__ in0, int w0, const T *__restrict__ in1,
                                                         int w1, T *__restrict__ out, int w_out, long long cap,
                                                         const int32_t *seg_off, const int32_t *seg_stock0,
                                                         const long long *seg_tick, const int32_t *cnt) {
    __shared__ T total;
    const int k = blockIdx.x;
    if (cnt && k >= cnt[0]) return;
    const long long len = seg_off[k + 1] - seg_off[k], s0 = seg_stock0[k], n = seg_tick[k];
    const T *a = in0 + (n % w0) * cap + s0, *b = in1 + (n % w1) * cap + s0;
    T *orow = out + (n % w_out) * cap + s0;
    if (threadIdx.x == 0) {
        T sum = 0;
        for (long long i = 0; i < len; i++) sum = kadd(sum, kmul(a[i], b[i]));
        total = sum;
    }
    __syncthreads();
    const T sum = total;
    for (long long i = threadIdx.x; i < len; i += blockDim.x) orow[i] = ksub(a[i], sum);
}

// STs <-> TS row copies around the cross-sectional kernels: rows
// [row0, row0 + length) of an [S/L][T_in][L] buffer to a [length][S] one, and
// back to an [S/L][length][L] buffer.
template <typename T>
__global__ void sts_rows_to_ts(const T *__restrict__ in, T *__restrict__ out, long long S, long long T_in,
                               long long row0, long long length, int L) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= length * S) return;
    const long long t = i / S, s = i % S;
    out[i] = in[(s / L) * T_in * L + (row0 + t) * L + s % L];
}
template <typename T>
__global__ void ts_rows_to_sts(const T *__restrict__ in, T *__restrict__ out, long long S, long long length, int L) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= length * S) return;
    const long long t = i / S, s = i % S;
    out[(s / L) * length * L + t * L + s % L] = in[i];
}
template <typename T>
inline int launch_sts_to_ts(const T *in, T *out, long long S, long long T_in, long long row0, long long length, int L,
                            cudaStream_t st) {
    const long long n = length * S;
    sts_rows_to_ts<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, S, T_in, row0, length, L);
    return (int)cudaGetLastError();
}
template <typename T>
inline int launch_ts_to_sts(const T *in, T *out, long long S, long long length, int L, cudaStream_t st) {
    const long long n = length * S;
    ts_rows_to_sts<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, S, length, L);
    return (int)cudaGetLastError();
}

constexpr long long kGridRows = 1ll << 30;  // rows of one launch

template <typename Kernel> inline int rank_smem_limit(Kernel kernel, size_t smem) {
    if (smem <= kSmemOptIn) return 0;
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// The block for rows of up to S stocks: go(items, max threads).  Batch rows
// are many, so they take few threads with many values each (throughput: the
// phases' fixed cost is a thread's); a stream's levels wait for one row, so
// they take 1024 threads before they take more values a thread (a level of one
// 4096-stock segment: 9 us, 22 us before).
template <bool LATENCY, typename Go> inline int rank_dispatch(long long S, Go go) {
    if (S > kRankMaxStocks) return (int)cudaErrorInvalidValue;
    using I4 = std::integral_constant<int, 4>;
    using I8 = std::integral_constant<int, 8>;
    using I16 = std::integral_constant<int, 16>;
    using T512 = std::integral_constant<int, 512>;
    using T1024 = std::integral_constant<int, 1024>;
    if constexpr (LATENCY) {
        if (S <= 4096) return go(I4(), T1024());
        if (S <= 8192) return go(I8(), T1024());
    } else {
        if (S <= 128) return go(I4(), T512());
        if (S <= 4096) return go(I8(), T512());
        if (S <= 8192) return go(I16(), T512());
    }
    return go(I16(), T1024());
}

template <typename T>
inline int launch_rank(const T *in, T *out, long long S, long long length, cudaStream_t st) {
    return rank_dispatch<false>(S, [&](auto items, auto maxt) {
        constexpr int I = decltype(items)::value, M = decltype(maxt)::value;
        const int nt = rank_threads((int)S, I);
        const size_t smem = rank_smem_bytes<T>(nt, I);
        if (int e = rank_smem_limit(rank_rows<T, I, M>, smem)) return e;
        for (long long t = 0; t < length; t += kGridRows)
            rank_rows<T, I, M>
                <<<(unsigned)std::min(length - t, kGridRows), nt, smem, st>>>(in + t * S, out + t * S, (int)S);
        return (int)cudaGetLastError();
    });
}

// Batch runs of several universes: the rows of one Rank stage of every job
// in one launch.  Job j ranks rows [row0, row0 + length) of the launch's
// row space, reading `in` and writing `out` ([length][S], TS).
struct RankRowsJob {
    const void *in;
    void *out;
    long long S, length, row0;
};

// A block has the threads of the longest row; a shorter row's surplus warps
// leave at once and its barriers count only the others.
template <typename T, int ITEMS, int MAXT>
__global__ void __launch_bounds__(MAXT, rank_min_blocks<T>(ITEMS, MAXT))
    rank_rows_multi(const RankRowsJob *__restrict__ jobs, int njobs, long long first_row) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long r = first_row + blockIdx.x;
    int lo = 0, hi = njobs - 1;  // the job whose rows hold r
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].row0 <= r) lo = mid;
        else hi = mid - 1;
    }
    const RankRowsJob jb = jobs[lo];
    const long long t = r - jb.row0, S = jb.S;
    if (t < 0 || t >= jb.length || S <= 0 || S > (long long)blockDim.x * ITEMS) return;
    const int nt = rank_threads((int)S, ITEMS);
    if ((int)threadIdx.x >= nt) return;
    rank_row<T, ITEMS>((const T *)jb.in + t * S, (int)S, nt, smem_raw, RankStore<T>{(T *)jb.out + t * S});
}

// max_S: the longest row of the jobs (sizes the blocks and their shared
// memory)
template <typename T>
inline int launch_rank_rows_multi(const RankRowsJob *d_jobs, int njobs, long long total_rows, long long max_S,
                                  cudaStream_t st) {
    if (njobs <= 0 || total_rows <= 0) return 0;
    return rank_dispatch<false>(max_S, [&](auto items, auto maxt) {
        constexpr int I = decltype(items)::value, M = decltype(maxt)::value;
        const int nt = rank_threads((int)max_S, I);
        const size_t smem = rank_smem_bytes<T>(nt, I);
        if (int e = rank_smem_limit(rank_rows_multi<T, I, M>, smem)) return e;
        for (long long r = 0; r < total_rows; r += kGridRows)
            rank_rows_multi<T, I, M>
                <<<(unsigned)std::min(total_rows - r, kGridRows), nt, smem, st>>>(d_jobs, njobs, r);
        return (int)cudaGetLastError();
    });
}

// rows whose addends exceed a block's shared memory are refused
template <typename T, typename Kernel> inline int scale_smem(Kernel kernel, long long S, size_t &smem) {
    if ((size_t)S * sizeof(T) > 200 * 1024) return (int)cudaErrorInvalidValue;
    smem = (size_t)scale_slots<T>(S) * sizeof(T);
    if (smem <= kSmemOptIn) return 0;
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <typename T>
inline int launch_scale(const T *in, T *out, long long S, long long length, cudaStream_t st) {
    size_t smem = 0;
    if (int e = scale_smem<T>(scale_rows<T>, S, smem)) return e;
    for (long long t = 0; t < length; t += kGridRows)
        scale_rows<T><<<(unsigned)std::min(length - t, kGridRows), S > 2048 ? 256 : 128, smem, st>>>(
            in + t * S, out + t * S, S);
    return (int)cudaGetLastError();
}

template <typename T>
inline int launch_diffwsum(const T *in0, const T *in1, T *out, long long S, long long length, cudaStream_t st) {
    long long grid = length < (long long)kun_num_sms() * 4 ? length : (long long)kun_num_sms() * 4;
    diffwsum_rows<T><<<(unsigned)grid, 256, 0, st>>>(in0, in1, out, S, length);
    return (int)cudaGetLastError();
}

template <typename T>
inline int launch_rank_segments(const T *in, int w_in, T *out, int w_out, long long cap, const int32_t *seg_off,
                                const int32_t *seg_stock0, const long long *seg_tick, int nseg, int max_len,
                                const int32_t *cnt, cudaStream_t st) {
    return rank_dispatch<true>(max_len, [&](auto items, auto maxt) {
        constexpr int I = decltype(items)::value, M = decltype(maxt)::value;
        const int nt = rank_threads(max_len, I);
        const size_t smem = rank_smem_bytes<T>(nt, I);
        if (int e = rank_smem_limit(rank_segments<T, I, M>, smem)) return e;
        rank_segments<T, I, M><<<(unsigned)nseg, nt, smem, st>>>(in, w_in, out, w_out, cap, seg_off, seg_stock0,
                                                                seg_tick, cnt);
        return (int)cudaGetLastError();
    });
}

// njobs Rank stages over (a part of) the step's segments in one launch (cnt:
// the step's device table, or null when the step has exactly nseg segments)
template <typename T>
inline int launch_rank_multi_segments(const RankJob *d_jobs, int njobs, long long cap, const int32_t *seg_off,
                                      const int32_t *seg_stock0, const long long *seg_tick, int nseg, int max_len,
                                      const int32_t *cnt, RankPart part, cudaStream_t st) {
    if (njobs <= 0 || nseg <= 0) return 0;
    if (njobs > 65535) return (int)cudaErrorInvalidValue;
    return rank_dispatch<true>(max_len, [&](auto items, auto maxt) {
        constexpr int I = decltype(items)::value, M = decltype(maxt)::value;
        const int nt = rank_threads(max_len, I);
        const size_t smem = rank_smem_bytes<T>(nt, I);
        if (int e = rank_smem_limit(rank_multi_segments<T, I, M>, smem)) return e;
        rank_multi_segments<T, I, M><<<dim3((unsigned)nseg, (unsigned)njobs), nt, smem, st>>>(
            d_jobs, cap, seg_off, seg_stock0, seg_tick, cnt, part);
        return (int)cudaGetLastError();
    });
}

template <typename T>
inline int launch_scale_segments(const T *in, int w_in, T *out, int w_out, long long cap, const int32_t *seg_off,
                                 const int32_t *seg_stock0, const long long *seg_tick, int nseg, int max_len,
                                 const int32_t *cnt, cudaStream_t st) {
    size_t smem = 0;
    if (int e = scale_smem<T>(scale_segments<T>, max_len, smem)) return e;
    scale_segments<T><<<(unsigned)nseg, 512, smem, st>>>(in, w_in, out, w_out, cap, seg_off, seg_stock0, seg_tick,
                                                         cnt, max_len);
    return (int)cudaGetLastError();
}

template <typename T>
inline int launch_diffwsum_segments(const T *in0, int w0, const T *in1, int w1, T *out, int w_out, long long cap,
                                    const int32_t *seg_off, const int32_t *seg_stock0, const long long *seg_tick,
                                    int nseg, int max_len, const int32_t *cnt, cudaStream_t st) {
    (void)max_len;
    diffwsum_segments<T><<<(unsigned)nseg, 256, 0, st>>>(in0, w0, in1, w1, out, w_out, cap, seg_off, seg_stock0,
                                                         seg_tick, cnt);
    return (int)cudaGetLastError();
}

}  // namespace kun
