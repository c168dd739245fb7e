// Utilities after the factor computation: corrWith / RankCorrWith (the
// cross-sectional correlation of every factor row with a label row, the IC)
// and aggregrate (per-stock group reductions over runs of equal labels).
// Reference: cpp/Kun/CorrWith.hpp:12-121, cpp/Kun/Aggregration.cpp:12-106,
// bound in Python at cpp/Python/PyBinding.cpp:396-506.
//
// corrWith: one block per (time row, input); the moments are summed per thread
// over a strided share of the stocks in two-float compensated fp32, then
// tree-reduced.  The label row's own moments do not depend on the input: one
// pass sums them for all.  The reference adds in stock order in plain fp32, so
// the results agree to rounding (its own tests hold 1e-4 relative to pandas).
// RankCorrWith ranks a row exactly as Rank does and sums the ranks from the
// registers they are found in.
//
// aggregrate: one thread per (stock, group, input) walks the group's rows in
// order, with the reference's reductions (Kahan sum, NaN-sticky min/max), so
// the outputs are the reference's bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "kun_runtime_internal.h"
#include "kun_xsec.cuh"

namespace kungpu {

constexpr int kCorrThreads = 256;
// (row, input) pairs up to which an unranked call is one launch, in which every
// input sums the label row again: launches cost more than that until the pairs
// are some blocks an SM (us, one launch and three: 1 input of 5000 x 20 54 and 71,
// 8 of 100 x 250 123 and 135, 8 of 5000 x 250 156 and 164, 32 of 5000 x 250 483
// and 437).  Calls of one or two inputs are at any length (3000 x 1250 71 and 86).
constexpr long long kCorrWhole = 2048;

// element (t, s) of a [T][S] (layout 1) or [S/L][T][L] (layout 0) buffer
__device__ __forceinline__ long long util_index(int layout, long long s, long long t, long long S, long long T,
                                                int L) {
    return layout == 1 ? t * S + s : (s / L) * T * L + t * L + s % L;
}

// Sums of a thread, normalised at every addition: values far from zero leave
// the correlation only what the sums hold beyond float (left unnormalised, their
// low parts' rounding made its error 1.8 to 2.8 times as large at 15000 stocks).
template <int N> struct CorrSums {
    kun::DFloat v[N];
    // every thread's sums over the block's first nt threads: a butterfly in each
    // warp, then one over the warps, or (IN_ORDER) the warps in order; thread 0
    // has the totals
    template <bool IN_ORDER> __device__ __forceinline__ void reduce(int nt) {
        __shared__ float sh[N][2][32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = nt >> 5;
        warp_totals();
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < N; q++) {
                sh[q][0][w] = v[q].hi;
                sh[q][1][w] = v[q].lo;
            }
        }
        __syncthreads();
        if (w != 0) return;
        if (IN_ORDER) {
            kun::DFloat total;  // lane q adds sum q
            for (int i = 0; i < nw && lane < N; i++) total = kun::kadd(total, kun::DFloat(sh[lane][0][i], sh[lane][1][i]));
#pragma unroll
            for (int q = 0; q < N; q++) v[q] = across(total, q);
        } else {
#pragma unroll
            for (int q = 0; q < N; q++) v[q] = lane < nw ? kun::DFloat(sh[q][0][lane], sh[q][1][lane]) : kun::DFloat();
            warp_totals();
        }
    }
    static __device__ __forceinline__ kun::DFloat across(kun::DFloat x, int from) {
        return kun::DFloat(__shfl_sync(0xffffffffu, x.hi, from), __shfl_sync(0xffffffffu, x.lo, from));
    }
    static __device__ __forceinline__ kun::DFloat pick(bool c, kun::DFloat x, kun::DFloat y) {
        return kun::DFloat(c ? x.hi : y.hi, c ? x.lo : y.lo);
    }
    // the warp's sums in every lane.  Of three, each lane goes on with the one
    // that its half and quarter keep: the butterfly's additions (which give the
    // same in either order) in 6 instead of 15.
    __device__ __forceinline__ void warp_totals() {
        const int lane = threadIdx.x & 31;
        if constexpr (N == 3) {
            const bool low = lane < 16, first = (lane & 8) == 0;
            const kun::DFloat a = across(pick(low, v[2], v[0]), lane ^ 16), b = across(v[1], lane ^ 16);
            const kun::DFloat x = kun::kadd(pick(low, v[0], v[2]), a), y = kun::kadd(v[1], b);
            const kun::DFloat send = pick(low && first, y, x), keep = pick(low && !first, y, x);
            kun::DFloat t = kun::kadd(keep, across(send, lane ^ 8));
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) t = kun::kadd(t, across(t, lane ^ o));
            v[0] = across(t, 0);
            v[1] = across(t, 8);
            v[2] = across(t, 16);
        } else {
#pragma unroll
            for (int q = 0; q < N; q++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v[q] = kun::kadd(v[q], across(v[q], lane ^ o));
        }
    }
};

// the label row's sum and sum of squares
__global__ void __launch_bounds__(kCorrThreads) corr_label_rows(const float *__restrict__ y, float4 *__restrict__ ysum,
                                                                long long S, long long T, int layout, int L) {
    const long long t = blockIdx.x;
    CorrSums<2> a;
    for (long long s = threadIdx.x; s < S; s += blockDim.x) {
        const float b = y[util_index(layout, s, t, S, T, L)];
        a.v[0] = kun::df_add_f(a.v[0], b);
        a.v[1] = kun::df_add_prod(a.v[1], b, b);
    }
    a.template reduce<true>(blockDim.x);
    if (threadIdx.x == 0) ysum[t] = make_float4(a.v[0].hi, a.v[0].lo, a.v[1].hi, a.v[1].lo);
}

// x, x*x and x*y sums of one (row, input)
struct CorrRow {
    float x[2], x2[2], xy[2];
};
template <int N> __device__ __forceinline__ void corr_add(CorrSums<N> &a, float x, float y) {
    a.v[0] = kun::df_add_f(a.v[0], x);
    a.v[1] = kun::df_add_prod(a.v[1], x, x);
    a.v[2] = kun::df_add_prod(a.v[2], x, y);
    if constexpr (N == 5) {  // and the label row's own
        a.v[3] = kun::df_add_f(a.v[3], y);
        a.v[4] = kun::df_add_prod(a.v[4], y, y);
    }
}
__device__ __forceinline__ CorrRow corr_row(const kun::DFloat *v) {
    return CorrRow{{v[0].hi, v[0].lo}, {v[1].hi, v[1].lo}, {v[2].hi, v[2].lo}};
}
// (XY - X*Y) / (sqrt(X2 - X*X) * sqrt(Y2 - Y*Y)) of the means, in double from
// the two-float sums (q: the label row's two)
__device__ __forceinline__ float corr_of(const CorrRow &r, float4 q, long long S) {
    const double n = (double)S;
    const double mx = ((double)r.x[0] + r.x[1]) / n, my = ((double)q.x + q.y) / n;
    const double mx2 = ((double)r.x2[0] + r.x2[1]) / n, my2 = ((double)q.z + q.w) / n;
    const double mxy = ((double)r.xy[0] + r.xy[1]) / n;
    return (float)((mxy - mx * my) / (sqrt(mx2 - mx * mx) * sqrt(my2 - my * my)));
}

// WHOLE: the label row's sums and the correlation too, in one launch
template <bool WHOLE>
__global__ void __launch_bounds__(kCorrThreads) corr_rows(const float *const *in, const float *__restrict__ y,
                                                          CorrRow *__restrict__ sums, float *const *out, long long S,
                                                          long long T, int layout, int L) {
    const long long t = blockIdx.x;
    const float *__restrict__ x = in[blockIdx.y];
    CorrSums<WHOLE ? 5 : 3> a;
    if (layout == 1) {
        const float *__restrict__ xr = x + t * S, *__restrict__ yr = y + t * S;
#pragma unroll 4
        for (long long s = threadIdx.x; s < S; s += kCorrThreads) corr_add(a, xr[s], yr[s]);
    } else {
        for (long long s = threadIdx.x; s < S; s += kCorrThreads) {
            const long long ix = util_index(layout, s, t, S, T, L);
            corr_add(a, x[ix], y[ix]);
        }
    }
    a.template reduce<true>(kCorrThreads);
    if (threadIdx.x != 0) return;
    if constexpr (WHOLE)
        out[blockIdx.y][t] = corr_of(corr_row(a.v), make_float4(a.v[3].hi, a.v[3].lo, a.v[4].hi, a.v[4].lo), S);
    else
        sums[(long long)blockIdx.y * T + t] = corr_row(a.v);
}

// the same with every input row's ranks in place of its values: they are
// summed where kun::rank_row finds them and never reach memory (5000 stocks x
// 1250 days x 32 inputs wrote and read 1.6 GB of them, in 33 launches: 5.4 ms,
// now 2.2 ms, bound by the ranking).  Ranks lie in (0, 1] and a thread has at
// most 16, so an addition takes the low parts together before it normalises:
// half the instructions, and with the butterfly over the warps an error no
// larger than that of the full additions of 256 threads (restated on the CPU, 100
// to 15000 stocks: 0.6 to 1.0 of it).  A sum that leaves the finite range, which
// only the label's values can bring about, ends as NaN either way.
struct CorrRankAdd {
    CorrSums<3> &a;
    const float *__restrict__ y;
    static __device__ __forceinline__ void add(kun::DFloat &s, float p, float e) {
        const kun::DFloat t = kun::df_two_sum(s.hi, p);
        s = kun::df_fast_two_sum(t.hi, __fadd_rn(__fadd_rn(s.lo, e), t.lo));
    }
    static __device__ __forceinline__ void add_prod(kun::DFloat &s, float x, float y) {
        const float p = __fmul_rn(x, y);
        add(s, p, __fmaf_rn(x, y, -p));
    }
    __device__ __forceinline__ void operator()(int i, float r) const {
        add(a.v[0], r, 0.f);
        add_prod(a.v[1], r, r);
        add_prod(a.v[2], r, y[i]);
    }
};
template <int ITEMS, int MAXT>
__global__ void __launch_bounds__(MAXT, kun::rank_min_blocks<float>(16, MAXT))
    corr_rank_rows(const float *const *in, const float *__restrict__ y, CorrRow *__restrict__ sums, int S, long long T) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long t = blockIdx.x;
    CorrSums<3> a;
    kun::rank_row<float, ITEMS>(in[blockIdx.y] + t * S, S, (int)blockDim.x, smem_raw, CorrRankAdd{a, y + t * S});
    a.template reduce<false>(blockDim.x);
    if (threadIdx.x == 0) sums[(long long)blockIdx.y * T + t] = corr_row(a.v);
}

// One thread a (row, input): a block's one thread doing it at the end of its row
// would hold the block for the double divisions.
__global__ void corr_finish(const CorrRow *__restrict__ sums, const float4 *__restrict__ ysum, float *const *out,
                            long long S, long long T) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < T) out[blockIdx.y][t] = corr_of(sums[(long long)blockIdx.y * T + t], ysum[t], S);
}

// First row of every run of equal consecutive labels (NaN equals nothing), in
// order: starts[g], and starts[groups] = length.  One block an input.
constexpr int kStartThreads = 1024;
template <typename T>
__global__ void __launch_bounds__(kStartThreads) group_starts(const void *const *labels,
                                                              long long *__restrict__ starts,
                                                              long long *__restrict__ groups, long long length) {
    const T *__restrict__ lab = (const T *)labels[blockIdx.x];
    long long *st = starts + blockIdx.x * (length + 1);
    __shared__ int warp_n[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    long long before = 0;
    for (long long r0 = 0; r0 < length; r0 += kStartThreads) {
        const long long r = r0 + tid;
        const bool head = r < length && (r == 0 || lab[r] != lab[r - 1]);
        const unsigned m = __ballot_sync(0xffffffffu, head);
        if (lane == 0) warp_n[warp] = __popc(m);
        __syncthreads();
        const int n = warp_n[lane];
        const long long at = before + __reduce_add_sync(0xffffffffu, lane < warp ? n : 0) + __popc(m & ((1u << lane) - 1));
        if (head) st[at] = r;
        before += __reduce_add_sync(0xffffffffu, n);
        __syncthreads();
    }
    if (tid == 0) {
        st[before] = length;
        groups[blockIdx.x] = before;
    }
}

// One thread a stock takes the groups that begin in the block's tile of rows,
// each from its first row to its last (which may lie in later blocks' rows),
// kAggAhead rows loaded ahead of the sums.  Groups do not depend on each
// other: one thread a stock walking all rows (40 blocks at 5000 stocks) waited
// for one load at a time, 1.1 ms an input of 2500 rows; now bound by memory, 6
// inputs in about 0.1 ms with monthly groups.  32 rows a tile, or 8 where those
// leave SMs without blocks: a thread's groups of one row wait for each other (60
// rows of 5000 stocks 49 us in tiles of 32, 40 in tiles of 8).
// OWN: of up to kAggThreads rows every block finds the groups itself, for the
// launch of group_starts is a tenth of so short a call (60 rows of 5000 stocks in
// groups of 21: 39 us with it, 34 without).
constexpr int kAggAhead = 8;
constexpr int kAggThreads = 128;
template <typename T, bool OWN>
__global__ void __launch_bounds__(kAggThreads) aggregate_groups(const void *const *in_, const void *const *labels,
                                                                T *const *outs_, const long long *starts_,
                                                                const long long *groups_, long long S,
                                                                long long length, int tile_rows) {
    __shared__ long long own[OWN ? kAggThreads + 1 : 1];
    __shared__ unsigned heads[kAggThreads / 32];
    long long groups;
    if (OWN) {
        const T *__restrict__ lab = (const T *)labels[blockIdx.z];
        const int r = threadIdx.x, lane = r & 31, w = r >> 5;
        const bool head = r < length && (r == 0 || lab[r] != lab[r - 1]);
        const unsigned m = __ballot_sync(0xffffffffu, head);
        if (lane == 0) heads[w] = m;
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int k = 0; k < kAggThreads / 32; k++) {
            const int n = __popc(heads[k]);
            before += k < w ? n : 0;
            all += n;
        }
        if (head) own[before + __popc(m & ((1u << lane) - 1))] = r;
        if (r == 0) own[all] = length;
        groups = all;
        __syncthreads();
    } else {
        groups = groups_[blockIdx.z];
    }
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const T *__restrict__ in = (const T *)in_[blockIdx.z] + s;
    T *const *outs = outs_ + 7 * blockIdx.z;
    const long long *starts = OWN ? own : starts_ + blockIdx.z * (length + 1);
    T *sum = outs[0], *mn = outs[1], *mx = outs[2], *first = outs[3], *last = outs[4], *cnt = outs[5],
      *mean = outs[6];
    for (long long tile = blockIdx.y; tile * tile_rows < length; tile += gridDim.y) {
        const long long r0 = tile * tile_rows, r1 = r0 + tile_rows < length ? r0 + tile_rows : length;
        long long g = 0, hi = groups;  // the first group that begins at r0 or later
        while (g < hi) {
            const long long m = (g + hi) >> 1;
            if (starts[m] < r0) g = m + 1;
            else hi = m;
        }
        for (; g < groups; g++) {
            const long long b = starts[g], e = starts[g + 1];
            if (b >= r1) break;
            kun::RAdd<T> radd;
            kun::RMin<T> rmin;
            kun::RMax<T> rmax;
            const T *p = in + b * S;
            const T f = *p;
            T l = f, c = T(0);
            for (long long left = e - b; left > 0; left -= kAggAhead, p += kAggAhead * S) {
                T x[kAggAhead];
#pragma unroll
                for (int u = 0; u < kAggAhead; u++) x[u] = u < left ? p[u * S] : T(0);
#pragma unroll
                for (int u = 0; u < kAggAhead; u++) {
                    if (u < left) {
                        c = kun::kadd(c, T(1));
                        l = x[u];
                        rmax.step(x[u]);
                        rmin.step(x[u]);
                        radd.step(x[u]);
                    }
                }
            }
            const long long o = g * S + s;
            if (sum) sum[o] = radd.value();
            if (mn) mn[o] = rmin.value();
            if (mx) mx[o] = rmax.value();
            if (first) first[o] = f;
            if (last) last[o] = l;
            if (cnt) cnt[o] = c;
            if (mean) mean[o] = kun::kdiv(radd.value(), c);
        }
    }
}

static KunStatus util_sync(Executor *ex, cudaStream_t st) {
    if (ex->has_user_stream) {
        cudaEventRecord(ex->bridge_out, st);
        cudaStreamWaitEvent(ex->user_stream, ex->bridge_out, 0);
    }
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        set_error("CUDA error: %s", cudaGetErrorString(e));
        return KUN_CUDA_ERROR;
    }
    return KUN_SUCCESS;
}

}  // namespace kungpu

using namespace kungpu;

// corrWith / RankCorrWith (GPU extension of the C API; the reference has it
// in C++ and Python).  inputs[n], corr_with and the n outputs (num_time
// floats each) are device memory; layout 1 = TS [T][S], 0 = STs [S/8][T][8].
KUN_EXPORT KunStatus kunCorrWith(KunExecutorHandle exec, int n, const float *const *inputs, const float *corr_with,
                                 float *const *outs, size_t num_stocks, size_t num_time, int layout,
                                 int rank_inputs) {
    clear_error();
    auto *ex = (Executor *)exec;
    if (!ex || n < 0 || (n > 0 && (!inputs || !outs)) || !corr_with) {
        set_error("corrWith: bad arguments");
        return KUN_INVALID_ARGUMENT;
    }
    if (n == 0) return KUN_SUCCESS;
    if (layout != 0 && layout != 1) {
        set_error("Unknown layout");
        return KUN_INVALID_ARGUMENT;
    }
    if (rank_inputs && layout != 1) {
        set_error("corrWith: rank_inputs needs the TS layout");
        return KUN_INVALID_ARGUMENT;
    }
    if (num_stocks == 0 || num_time == 0 || num_time > 0x7fffffff || n > 65535) {
        set_error("corrWith: bad shape");
        return KUN_INVALID_ARGUMENT;
    }
    std::lock_guard<std::mutex> lk(ex->mu);
    cudaSetDevice(ex->device);
    cudaStream_t st = ex->stream();
    if (ex->has_user_stream) {
        cudaEventRecord(ex->bridge_in, ex->user_stream);
        cudaStreamWaitEvent(st, ex->bridge_in, 0);
    }
    if (rank_inputs && num_stocks > (size_t)kun::kRankMaxStocks) {
        set_error("corrWith: rank failed: %s", cudaGetErrorString(cudaErrorInvalidValue));
        return KUN_CUDA_ERROR;
    }
    // device copies of the pointer arrays and the rows' sums in the arena
    auto up = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t ptrs = up((size_t)n * sizeof(void *)), ysums = up(num_time * sizeof(float4));
    if (!ex->arena.ensure(2 * ptrs + ysums + (size_t)n * num_time * sizeof(CorrRow))) {
        set_error("out of device memory for corrWith");
        return KUN_OUT_OF_MEMORY;
    }
    char *base = (char *)ex->arena.ptr;
    const float **d_in = (const float **)base;
    float **d_out = (float **)(base + ptrs);
    float4 *d_ysum = (float4 *)(base + 2 * ptrs);
    CorrRow *d_sums = (CorrRow *)(base + 2 * ptrs + ysums);
    const long long S = (long long)num_stocks, T = (long long)num_time;
    cudaMemcpyAsync(d_in, inputs, (size_t)n * sizeof(void *), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_out, outs, (size_t)n * sizeof(void *), cudaMemcpyHostToDevice, st);
    const bool whole = !rank_inputs && (n <= 2 || n * T <= kCorrWhole);
    if (!whole) corr_label_rows<<<(unsigned)T, kCorrThreads, 0, st>>>(corr_with, d_ysum, S, T, layout, 8);
    const dim3 grid((unsigned)T, (unsigned)n);
    if (rank_inputs) {
        const int rc = kun::rank_dispatch<false>(S, [&](auto items, auto maxt) {
            constexpr int I = decltype(items)::value, M = decltype(maxt)::value;
            const int nt = kun::rank_threads((int)S, I);
            const size_t smem = kun::rank_smem_bytes<float>(nt, I);
            if (int e = kun::rank_smem_limit(corr_rank_rows<I, M>, smem)) return e;
            corr_rank_rows<I, M><<<grid, nt, smem, st>>>(d_in, corr_with, d_sums, (int)S, T);
            return (int)cudaGetLastError();
        });
        if (rc) {
            set_error("corrWith: rank failed: %s", cudaGetErrorString((cudaError_t)rc));
            return KUN_CUDA_ERROR;
        }
    } else if (whole) {
        corr_rows<true><<<grid, kCorrThreads, 0, st>>>(d_in, corr_with, nullptr, d_out, S, T, layout, 8);
    } else {
        corr_rows<false><<<grid, kCorrThreads, 0, st>>>(d_in, corr_with, d_sums, nullptr, S, T, layout, 8);
    }
    if (!whole) corr_finish<<<dim3((unsigned)((T + 127) / 128), (unsigned)n), 128, 0, st>>>(d_sums, d_ysum, d_out, S, T);
    if (cudaError_t e = cudaGetLastError()) {
        set_error("corrWith: %s", cudaGetErrorString(e));
        return KUN_CUDA_ERROR;
    }
    return util_sync(ex, st);
}

// aggregrate (GPU extension; PyBinding.cpp:449-506): for each of n inputs
// ([length][S], TS), labels[k] (length values) and outs[k*7 + kind] (kind =
// sum, min, max, first, last, count, mean; NULL to skip; [groups][S]).
// dtype 0 = float, 1 = double.  All pointers are device memory.
KUN_EXPORT KunStatus kunAggregrate(KunExecutorHandle exec, int n, const void *const *inputs,
                                   const void *const *labels, void *const *outs, size_t num_stocks, size_t length,
                                   int dtype) {
    clear_error();
    auto *ex = (Executor *)exec;
    if (!ex || n < 0 || (n > 0 && (!inputs || !labels || !outs)) || (dtype != 0 && dtype != 1)) {
        set_error("aggregrate: bad arguments");
        return KUN_INVALID_ARGUMENT;
    }
    if (n == 0) return KUN_SUCCESS;
    if (num_stocks == 0 || length == 0) {
        set_error("aggregrate: bad shape");
        return KUN_INVALID_ARGUMENT;
    }
    std::lock_guard<std::mutex> lk(ex->mu);
    cudaSetDevice(ex->device);
    cudaStream_t st = ex->stream();
    if (ex->has_user_stream) {
        cudaEventRecord(ex->bridge_in, ex->user_stream);
        cudaStreamWaitEvent(st, ex->bridge_in, 0);
    }
    auto up = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    const size_t ptrs = up((size_t)n * 9 * sizeof(void *)), counts = up((size_t)n * sizeof(long long));
    if (!ex->arena.ensure(ptrs + counts + (size_t)n * (length + 1) * sizeof(long long))) {
        set_error("out of device memory for aggregrate");
        return KUN_OUT_OF_MEMORY;
    }
    char *base = (char *)ex->arena.ptr;
    void **d_ptrs = (void **)base;  // inputs, labels, outputs
    long long *d_groups = (long long *)(base + ptrs), *d_starts = (long long *)(base + ptrs + counts);
    std::vector<const void *> table(inputs, inputs + n);
    table.insert(table.end(), labels, labels + n);
    table.insert(table.end(), outs, outs + 7 * (size_t)n);
    cudaMemcpyAsync(d_ptrs, table.data(), table.size() * sizeof(void *), cudaMemcpyHostToDevice, st);
    auto go = [&](auto zero) {
        using T = decltype(zero);
        const long long S = (long long)num_stocks, rows = (long long)length;
        const long long stock_blocks = (S + kAggThreads - 1) / kAggThreads;
        const int tile_rows = stock_blocks * ((rows + 31) / 32) * n < 4LL * kun::kun_num_sms() ? 8 : 32;
        const long long tiles = (rows + tile_rows - 1) / tile_rows;
        const bool own = rows <= kAggThreads;
        if (!own) group_starts<T><<<(unsigned)n, kStartThreads, 0, st>>>(d_ptrs + n, d_starts, d_groups, rows);
        for (int k = 0; k < n; k += 65535) {
            const dim3 grid((unsigned)stock_blocks, (unsigned)std::min(tiles, 65535LL),
                            (unsigned)std::min(n - k, 65535));
            T *const *to = (T *const *)(d_ptrs + 2 * (size_t)n) + 7 * (size_t)k;
            if (own)
                aggregate_groups<T, true><<<grid, kAggThreads, 0, st>>>(d_ptrs + k, d_ptrs + n + k, to, nullptr, nullptr,
                                                                        S, rows, tile_rows);
            else
                aggregate_groups<T, false><<<grid, kAggThreads, 0, st>>>(
                    d_ptrs + k, nullptr, to, d_starts + k * (rows + 1), d_groups + k, S, rows, tile_rows);
        }
    };
    if (dtype == 0)
        go(0.f);
    else
        go(0.0);
    if (cudaError_t e = cudaGetLastError()) {
        set_error("aggregrate: %s", cudaGetErrorString(e));
        return KUN_CUDA_ERROR;
    }
    return util_sync(ex, st);
}
