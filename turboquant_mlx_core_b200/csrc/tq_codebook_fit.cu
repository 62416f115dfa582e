// Lloyd-Max codebook fit on the device (generate_codebook_from_data, src/codebook.cpp:99-143 and
// 158-267) and the sample extraction of the converter's per-layer fit (src/converter.cpp:291-368).
//
// An iteration needs, for every boundary, the count and the sum of the values at or below it.  Going over all samples for
// that took 110 us per iteration at 16.8 M samples, a hundred times.  Instead the samples are bucketed ONCE by the leading
// bits of their order-preserving key (sign, exponent, a few mantissa bits), with running counts and a sum per bucket; a
// boundary then only looks at the values of its own bucket, and all iterations run in one launch of one CTA, a warp per
// boundary and bin (3 to 6 us each).
//   fit_look_kernel       whether the samples repeat themselves (then as below)
//   fit_count_window_kernel    bucket counts, largest magnitude       (one pass over the samples; fit_count_kernel for few of them)
//   fit_groups / fit_offsets   exclusive scan of the counts, 256 buckets per group
//   fit_scatter_window_kernel  samples into their buckets             (one pass; fit_scatter_kernel)
//   fit_sums_kernel       sum of every bucket
//   fit_iterate_kernel    the iterations
// A value equal to a boundary goes to the lower bin, as std::lower_bound in the reference's CPU path and quantize() have
// it.  All values of a bucket have one sign and exponent, so a bucket's sum, and the sum of its values up to a boundary, is an
// exact 64-bit integer of significands.  A bin is the double sum of the buckets between its boundaries and those two partial
// ones, in a fixed order: only its own values enter, as in the reference's double sums, whatever the magnitudes of the
// others (running sums over all buckets would lose a bin beside an outlier), and results are run-to-run identical.
// Samples that repeat themselves skip all that, and a boundary whose bucket holds more than kFitMaxBucket values, or samples
// that are not finite, stop fit_iterate_kernel; the remaining iterations then go over all samples:
//   fit_partial_kernel   every thread bins its values by lower_bound over the current boundaries into a PRIVATE histogram in
//                        shared memory ([bin][thread]: no atomics, no bank conflicts), sums in double; the block then folds
//                        its 256 histograms in a fixed order and writes one (sum, count) pair per bin;
//   fit_update_kernel    one warp folds the blocks' pairs in block order, moves each non-empty bin's centroid to its mean,
//                        recomputes the midpoints and raises a "converged" flag when no centroid moved by 1e-6 or more
//                        (src/codebook.cpp:68, 128-131).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <functional>

#include "tq_common.cuh"
#include "tq_host.hpp"
#include "tq_kernels.cuh"

namespace tq {

namespace {

constexpr int kFitThreads = 256;
constexpr int kFitMaxBins = 32;
constexpr float kFitShiftThreshold = 1e-6f;   // src/codebook.cpp:68

struct FitState {
    float centroids[kFitMaxBins];
    float boundaries[kFitMaxBins];   // n - 1 used
    int n;
    int converged;
    int iterations_run;
    int go_over_all;                 // fit_iterate_kernel stopped: the remaining iterations go over all samples
    unsigned int max_bits;           // bits of the largest magnitude
    int window_low;                  // lowest exponent of the window (fit_count_window_kernel)
};

constexpr int kFitGroup = 256;              // buckets of a group
constexpr int kFitSumBuckets = 32;          // buckets whose sums a block takes
constexpr int kFitBatch = 8;                // values of a bucket that a lane requests at once
constexpr int kFitLongBatch = 16;           // ... of a long one, in the iterations
constexpr unsigned int kFitMaxBucket = 32768;   // values of a bucket that the iterations look through
constexpr int kFitLooked = 4096, kFitSlots = 8192;   // samples that fit_look_kernel looks at, its counters
constexpr unsigned int kFitCrowd = 2 * kFitMaxBucket;

// Order-preserving key of a float: smaller values have smaller keys (-0 and +0 differ by one, which no sum notices).
__device__ __forceinline__ unsigned int fit_key(float x) {
    const unsigned int u = __float_as_uint(x);
    return u ^ ((u & 0x80000000u) ? 0xffffffffu : 0x80000000u);
}
// The values of a bucket agree in all bits above `shift` (the sign, the exponent, 3 of the mantissa at least), so a value is
// (base + its bits below `shift`) units; the unit carries the sign.
struct FitBucket {
    unsigned int base;
    double unit;
};
__device__ __forceinline__ FitBucket fit_bucket(int bucket, int shift) {
    const unsigned int key = static_cast<unsigned int>(bucket) << shift;
    const unsigned int u = (key & 0x80000000u) ? key ^ 0x80000000u : ~(key | ((1u << shift) - 1u));
    const unsigned int e = (u >> 23) & 0xffu;
    const double unit = __longlong_as_double(static_cast<long long>(max(e, 1u) - 150u + 1023u) << 52);
    return FitBucket{(u & 0x7fffffu) | (e != 0u ? 0x800000u : 0u), (u & 0x80000000u) ? -unit : unit};
}

// Samples that repeat themselves: the atomic additions of a bucket's samples follow one another (3 ns each: 16.8 M equal
// samples took 55 ms, half of them zero 39 ms, where the passes over all samples take 1 and 11), and the iterations stop
// at such a bucket anyway.  One CTA looks at kFitLooked samples, evenly spread: where one bucket must hold more than
// kFitCrowd, the kernels after it return at once.  (kFitSlots counters: two buckets that share one need twice the luck.)
// It also chooses the window of the two kernels behind it: `window` exponents down from the largest one of which it sees two samples.
__global__ void __launch_bounds__(1024) fit_look_kernel(const float* __restrict__ data, unsigned int n, int shift, int window, FitState* __restrict__ state) {
    __shared__ unsigned int s_count[kFitSlots], s_exp[256];
    for (int i = threadIdx.x; i < kFitSlots; i += 1024) s_count[i] = 0u;
    if (threadIdx.x < 256) s_exp[threadIdx.x] = 0u;
    __syncthreads();
    unsigned int most = 0;
    const unsigned int step = n / kFitLooked;
#pragma unroll
    for (int k = 0; k < kFitLooked / 1024; ++k) {
        const float x = __ldg(data + static_cast<size_t>(k * 1024 + threadIdx.x) * step);
        const unsigned int bucket = fit_key(x) >> shift;
        atomicAdd(&s_exp[(__float_as_uint(x) >> 23) & 0xffu], 1u);
        most = max(most, atomicAdd(&s_count[bucket % kFitSlots], 1u) + 1u);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && most >= 16u && static_cast<unsigned long long>(most) * step > kFitCrowd) state->go_over_all = 1;
    __syncthreads();
    if (threadIdx.x < 32) {
        int top = -1;
        for (int e = threadIdx.x; e < 256; e += 32)
            if (s_exp[e] >= 2u) top = e;
        top = __reduce_max_sync(0xffffffffu, top);
        if (threadIdx.x == 0) state->window_low = max(0, min(top, 254) - window + 1);
    }
}

// Counting and scattering with most of the counters on the SM.  An atomic addition in L2 for every sample took 250 to 420 us per
// pass over 16.8 M of them (the scatter waits for its answer), of which reading them is 10.  A CTA per SM keeps counters for
// the buckets of a window, 2^(shift - 23) .. of `window` exponents and both signs (all but 0.1 % of normal samples), and
// adds a bucket's count up in L2 once; what that addition returns is where the CTA's samples of the bucket begin, so
// the scatter, which deals the samples to CTAs in the same way, needs no other word from the CTAs around it.  Samples outside of
// the window are counted in L2.
constexpr int kWindowSlots = 49152;           // counters of a CTA: 192 KB
constexpr int kWindowExponents = 32;          // no more exponents than that: below 2^-31 of the largest there is next to nothing
constexpr unsigned int kWindowTile = 8192;    // samples that a CTA takes at a time
// Used wherever the samples are looked at first (from kFitCrowd on): 262144 / 1 M / 4.2 M / 16.8 M normal samples are counted in
// 5 / 8 / 14 / 40 us (37 / 104 / 135 / 186 in L2) and scattered in 9 / 13 / 30 / 142 (39 / 113 / 143 / 299).
struct FitWindow {
    unsigned int low, slots;   // magnitudes (shifted) from `low` on, `slots` of them, of either sign
    int shift;
    __device__ __forceinline__ FitWindow(const FitState* state, int shift_, int window)
        : low(static_cast<unsigned int>(state->window_low) << (23 - shift_)), slots(static_cast<unsigned int>(window) << (23 - shift_)), shift(shift_) {}
    // The slot of a sample, or 0xffffffff.
    __device__ __forceinline__ unsigned int slot(float x) const {
        const unsigned int u = __float_as_uint(x), m = ((u & 0x7fffffffu) >> shift) - low;
        return m < slots ? m + ((u >> 31) ? slots : 0u) : 0xffffffffu;
    }
    __device__ __forceinline__ unsigned int bucket(unsigned int slot) const {
        const bool negative = slot >= slots;
        const unsigned int m = (negative ? slot - slots : slot) + low + (0x80000000u >> shift);
        return negative ? (0xffffffffu >> shift) - m : m;
    }
};
__global__ void __launch_bounds__(1024) fit_count_window_kernel(const float* __restrict__ data, unsigned int n, int shift, int window,
                                                                unsigned int* __restrict__ count, unsigned int* __restrict__ begin, FitState* __restrict__ state) {
    if (state->go_over_all) return;
    extern __shared__ unsigned int s_counter[];
    const FitWindow w(state, shift, window);
    for (unsigned int i = threadIdx.x; i < 2 * w.slots; i += 1024) s_counter[i] = 0u;
    __syncthreads();
    unsigned int top = 0;
    for (unsigned long long i0 = static_cast<unsigned long long>(blockIdx.x) * kWindowTile; i0 < n; i0 += static_cast<unsigned long long>(gridDim.x) * kWindowTile) {
        float x[kWindowTile / 1024];
        const unsigned int i = static_cast<unsigned int>(i0) + threadIdx.x;
#pragma unroll
        for (int k = 0; k < static_cast<int>(kWindowTile / 1024); ++k)
            if (i + 1024u * k < n) x[k] = __ldcs(data + i + 1024u * k);
#pragma unroll
        for (int k = 0; k < static_cast<int>(kWindowTile / 1024); ++k)
            if (i + 1024u * k < n) {
                top = max(top, __float_as_uint(x[k]) & 0x7fffffffu);
                const unsigned int slot = w.slot(x[k]);
                if (slot != 0xffffffffu) atomicAdd(&s_counter[slot], 1u);
                else atomicAdd(&count[fit_key(x[k]) >> shift], 1u);
            }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&state->max_bits, top);
    __syncthreads();
    unsigned int* const mine = begin + static_cast<size_t>(blockIdx.x) * 2 * w.slots;
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < 2 * w.slots; i += 1024) {
        const unsigned int c = s_counter[i];
        if (c != 0u) mine[i] = atomicAdd(&count[w.bucket(i)], c);
    }
}
__global__ void __launch_bounds__(1024) fit_scatter_window_kernel(const float* __restrict__ data, unsigned int n, int shift, int window,
                                                                  const unsigned int* __restrict__ offset, const unsigned int* __restrict__ begin,
                                                                  unsigned int* __restrict__ cursor, float* __restrict__ sorted,
                                                                  const FitState* __restrict__ state) {
    if (state->go_over_all) return;
    extern __shared__ unsigned int s_counter[];
    const FitWindow w(state, shift, window);
    const unsigned int* const mine = begin + static_cast<size_t>(blockIdx.x) * 2 * w.slots;   // (not set where the CTA has no sample)
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < 2 * w.slots; i += 1024) s_counter[i] = mine[i] + offset[w.bucket(i)];
    __syncthreads();
    for (unsigned long long i0 = static_cast<unsigned long long>(blockIdx.x) * kWindowTile; i0 < n; i0 += static_cast<unsigned long long>(gridDim.x) * kWindowTile) {
        float x[kWindowTile / 1024];
        const unsigned int i = static_cast<unsigned int>(i0) + threadIdx.x;
#pragma unroll
        for (int k = 0; k < static_cast<int>(kWindowTile / 1024); ++k)
            if (i + 1024u * k < n) x[k] = __ldcs(data + i + 1024u * k);
#pragma unroll
        for (int k = 0; k < static_cast<int>(kWindowTile / 1024); ++k)
            if (i + 1024u * k < n) {
                const unsigned int slot = w.slot(x[k]);
                sorted[atomicAdd(slot != 0xffffffffu ? &s_counter[slot] : &cursor[fit_key(x[k]) >> shift], 1u)] = x[k];
            }
    }
}

__global__ void __launch_bounds__(256) fit_count_kernel(const float* __restrict__ data, unsigned int n, int shift, unsigned int* __restrict__ count,
                                                        FitState* __restrict__ state) {
    if (state->go_over_all) return;
    unsigned int top = 0;
    for (unsigned int i = blockIdx.x * 1024u + threadIdx.x; i < n; i += gridDim.x * 1024u) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned int at = i + 256u * k;
            if (at < n && at >= i) {
                const float x = __ldg(data + at);
                top = max(top, __float_as_uint(x) & 0x7fffffffu);
                atomicAdd(&count[fit_key(x) >> shift], 1u);
            }
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&state->max_bits, top);
}

// Inclusive scan over the 256 threads of a block.
__device__ __forceinline__ unsigned int block_scan256(unsigned int v, unsigned int* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; ++w) v += s_warp[w];
    __syncthreads();
    return v;
}
__global__ void __launch_bounds__(256) fit_groups_kernel(const unsigned int* __restrict__ count, unsigned int* __restrict__ group) {
    __shared__ unsigned int s_warp[8];
    const unsigned int v = block_scan256(count[blockIdx.x * kFitGroup + threadIdx.x], s_warp);
    if (threadIdx.x == 255) group[blockIdx.x] = v;
}
// Exclusive offsets of the buckets of a group; the groups before it are added up here (a few thousand at most).
__global__ void __launch_bounds__(256) fit_offsets_kernel(const unsigned int* __restrict__ count, const unsigned int* __restrict__ group,
                                                          unsigned int* __restrict__ offset, unsigned int* __restrict__ cursor) {
    __shared__ unsigned int s_warp[8];
    unsigned int before = 0;
    for (unsigned int g = threadIdx.x; g < blockIdx.x; g += 256) before += group[g];
    before = block_scan256(before, s_warp);
    __shared__ unsigned int s_before;
    if (threadIdx.x == 255) s_before = before;
    __syncthreads();
    const int b = blockIdx.x * kFitGroup + threadIdx.x;
    const unsigned int c = count[b], at = s_before + block_scan256(c, s_warp) - c;
    offset[b] = at;
    cursor[b] = at;
}
__global__ void __launch_bounds__(256) fit_scatter_kernel(const float* __restrict__ data, unsigned int n, int shift, unsigned int* __restrict__ cursor,
                                                          float* __restrict__ sorted, const FitState* __restrict__ state) {
    if (state->go_over_all) return;
    for (unsigned int i = blockIdx.x * 1024u + threadIdx.x; i < n; i += gridDim.x * 1024u) {
        float x[4];
        unsigned int pos[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned int at = i + 256u * k;
            const bool in = at < n && at >= i;
            x[k] = in ? __ldg(data + at) : 0.f;
            pos[k] = in ? atomicAdd(&cursor[fit_key(x[k]) >> shift], 1u) : 0xffffffffu;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (pos[k] != 0xffffffffu) sorted[pos[k]] = x[k];
    }
}
// Bucket sums, and the double sum of every kFitSumBuckets of them.  A block looks at up to eight ranges of so many buckets, far apart (the
// samples lie in about a hundred groups of 256 buckets; with a block per group those few blocks took 450 us for 16.8 M samples):
// a warp each, which writes the zeros of a range without samples, most of them, and then all warps take the others, a bucket each.
// Bound by the latency of the buckets' loads: 16.8 M normal samples 39 us; with a block per range, 32 768 of which nine tenths
// write zeros, 67.
constexpr int kFitSumRanges = 8;
static_assert(kFitSumBuckets == 32, "a lane per bucket of a range");
__global__ void __launch_bounds__(256) fit_sums_kernel(const float* __restrict__ sorted, const unsigned int* __restrict__ count,
                                                       const unsigned int* __restrict__ offset, int shift, double* __restrict__ sum,
                                                       double* __restrict__ part, const FitState* __restrict__ state, int ranges) {
    __shared__ double s_warp[8];
    __shared__ int s_some[kFitSumRanges];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int below = (1u << shift) - 1u;
    if (warp < ranges) {
        const int mine = (blockIdx.x + warp * gridDim.x) * kFitSumBuckets + lane;
        const unsigned int c_mine = count[mine];
        if (state->go_over_all) return;
        const bool some = __any_sync(0xffffffffu, c_mine != 0u);
        if (!some) {
            sum[mine] = 0.0;
            if (lane == 0) part[mine / kFitSumBuckets] = 0.0;
        }
        if (lane == 0) s_some[warp] = some ? 1 : 0;
    } else if (state->go_over_all) {
        return;
    }
    __syncthreads();
    for (int r = 0; r < ranges; ++r) {
        if (s_some[r] == 0) continue;
        const int range = blockIdx.x + r * gridDim.x;
        const unsigned int c_lane = count[range * kFitSumBuckets + lane], at_lane = offset[range * kFitSumBuckets + lane];
        double total = 0.0;
        for (int k = warp; k < kFitSumBuckets; k += 8) {
            const int b = range * kFitSumBuckets + k;
            const unsigned int c = __shfl_sync(0xffffffffu, c_lane, k), at = __shfl_sync(0xffffffffu, at_lane, k);
            long long s = 0;
            for (unsigned int i = lane; i < c; i += 32 * kFitBatch) {
                float x[kFitBatch];
#pragma unroll
                for (int j = 0; j < kFitBatch; ++j) x[j] = i + 32u * j < c ? sorted[at + i + 32u * j] : 0.f;
                unsigned int t = 0;   // 8 x 2^20 at most
#pragma unroll
                for (int j = 0; j < kFitBatch; ++j) t += __float_as_uint(x[j]) & below;
                s += t;
            }
            double v = 0.0;
            if (c != 0) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                const FitBucket f = fit_bucket(b, shift);
                v = static_cast<double>(s + static_cast<long long>(c) * f.base) * f.unit;
                total += v;
            }
            if (lane == 0) sum[b] = v;
        }
        if (lane == 0) s_warp[warp] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) total += s_warp[w];
            part[range] = total;
        }
        __syncthreads();
    }
}
// All iterations of a fit in one CTA, a CTA per fit: warp w follows boundary w, the upper one of bin w.  Bound by the latency of a
// chain of L2 reads, reductions and barriers: a bucket's place, its values, the sums around it and between the boundaries are a few
// hundred to 2000 cycles each.  Long buckets are read 16 values a lane at a time (eight: six such reads one after the other for 1500
// values; 24 slow those down whose boundaries lie in small buckets), the rest and small buckets eight, which issues less.  100 iterations of a
// layer's two fits over 16.8 M samples each, side by side, 497 us (eight at a time throughout 555; 24 470); samples over 60 decades, whose boundaries lie in
// small buckets, cost 2 % more for it, 4 M of them 453 -> 463 us a fit.  (Significands as 64-bit sums of doubles' conversions took 400 to 660 us;
// the bits below a bucket's prefix are 32-bit sums.  Two warps per boundary that keep their bucket's samples in registers: no change.)
// `group_sum`: filled here from the parts.
struct FitJob {
    const float* sorted;
    const unsigned int *count, *offset;
    const double *sum, *part;
    double* group_sum;
    FitState* state;
    unsigned int n;
    int n_groups, shift, iterations;
};
constexpr int kFitJobs = 2;
struct FitJobs {
    FitJob job[kFitJobs];
};
__global__ void __launch_bounds__(1024) fit_iterate_kernel(const __grid_constant__ FitJobs jobs) {
    const FitJob& f = jobs.job[blockIdx.x];
    const float* __restrict__ sorted = f.sorted;
    const unsigned int *__restrict__ count = f.count, *__restrict__ offset = f.offset;
    const double *__restrict__ sum = f.sum, *__restrict__ part = f.part;
    double* __restrict__ group_sum = f.group_sum;
    FitState* __restrict__ state = f.state;
    const unsigned int n = f.n;
    const int n_groups = f.n_groups, shift = f.shift, iterations = f.iterations;
    __shared__ float s_c[kFitMaxBins], s_b[kFitMaxBins];
    // Per boundary: its bucket, that bucket's unit and sum, the sums of its group's buckets before and after it; the samples up
    // to the boundary, those before the bucket included, and the significands of the ones in the bucket.
    __shared__ int s_bucket[kFitMaxBins];
    __shared__ double s_unit[kFitMaxBins], s_own[kFitMaxBins], s_before[kFitMaxBins], s_after[kFitMaxBins];
    __shared__ unsigned int s_le[kFitMaxBins];
    __shared__ long long s_low[kFitMaxBins];
    __shared__ double s_mid[kFitMaxBins];      // per bin: the groups between its boundaries' (or the buckets, where they share one)
    __shared__ int s_stop, s_converged, s_moved, s_near;
    if (state->go_over_all) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nc = state->n;
    if (tid < nc) s_c[tid] = state->centroids[tid];
    if (tid < nc - 1) s_b[tid] = state->boundaries[tid];
    const bool finite = state->max_bits < 0x7f800000u;
    if (tid == 0) {
        s_stop = finite ? 0 : 1;
        s_converged = s_moved = s_near = 0;
    }
    constexpr int kParts = kFitGroup / kFitSumBuckets;
    for (int g = tid; g < n_groups; g += 1024) {
        double v[kParts], s = 0.0;
#pragma unroll
        for (int k = 0; k < kParts; ++k) v[k] = part[g * kParts + k];
#pragma unroll
        for (int k = 0; k < kParts; ++k) s += v[k];
        group_sum[g] = s;
    }
    __syncthreads();   // (also makes group_sum visible within the block)
    int bucket = -1;                       // of the boundary, as of its last iteration
    unsigned int b_at = 0, b_count = 0, base = 0;
    int it = 0;
    // (s_stop is set between the barriers of an iteration, so only the check behind the first of them reads it)
    for (; finite && it < iterations && !s_converged; ++it) {
        if (warp < nc - 1) {
            const float bound = s_b[warp] + 0.0f;   // -0 as +0: the two zeros lie in neighbouring buckets
            const int now = static_cast<int>(fit_key(bound) >> shift);
            const bool changed = now != bucket;
            bool moved = false;
            double near[kFitGroup / 32];         // the group's buckets: requested before the bucket's samples, added up after them
            if (changed) {
                moved = bucket < 0 || now / kFitGroup != bucket / kFitGroup || s_near != 0;
                bucket = now;
                b_at = offset[now];
                b_count = count[now];
                base = fit_bucket(now, shift).base;
#pragma unroll
                for (int k = 0; k < kFitGroup / 32; ++k) near[k] = sum[now / kFitGroup * kFitGroup + 32 * k + lane];
            }
            unsigned int c = 0, t = 0;   // t: 1024 x 2^20 at most
            if (b_count <= kFitMaxBucket) {
                const auto look = [&](auto batch, unsigned int i) {
                    constexpr int B = decltype(batch)::value;
                    float x[B];
#pragma unroll
                    for (int j = 0; j < B; ++j) x[j] = i + 32u * j < b_count ? sorted[b_at + i + 32u * j] : INFINITY;
#pragma unroll
                    for (int j = 0; j < B; ++j) {
                        const bool le = !(bound < x[j]);   // (the padding is not)
                        c += le ? 1u : 0u;
                        t += le ? __float_as_uint(x[j]) & ((1u << shift) - 1u) : 0u;
                    }
                };
                unsigned int at = 0;
                for (; at + 32u * (kFitLongBatch - kFitBatch) < b_count; at += 32u * kFitLongBatch) look(std::integral_constant<int, kFitLongBatch>{}, at + lane);
                for (; at < b_count; at += 32u * kFitBatch) look(std::integral_constant<int, kFitBatch>{}, at + lane);
            }
            c = __reduce_add_sync(0xffffffffu, c);
            const unsigned int t_high = __reduce_add_sync(0xffffffffu, t >> 16), t_low = __reduce_add_sync(0xffffffffu, t & 0xffffu);
            if (changed) {
                double low[kFitGroup / 32];
#pragma unroll
                for (int k = 0; k < kFitGroup / 32; ++k) {
                    const int b = now / kFitGroup * kFitGroup + 32 * k + lane;
                    if (b == now) s_own[warp] = near[k];
                    low[k] = b < now ? near[k] : 0.0;
                    near[k] = b > now ? near[k] : 0.0;
                }
#pragma unroll
                for (int h = kFitGroup / 64; h > 0; h >>= 1)
#pragma unroll
                    for (int k = 0; k < h; ++k) {
                        low[k] += low[k + h];
                        near[k] += near[k + h];
                    }
                const double before = low[0], after = near[0];
                // the lower half of the lanes adds up `before`, the upper half `after`
                double v = (lane & 16) ? after : before;
                v += __shfl_xor_sync(0xffffffffu, (lane & 16) ? before : after, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 16) s_after[warp] = v;
                if (lane == 0) {
                    s_before[warp] = v;
                    s_bucket[warp] = now;
                    s_unit[warp] = fit_bucket(now, shift).unit;
                    if (moved) s_moved = 1;
                    if (b_count > kFitMaxBucket) s_stop = 1;
                }
            }
            if (lane == 0) {
                s_le[warp] = b_at + c;
                s_low[warp] = (static_cast<long long>(t_high) << 16) + t_low + static_cast<long long>(c) * base;
            }
        }
        __syncthreads();
        if (s_stop) break;   // nothing of this iteration has been applied
        if (s_moved) {       // a boundary is in another group than before: the sums of the groups in between
            if (warp < nc) {
                const int lo = warp > 0 ? s_bucket[warp - 1] : -1, hi = warp < nc - 1 ? s_bucket[warp] : n_groups * kFitGroup;
                const int g_lo = warp > 0 ? lo / kFitGroup : -1, g_hi = hi / kFitGroup;
                const bool groups = g_lo != g_hi;
                const double* const from = groups ? group_sum : sum;
                const int end = groups ? g_hi : hi;
                double mid = 0.0;
                for (int i = (groups ? g_lo : lo) + 1 + lane; i < end; i += 32 * kFitBatch) {
                    double v[kFitBatch];
#pragma unroll
                    for (int j = 0; j < kFitBatch; ++j) v[j] = i + 32 * j < end ? from[i + 32 * j] : 0.0;
#pragma unroll
                    for (int j = 0; j < kFitBatch; ++j) mid += v[j];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mid += __shfl_xor_sync(0xffffffffu, mid, o);
                if (lane == 0) {
                    s_mid[warp] = mid;
                    if (!groups) s_near = 1;   // (stays: every further move counts then)
                }
            }
            __syncthreads();
        }
        if (warp == 0) {
            float shift_of = 0.f, c_new = lane < nc ? s_c[lane] : 0.f;
            if (lane < nc) {
                const bool has_lo = lane > 0, has_hi = lane < nc - 1;
                const unsigned int above = has_hi ? s_le[lane] : n, below = has_lo ? s_le[lane - 1] : 0u;
                if (above > below) {   // an empty bin keeps its centroid
                    const int lo = has_lo ? s_bucket[lane - 1] : -1, hi = has_hi ? s_bucket[lane] : n_groups * kFitGroup;
                    const bool groups = !has_lo || lo / kFitGroup != hi / kFitGroup;
                    double total;
                    if (lo == hi) {
                        total = static_cast<double>(s_low[lane] - s_low[lane - 1]) * s_unit[lane];
                    } else {
                        total = s_mid[lane];
                        // (both terms are whole numbers of the bucket's unit: exact)
                        if (has_lo) total += s_own[lane - 1] - static_cast<double>(s_low[lane - 1]) * s_unit[lane - 1] + (groups ? s_after[lane - 1] : 0.0);
                        if (has_hi) total += static_cast<double>(s_low[lane]) * s_unit[lane] + (groups ? s_before[lane] : 0.0);
                    }
                    const float mean = static_cast<float>(total / static_cast<double>(above - below));
                    shift_of = fabsf(mean - c_new);
                    c_new = mean;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) shift_of = fmaxf(shift_of, __shfl_xor_sync(0xffffffffu, shift_of, o));
            const float c_next = __shfl_down_sync(0xffffffffu, c_new, 1);
            if (lane < nc) s_c[lane] = c_new;
            if (lane + 1 < nc) s_b[lane] = __fmul_rn(__fadd_rn(c_new, c_next), 0.5f);
            if (lane == 0) {
                s_moved = 0;   // (the others have read it, or read the zero that it still is)
                if (shift_of < kFitShiftThreshold) s_converged = 1;
            }
        }
        __syncthreads();
    }
    if (tid < nc) state->centroids[tid] = s_c[tid];
    if (tid < nc - 1) state->boundaries[tid] = s_b[tid];
    if (tid == 0) {
        state->iterations_run += it;
        state->converged = s_converged;
        state->go_over_all = s_stop;
    }
}

__global__ void __launch_bounds__(kFitThreads) fit_partial_kernel(const float* __restrict__ data, long n_values,
                                                                   const FitState* __restrict__ state, double* __restrict__ part_sum,
                                                                   unsigned long long* __restrict__ part_count) {
    if (state->converged) return;
    extern __shared__ __align__(16) unsigned char fit_smem[];
    double* const h_sum = reinterpret_cast<double*>(fit_smem);                                             // [bin][thread]
    unsigned int* const h_cnt = reinterpret_cast<unsigned int*>(fit_smem + sizeof(double) * kFitMaxBins * kFitThreads);
    __shared__ float s_b[kFitMaxBins];
    const int tid = threadIdx.x;
    const int nc = state->n;
    if (tid < kFitMaxBins) s_b[tid] = tid < nc - 1 ? state->boundaries[tid] : INFINITY;
    for (int b = 0; b < nc; ++b) {
        h_sum[b * kFitThreads + tid] = 0.0;
        h_cnt[b * kFitThreads + tid] = 0u;
    }
    __syncthreads();
    // blocks take chunks of 2^14 values in turn; a thread's 32-bit count holds n / (blocks * 256) values
    const long chunk = 1L << 14;
    for (long c0 = static_cast<long>(blockIdx.x) * chunk; c0 < n_values; c0 += static_cast<long>(gridDim.x) * chunk) {
        const long c1 = c0 + chunk < n_values ? c0 + chunk : n_values;
        for (long i = c0 + tid; i < c1; i += kFitThreads) {
            const float x = __ldg(data + i);
            // number of boundaries strictly below x = std::lower_bound's index; the padding is +inf
            int idx = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (s_b[idx + step - 1] < x) idx += step;
            if (idx >= nc) idx = nc - 1;
            h_sum[idx * kFitThreads + tid] += static_cast<double>(x);
            h_cnt[idx * kFitThreads + tid] += 1u;
        }
    }
    __syncthreads();
    // fold the 256 private histograms: warp w takes bins w, w + 8, ...; lane l adds threads l, l + 32, ...
    const int lane = tid & 31, warp = tid >> 5;
    for (int b = warp; b < nc; b += kFitThreads / 32) {
        double s = 0.0;
        unsigned long long c = 0;
        for (int t = lane; t < kFitThreads; t += 32) {
            s += h_sum[b * kFitThreads + t];
            c += h_cnt[b * kFitThreads + t];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_down_sync(0xffffffffu, s, o);
            c += __shfl_down_sync(0xffffffffu, c, o);
        }
        if (lane == 0) {
            part_sum[static_cast<size_t>(blockIdx.x) * kFitMaxBins + b] = s;
            part_count[static_cast<size_t>(blockIdx.x) * kFitMaxBins + b] = c;
        }
    }
}

__global__ void __launch_bounds__(32) fit_update_kernel(FitState* __restrict__ state, const double* __restrict__ part_sum,
                                                        const unsigned long long* __restrict__ part_count, int n_blocks) {
    if (state->converged) return;
    const int b = threadIdx.x;
    const int nc = state->n;
    float shift = 0.f;
    float c_new = b < nc ? state->centroids[b] : 0.f;
    if (b < nc) {
        double s = 0.0;
        unsigned long long c = 0;
        for (int k = 0; k < n_blocks; ++k) {
            s += part_sum[static_cast<size_t>(k) * kFitMaxBins + b];
            c += part_count[static_cast<size_t>(k) * kFitMaxBins + b];
        }
        if (c > 0) {   // an empty bin keeps its centroid
            c_new = static_cast<float>(s / static_cast<double>(c));
            shift = fabsf(c_new - state->centroids[b]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) shift = fmaxf(shift, __shfl_xor_sync(0xffffffffu, shift, o));
    const float c_next = __shfl_down_sync(0xffffffffu, c_new, 1);
    if (b < nc) state->centroids[b] = c_new;
    if (b + 1 < nc) state->boundaries[b] = __fmul_rn(__fadd_rn(c_new, c_next), 0.5f);
    if (b == 0) {
        state->iterations_run += 1;
        if (shift < kFitShiftThreshold) state->converged = 1;
    }
}

// Rotated, scaled samples of a weight matrix and the residuals the shared primary codebook leaves
// (src/converter.cpp:303-357; the arithmetic is the quantiser's, src/quantizer.cpp:43-62, 117-120).
// One warp per (row, WHT block).  residual may be NULL.
// Bound by instruction issue: 4096 x 4096, block 512, 184 us with 4-byte accesses 64 bytes apart and the boundaries compared one
// after the other, 62 here.
struct SampleTables {
    float cp[32], bp[31];   // the shared codebook's, ascending; boundaries padded with +infinity
    int n_p;
};

template <int E>
__global__ void __launch_bounds__(128) layer_samples_kernel(const float* __restrict__ w, const float* __restrict__ orig_norm, long rows,
                                                            int blocks_per_row, uint32_t seed_p, float scale, float inv_sqrt, int wide,
                                                            const SampleTables tb, float* __restrict__ scaled,
                                                            float* __restrict__ residual) {
    __shared__ SampleTables t;
    if (threadIdx.x == 0) t = tb;
    __syncthreads();
    constexpr int BS = 32 * E;
    const int lane = threadIdx.x & 31;
    const long warp0 = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long n_warps = (static_cast<long>(gridDim.x) * blockDim.x) >> 5;
    const long total = rows * blocks_per_row;
    const int in = blocks_per_row * BS;
    float sp[E];
#pragma unroll
    for (int j = 0; j < E; ++j) sp[j] = sign_value(seed_p, static_cast<uint32_t>(lane * E + j));
    for (long blk = warp0; blk < total; blk += n_warps) {
        const long row = blk / blocks_per_row;
        const int bcol = static_cast<int>(blk - row * blocks_per_row) * BS + lane * E;
        const size_t base = static_cast<size_t>(row) * in + bcol;
        const float safe = fmaxf(orig_norm[row], 1e-10f);
        float v[E];
        load_lane<E>(v, w + base, wide != 0);
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = __fmul_rn(__fdiv_rn(v[j], safe), sp[j]);
        warp_fwht<E>(v, lane);
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = __fmul_rn(__fmul_rn(v[j], inv_sqrt), scale);
        store_lane<E>(scaled + base, v, wide != 0);
        if (residual != nullptr) {
#pragma unroll
            for (int j = 0; j < E; ++j) v[j] = __fsub_rn(v[j], t.cp[bin_of_sorted(v[j], t.bp, t.n_p > 16)]);
            store_lane<E>(residual + base, v, wide != 0);
        }
    }
}

}  // namespace

namespace {

// One fit on its way: what is queued on the stream, and the memory that it uses.
class FitRun {
public:
    // lender: a fit that is queued before this one on the same stream; its memory for the CTAs' places serves both.
    FitRun(const FitRequest& r, cudaStream_t stream, const FitRun* lender = nullptr) : r_(r), stream_(stream), nc_(1 << r.bits) {
        TQ_REQUIRE(r.bits >= 1 && r.bits <= 5, "Unsupported bit width; must be 1-5");
        h_.n = nc_;
        for (int i = 0; i < nc_; ++i) h_.centroids[i] = r.init_centroids[i];
        for (int i = 0; i + 1 < nc_; ++i) h_.boundaries[i] = (r.init_centroids[i] + r.init_centroids[i + 1]) * 0.5f;
        active_ = r.n > 0 && r.iterations > 0;
        if (!active_) return;
        TQ_CUDA(cudaGetDevice(&dev_));
        sms_ = sm_count(dev_);
        TQ_REQUIRE(r.n < (1L << 40), "tq_codebook_fit: at most 2^40 samples");
        state_buf_.reserve(sizeof(FitState), stream);
        TQ_CUDA(cudaMemcpyAsync(state(), &h_, sizeof h_, cudaMemcpyHostToDevice, stream));
        h_.go_over_all = 1;
        // Mantissa bits of a bucket's key: a few hundred values in the buckets where boundaries lie (16.8 M normal samples:
        // 11 bits, about 600), between 2^12 and 2^21 buckets.
        int log2_n = 0;
        while ((1L << log2_n) < r.n) ++log2_n;
        const int key_bits = 9 + std::min(12, std::max(3, log2_n - 13));
        shift_ = 32 - key_bits;
        n_buckets_ = 1 << key_bits;
        n_groups_ = n_buckets_ / kFitGroup;
        const int n_parts = n_buckets_ / kFitSumBuckets;
        const size_t bucket_bytes = static_cast<size_t>(n_buckets_) * (8 + 3 * 4) + static_cast<size_t>(n_parts + n_groups_) * 8 + static_cast<size_t>(n_groups_) * 4;
        // exponents of the window; without memory for the CTAs' places all counters are in L2
        window_ = std::min(kWindowExponents, kWindowSlots >> (24 - shift_));
        window_ctas_ = static_cast<int>(std::min<long>(sms_, (r.n + kWindowTile - 1) / kWindowTile));
        bucketed_ = r.n < (1L << 31);
        windowed_ = bucketed_ && r.n >= static_cast<long>(kFitCrowd);
        const bool lent = windowed_ && lender != nullptr && lender->windowed_ && lender->begin_bytes() >= begin_bytes();
        for (;;) {
            // (one block for the buckets and the places behind them: a cudaMalloc less in a first call)
            const size_t places_at = (bucket_bytes + 255) / 256 * 256;
            try {
                if (bucketed_) bucket_buf_.reserve(windowed_ && !lent ? places_at + begin_bytes() : bucket_bytes, stream);
                if (bucketed_ && r.room == nullptr) sorted_buf_.reserve(static_cast<size_t>(r.n) * 4, stream);
            } catch (const OutOfMemory&) {
                bucket_buf_.set_idle();
                bucket_buf_.release();
                if (windowed_) windowed_ = false;
                else bucketed_ = false;   // the passes over all samples need next to nothing
                continue;
            }
            if (windowed_) begin_ = lent ? lender->begin_ : reinterpret_cast<unsigned int*>(bucket_buf_.as<uint8_t>() + places_at);
            break;
        }
    }
    bool iterated() const { return iterated_; }
    bool short_of_memory() const { return active_ && (!bucketed_ || (!windowed_ && r_.n >= static_cast<long>(kFitCrowd))) && r_.n < (1L << 31); }

    // Queues what comes before the iterations; fills in the job and returns true where there are buckets to iterate on.
    bool enqueue_buckets(FitJob& job) {
        if (!active_ || !bucketed_) return false;
        const int n_parts = n_buckets_ / kFitSumBuckets;
        double* const d_sum = bucket_buf_.as<double>();
        double* const d_part = d_sum + n_buckets_;
        double* const d_group_sum = d_part + n_parts;
        unsigned int* const d_count = reinterpret_cast<unsigned int*>(d_group_sum + n_groups_);
        unsigned int* const d_offset = d_count + n_buckets_;
        unsigned int* const d_cursor = d_offset + n_buckets_;
        unsigned int* const d_group = d_cursor + n_buckets_;
        float* const d_sorted = r_.room != nullptr ? r_.room : sorted_buf_.as<float>();
        const unsigned int un = static_cast<unsigned int>(r_.n);
        const int grid = static_cast<int>(std::min<long>((r_.n + 1023) / 1024, 16L * sms_));
        TQ_CUDA(cudaMemsetAsync(d_count, 0, static_cast<size_t>(n_buckets_) * 4, stream_));
        if (windowed_) {
            static bool configured[64] = {false};
            if (dev_ < 0 || dev_ >= 64 || !configured[dev_]) {
                TQ_CUDA(cudaFuncSetAttribute(fit_count_window_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindowSlots * 4));
                TQ_CUDA(cudaFuncSetAttribute(fit_scatter_window_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindowSlots * 4));
                if (dev_ >= 0 && dev_ < 64) configured[dev_] = true;
            }
        }
        if (un >= kFitCrowd) fit_look_kernel<<<1, 1024, 0, stream_>>>(r_.data, un, shift_, window_, state());
        if (windowed_) fit_count_window_kernel<<<window_ctas_, 1024, window_bytes(), stream_>>>(r_.data, un, shift_, window_, d_count, begin_, state());
        else fit_count_kernel<<<grid, 256, 0, stream_>>>(r_.data, un, shift_, d_count, state());
        fit_groups_kernel<<<n_groups_, 256, 0, stream_>>>(d_count, d_group);
        fit_offsets_kernel<<<n_groups_, 256, 0, stream_>>>(d_count, d_group, d_offset, d_cursor);
        if (windowed_) fit_scatter_window_kernel<<<window_ctas_, 1024, window_bytes(), stream_>>>(r_.data, un, shift_, window_, d_offset, begin_, d_cursor, d_sorted, state());
        else fit_scatter_kernel<<<grid, 256, 0, stream_>>>(r_.data, un, shift_, d_cursor, d_sorted, state());
        int ranges = kFitSumRanges;   // fewer where the blocks would not fill the device: 1 M samples of all exponents, 2048 ranges, 188 us, 193 with eight
        while (ranges > 1 && n_parts / ranges < 8 * sms_) ranges /= 2;
        fit_sums_kernel<<<n_parts / ranges, 256, 0, stream_>>>(d_sorted, d_count, d_offset, shift_, d_sum, d_part, state(), ranges);
        TQ_CUDA(cudaGetLastError());
        job = FitJob{d_sorted, d_count, d_offset, d_sum, d_part, d_group_sum, state(), un, n_groups_, shift_, r_.iterations};
        iterated_ = true;
        return true;
    }

    // Waits for the iterations, makes those that are left over all samples, and hands the results out; the iterations run.
    // samples_again: queues what fills the samples in once more, where they have been overwritten.
    int finish(const std::function<void()>* samples_again = nullptr) {
        if (active_) {
            if (iterated_) read_state();
            if (h_.go_over_all && !h_.converged && h_.iterations_run < r_.iterations) {
                if (samples_again != nullptr) (*samples_again)();
                go_over_all();
            }
            for (DeviceBuffer* b : {&state_buf_, &bucket_buf_, &sorted_buf_}) b->set_idle();
        }
        for (int i = 0; i < nc_; ++i) r_.centroids_out[i] = h_.centroids[i];
        if (r_.boundaries_out)
            for (int i = 0; i + 1 < nc_; ++i) r_.boundaries_out[i] = (h_.centroids[i] + h_.centroids[i + 1]) * 0.5f;   // src/codebook.cpp:135-139
        return h_.iterations_run;
    }

private:
    FitState* state() { return state_buf_.as<FitState>(); }
    size_t window_bytes() const { return (static_cast<size_t>(window_) << (24 - shift_)) * sizeof(unsigned int); }
    size_t begin_bytes() const { return window_bytes() * window_ctas_; }
    void read_state() {
        TQ_CUDA(cudaMemcpyAsync(&h_, state(), sizeof h_, cudaMemcpyDeviceToHost, stream_));
        TQ_CUDA(cudaStreamSynchronize(stream_));
    }
    void go_over_all() {
        const long chunks = (r_.n + (1L << 14) - 1) >> 14;
        const int blocks = static_cast<int>(std::min<long>(chunks, 2L * sms_));
        const size_t smem = (sizeof(double) + sizeof(unsigned int)) * kFitMaxBins * kFitThreads;
        static bool configured[64] = {false};
        if (dev_ < 0 || dev_ >= 64 || !configured[dev_]) {
            TQ_CUDA(cudaFuncSetAttribute(fit_partial_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
            if (dev_ >= 0 && dev_ < 64) configured[dev_] = true;
        }
        DeviceBuffer part_buf;
        part_buf.reserve((sizeof(double) + sizeof(unsigned long long)) * kFitMaxBins * blocks, stream_);
        double* const d_psum = part_buf.as<double>();
        unsigned long long* const d_pcnt = reinterpret_cast<unsigned long long*>(d_psum + kFitMaxBins * blocks);
        // all pairs of launches are enqueued at once; those after convergence return at their first instruction
        for (int it = h_.iterations_run; it < r_.iterations; ++it) {
            fit_partial_kernel<<<blocks, kFitThreads, smem, stream_>>>(r_.data, r_.n, state(), d_psum, d_pcnt);
            fit_update_kernel<<<1, 32, 0, stream_>>>(state(), d_psum, d_pcnt, blocks);
        }
        TQ_CUDA(cudaGetLastError());
        read_state();
        part_buf.set_idle();
    }

    const FitRequest r_;
    const cudaStream_t stream_;
    const int nc_;
    FitState h_{};
    DeviceBuffer state_buf_, bucket_buf_, sorted_buf_;
    bool active_ = false, bucketed_ = false, windowed_ = false, iterated_ = false;
    int dev_ = 0, sms_ = 148, shift_ = 0, n_buckets_ = 0, n_groups_ = 0, window_ = 0, window_ctas_ = 0;
    unsigned int* begin_ = nullptr;   // where each CTA's samples of a bucket begin
};

}  // namespace

// Fits `bits`-bit centroids to data[n] starting from init_centroids (2^bits values, ascending).
// centroids_out / boundaries_out: host arrays of 2^bits and 2^bits - 1 floats.  Returns the iterations run.
int launch_codebook_fit(const FitRequest& r, cudaStream_t stream) {
    FitRun run(r, stream);
    FitJobs jobs{};
    if (run.enqueue_buckets(jobs.job[0])) {
        fit_iterate_kernel<<<1, 1024, 0, stream>>>(jobs);
        TQ_CUDA(cudaGetLastError());
    }
    return run.finish();
}

// Two fits; their iterations run side by side (a CTA each, in one launch), as long as the device has memory for both.  Beyond what
// one fit takes that is the second one's buckets, and what it holds of the first one's samples (b.room).
void launch_codebook_fits(const FitRequest& a, const FitRequest& b, const std::function<void()>& samples_again, cudaStream_t stream) {
    constexpr long kTogether = 1L << 25;   // samples: up to there the memory is kept for the next call (tq_memory.cu)
    if (std::max(a.n, b.n) <= kTogether) {
        FitRun first(a, stream), second(b, stream, &first);
        if (!first.short_of_memory() && !second.short_of_memory()) {
            FitJobs jobs{};
            int n = 0;
            if (first.enqueue_buckets(jobs.job[n])) ++n;
            const bool overwritten = second.enqueue_buckets(jobs.job[n]) && b.room != nullptr;
            if (second.iterated()) ++n;
            if (n != 0) {
                fit_iterate_kernel<<<n, 1024, 0, stream>>>(jobs);
                TQ_CUDA(cudaGetLastError());
            }
            second.finish();   // (its samples in the room that they share, if any, are not needed any more)
            first.finish(overwritten ? &samples_again : nullptr);
            return;
        }
    }
    launch_codebook_fit(a, stream);
    launch_codebook_fit(b, stream);
}

void launch_layer_samples(const float* d_weight, const float* d_row_norms, long rows, int in, uint32_t block, uint32_t seed_p,
                          const float* primary_centroids, int n_primary, float* d_scaled, float* d_residual, cudaStream_t stream) {
    TQ_REQUIRE(is_pow2(block) && block >= 32 && block <= 1024, "block_size must be a power of two in [32, 1024]");
    TQ_REQUIRE(in % static_cast<int>(block) == 0, "in_features must be divisible by block_size");
    TQ_REQUIRE(n_primary >= 2 && n_primary <= 32, "bad codebook size");
    if (rows == 0) return;
    SampleTables tb{};
    tb.n_p = n_primary;
    for (int i = 0; i < n_primary; ++i) tb.cp[i] = primary_centroids[i];
    for (float& b : tb.bp) b = INFINITY;
    for (int i = 0; i + 1 < n_primary; ++i) tb.bp[i] = (primary_centroids[i] + primary_centroids[i + 1]) * 0.5f;
    const float scale = std::sqrt(static_cast<float>(in));
    const float inv_sqrt = 1.0f / std::sqrt(static_cast<float>(block));
    const int bpr = in / static_cast<int>(block);
    const long total = rows * bpr;
    const long want = (total + 3) / 4;
    const int grid = static_cast<int>(want < 148L * 16 ? want : 148L * 16);
    const int wide = (reinterpret_cast<uintptr_t>(d_weight) | reinterpret_cast<uintptr_t>(d_scaled) | reinterpret_cast<uintptr_t>(d_residual)) % 16 == 0 ? 1 : 0;
#define TQ_S_CASE(EV)                                                                                                              \
    case 32 * EV:                                                                                                                  \
        layer_samples_kernel<EV><<<grid, 128, 0, stream>>>(d_weight, d_row_norms, rows, bpr, seed_p, scale, inv_sqrt, wide, tb, d_scaled, \
                                                           d_residual);                                                            \
        break;
    switch (block) {
        TQ_S_CASE(1) TQ_S_CASE(2) TQ_S_CASE(4) TQ_S_CASE(8) TQ_S_CASE(16) TQ_S_CASE(32)
        default: throw Error("unsupported WHT block size");
    }
#undef TQ_S_CASE
    TQ_CUDA(cudaGetLastError());
}

}  // namespace tq
