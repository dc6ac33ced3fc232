// lists.cuh — device-side re-binning and ordering of class lists.
#pragma once

#include "rank.cuh"

namespace opsg {

// Device-side re-binning of a class list into kWays sub-lists (out + w*stride), with
// the row counts added to out_counts[w].  Row order inside a sub-list follows the
// warp-aggregated atomics, which is fine: every sub-list kernel schedules rows itself.
template <int kWays, typename Pick>
__global__ void k_split_list(const int *__restrict__ list, const int *count_ptr, Pick pick, int *out, int stride,
                             int *out_counts)
{
    const int count = *count_ptr;
    const int lane = lane_id();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i - lane < count; i += gridDim.x * blockDim.x) {
        const bool in = i < count;
        int r = 0, w = -1;
        if (in) {
            r = list[i];
            w = pick(r);
        }
#pragma unroll
        for (int c = 0; c < kWays; ++c) {
            const unsigned m = __ballot_sync(kFull, w == c);
            if (!m) continue;
            int b = 0;
            if (lane == 0) b = atomicAdd(&out_counts[c], __popc(m));
            b = __shfl_sync(kFull, b, 0);
            if (w == c) out[(size_t)c * stride + b + __popc(m & lanemask_lt())] = r;
        }
    }
}

// Flags of a row beside the next one (regular.cuh): row r + 1 follows row r; row r belongs
// to a group of rows of one pattern.
constexpr unsigned char kLinked = 1;
constexpr unsigned char kGrouped = 2;

// Numeric re-binning of the E1 rows by their output size (known after the symbolic
// phase): 0 / 3 = the rank shapes of a warp / 64 threads (fewer than two products per
// output), 1 = warp hash (at most kSplitNnz outputs: hashing folds the many products per
// output cheaply), 2 = the 128-thread rank shape.
constexpr int kSplitNnz = 256;
static_assert(RankW::kCap >= kWarpFlopMax && RankE1::kCap >= kEsc1FlopMax && RankE1::kAEntries >= kEsc1AMax &&
                  RankLarge::kCap >= kEsc2FlopMax && RankLarge::kAEntries >= kEsc2AMax,
              "every class's rows fit its shapes");
static_assert(RankS::kCap >= kE1SmallMax && RankS::kAEntries >= kE1SmallAMax && RankM::kCap >= kE1HalfMax &&
                  RankM::kAEntries >= kE1HalfAMax && RankMid::kCap >= kE2MidMax && RankMid::kAEntries >= kE2MidAMax,
              "every size's rows fit its shape");
static_assert(2 * (kSplitNnz + 1) > kE1HalfMax, "rows of list 2 have the E1 shape");

struct PickE1 {
    const int *c_rpt;
    const int *row_flop;
    const int *arpt;
    __device__ int operator()(int r) const
    {
        const int nnz = c_rpt[r + 1] - c_rpt[r];
        const int f = row_flop[r];
        if (f <= kE1HalfMax && f < 2 * nnz) {
            const int shape = e1_shape(f, arpt[r + 1] - arpt[r]);
            return shape == 0 ? 0 : (shape == 1 ? 3 : 2);
        }
        return nnz <= kSplitNnz ? 1 : 2;
    }
};

// E1 rows of a one-pass call: 1 = not staged, else (a staging slot of one or more products)
// 0, 3, 2 = the rank shape of a warp, 64 threads, 128 threads.
struct PickStaged {
    const int *soff;
    const int *row_flop;
    const int *arpt;
    __device__ int operator()(int r) const
    {
        if (soff[r + 1] <= soff[r]) return 1;
        const int shape = e1_shape(row_flop[r], arpt[r + 1] - arpt[r]);
        return shape == 0 ? 0 : (shape == 1 ? 3 : 2);
    }
};

// E2 rows by size: 0 = mid shape (RankMid), 1 = large shape (RankLarge).
struct PickE2 {
    const int *arpt;
    const int *row_flop;
    __device__ int operator()(int r) const
    {
        const bool mid = row_flop[r] <= kE2MidMax && arpt[r + 1] - arpt[r] <= kE2MidAMax;
        return mid ? 0 : 1;
    }
};

// Orders a class list by product count, largest first, so that with dynamic row
// scheduling the longest rows start first (longest-processing-time order).  One CTA;
// lists longer than kLptMax stay as they are.
constexpr int kLptMax = 4096;

static __global__ void __launch_bounds__(1024) k_sort_heavy_first(int *list, const int *count_ptr,
                                                           const int *__restrict__ row_flop)
{
    // Rows are grouped by product count in quarter-octave buckets, largest first: one
    // histogram, one scan, one scatter.  Scheduling only needs the heavy rows early; the
    // order inside a bucket is free (every row's result is independent of it).
    constexpr int kBuckets = 128;
    __shared__ int s_rows[kLptMax];
    __shared__ unsigned char s_bucket[kLptMax];
    __shared__ int s_next[kBuckets];
    const int n = *count_ptr;
    if (n <= 1 || n > kLptMax) return;
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x) s_next[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int r = list[i];
        const unsigned f = (unsigned)max(row_flop[r], 1);
        const int lz = 31 - __clz(f);  // floor(log2 f)
        const int frac = lz >= 2 ? (int)((f >> (lz - 2)) & 3u) : 0;
        const int b = kBuckets - 1 - min(kBuckets - 1, 4 * lz + frac);
        s_rows[i] = r;
        s_bucket[i] = (unsigned char)b;
        atomicAdd(&s_next[b], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int b = 0; b < kBuckets; ++b) {
            const int c = s_next[b];
            s_next[b] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) list[atomicAdd(&s_next[s_bucket[i]], 1)] = s_rows[i];
}

}  // namespace opsg
