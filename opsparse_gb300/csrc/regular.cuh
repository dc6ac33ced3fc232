// regular.cuh — rows of C on structured grids: consecutive rows whose A entries and whose B
// rows move on by one column from row to row (stencils and other banded operators) share
// one pattern, so it is worked out once for a group of rows.  Replaces, for those
// rows, OpSparse's shared-hash kernels of its middle bins (kernels/symbolic.cuh:74-130,
// kernels/numeric.cuh:109-205), which hash every product of every row.
//
// Row r + 1 follows row r ("link") when A's row r + 1 is A's row r moved by one column and
// every B row j that A's row r selects is followed by B's row j + 1, its columns moved by one.
// The product of such rows has the same pattern moved by one, and product number q of each
// of them goes to the same position.  The relation is checked exactly, entry by entry.
//
//   k_setup        A's part of the link, for the rows that fold many products per entry
//   k_shift_links  B's part: b_link[j]
//   k_row_links    both: link[r]
//   k_form_groups  runs of links cut into groups of up to kGroupRows rows; marks their rows
//   k_group_count  one row counted, all counts written
//   k_group_rows   numeric: a CTA per group.  The pattern's schedule lists every entry's
//                  products in ascending j, once.  32 rows at a time, A's and B's values are
//                  staged in shared memory (a B row once for all rows and A entries that
//                  reach it) and a lane is a row: a warp walks its share of the schedule with
//                  one FMA per product of 32 rows and the accumulator in a register (FP32: 64
//                  rows, two a lane).  A remainder of at most 16 or 8 rows takes 2 or 4
//                  entries per warp.
//
// What bounds it: FP64 issue (a warp's FMA occupies the SM for about 20 cycles; a 78-row
// run of the 27-point stencil takes 2.5 FMAs per product, 0.80 ms for an 80^3 grid); FP32
// instruction issue (the compensated sum and three shared loads a product), so a lane takes
// two rows there and the compensated sums of both in packed instructions: 61x47x53 grid, the
// kernel 216 -> 175 us, 199 -> 133 million warp instructions, 81% -> 66% of the issue slots
// (barriers and the fixed latency of the packed instructions first), the numeric phase 331 ->
// 283 us.  What is done once a chunk counts as much: with every warp at every pencil of the
// staging and a search per warp for its share a row per lane took 262 million warp
// instructions and 268 us.  The warp hash, which probes and updates shared memory for every
// product, took 1.91 ms (FP32, 61x47x53 grid: 548 us), the window count of every row 0.58 ms
// against 0.11 for links, groups and counts.  Rows that one-pass calls would stage (products
// over 32,768 columns or more) gain as much: 25x100x100 grid, FP64, one call 0.85 ms, two
// phases 0.72 ms, against 4.7 and 1.7 ms by sort and hash kernels.
#pragma once

#include <type_traits>

#include "lists.cuh"

namespace opsg {

constexpr int kGroupRows = 256;     // rows of a group, at most
constexpr int kGroupLanes = 32;     // rows computed together: a lane each
// Runs of fewer rows stay with their class: on runs of 17 rows a 60x60x19 grid took 572 us
// grouped and 537 hashed (FP64, two phases), on runs of 28 rows a 30^3 grid 276 and 345.
constexpr int kGroupMin = 20;
constexpr int kGroupRestMin = 6;    // rows after the last 32 of a run that still join its group
constexpr int kGroupAMax = 32;      // A entries of a grouped row: a bit each in an entry's mask
constexpr int kGroupWindow = 1024;  // rows whose runs one warp cuts
constexpr int kGroupStage = 9216;   // B values staged for 32 rows, at most
constexpr int kGroupThreads = 512;
constexpr int kGroupFlush = 4;      // entries a warp gathers before it writes them
constexpr int kGroupParts = kGroupThreads / 8;  // shares of the schedule, at most
constexpr int kGroupTop = 1024;     // words of the pattern's trie level 0, at most

// b_link[j] = 1 where row j + 1 is row j moved by one column and all its columns are in
// [0, cols).  Eight lanes per row.  Rows whose number is a multiple of kAscendEvery have to
// ascend as well: a column that a row holds twice (outside the library's contract) would leave
// products without a place in the groups' schedule, and a group's entries each reach one of
// these rows.  (Asked of every row, the kernel took 31 us for 25 on an 80^3 grid.)
constexpr int kAscendEvery = 16;
static_assert(kGroupMin - 1 >= kAscendEvery, "the links of a group's rows pass such a row");

static __global__ void __launch_bounds__(256) k_shift_links(const int *__restrict__ rpt, const int *__restrict__ col,
                                                            int rows, int cols, unsigned char *__restrict__ b_link)
{
    const int sub = threadIdx.x & 7;
    for (long long j = (blockIdx.x * 256ll + threadIdx.x) >> 3; j < rows; j += gridDim.x * 32ll) {
        bool ok = j + 1 < rows;
        if (ok) {
            const int b0 = __ldg(rpt + j), b1 = __ldg(rpt + j + 1), b2 = __ldg(rpt + j + 2);
            const int n = b1 - b0;
            ok = b2 - b1 == n && n <= kGroupStage / kGroupLanes;
            if (ok) {
                for (int i = sub; i < n; i += 8) {
                    const int c = __ldg(col + b0 + i), d = __ldg(col + b1 + i);
                    ok &= d == c + 1 && d < cols && c >= 0;
                    if (j % kAscendEvery == 0 && i + 1 < n) ok &= c < __ldg(col + b0 + i + 1);
                }
            }
        }
        const bool all = __all_sync(255u << (threadIdx.x & 24), ok);
        if (sub == 0) b_link[j] = all ? 1 : 0;
    }
}

// link[r] (in: A's part) and the B part of every B row the row selects, where the row's B
// values fit the staging area.  Eight lanes per row.
static __global__ void __launch_bounds__(256) k_row_links(const int *__restrict__ arpt, const int *__restrict__ acol,
                                                          const int *__restrict__ brpt, int M,
                                                          const unsigned char *__restrict__ b_link,
                                                          unsigned char *__restrict__ link)
{
    const int sub = threadIdx.x & 7;
    for (long long r = (blockIdx.x * 256ll + threadIdx.x) >> 3; r < M; r += gridDim.x * 32ll) {
        bool ok = link[r] & kLinked;
        int pencils = 0, longest = 0, inner = 0;
        const unsigned row_lanes = 255u << (threadIdx.x & 24);
        if (ok) {
            const int a0 = __ldg(arpt + r), a1 = __ldg(arpt + r + 1);
            for (int p = a0 + sub; p < a1; p += 8) {
                const int j = __ldg(acol + p);
                ok &= __ldg(b_link + j) != 0;
                longest = max(longest, __ldg(brpt + j + 1) - __ldg(brpt + j));
                if (p + 1 < a1 && __ldg(acol + p + 1) == j + 1) ++inner;
                else ++pencils;
            }
        }
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            pencils += __shfl_xor_sync(row_lanes, pencils, d);
            inner += __shfl_xor_sync(row_lanes, inner, d);
            longest = max(longest, __shfl_xor_sync(row_lanes, longest, d));
        }
        ok &= (pencils * kGroupLanes + inner) * (longest | 1) + 8 * pencils <= kGroupStage;
        const bool all = __all_sync(row_lanes, ok);
        if (sub == 0 && !all) link[r] = 0;
    }
}

// Cuts the runs of links into groups (first row, rows) and marks their rows.  A warp takes
// kGroupWindow rows; runs end at its window.  soff (one-pass calls, else null): the products
// each row stages; a grouped row stages none, whatever its span, and leaves the totals.
static __global__ void __launch_bounds__(128) k_form_groups(int M, unsigned char *__restrict__ link,
                                                            int2 *__restrict__ groups, int *__restrict__ soff,
                                                            DevInfo *info)
{
    const int lane = lane_id();
    unsigned long long products = 0;  // that the lane's grouped rows would have staged
    int rows = 0;                     // of those rows
    const int w0 = ((blockIdx.x * 128 + threadIdx.x) >> 5) * kGroupWindow;
    if (w0 >= M) return;
    unsigned mine = 0u;  // lane i: links of rows w0 + 32 i .. + 31
    for (int i = 0; i < kGroupWindow / 32; ++i) {
        const int r = w0 + 32 * i + lane;
        const bool l = r < M && r + 1 < w0 + kGroupWindow && (link[r] & kLinked);
        const unsigned m = __ballot_sync(kFull, l);
        if (lane == i) mine = m;
    }
    int at = 0;  // rows of the window looked at so far
    while (at < kGroupWindow) {
        // next linked row from `at` on
        unsigned m = mine;
        const int w = at >> 5;
        if (lane < w) m = 0u;
        if (lane == w) m &= kFull << (at & 31);
        const unsigned any = __ballot_sync(kFull, m != 0u);
        if (!any) break;
        const int wl = __ffs(any) - 1;
        const int s = 32 * wl + __ffs(__shfl_sync(kFull, m, wl)) - 1;
        // first row from s on without a link: the run's last row
        m = ~mine;
        if (lane < (s >> 5)) m = 0u;
        if (lane == (s >> 5)) m &= kFull << (s & 31);
        const unsigned any0 = __ballot_sync(kFull, m != 0u);  // never 0: the window's last row has no link
        const int we = __ffs(any0) - 1;
        const int e = 32 * we + __ffs(__shfl_sync(kFull, m, we)) - 1;
        const int len = e - s + 1;
        const int rest = len % kGroupLanes;
        const int grouped = len < kGroupMin ? 0 : len - (rest < kGroupRestMin ? rest : 0);
        const int n = (grouped + kGroupRows - 1) / kGroupRows;
        if (n > 0) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&info->groups, n);
            base = __shfl_sync(kFull, base, 0);
            if (lane < n) groups[base + lane] = make_int2(w0 + s + kGroupRows * lane, min(kGroupRows, grouped - kGroupRows * lane));
            for (int i = lane; i < grouped; i += 32) {
                const int r = w0 + s + i;
                link[r] |= kGrouped;
                if (soff && soff[r] > 0) {
                    products += (unsigned long long)soff[r];
                    ++rows;
                    soff[r] = 0;
                }
            }
        }
        at = e + 1;
    }
    if (!soff) return;
    products = warp_sum_u64(products);
    rows = (int)__reduce_add_sync(kFull, (unsigned)rows);
    if (lane == 0 && rows > 0) {
        atomicAdd(&info->staged_flop, 0ull - products);
        atomicSub(&info->e1_one, rows);
    }
}

// Rows of a class list outside the groups: 0 kept, -1 dropped.
struct PickUngrouped {
    const unsigned char *link;
    __device__ int operator()(int r) const { return (link[r] & kGrouped) ? -1 : 0; }
};

// Counting: the group's first row by column rank, its count for every row.
static __global__ void __launch_bounds__(RankE1::kThreads, RankE1::kMinBlocks)
    k_group_count(SpgemmArgs<double> g, const int2 *__restrict__ groups)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const RankSmem<RankE1, double> sm(smem_raw);
    const int count = g.info->groups;
    const int levels = rank_levels(g.N, RankE1::kTop);
    unsigned long long nnz_acc = 0;
    int n_late = 0;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int2 gr = groups[i];
        const unsigned long long before = nnz_acc;
        rank_row<RankE1, false, double>(g, gr.x, sm, levels, nnz_acc, &n_late);  // ends with a barrier
        if (threadIdx.x == 0) nnz_acc = before + (unsigned long long)gr.y * (nnz_acc - before);
        const int c = g.c_rpt[gr.x];
        for (int r = threadIdx.x + 1; r < gr.y; r += RankE1::kThreads) g.c_rpt[gr.x + r] = c;
    }
    if (threadIdx.x == 0 && nnz_acc) atomicAdd(&g.info->total_nnz, nnz_acc);
}

// Copies one value to shared memory without a register.
template <typename T>
__device__ __forceinline__ void copy_async(T *dst, const T *src)
{
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "one 4- or 8-byte value");
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"((int)sizeof(T)) : "memory");
}

// Copies 16 bytes (both addresses aligned to them).
template <typename T>
__device__ __forceinline__ void copy_async16(T *dst, const T *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

template <typename T>
struct GroupSmem {
    // rows walked together, at most: FP32 takes two per lane where their B values fit
    static constexpr int kRows = sizeof(T) == 4 ? 2 * kGroupLanes : kGroupLanes;
    static constexpr int kStage = sizeof(T) == 4 ? 17408 : kGroupStage;
    T b[kStage];                                // B values: slot rows of one pitch
    // A values, rows of lenA | 1; of rows r and r + 32 in pairs where a lane takes two
    alignas(16) T a[kRows * (kGroupAMax + 1)];
    union {
        T tile[kGroupThreads / 32][kGroupFlush * (kRows + 4)];  // a warp's entries by (entry, row)
        struct {  // while the pattern is worked out
            unsigned bits[2][kEsc1FlopMax];     // trie levels, then the entries' masks of A entries
            unsigned pre[2][kEsc1FlopMax];
        };
    };
    unsigned sched[kEsc1FlopMax];      // products by entry: stage offset << 6 | last of its entry << 5 | A entry
    int col[kEsc1FlopMax];             // the first row's columns
    unsigned start[kEsc1FlopMax + 4];  // an entry's first product in sched
    int e_start[kGroupAMax + 1];       // first product of an A entry
    int e_b0[kGroupAMax];              // its B row's first entry in B
    int e_len[kGroupAMax];             // and length
    int e_base[kGroupAMax];            // and its place in b
    int p_entry[kGroupAMax];           // pencils (runs of entries whose B rows follow one another): first entry
    int p_entries[kGroupAMax];         // and entries
    int part[kGroupParts + 1];         // first entry at or after each part of the products
    int wsum[32];
    int next;
};
constexpr int kGroupCtas = 2;  // per SM
static_assert(kGroupCtas * (sizeof(GroupSmem<double>) + 1024) <= 227 * 1024 &&
                  kGroupCtas * (sizeof(GroupSmem<float>) + 1024) <= 227 * 1024 && kGroupTop <= kEsc1FlopMax,
              "the CTAs of an SM fit its shared memory");

// Two rows' FP32 accumulators: Acc<float>'s steps on both at once (the packed instructions
// round each half as their scalar forms do).
struct AccPair {
    unsigned long long x, y;  // running sums, running compensations
    __device__ __forceinline__ static unsigned long long pack(float lo, float hi)
    {
        unsigned long long v;
        asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
        return v;
    }
    __device__ __forceinline__ static float2 unpack(unsigned long long v)
    {
        float2 f;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
        return f;
    }
    __device__ __forceinline__ static unsigned long long add(unsigned long long a, unsigned long long b)
    {
        unsigned long long v;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
        return v;
    }
    __device__ __forceinline__ static unsigned long long sub(unsigned long long a, unsigned long long b)
    {
        unsigned long long v;
        asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
        return v;
    }
    __device__ __forceinline__ static unsigned long long mul(unsigned long long a, unsigned long long b)
    {
        unsigned long long v;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
        return v;
    }
    __device__ __forceinline__ static unsigned long long fma(unsigned long long a, unsigned long long b,
                                                             unsigned long long c)
    {
        unsigned long long v;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
        return v;
    }
    __device__ __forceinline__ void step(unsigned long long a, unsigned long long b)
    {
        // TwoProduct: h + r == a*b.  h is negated by its sign bits: with a packed subtraction
        // from zero in its place the compiled code lost r (tested against the scalar steps).
        const unsigned long long h = mul(a, b);
        const unsigned long long r = fma(a, b, h ^ 0x8000000080000000ull);
        const unsigned long long s = add(x, h);  // TwoSum: s + q == x + h
        const unsigned long long z = sub(s, x);
        const unsigned long long q = add(sub(x, sub(s, z)), sub(h, z));
        x = s;
        y = add(y, add(q, r));
    }
    __device__ __forceinline__ float2 fin() const { return unpack(add(x, y)); }
};

// The entries of n rows (n <= SW, or 2 * SW in pairs): part threadIdx.x / SW of the schedule
// by SW lanes, a lane per row or per rows r and r + SW, written to C kGroupFlush entries of a
// row at a time.
template <int SW, bool kPair, typename T>
__device__ __forceinline__ void group_fold(GroupSmem<T> &s, int total, int n, int row0, int pa, int pb, int *pc, T *pv)
{
    using AccT = Acc<T>;
    constexpr int kParts = kGroupThreads / SW;
    constexpr int kWidth = kPair ? 2 * SW : SW;  // rows
    const int lane = lane_id();
    const int row = lane % SW;
    const unsigned lanes = SW == 32 ? kFull : ((1u << (SW & 31)) - 1u) << (lane & ~(SW - 1));
    const int part = (int)threadIdx.x / SW;
    const int o0 = s.part[part * (kGroupParts / kParts)], o_end = s.part[(part + 1) * (kGroupParts / kParts)];
    int e = (int)s.start[o0];
    const int e_end = (int)s.start[o_end];
    const T *a = s.a + min(row, n - 1) * (kPair ? 2 * pa : pa);
    const T *b = s.b + min(row, n - 1) * pb;
    [[maybe_unused]] const T *b1 = s.b + min(row + SW, n - 1) * pb;
    T *tile = s.tile[threadIdx.x >> 5] + (lane / SW) * kGroupFlush * (kWidth + 1);
    T *put = tile + row;  // this row's next entry
    // the lane's part of a flush: entry fx of rows fr, fr + SW / kGroupFlush, ...
    const int fx = row % kGroupFlush, fr = row / kGroupFlush;
    const int *fcol = s.col + o0 + fx;
    pc += fr * total + o0 + fx;
    pv += fr * total + o0 + fx;
    auto flush = [&]() {
        __syncwarp(lanes);
        if (tile + fx * (kWidth + 1) + row < put) {  // the entry is held (put = tile + held * (kWidth + 1) + row)
            const int c = *fcol + row0;
            const T *from = tile + fx * (kWidth + 1);
            int at = 0;
#pragma unroll
            for (int r = fr; r < kWidth; r += SW / kGroupFlush, at += SW / kGroupFlush * total) {
                if (r < n) {
                    pc[at] = c + r;
                    pv[at] = from[r];
                }
            }
        }
        __syncwarp(lanes);
        put = tile + row;
        fcol += kGroupFlush;
        pc += kGroupFlush;
        pv += kGroupFlush;
    };
    // a product's operands: of the lane's row, or of its two
    using Operand = std::conditional_t<kPair, unsigned long long, T>;
    std::conditional_t<kPair, AccPair, typename AccT::S> acc{};
    auto load = [&](unsigned x, Operand &av, Operand &bv) {
        if constexpr (kPair) {
            av = reinterpret_cast<const unsigned long long *>(a)[x & 31u];
            bv = AccPair::pack(b[x >> 6], b1[x >> 6]);
        } else {
            av = a[x & 31u];
            bv = b[x >> 6];
        }
    };
    auto product = [&](unsigned x, Operand av, Operand bv) {
        if constexpr (kPair) acc.step(av, bv);
        else acc = AccT::step(acc, av, bv);
        if (x & 32u) {
            if constexpr (kPair) {
                const float2 v = acc.fin();
                put[0] = v.x;
                put[SW] = v.y;
            } else {
                *put = AccT::fin(acc);
            }
            acc = {};
            put += kWidth + 1;
            if (put == tile + row + kGroupFlush * (kWidth + 1)) flush();
        }
    };
    for (; e + 4 <= e_end; e += 4) {
        unsigned x[4];
        Operand av[4], bv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = s.sched[e + u];
#pragma unroll
        for (int u = 0; u < 4; ++u) load(x[u], av[u], bv[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) product(x[u], av[u], bv[u]);
    }
    for (; e < e_end; ++e) {
        const unsigned x = s.sched[e];
        Operand av, bv;
        load(x, av, bv);
        product(x, av, bv);
    }
    if (put != tile + row) flush();
}

template <typename T>
__global__ void __launch_bounds__(kGroupThreads, kGroupCtas) k_group_rows(SpgemmArgs<T> g, const int2 *__restrict__ groups,
                                                                 int *cursor)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GroupSmem<T> &s = *reinterpret_cast<GroupSmem<T> *>(smem_raw);
    constexpr int NT = kGroupThreads;
    constexpr int NW = NT / 32;
    constexpr int PER = kEsc1FlopMax / NT;       // products per thread
    constexpr int kQuad = 16 / (int)sizeof(T);   // values of a 16-byte copy
    const int t = threadIdx.x;
    const int lane = lane_id();
    const int warp = t >> 5;
    const int count = g.info->groups;
    const int levels = rank_levels(g.N, kGroupTop);
    const int a_nnz = __ldg(g.arpt + g.M), b_nnz = __ldg(g.brpt + g.K);
    for (;;) {
        if (t == 0) s.next = atomicAdd(cursor, 1);
        __syncthreads();
        const int it = s.next;
        if (it >= count) break;
        const int2 gr = groups[it];
        const int a0 = __ldg(g.arpt + gr.x);
        const int len_a = __ldg(g.arpt + gr.x + 1) - a0;
        const int off = __ldg(g.c_rpt + gr.x);
        const int pa = len_a | 1;
        // the pattern's A entries and pencils; every warp works them out, warp 0 stores them
        int j = -2, b0 = 0, bl = 0;
        if (lane < len_a) {
            j = __ldg(g.acol + a0 + lane);
            b0 = __ldg(g.brpt + j);
            bl = __ldg(g.brpt + j + 1) - b0;
        }
        const int jp = __shfl_up_sync(kFull, j, 1), lp = __shfl_up_sync(kFull, bl, 1);
        const bool head = lane < len_a && (lane == 0 || jp != j - 1);
        const unsigned heads = __ballot_sync(kFull, head);
        const int pencils = __popc(heads);
        const int longest = (int)__reduce_max_sync(kFull, (unsigned)bl);
        // what the reads and the shared memory below rest on; the groups were formed so
        const bool same = (unsigned)(len_a - 1) < (unsigned)kGroupAMax &&
                          (unsigned)longest <= kGroupStage / kGroupLanes &&
                          (len_a + pencils * (kGroupLanes - 1)) * (longest | 1) + 8 * pencils <= kGroupStage &&
                          gr.y * len_a <= a_nnz - a0 && gr.y * bl <= b_nnz - b0 &&
                          (lane >= len_a || head || lp == bl);
        if (!__all_sync(kFull, same)) {  // not the matrices that were classified (on every warp alike)
            if (t == 0) atomicOr(&g.info->flags, kErrCountMismatch);
            __syncthreads();  // s.next is read
            continue;
        }
        // B rows of one odd length: a pencil's rows lie in b as they lie in B, copied 16 bytes
        // at a time; else every B row gets a row of an odd pitch
        const bool packed = (longest & 1) && __all_sync(kFull, lane >= len_a || bl == longest);
        const int pb = longest | 1;
        const int p = __popc(heads & (lanemask_lt() | (1u << lane))) - 1;  // pencils before and with this entry, less 1
        // rows walked together: two per lane where there are more than 32 and their values fit
        constexpr int kRows = GroupSmem<T>::kRows;
        const bool wide = kRows > kGroupLanes && gr.y > kGroupLanes &&
                          (len_a + pencils * (kRows - 1)) * pb + 8 * pencils <= GroupSmem<T>::kStage;
        auto rows_at = [&](int rest) {  // 17 to 24 rows as 16 and the rest: three quarters of the work of 32
            return rest > 24 ? min(wide ? kRows : kGroupLanes, rest) : min(16, rest);
        };
        int base = (lane + p * ((wide ? kRows : kGroupLanes) - 1)) * pb;
        if (packed) {  // as many values into 16 bytes as the pencil's first value lies in memory
            const int h = 31 - __clz(heads & (lanemask_lt() | (1u << lane)));  // the pencil's first entry
            const int first = __shfl_sync(kFull, b0, h);
            const int want = (int)(((size_t)(g.bval + first) / sizeof(T)) % kQuad);
            const int k = lane - h;
            // (8 values a pencil cover the rounding and the shift)
            base = (base - k * pb + p * 8 + kQuad - 1) / kQuad * kQuad + want + k * pb;
        }
        const int p_incl = warp_incl_scan(bl);
        if (warp == 0) {
            if (lane < len_a) {
                s.e_start[lane + 1] = p_incl;
                s.e_b0[lane] = b0;
                s.e_len[lane] = bl;
                s.e_base[lane] = base;
            }
            if (head) {
                const unsigned after = heads & ~(lanemask_lt() | (1u << lane));
                s.p_entry[p] = lane;
                s.p_entries[p] = (after ? __ffs(after) - 1 : len_a) - lane;
            }
            if (lane == 0) s.e_start[0] = 0;
        }
        int words = (int)(((unsigned)g.N - 1u) >> (5 * levels)) + 1;
        rank_clear<NT>(s.bits[0], words, t);
        rank_clear<NT>(s.bits[1], kEsc1FlopMax, t);
        __syncthreads();
        const int products = min(s.e_start[len_a], kEsc1FlopMax);
        // A's and B's values of rows [r0, r0 + n) of the group
        auto stage = [&](int r0, int n) {
            for (int i = warp; i < n; i += NW) {
                T *to = s.a + i * pa + lane;
                if (n > kGroupLanes) to = s.a + 2 * ((i % kGroupLanes) * pa + lane) + i / kGroupLanes;
                if (lane < len_a) copy_async(to, g.aval + a0 + (long long)(r0 + i) * len_a + lane);
            }
            // a pencil by one warp, or by as many as there are to a pencil
            const int parts = max(1, NW / pencils);
            for (int w = warp; w < pencils * parts; w += NW) {
                const int q = w % pencils, part = w / pencils;
                const int e = s.p_entry[q], rows = s.p_entries[q] - 1 + n, len = s.e_len[e];
                const T *src = g.bval + s.e_b0[e] + (long long)r0 * len;
                T *dst = s.b + s.e_base[e];
                if (packed) {
                    const int values = rows * len;
                    const int lead = min(values, (int)((kQuad - ((size_t)src / sizeof(T)) % kQuad) % kQuad));
                    const int quads = (values - lead) / kQuad;
                    for (int i = part * 32 + lane; i < quads; i += parts * 32)
                        copy_async16(dst + lead + i * kQuad, src + lead + i * kQuad);
                    const int rest = values - quads * kQuad;  // before and after the whole quads
                    if (part == 0 && lane < rest) {
                        const int i = lane < lead ? lane : lane + quads * kQuad;
                        copy_async(dst + i, src + i);
                    }
                } else {
                    for (int i = part; i < rows; i += parts)
                        for (int c = lane; c < len; c += 32) copy_async(dst + i * pb + c, src + i * len + c);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        stage(0, rows_at(gr.y));
        // the pattern: products' columns, entries and positions
        unsigned col[PER], idx[PER];
        int own[PER], at[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int q = t + k * NT;
            col[k] = 0u;
            own[k] = 0;
            at[k] = 0;
            if (q < products) {
                int lo = 0, hi = len_a;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (s.e_start[mid] <= q) lo = mid;
                    else hi = mid;
                }
                own[k] = lo;
                const int c = q - s.e_start[lo];
                at[k] = s.e_base[lo] + c;
                col[k] = min((unsigned)__ldg(g.bcol + s.e_b0[lo] + c), (unsigned)g.N - 1u);
            }
            idx[k] = col[k] >> (5 * levels);
        }
        int total = 0;
        for (int l = 0; l < levels; ++l) {
            unsigned *bits = s.bits[l & 1], *pre = s.pre[l & 1];
            const int shift = 5 * (levels - 1 - l);
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (t + k * NT < products) atomicOr(bits + idx[k], 1u << ((col[k] >> shift) & 31u));
            __syncthreads();
            if (l > 0) rank_clear<NT>(s.bits[(l + 1) & 1], kEsc1FlopMax, t);
            total = rank_prefix<NT>(bits, pre, words, t, warp, lane, s.wsum);
            words = total;
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (t + k * NT < products)
                    idx[k] = pre[idx[k]] + __popc(bits[idx[k]] & ((1u << ((col[k] >> shift) & 31u)) - 1u));
        }
        // an entry's products in ascending j: its mask of A entries is one more level
        unsigned *mask = s.bits[levels & 1];  // zeroed above (levels >= 2) or at the group's start
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (t + k * NT < products) {
                atomicOr(mask + idx[k], 1u << own[k]);
                s.col[idx[k]] = (int)col[k];
            }
        }
        __syncthreads();
        const int listed = rank_prefix<NT>(mask, s.start, total, t, warp, lane, s.wsum);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (t + k * NT < products) {
                const unsigned m = mask[idx[k]], below = m & ((1u << own[k]) - 1u);
                const unsigned last = (m >> own[k]) == 1u ? 32u : 0u;
                s.sched[s.start[idx[k]] + __popc(below)] = ((unsigned)at[k] << 6) | last | (unsigned)own[k];
            }
        }
        if (t == 0) s.start[total] = (unsigned)products;
        if (t <= kGroupParts) {
            const int p = (int)((long long)products * t / kGroupParts);
            int lo = 0, hi = total;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if ((int)s.start[mid] < p) lo = mid + 1;
                else hi = mid;
            }
            s.part[t] = lo;
        }
        const bool fits = __ldg(g.c_rpt + gr.x + gr.y) - off == gr.y * total && listed == s.e_start[len_a];
        if (t == 0 && !fits) atomicOr(&g.info->flags, kErrCountMismatch);
        int n = 0;
        for (int r0 = 0; r0 < gr.y; r0 += n) {
            n = rows_at(gr.y - r0);
            if (r0 > 0) stage(r0, n);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (fits) {
                int *pc = g.c_col + off + r0 * total;
                T *pv = g.c_val + off + r0 * total;
                if constexpr (kRows > kGroupLanes) {
                    if (n > kGroupLanes) group_fold<32, true, T>(s, total, n, r0, pa, pb, pc, pv);
                }
                if (n <= 8) group_fold<8, false, T>(s, total, n, r0, pa, pb, pc, pv);
                else if (n <= 16) group_fold<16, false, T>(s, total, n, r0, pa, pb, pc, pv);
                else if (n <= kGroupLanes) group_fold<32, false, T>(s, total, n, r0, pa, pb, pc, pv);
            }
            __syncthreads();  // the staged values are done with
        }
    }
}

}  // namespace opsg
