// rank.cuh — rows of C by column rank: no sort and no hash table.  A group of threads (a
// warp for rows of at most 256 products, a CTA above) computes one row.  Replaces OpSparse's
// shared-hash kernels of its small to large bins (kernels/symbolic.cuh:74-261,
// kernels/numeric.cuh:109-302), which probe a hash table per product and sort it afterwards.
//
// Per row, over chunks of 32 products (product q is the q-th of A's row in ascending j):
//   1. list A's entries whose B rows are not empty, with the exclusive scan of the B rows'
//      lengths; chunk table: the entry that holds the first product of each chunk;
//   2. expand: the entries that start inside a chunk are one bit each, OR-ed over the warp
//      in one instruction; a lane's entry is the population count of the bits up to its
//      own, where a search per product takes five dependent shuffles;
//   3. rank the columns in a bitmap trie of fan-out 32: level 0 has one bit per 32^(L-1)
//      columns, each set bit owns one 32-bit word of the next level, and level L-1 has one
//      bit per column.  Marking a product is one shared-memory OR per level, a level's
//      word of a column is the column's rank in the level above (prefix popcounts of its
//      words), and the rank in the last level is the entry's position in C's row.  A level
//      holds at most as many words as the row has products, whatever B's width, so the
//      sweeps cost a few words per thread; L is the smallest depth that keeps level 0 within
//      kTop words (one level up to 8,192 columns for a warp, two up to 262,144);
//   symbolic: 4. the row's count is its products less the late ones (whose OR found its
//                bit already set);
//   numeric:  4. a product whose column is not repeated is its entry.  The products of
//                repeated columns fold in product order, 32 at a time, those of one A entry
//                in one step (a B row holds a column once); a CTA lists them first, by the
//                warp that folds their position.  One FMA per product, the
//                oracle's sequence bit for bit;
//             5. C's row is written in column order from shared memory.
//
// What bounds it: instruction issue (about 290 warp instructions per 32 products of a short
// row, 255 of a long one; 140 to count) at 45-60% of the issue slots, and the latency of
// three dependent loads (A's column, B's row extent, B's column).  Measured on a GB300
// against the register, CTA and radix sorts that it replaced: rows of 129-512 products of a
// batch 331 -> 255 us, 513-1,024 141 -> 110, rows of 1,025-4,096 products 82 -> 36 us
// (web graph of 300,000 rows, FP32), 4,097-13,312 55 -> 43 (only 40 rows: one chain each).
#pragma once

#include <climits>

#include "kernels.cuh"

namespace opsg {

// NT threads compute a row of at most NT * PER products (product q = tid + k * NT is a
// thread's k-th), GROUPS rows at a time per CTA (GROUPS > 1: warps).  ACAP bounds the A
// entries with a non-empty B row, MINB the CTAs per SM the registers must allow, TOP the
// words of level 0.  RELOAD64: 64-bit values of B are loaded when they are folded, not held
// in registers from the expansion on.
template <int NT, int PER, int ACAP, int GROUPS, int MINB, int TOP, bool RELOAD64 = false>
struct RankShape {
    static_assert((NT & (NT - 1)) == 0 && NT >= 32 && (GROUPS == 1 || NT == 32), "rows of several warps take a whole CTA");
    static constexpr int kGroup = NT;
    static constexpr int kPer = PER;
    static constexpr int kGroups = GROUPS;
    static constexpr int kThreads = NT * GROUPS;
    static constexpr int kMinBlocks = MINB;
    static constexpr int kWarps = NT / 32;
    static constexpr int kCap = NT * PER;
    static constexpr int kAEntries = ACAP;
    static constexpr int kTop = TOP;
    // the widest shape writes entries of unrepeated columns straight to C (its shared memory
    // holds values of repeated columns only) and reloads its operands
    static constexpr bool kWide = kCap > 4096;
    template <typename T>
    static constexpr bool reload()
    {
        return kWide || (RELOAD64 && sizeof(T) == 8);
    }
    static constexpr int kLevel0 = !kWide && kCap > TOP ? kCap : TOP;
    static_assert(kCap % 128 == 0 && TOP % 4 == 0 && kCap < 65536 && ACAP < 4096, "packed scan, 16-bit product numbers");

    static constexpr size_t up16(size_t x) { return (x + 15) / 16 * 16; }
    static constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
    // [B offset | A value (wide: A position) | first product per entry] [chunk table] [scan]
    // [repeated positions] [wide: their prefixes] [levels; later: values | columns by
    // position | list of products, their entries and positions | counts]
    static constexpr size_t kOffAt = 0;
    static constexpr size_t kAvalAt = kOffAt + up16(4 * (size_t)ACAP);
    static constexpr size_t kStartAt = kAvalAt + up16((kWide ? 4 : 8) * (size_t)ACAP);
    static constexpr size_t kFirstAt = kStartAt + up16(2 * (size_t)ACAP);
    static constexpr size_t kScanAt = kFirstAt + up16(2 * (size_t)(kCap / 32));
    static constexpr size_t kMultiAt = kScanAt + 160;
    static constexpr size_t kMultiPreAt = kMultiAt + up16(4 * (size_t)(kCap / 32));
    static constexpr size_t kRegionAt = kMultiPreAt + (kWide ? up16(4 * (size_t)(kCap / 32)) : 0);
    // a level: one word of bits and the set bits before it per word
    static constexpr size_t kLevelBytes = 8 * ((size_t)kLevel0 + (size_t)kCap);
    static constexpr size_t kColumnAt = kRegionAt + (kWide ? 4 : 8) * (size_t)kCap;
    static constexpr size_t kListAt = kColumnAt + (kWide ? 0 : 4 * (size_t)kCap);
    // counts of listed products per warp that folds them and chunk; an odd number of words
    // between warps keeps a chunk's counts in different banks
    // a listed product, its entry and its position share a word where 10, 12 and 10 bits do
    static constexpr bool kPacked = kCap <= 1024;
    static constexpr size_t kCountAt = kListAt + (kPacked ? 4 : 6) * (size_t)kCap;
    static constexpr int kCountStride = PER * kWarps + 2;
    static_assert(NT == 32 || PER * kWarps % 4 == 0, "an odd number of words");
    template <bool kNum>
    static constexpr size_t group_bytes()
    {
        return cmax(kRegionAt + kLevelBytes,
                    kNum ? (NT > 32 ? kCountAt + up16(2 * (size_t)kWarps * kCountStride) : kListAt) : 0);
    }
    template <bool kNum>
    static constexpr size_t smem()
    {
        return GROUPS * group_bytes<kNum>();
    }
};

// Rows of at most 128, 256, 512, 1,024, 4,096 and 13,312 products.  The kernels are bound by
// latency at 40-60% of the warps an SM holds, so the A entries of the shapes in between are
// few enough (128, 192 and 512; longer rows take the next shape) for their shared memory and
// registers to let 36, 34 and 32 warps run: rows of 352 products 54.6 -> 49.3 us for 10,000
// (FP64), of 176 products 48.8 -> 45.0 us for 20,000, of 64 products 36.5 -> 33.8 us for
// 30,000, against 28, 26, 24 and 32 warps.
using RankW = RankShape<32, 4, 128, 4, 10, 256>;
using RankS = RankShape<32, 8, 128, 4, 9, 256, true>;
using RankM = RankShape<64, 8, 192, 1, 17, 512, true>;
using RankE1 = RankShape<128, 8, 512, 1, 8, 1024>;
using RankMid = RankShape<512, 8, 1280, 1, 2, 2048>;
using RankLarge = RankShape<1024, 13, 2560, 1, 1, 1024>;

// Trie depth for B's width: the smallest with at most `top` words in level 0.
__host__ __device__ __forceinline__ int rank_levels(int N, int top)
{
    int l = 1;
    while (((((unsigned)(N > 1 ? N : 1)) - 1u) >> (5 * l)) >= (unsigned)top) ++l;
    return l;
}

template <int NT>
__device__ __forceinline__ void group_sync()
{
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
}

// Shared memory of one group.
template <typename Sh, typename T>
struct RankSmem {
    using S = typename Acc<T>::S;
    unsigned char *p;
    __device__ __forceinline__ explicit RankSmem(unsigned char *base) : p(base) {}
    template <typename X>
    __device__ __forceinline__ X *at(size_t o) const
    {
        return reinterpret_cast<X *>(p + o);
    }
    // B position of an entry's first product, less its number
    __device__ __forceinline__ int *off() const { return at<int>(Sh::kOffAt); }
    // number of the entry's first product
    __device__ __forceinline__ unsigned short *start() const { return at<unsigned short>(Sh::kStartAt); }
    // entry of product 32 * c
    __device__ __forceinline__ unsigned short *first() const { return at<unsigned short>(Sh::kFirstAt); }
    __device__ __forceinline__ int *wsum() const { return at<int>(Sh::kScanAt); }  // scan: one slot per warp
    __device__ __forceinline__ int *late() const { return at<int>(Sh::kScanAt + 128); }
    // positions of repeated columns, a bit each
    __device__ __forceinline__ unsigned *multi() const { return at<unsigned>(Sh::kMultiAt); }
    __device__ __forceinline__ unsigned *multi_pre() const { return at<unsigned>(Sh::kMultiPreAt); }
    // levels alternate between two spaces; the wide shape's first space holds level 0 only
    __device__ __forceinline__ static bool second(int l) { return Sh::kWide ? l > 0 : (l & 1) != 0; }
    __device__ __forceinline__ unsigned *bits(int l) const
    {
        return at<unsigned>(Sh::kRegionAt + (second(l) ? 8 * (size_t)Sh::kLevel0 : 0));
    }
    __device__ __forceinline__ static int words(int l) { return second(l) ? Sh::kCap : Sh::kLevel0; }
    __device__ __forceinline__ S *val() const { return at<S>(Sh::kRegionAt); }
    __device__ __forceinline__ int *column() const { return at<int>(Sh::kColumnAt); }
    // listed products: number | entry << 10 | position << 22, or number | entry << 16 and the
    // position apart
    __device__ __forceinline__ unsigned *list() const { return at<unsigned>(Sh::kListAt); }
    __device__ __forceinline__ unsigned short *list_pos() const
    {
        return at<unsigned short>(Sh::kListAt + 4 * (size_t)Sh::kCap);
    }
    __device__ __forceinline__ unsigned short *counts() const { return at<unsigned short>(Sh::kCountAt); }
    __device__ __forceinline__ T a_value(const SpgemmArgs<T> &g, int e) const
    {
        if constexpr (Sh::kWide) return __ldg(g.aval + at<int>(Sh::kAvalAt)[e]);
        else return at<T>(Sh::kAvalAt)[e];
    }
};

// Zeroes the first `words` words (rounded up to 16 bytes).
template <int NT>
__device__ __forceinline__ void rank_clear(unsigned *bits, int words, int t)
{
    uint4 *b4 = reinterpret_cast<uint4 *>(bits);
    for (int i = t; i * 4 < words; i += NT) b4[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Inclusive warp scan: two instructions a step (the shuffle's own in-range predicate).
__device__ __forceinline__ int warp_incl_scan(int v)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
        asm volatile(
            "{ .reg .pred p; .reg .s32 t; shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff; @p add.s32 %0, %0, t; }"
            : "+r"(v)
            : "r"(d));
    return v;
}

// Sum of the earlier warps' v (one value per warp, the same on its lanes), and *total over
// all.  A barrier must lie between two uses of wsum.
template <int NT>
__device__ __forceinline__ int group_before(int v, int warp, int lane, int *wsum, int *total)
{
    if constexpr (NT == 32) {
        *total = v;
        return 0;
    } else {
        if (lane == 0) wsum[warp] = v;
        __syncthreads();
        const int x = lane < NT / 32 ? wsum[lane] : 0;
        *total = (int)__reduce_add_sync(kFull, (unsigned)x);
        return (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? x : 0));
    }
}

// pre[w] = set bits before word w, for the level's `words` words; returns all set bits on
// every thread.  Ends with a barrier.
template <int NT>
__device__ __forceinline__ int rank_prefix(const unsigned *bits, unsigned *pre, int words, int t, int warp, int lane,
                                           int *wsum)
{
    const uint4 *b4 = reinterpret_cast<const uint4 *>(bits);
    uint4 *p4 = reinterpret_cast<uint4 *>(pre);
    int total = 0;
    if (words <= 4 * NT) {  // a quad per thread
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (t * 4 < words) v = b4[t];
        const int n1 = __popc(v.x), n2 = n1 + __popc(v.y), n3 = n2 + __popc(v.z), n4 = n3 + __popc(v.w);
        const int incl = warp_incl_scan(n4);
        const int e0 = group_before<NT>(__shfl_sync(kFull, incl, 31), warp, lane, wsum, &total) + incl - n4;
        if (t * 4 < words) p4[t] = make_uint4(e0, e0 + n1, e0 + n2, e0 + n3);
    } else {
        const int quads = (words + 3) >> 2;
        const int per = (quads + NT - 1) / NT;  // consecutive quads of this thread
        const int q0 = min(quads, t * per), q1 = min(quads, q0 + per);
        int mine = 0;
        for (int q = q0; q < q1; ++q) {
            const uint4 v = b4[q];
            mine += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
        const int incl = warp_incl_scan(mine);
        unsigned run =
            (unsigned)(group_before<NT>(__shfl_sync(kFull, incl, 31), warp, lane, wsum, &total) + incl - mine);
        for (int q = q0; q < q1; ++q) {
            const uint4 v = b4[q];
            const unsigned e1 = run + __popc(v.x), e2 = e1 + __popc(v.y), e3 = e2 + __popc(v.z);
            p4[q] = make_uint4(run, e1, e2, e3);
            run = e3 + __popc(v.w);
        }
    }
    group_sync<NT>();
    return total;
}

// Folds listed products, 32 at a time in product order (lanes with `in` hold one of entry e
// and position pos, at slot v).  All lanes call it.  Few repeated positions (a warp's row):
// the products of one A entry never share a position, so they fold in one step.
template <typename T>
__device__ __forceinline__ void rank_fold_entries(bool in, int e, typename Acc<T>::S *v, T a, T b)
{
    unsigned pending = __ballot_sync(kFull, in);
    while (pending) {
        const int lead = __shfl_sync(kFull, e, __ffs(pending) - 1);
        const bool mine = in && e == lead;
        if (mine) *v = Acc<T>::step(*v, a, b);
        pending &= ~__ballot_sync(kFull, mine);
        __syncwarp();
    }
}

// Long runs of one position (a CTA's row): a position's lowest lane folds its lanes in
// order from a register, so a step costs the FMA and not a round trip to shared memory.
template <typename T>
__device__ __forceinline__ void rank_fold_positions(bool in, unsigned pos, typename Acc<T>::S *v, T a, T b)
{
    if (!__any_sync(kFull, in)) return;
    const unsigned m = __match_any_sync(kFull, in ? pos : 0xffffffffu);
    const bool lead = in && lane_id() == __ffs(m) - 1;
    typename Acc<T>::S s = lead ? *v : Acc<T>::zero();
    s = fold_group<T>(s, lead ? m : 0u, a, b);
    if (lead) *v = s;
    __syncwarp();
}

// A warp's row of at most 32 entries with repeated columns: lane p keeps entry p in a
// register.  Five ballots of a chunk's position bits give each lane the mask of its products,
// whose operands it takes by shuffle in product order.
template <typename T>
__device__ __forceinline__ void rank_fold_lanes(bool in, unsigned pos, typename Acc<T>::S &s, T a, T b)
{
    unsigned mine = __ballot_sync(kFull, in);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const unsigned m = __ballot_sync(kFull, (pos >> i) & 1u);
        mine &= ((lane_id() >> i) & 1) ? m : ~m;
    }
    s = fold_group<T>(s, mine, a, b);
}

// One row r of at most Sh::kCap products and Sh::kAEntries A entries with products, by the
// group.  Symbolic and one-pass calls write the row's count to c_rpt[r] and add it to
// nnz_acc (thread 0).  *n_late_out: the row's late products.  Every thread of the group
// calls it; it ends with a barrier.
template <typename Sh, bool kNum, typename T>
__device__ __forceinline__ void rank_row(const SpgemmArgs<T> &g, int r, const RankSmem<Sh, T> &sm, int levels,
                                         unsigned long long &nnz_acc, int *n_late_out)
{
    using AccT = Acc<T>;
    using S = typename AccT::S;
    constexpr int NT = Sh::kGroup;
    constexpr int PER = Sh::kPer;
    constexpr int NW = Sh::kWarps;
    constexpr bool kReload = Sh::template reload<T>();
    const int lane = lane_id();
    const int t = NT == 32 ? lane : (int)threadIdx.x;
    const int warp = NT == 32 ? 0 : t >> 5;
    const int a0 = __ldg(g.arpt + r), a1 = __ldg(g.arpt + r + 1);
    const int row_products = min(__ldg(g.row_flop + r), Sh::kCap);
    int off = 0, n_expect = 0;
    if constexpr (kNum) {
        if (g.soff) {  // one-pass: the row's staging slot, count unknown
            off = __ldg(g.soff + r);
            n_expect = INT_MAX;
        } else {
            off = __ldg(g.c_rpt + r);
            n_expect = __ldg(g.c_rpt + r + 1) - off;
        }
    }
    int words = (int)(((unsigned)g.N - 1u) >> (5 * levels)) + 1;
    rank_clear<NT>(sm.bits(0), words, t);
    if (levels > 1) rank_clear<NT>(sm.bits(1), row_products, t);
    if constexpr (kNum) {
        static_assert(Sh::kCap / 32 <= NT, "a word per thread");
        if (t < Sh::kCap / 32) sm.multi()[t] = 0u;
    }
    if (t == 0) sm.late()[0] = 0;

    // 1. entries with products, their first products and the chunk table
    int entries = 0, products = 0;
    for (int w0 = a0; w0 < a1; w0 += NT) {
        const int q = w0 + t;
        int b0 = 0, bl = 0;
        T av = T(0);
        if (q < a1) {
            const int j = __ldg(g.acol + q);
            if constexpr (kNum && !Sh::kWide) av = __ldg(g.aval + q);
            b0 = __ldg(g.brpt + j);
            bl = __ldg(g.brpt + j + 1) - b0;
        }
        // one scan of (products, entries)
        const int v = (bl << 12) | (bl > 0 ? 1 : 0);
        const int incl = warp_incl_scan(v);
        int total = 0;
        const int before =
            group_before<NT>(__shfl_sync(kFull, incl, 31), warp, lane, sm.wsum(), &total) + incl - v;
        const int s = products + (before >> 12);
        const int e = entries + (before & 4095);
        if (bl > 0 && e < Sh::kAEntries && (unsigned)s < (unsigned)Sh::kCap && s + bl <= Sh::kCap) {
            sm.off()[e] = b0 - s;
            if constexpr (Sh::kWide) sm.template at<int>(Sh::kAvalAt)[e] = q;
            else if constexpr (kNum) sm.template at<T>(Sh::kAvalAt)[e] = av;
            sm.start()[e] = (unsigned short)s;
            for (int c = (s + 31) >> 5; c * 32 < s + bl; ++c) sm.first()[c] = (unsigned short)e;
        }
        products += total >> 12;
        entries += total & 4095;
        group_sync<NT>();
    }
    // the same on every lane, and known to be (a reduction): the branches on it are uniform
    int n = (int)__reduce_max_sync(kFull, (unsigned)row_products);
    if (products != n || entries > Sh::kAEntries) {  // not the matrices that were classified
        if (t == 0) atomicOr(&g.info->flags, kErrCountMismatch);
        n = 0;
    }
    // this warp's chunk k holds products k * NT + c0 + lane; lanes past the row's end hold
    // column 0, mark nothing and look up ranks that nobody uses
    const int c0 = NT == 32 ? 0 : (int)__reduce_max_sync(kFull, (unsigned)(warp * 32));

    // 2. expansion, and level 0's marks
    unsigned col[PER], idx[PER];
    int own[PER];
    T bv[PER];
    unsigned late = 0u;
    {
        bool bad = false;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            col[k] = 0u;
            idx[k] = 0u;
            own[k] = 0;
            bv[k] = T(0);
            const int c = k * NT + c0;
            if (c < n) {
                const int e0 = sm.first()[c >> 5];
                const int e = e0 + 1 + lane;
                const unsigned s = e < entries ? (unsigned)sm.start()[e] - (unsigned)c : 32u;
                const unsigned heads = __reduce_or_sync(kFull, s < 32u ? 1u << s : 0u);
                own[k] = e0 + __popc(heads & ((2u << lane) - 1u));
                if (c + lane < n) {
                    const int kb = sm.off()[own[k]] + c + lane;
                    col[k] = (unsigned)__ldg(g.bcol + kb);
                    if constexpr (kNum && !kReload) bv[k] = __ldg(g.bval + kb);
                }
            }
        }
        unsigned *bits = sm.bits(0);
        const int shift = 5 * (levels - 1);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int c = k * NT + c0;
            if (c >= n) break;
            if (col[k] >= (unsigned)g.N) {
                bad = true;
                col[k] = 0u;
            }
            const unsigned x = col[k] >> shift;
            const unsigned bit = (c + lane < n ? 1u : 0u) << (x & 31u);
            idx[k] = x >> 5;
            if (levels > 1) atomicOr(bits + idx[k], bit);
            else if (atomicOr(bits + idx[k], bit) & bit) late |= 1u << k;
        }
        if (bad) atomicOr(&g.info->flags, kErrBadColumn);
    }

    // 3. ranks, level by level
    int total = 0;
    for (int l = 1; l < levels; ++l) {
        group_sync<NT>();
        if (l > 1 && !Sh::kWide) rank_clear<NT>(sm.bits(l), n, t);  // level l - 2's space, done with
        const unsigned *up = sm.bits(l - 1);
        const unsigned *pre = up + RankSmem<Sh, T>::words(l - 1);
        total = rank_prefix<NT>(up, sm.bits(l - 1) + RankSmem<Sh, T>::words(l - 1), words, t, warp, lane, sm.wsum());
        words = total;
        unsigned *bits = sm.bits(l);
        const int shift = 5 * (levels - 1 - l);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (k * NT + c0 >= n) break;
            const unsigned below = (1u << ((col[k] >> (shift + 5)) & 31u)) - 1u;
            idx[k] = pre[idx[k]] + __popc(up[idx[k]] & below);
        }
        if (Sh::kWide && l > 1) {  // all ranks are looked up before the space is marked again
            __syncthreads();
            rank_clear<NT>(bits, n, t);
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int c = k * NT + c0;
            if (c >= n) break;
            const unsigned bit = (c + lane < n ? 1u : 0u) << ((col[k] >> shift) & 31u);
            if (l < levels - 1) atomicOr(bits + idx[k], bit);
            else if (atomicOr(bits + idx[k], bit) & bit) late |= 1u << k;
        }
    }
    int n_late = (int)__reduce_add_sync(kFull, (unsigned)__popc(late));
    if constexpr (NT > 32) {
        if (lane == 0 && n_late) atomicAdd(sm.late(), n_late);
    }
    group_sync<NT>();
    if constexpr (!kNum) {
        if constexpr (NT > 32) n_late = sm.late()[0];
        *n_late_out = n_late;
        if (t == 0) {
            g.c_rpt[r] = n - n_late;
            nnz_acc += (unsigned long long)(n - n_late);
        }
        group_sync<NT>();
    } else {
        auto b_value = [&](int k) -> T {
            if constexpr (kReload) return __ldg(g.bval + sm.off()[own[k]] + t + k * NT);
            else return bv[k];
        };
        // positions
        {
            unsigned *up = sm.bits(levels - 1);
            unsigned *pre = up + RankSmem<Sh, T>::words(levels - 1);
            total = rank_prefix<NT>(up, pre, words, t, warp, lane, sm.wsum());
            if constexpr (NT > 32) n_late = sm.late()[0];
            *n_late_out = n_late;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (k * NT + c0 >= n) break;
                idx[k] = pre[idx[k]] + __popc(up[idx[k]] & ((1u << (col[k] & 31u)) - 1u));
            }
        }
        if constexpr (NT == 32) {
            if (n_late > 0 && total <= 32) {
                S s = AccT::zero();
                int *pc = g.c_col + off;
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    if (k * NT >= n) break;
                    const bool in = t + k * NT < n;
                    if (in && !((late >> k) & 1u) && (int)idx[k] < n_expect) pc[idx[k]] = (int)col[k];
                    rank_fold_lanes<T>(in, idx[k], s, in ? sm.a_value(g, own[k]) : T(0), in ? b_value(k) : T(0));
                }
                if (lane < min(total, n_expect)) g.c_val[off + lane] = AccT::fin(s);
                if (lane == 0) {
                    if (g.soff) {
                        g.c_rpt[r] = total;
                        nnz_acc += (unsigned long long)total;
                    } else if (total != n_expect) {
                        atomicOr(&g.info->flags, kErrCountMismatch);
                    }
                }
                __syncwarp();
                return;
            }
        }
        if (n_late > 0) {  // the late products' positions are repeated
            unsigned m = late;
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if ((m >> k) & 1u) atomicOr(sm.multi() + (idx[k] >> 5), 1u << (idx[k] & 31u));
        }
        group_sync<NT>();  // the levels are done with: their space holds the entries from here on
        S *val = sm.val();
        if constexpr (Sh::kWide) {
            if (n_late > 0)
                rank_prefix<NT>(sm.multi(), sm.multi_pre(), (total + 31) >> 5, t, warp, lane, sm.wsum());
        }
        // the value of position pos (wide shape: of a repeated one, in their order)
        auto slot = [&](unsigned pos) -> S * {
            if constexpr (!Sh::kWide) return val + pos;
            return val + sm.multi_pre()[pos >> 5] + __popc(sm.multi()[pos >> 5] & ((1u << (pos & 31u)) - 1u));
        };
        unsigned listed = 0u;  // products of repeated columns
        if (n_late > 0) {
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (k * NT + c0 >= n) break;
                if (t + k * NT < n && ((sm.multi()[idx[k] >> 5] >> (idx[k] & 31u)) & 1u)) listed |= 1u << k;
            }
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (k * NT + c0 >= n) break;
            if (t + k * NT < n && !((late >> k) & 1u)) {  // one product of each column
                const bool direct = !((listed >> k) & 1u);
                S s = AccT::zero();
                if (direct) s = AccT::step(s, sm.a_value(g, own[k]), b_value(k));
                if constexpr (Sh::kWide) {
                    if ((int)idx[k] < n_expect) {
                        g.c_col[off + (int)idx[k]] = (int)col[k];
                        if (direct) g.c_val[off + (int)idx[k]] = AccT::fin(s);
                    }
                    if (!direct) *slot(idx[k]) = s;
                } else {
                    val[idx[k]] = s;
                    sm.column()[idx[k]] = (int)col[k];
                }
            }
        }
        if constexpr (NT == 32) {
            __syncwarp();
            if (n_late > 0) {
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    if (k * NT >= n) break;
                    const bool in = (listed >> k) & 1u;
                    rank_fold_entries<T>(in, own[k], val + idx[k], in ? sm.a_value(g, own[k]) : T(0),
                                         in ? b_value(k) : T(0));
                }
            }
        } else if (n_late > 0) {
            // Listed products by the warp that folds them (the low bits of their position), in
            // product order: a count per warp and chunk, their prefixes, the list.  The lanes
            // of a chunk that share a warp come from a ballot per bit; the same ballots give
            // lane w the products of warp w.  (With one list that every warp walked for its
            // share a row's listing cost as many walks as it has warps: the 40 longest rows of
            // a web graph 72 -> 43 us, graph of 200,000 nodes times its transpose 2.51 -> 2.37
            // ms.)
            unsigned short *counts = sm.counts();
            auto by_warp = [&](bool in, unsigned pos, unsigned &same, unsigned &lanes) {
                same = lanes = __ballot_sync(kFull, in);
#pragma unroll
                for (int i = 0; (1 << i) < NW; ++i) {
                    const unsigned m = __ballot_sync(kFull, (pos >> i) & 1u);
                    same &= ((pos >> i) & 1u) ? m : ~m;
                    lanes &= ((lane >> i) & 1) ? m : ~m;
                }
            };
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                unsigned same, lanes = 0u;
                if (k * NT + c0 < n) by_warp((listed >> k) & 1u, idx[k], same, lanes);
                if (lane < NW) counts[lane * Sh::kCountStride + k * NW + warp] = (unsigned short)__popc(lanes);
            }
            __syncthreads();
            {
                constexpr int kEach = (PER * NW + 31) / 32;
                unsigned short *mine = counts + warp * Sh::kCountStride;
                int v[kEach], sum = 0;
#pragma unroll
                for (int i = 0; i < kEach; ++i) {
                    const int q = lane * kEach + i;
                    v[i] = q < PER * NW ? (int)mine[q] : 0;
                    sum += v[i];
                }
                const int incl = warp_incl_scan(sum);
                int run = incl - sum;
#pragma unroll
                for (int i = 0; i < kEach; ++i) {
                    const int q = lane * kEach + i;
                    if (q < PER * NW) mine[q] = (unsigned short)run;
                    run += v[i];
                }
                if (lane == 31) sm.wsum()[warp] = incl;
            }
            __syncthreads();
            const int held = lane < NW ? sm.wsum()[lane] : 0;
            const int first = warp_incl_scan(held) - held;  // lane w: warp w's first item
            const int i_begin = __shfl_sync(kFull, first, warp), i_end = i_begin + __shfl_sync(kFull, held, warp);
            unsigned *list = sm.list();
            [[maybe_unused]] unsigned short *list_pos = sm.list_pos();
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (k * NT + c0 >= n) break;
                const bool in = (listed >> k) & 1u;
                unsigned same, lanes;
                by_warp(in, idx[k], same, lanes);
                const int w = (int)(idx[k] % NW);
                const int i = __shfl_sync(kFull, first, w) + __popc(same & lanemask_lt());
                if (in) {
                    const int at = i + counts[w * Sh::kCountStride + k * NW + warp];
                    const unsigned p = (unsigned)(t + k * NT), x = (unsigned)own[k];
                    if constexpr (Sh::kPacked) {
                        list[at] = p | (x << 10) | (idx[k] << 22);
                    } else {
                        list[at] = p | (x << 16);
                        list_pos[at] = (unsigned short)idx[k];
                    }
                }
            }
            __syncthreads();
            // each warp folds its items, the operands of the next 32 loaded ahead
            auto item = [&](int i, unsigned &pos, int &e, T &a, T &b) -> bool {
                if (i >= i_end) return false;
                const unsigned x = list[i];
                unsigned p;
                if constexpr (Sh::kPacked) {
                    p = x & 1023u;
                    e = (int)((x >> 10) & 4095u);
                    pos = x >> 22;
                } else {
                    p = x & 0xffffu;
                    e = (int)(x >> 16);
                    pos = list_pos[i];
                }
                a = sm.a_value(g, e);
                b = __ldg(g.bval + sm.off()[e] + (int)p);
                return true;
            };
            unsigned pos = 0u, pos_n = 0u;
            int e = 0, e_n = 0;
            T a = T(0), b = T(0), a_n = T(0), b_n = T(0);
            bool in = item(i_begin + lane, pos, e, a, b);
            for (int i0 = i_begin; i0 < i_end; i0 += 32) {
                const bool in_n = item(i0 + 32 + lane, pos_n, e_n, a_n, b_n);
                rank_fold_positions<T>(in, pos, slot(pos), a, b);
                in = in_n;
                pos = pos_n;
                e = e_n;
                a = a_n;
                b = b_n;
            }
        }
        group_sync<NT>();
        // 5. the row in column order
        const int count = min(total, n_expect);
        if (t == 0 && !g.soff && total != n_expect) atomicOr(&g.info->flags, kErrCountMismatch);
        if constexpr (Sh::kWide) {
            if (n_late > 0) {
                for (int i = t; i < count; i += NT)
                    if ((sm.multi()[i >> 5] >> (i & 31)) & 1u) g.c_val[off + i] = AccT::fin(*slot((unsigned)i));
            }
        } else {
            int *pc = g.c_col + off;
            T *pv = g.c_val + off;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (k * NT >= count) break;
                const int i = t + k * NT;
                if (i < count) {
                    pc[i] = sm.column()[i];
                    pv[i] = AccT::fin(val[i]);
                }
            }
        }
        if (g.soff && t == 0) {
            g.c_rpt[r] = total;
            nnz_acc += (unsigned long long)total;
        }
        group_sync<NT>();
    }
}

// Rows by late products: none, at most kRankLateFew, more (counted for diagnosis where B
// has at most kRankCountCols columns).
constexpr int kRankLateFew = 128;
constexpr int kRankCountCols = 65536;

// Rows a group takes before its CTA ends, beside D rows: the D rows' chain of short launches,
// on a stream of higher priority, then places its CTAs between those of a long list (with
// CTAs that stay until their list is empty its every launch waited for a whole list: graph
// of 200,000 nodes times its transpose 2.83 -> 2.65 ms).  Without D rows staying is faster
// (Galerkin product 0.97 ms against 1.01).
template <typename Sh>
constexpr int rank_rows_per_group()
{
    return Sh::kCap <= 256 ? 16 : (Sh::kCap <= 1024 ? 4 : (Sh::kWide ? 1 : 2));
}

// One row per group at a time.  Warp shapes walk the list with a fixed stride; CTA shapes
// draw rows from the cursor (lists are longest first where it matters).  The row count is
// read from device memory, so lists split on the device need no host round trip; the grid
// covers the rows the list may hold.
template <typename Sh, bool kNum, typename T, bool kDiag = false>
__global__ void __launch_bounds__(Sh::kThreads, Sh::kMinBlocks)
    k_rank_rows(SpgemmArgs<T> g, const int *__restrict__ list, const int *count_ptr, int *cursor,
                int max_rows)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int count = *count_ptr;
    const int levels = rank_levels(g.N, Sh::kTop);
    unsigned long long nnz_acc = 0;
    int n_late = 0;
    if constexpr (Sh::kGroups > 1) {
        const int warp = threadIdx.x >> 5;
        const RankSmem<Sh, T> sm(smem_raw + (size_t)warp * Sh::template group_bytes<kNum>());
        const int nwarps = gridDim.x * Sh::kGroups;
        for (int it = blockIdx.x * Sh::kGroups + warp; it < count; it += nwarps)
            rank_row<Sh, kNum, T>(g, __ldg(list + it), sm, levels, nnz_acc, &n_late);
        if (!kNum || g.soff) {
            __shared__ unsigned s_nnz;
            if (threadIdx.x == 0) s_nnz = 0u;
            __syncthreads();
            if (lane_id() == 0 && nnz_acc) atomicAdd(&s_nnz, (unsigned)nnz_acc);
            __syncthreads();
            if (threadIdx.x == 0 && s_nnz) atomicAdd(&g.info->total_nnz, (unsigned long long)s_nnz);
        }
    } else {
        __shared__ int s_row;
        const RankSmem<Sh, T> sm(smem_raw);
        int paths[3] = {0, 0, 0};
        for (int i = 0; i < max_rows; ++i) {
            if (threadIdx.x == 0) s_row = atomicAdd(cursor, 1);
            __syncthreads();
            const int it = s_row;
            if (it >= count) break;
            rank_row<Sh, kNum, T>(g, __ldg(list + it), sm, levels, nnz_acc, &n_late);  // ends with a barrier
            if constexpr (kDiag) ++paths[n_late == 0 ? 0 : (n_late <= kRankLateFew ? 1 : 2)];
        }
        if (threadIdx.x == 0) {
            if ((!kNum || g.soff) && nnz_acc) atomicAdd(&g.info->total_nnz, nnz_acc);
            if constexpr (kDiag) {
                if (g.N <= kRankCountCols)
                    for (int i = 0; i < 3; ++i)
                        if (paths[i]) atomicAdd(&g.info->rank_rows[i], paths[i]);
            }
        }
    }
}

// Small problems, every row of at most RankS::kCap products (E1 rows of at most
// RankS::kAEntries A entries) by one kernel, a warp per row in row order: the classes' kernels,
// each a launch and two events on a stream of its own, take longer to launch than to run.
// Symbolic: the rows that k_setup left to count (not those of at most r8 products and A
// entries).  Does nothing where k_setup found a bad column of A or a row too large for it: the
// usual pipeline then goes on from k_setup's classes.
template <bool kNum, typename T>
__global__ void __launch_bounds__(RankS::kThreads, RankS::kMinBlocks) k_rank_all(SpgemmArgs<T> g, int r8)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (!kNum && (g.info->flags || beyond_small(*g.info))) return;
    const int warp = threadIdx.x >> 5;
    const RankSmem<RankS, T> sm(smem_raw + (size_t)warp * RankS::template group_bytes<kNum>());
    const int levels = rank_levels(g.N, RankS::kTop);
    unsigned long long nnz_acc = 0;
    int n_late = 0;
    const int nwarps = gridDim.x * RankS::kGroups;
    for (int r = blockIdx.x * RankS::kGroups + warp; r < g.M; r += nwarps) {
        const int f = __ldg(g.row_flop + r);
        if (f == 0 || f > RankS::kCap) continue;
        const int len_a = __ldg(g.arpt + r + 1) - __ldg(g.arpt + r);
        if (!kNum && f <= r8 && len_a <= r8) continue;
        if (f > RankS::kAEntries && len_a > RankS::kAEntries) continue;
        rank_row<RankS, kNum, T>(g, r, sm, levels, nnz_acc, &n_late);
    }
    if constexpr (!kNum) {
        if (lane_id() == 0 && nnz_acc) atomicAdd(&g.info->total_nnz, nnz_acc);
    }
}

}  // namespace opsg
