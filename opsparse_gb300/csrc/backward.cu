// backward.cu — gradients of loss = sum(dC .* C) for C = A*B on fixed sparsity patterns.
// OpSparse has no backward pass; this is new.
//
//   dA_ij = sum_{k in B(j,:)} B_jk * dC_ik      (one value per entry of A)
//   dB_jk = sum_{i : j in A(i,:)} A_ij * dC_ik   (one value per entry of B)
//
// Both re-walk the forward's product enumeration (i, j in A(i,:), k in B(j,:)); every
// product needs the position of (i, k) in C's row i.  Each value is folded in a fixed
// order with the same accumulation policy as the forward (FP64: one FMA per term; FP32:
// Dot2): dA over k in B's row order, dB over i ascending.  dB is computed per entry of B
// over the A entries of column j (a stable transpose of A), so no atomics are needed and
// results are deterministic.
//
// Plan (built once per pattern, kept on the handle):
//   arow[p]     row of A entry p;
//   pos_base[p] index of A entry p's first product in the global (row, A entry, B entry)
//               enumeration = exclusive scan of the B-row lengths over A's entries;
//   at_ptr/at_ent  A's entries ordered by (column, row): CUB radix sort by column, which
//               is stable, over entries in row-major order;
//   at_src[e]   what the e-th of them needs to find its products' positions in C: the index
//               of its first product (with the map below), else its row;
//   brow[q]     row of B entry q;
//   long_b      the chunks of B entries whose column of A is long (k_grad_b_long);
//   pmap[q]     position in C of product q, found once by binary search in C's sorted
//               row — only when products * 4 bytes fits the handle's map budget.  Without
//               it every product's position is searched again on each call.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "internal.hpp"

using namespace opsg;
using namespace opsg_internal;

namespace {

constexpr int kGradBatch = 8;      // chain steps whose operands are loaded together
constexpr int kGradShortMax = 64;  // chains longer than this are folded by a warp
// dB walks A's rows in blocks of about kGradBlock entries of C (112 MB in FP64, within L2; in
// FP32 half of it), but in no more than kGradBlocksMax and only as many as leave a block
// kGradBlockMean entries of A's columns on average: of a C of more than 8 x 14.7 million
// entries, or of short columns, the blocks are larger and reach beyond L2.  Graph of 200,000 nodes times its transpose (40 million entries): the
// gradient kernel 557 us in one block, 470 in five, 391 in three, 375 in three with half the
// operands loaded ahead (a block's part of a column is short), the step 3.21 -> 3.00 ms;
// uniform 100,000 x 60,000 x 100,000 FP32, the step 1.18 -> 0.80 ms with what a thread per
// entry gives.
constexpr int kGradBlock = 14 << 20;
constexpr int kGradBlocksMax = 8;
constexpr int kGradBlockMean = 2;

// First index in a[0, n) with a[idx] >= key.
__device__ __forceinline__ int lower_bound_i32(const int *__restrict__ a, int n, int key)
{
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(a + mid) < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Position of (i, key) in C, or -1 (and an error flag) if C's row i lacks the key.
__device__ __forceinline__ int c_position(const int *__restrict__ c_rpt, const int *__restrict__ c_col, int i,
                                          int key, int *flags)
{
    const int c0 = __ldg(c_rpt + i);
    const int n = __ldg(c_rpt + i + 1) - c0;
    const int t = lower_bound_i32(c_col + c0, n, key);
    if (t >= n || __ldg(c_col + c0 + t) != key) {
        atomicOr(flags, kErrCountMismatch);
        return -1;
    }
    return c0 + t;
}

__global__ void k_blen_of_a(const int *__restrict__ acol, const int *__restrict__ brpt, long long nnz,
                            long long *__restrict__ out)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nnz; p += (long long)gridDim.x * blockDim.x) {
        const int j = __ldg(acol + p);
        out[p] = __ldg(brpt + j + 1) - __ldg(brpt + j);
    }
}

__global__ void k_iota(int *out, long long n)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        out[p] = (int)p;
}

// arow[p] = row of A's entry p < nnz_a, brow[q] = row of B's entry q < nnz_b; one warp per row.
// *count = 0.
__global__ void k_expand_rows(const int *__restrict__ arpt, int M, long long nnz_a, int *__restrict__ arow,
                              const int *__restrict__ brpt, int K, long long nnz_b, int *__restrict__ brow, int *count)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = 0;
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long w = w0; w < (long long)M + K; w += nw) {
        const bool of_a = w < M;
        const int i = (int)(of_a ? w : w - M);
        const int *rpt = of_a ? arpt : brpt;
        int *row = of_a ? arow : brow;
        const long long nnz = of_a ? nnz_a : nnz_b;
        const int p0 = __ldg(rpt + i), p1 = __ldg(rpt + i + 1);
        for (int p = p0 + lane_id(); p < p1 && p < nnz; p += 32) row[p] = i;
    }
}

// at_ptr[j] = first position of column j in the column-sorted key array.
__global__ void k_col_starts(const int *__restrict__ sorted_cols, long long nnz, int K, int *__restrict__ at_ptr)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p <= nnz; p += (long long)gridDim.x * blockDim.x) {
        const int cur = p < nnz ? __ldg(sorted_cols + p) : K;
        const int prev = p > 0 ? __ldg(sorted_cols + p - 1) : -1;
        for (int j = prev + 1; j <= cur; ++j) at_ptr[j] = (int)p;
    }
}

// The chunks of up to 32 entries of one row of B whose column of A is too long for a thread
// (k_grad_b_long); their order does not matter to the results.
__global__ void k_list_long_b(long long nnz_b, const int *__restrict__ brow, const int *__restrict__ brpt,
                              const int *__restrict__ at_ptr, int *__restrict__ list, int *count)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nnz_b; q += (long long)gridDim.x * blockDim.x) {
        const int j = __ldg(brow + q);
        if (__ldg(at_ptr + j + 1) - __ldg(at_ptr + j) > kGradShortMax && (q - __ldg(brpt + j)) % 32 == 0)
            list[atomicAdd(count, 1)] = (int)q;
    }
}

// at_src[e]: first product of the e-th column-ordered A entry (with a map), else its row.
template <bool kMap>
__global__ void k_column_sources(const int *__restrict__ at_ent, long long nnz, const long long *__restrict__ pos_base,
                                 const int *__restrict__ arow, int *__restrict__ at_src)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nnz; e += (long long)gridDim.x * blockDim.x) {
        const int p = __ldg(at_ent + e);
        at_src[e] = kMap ? (int)__ldg(pos_base + p) : __ldg(arow + p);
    }
}

// at_blk[j] = first entry of A's column j in a row from which on C holds at least `entries`
// entries.
__global__ void k_column_block(int K, const int *__restrict__ at_ptr, const int *__restrict__ at_ent,
                               const int *__restrict__ arow, const int *__restrict__ c_rpt, int M, int entries,
                               int *__restrict__ at_blk)
{
    const int row = lower_bound_i32(c_rpt, M + 1, entries);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < K; j += gridDim.x * blockDim.x) {
        int lo = __ldg(at_ptr + j), hi = __ldg(at_ptr + j + 1);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(arow + __ldg(at_ent + mid)) < row) lo = mid + 1;
            else hi = mid;
        }
        at_blk[j] = lo;
    }
}

// pmap[pos_base[p] + t] = position in C of product (row(p), B entry brpt[j]+t); one warp
// per row of A, products walked in chunks of 32.
__global__ void __launch_bounds__(256) k_build_pmap(const int *__restrict__ arpt, const int *__restrict__ acol,
                                                     const int *__restrict__ brpt, const int *__restrict__ bcol, int M,
                                                     const int *__restrict__ c_rpt, const int *__restrict__ c_col,
                                                     const long long *__restrict__ pos_base, int *__restrict__ pmap,
                                                     int *flags)
{
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = w0; i < M; i += nw) {
        const int a0 = __ldg(arpt + i), a1 = __ldg(arpt + i + 1);
        warp_products<false, double>(a0, a1, 32, acol, nullptr, brpt, [&](bool valid, int k, double, int p) {
            if (valid) {
                const int j = __ldg(acol + p);
                const int pos = c_position(c_rpt, c_col, (int)i, __ldg(bcol + k), flags);
                pmap[__ldg(pos_base + p) + (k - __ldg(brpt + j))] = pos;
            }
        });
    }
}

// The position in C of product (row i, B entry q) of A entry p: from the map, or by a
// binary search of C's row i.
template <bool kMap>
__device__ __forceinline__ int prod_pos(const int *__restrict__ pmap, long long base, int t,
                                        const int *__restrict__ c_rpt, const int *__restrict__ c_col, int i, int key,
                                        int *flags)
{
    if constexpr (kMap) return __ldg(pmap + base + t);
    return c_position(c_rpt, c_col, i, key, flags);
}

// dA, chains of at most kGradShortMax terms: one thread per A entry p = (i, j), folding
// B row j in order, kGradBatch terms' operands loaded ahead of their FMAs.  Longer chains
// are listed for k_grad_a_long.  (A warp that walks 32 entries' products together, through
// shared memory, reads positions and values in order but took 438 us against 258 on a
// graph of 200,000 nodes times its transpose; four terms ahead instead of eight, 253.)
template <typename T, bool kMap>
__global__ void __launch_bounds__(256) k_grad_a_short(const int *__restrict__ acol, long long nnz_a,
                                                       const int *__restrict__ arow, const int *__restrict__ brpt,
                                                       const int *__restrict__ bcol, const T *__restrict__ bval,
                                                       const int *__restrict__ c_rpt, const int *__restrict__ c_col,
                                                       const T *__restrict__ dc, const long long *__restrict__ pos_base,
                                                       const int *__restrict__ pmap, T *__restrict__ da,
                                                       int *__restrict__ long_list, int *long_count, int *flags)
{
    using AccT = Acc<T>;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nnz_a;
         p += (long long)gridDim.x * blockDim.x) {
        const int j = __ldg(acol + p);
        const int b0 = __ldg(brpt + j), b1 = __ldg(brpt + j + 1);
        if (b1 - b0 > kGradShortMax) {
            long_list[atomicAdd(long_count, 1)] = (int)p;
            continue;
        }
        const long long base = kMap ? __ldg(pos_base + p) : 0;
        const int i = kMap ? 0 : __ldg(arow + p);
        typename AccT::S s = AccT::zero();
        for (int q0 = b0; q0 < b1; q0 += kGradBatch) {
            int pos[kGradBatch];
            T bv[kGradBatch], d[kGradBatch];
#pragma unroll
            for (int u = 0; u < kGradBatch; ++u)
                pos[u] = q0 + u < b1 ? prod_pos<kMap>(pmap, base, q0 + u - b0, c_rpt, c_col, i,
                                                      kMap ? 0 : __ldg(bcol + q0 + u), flags)
                                     : -1;
#pragma unroll
            for (int u = 0; u < kGradBatch; ++u) {
                bv[u] = q0 + u < b1 ? __ldg(bval + q0 + u) : T(0);
                d[u] = pos[u] >= 0 ? __ldg(dc + pos[u]) : T(0);
            }
#pragma unroll
            for (int u = 0; u < kGradBatch; ++u)
                if (q0 + u < b1) s = AccT::step(s, bv[u], d[u]);
        }
        da[p] = AccT::fin(s);
    }
}

// dA, long chains: one warp per listed A entry.  The lanes load the operands of the next
// two batches of 32 terms (positions and B values coalesced, dC gathered in parallel)
// while lane 0 folds the current 32 from shared memory, in order.
template <typename T, bool kMap>
__global__ void __launch_bounds__(256) k_grad_a_long(const int *__restrict__ acol, const int *__restrict__ arow,
                                                      const int *__restrict__ brpt, const int *__restrict__ bcol,
                                                      const T *__restrict__ bval, const int *__restrict__ c_rpt,
                                                      const int *__restrict__ c_col, const T *__restrict__ dc,
                                                      const long long *__restrict__ pos_base,
                                                      const int *__restrict__ pmap, T *__restrict__ da,
                                                      const int *__restrict__ long_list, const int *long_count,
                                                      int *flags)
{
    using AccT = Acc<T>;
    __shared__ T s_b[256 / 32][2][32];
    __shared__ T s_d[256 / 32][2][32];
    const int lane = lane_id();
    const int warp = threadIdx.x >> 5;
    const int count = *long_count;
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long it = w0; it < count; it += nw) {
        const int p = __ldg(long_list + it);
        const int j = __ldg(acol + p);
        const int b0 = __ldg(brpt + j), b1 = __ldg(brpt + j + 1);
        const long long base = kMap ? __ldg(pos_base + p) : 0;
        const int i = kMap ? 0 : __ldg(arow + p);
        auto gather = [&](int q, T &bv, T &d) {
            bv = T(0);
            d = T(0);
            if (q < b1) {
                const int pos = prod_pos<kMap>(pmap, base, q - b0, c_rpt, c_col, i, kMap ? 0 : __ldg(bcol + q), flags);
                bv = __ldg(bval + q);
                d = pos >= 0 ? __ldg(dc + pos) : T(0);
            }
        };
        T nb, nd, nb2, nd2;
        gather(b0 + lane, nb, nd);
        gather(b0 + 32 + lane, nb2, nd2);
        typename AccT::S s = AccT::zero();
        int buf = 0;
        for (int q = b0; q < b1; q += 32) {
            s_b[warp][buf][lane] = nb;
            s_d[warp][buf][lane] = nd;
            __syncwarp();
            nb = nb2;
            nd = nd2;
            gather(q + 64 + lane, nb2, nd2);
            if (lane == 0) {
                const int m = min(32, b1 - q);
                for (int u = 0; u < m; ++u) s = AccT::step(s, s_b[warp][buf][u], s_d[warp][buf][u]);
            }
            buf ^= 1;
        }
        if (lane == 0) da[p] = AccT::fin(s);
        __syncwarp();
    }
}

// dB, columns of A with at most kGradShortMax entries: one thread per B entry q = (j, k),
// folding the A entries of column j in ascending row order, kGradBatch terms' operands
// loaded ahead of their FMAs.  The threads of one row of B read the same column entries (one
// request each) and neighbouring positions.  Bound by the gathers of dC, a 32-byte sector a
// product: a warp per row of B left the lanes beyond the row's length idle, and took one
// dependent load more to find each product's position (uniform FP32 products 49 -> 26 us).
// kBlocked: the launch walks one block of A's rows, entries [e_lo[j], e_hi[j]) of the column,
// so that the rows of dC it gathers from stay in L2; the fold's state is kept in between.
template <typename T, bool kMap, bool kBlocked>
__global__ void __launch_bounds__(256) k_grad_b_short(long long nnz_b, const int *__restrict__ brow,
                                                       const int *__restrict__ brpt, const int *__restrict__ bcol,
                                                       const T *__restrict__ aval, const int *__restrict__ at_ptr,
                                                       const int *__restrict__ at_ent, const int *__restrict__ at_src,
                                                       const int *__restrict__ c_rpt, const int *__restrict__ c_col,
                                                       const T *__restrict__ dc, const int *__restrict__ pmap,
                                                       T *__restrict__ db, int *flags, const int *__restrict__ e_lo,
                                                       const int *__restrict__ e_hi, typename Acc<T>::S *state,
                                                       bool first, bool last)
{
    using AccT = Acc<T>;
    constexpr int kBatch = kBlocked ? kGradBatch / 2 : kGradBatch;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nnz_b;
         q += (long long)gridDim.x * blockDim.x) {
        const int j = __ldg(brow + q);
        int e0 = __ldg(at_ptr + j), e1 = __ldg(at_ptr + j + 1);
        if (e1 - e0 > kGradShortMax) continue;  // k_grad_b_long's
        if constexpr (kBlocked) {
            e0 = __ldg(e_lo + j);
            e1 = __ldg(e_hi + j);
            if (e0 == e1 && !first && !last) continue;
        }
        const int b0 = __ldg(brpt + j);
        const int t = (int)(q - b0);
        if (t < 0 || t >= __ldg(brpt + j + 1) - b0) {  // not the pattern of the plan
            atomicOr(flags, kErrCountMismatch);
            continue;
        }
        const int key = kMap ? 0 : __ldg(bcol + q);
        typename AccT::S s = AccT::zero();
        if constexpr (kBlocked)
            if (!first) s = state[q];
        for (int eb = e0; eb < e1; eb += kBatch) {
            int pos[kBatch];
            T a[kBatch], d[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                pos[u] = -1;
                a[u] = T(0);
                if (eb + u < e1) {
                    const int src = __ldg(at_src + eb + u);
                    a[u] = __ldg(aval + __ldg(at_ent + eb + u));
                    pos[u] = prod_pos<kMap>(pmap, src, t, c_rpt, c_col, src, key, flags);
                }
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) d[u] = pos[u] >= 0 ? __ldg(dc + pos[u]) : T(0);
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (eb + u < e1) s = AccT::step(s, a[u], d[u]);
        }
        if (!kBlocked || last) db[q] = AccT::fin(s);
        else state[q] = s;
    }
}

// dB, longer columns: one warp per listed chunk of up to 32 entries of one row j of B, lanes
// over the entries q, each folding the A entries of column j in ascending row order.  All
// lanes walk the same column entries, so the warp loads 32 of them at once (one per lane) and
// shares them by shuffle; each lane then loads kGradBatch terms' positions and dC values
// ahead of its FMAs.  Of the plan's entries of row j, those outside B's row are refused.
template <typename T, bool kMap>
__global__ void __launch_bounds__(256) k_grad_b_long(const int *__restrict__ list, int count, long long nnz_b,
                                                      const int *__restrict__ brow, const int *__restrict__ brpt,
                                                      const int *__restrict__ bcol, const T *__restrict__ aval,
                                                      const int *__restrict__ at_ptr, const int *__restrict__ at_ent,
                                                      const int *__restrict__ at_src, const int *__restrict__ c_rpt,
                                                      const int *__restrict__ c_col, const T *__restrict__ dc,
                                                      const int *__restrict__ pmap, T *__restrict__ db, int *flags)
{
    using AccT = Acc<T>;
    const int lane = lane_id();
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long it = w0; it < count; it += nw) {
        const int qb = __ldg(list + it);
        const int j = __ldg(brow + qb);
        const int b0 = __ldg(brpt + j), b1 = __ldg(brpt + j + 1);
        const int e0 = __ldg(at_ptr + j), e1 = __ldg(at_ptr + j + 1);
        const int q = qb + lane;
        const bool qv = q >= b0 && q < b1;
        if (!qv && q < nnz_b && __ldg(brow + q) == j) atomicOr(flags, kErrCountMismatch);
        const int key = (!kMap && qv) ? __ldg(bcol + q) : 0;
        typename AccT::S s = AccT::zero();
        for (int eb = e0; eb < e1; eb += 32) {
            // one column entry per lane: its value, and its product base or its row
            int se = 0;
            T ae = T(0);
            if (eb + lane < e1) {
                se = __ldg(at_src + eb + lane);
                ae = __ldg(aval + __ldg(at_ent + eb + lane));
            }
            const int m = min(32, e1 - eb);
            for (int t0 = 0; t0 < m; t0 += kGradBatch) {
                int pos[kGradBatch];
                T a[kGradBatch], d[kGradBatch];
#pragma unroll
                for (int u = 0; u < kGradBatch; ++u) {
                    const int lu = min(t0 + u, 31);
                    const int su = __shfl_sync(kFull, se, lu);
                    a[u] = shfl(ae, lu);
                    pos[u] = (qv && t0 + u < m) ? prod_pos<kMap>(pmap, su, q - b0, c_rpt, c_col, su, key, flags) : -1;
                }
#pragma unroll
                for (int u = 0; u < kGradBatch; ++u) d[u] = pos[u] >= 0 ? __ldg(dc + pos[u]) : T(0);
#pragma unroll
                for (int u = 0; u < kGradBatch; ++u)
                    if (t0 + u < m) s = AccT::step(s, a[u], d[u]);
            }
        }
        if (qv) db[q] = AccT::fin(s);
    }
}

int grid_of(long long work, int per_block, int cap)
{
    const long long b = (work + per_block - 1) / per_block;
    return (int)std::max<long long>(1, std::min<long long>(b, cap));
}

// Builds (or reuses) the plan for this pattern.
int build_plan(ops_handle_s *h, int M, int K, int N, const int *a_rpt, const int *a_col, long long nnz_a,
               const int *b_rpt, const int *b_col, long long nnz_b, const int *c_rpt, const int *c_col,
               cudaStream_t st)
{
    BackwardPlan &pl = h->bwd;
    if (pl.valid && pl.M == M && pl.K == K && pl.N == N && pl.nnz_a == nnz_a && pl.nnz_b == nnz_b &&
        pl.a_rpt == a_rpt && pl.a_col == a_col && pl.b_rpt == b_rpt && pl.b_col == b_col && pl.c_rpt == c_rpt &&
        pl.c_col == c_col)
        return OPS_OK;
    if (pl.mem) {
        OPS_CUDA(h, cudaFreeAsync(pl.mem, st));
        pl.mem = nullptr;
    }
    if (pl.at_blk) {
        OPS_CUDA(h, cudaFreeAsync(pl.at_blk, st));
        pl.at_blk = nullptr;
    }
    if (pl.pmap) {
        OPS_CUDA(h, cudaFreeAsync(pl.pmap, st));
        pl.pmap = nullptr;
    }
    pl.valid = false;
    const int sms = h->num_sms;
    const size_t na = (size_t)std::max<long long>(nnz_a, 1);
    // temporaries: B-row length per A entry (int64), sort keys/values, CUB scratch
    size_t sort_tmp = 0, scan_tmp = 0;
    OPS_CUDA(h, cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (int *)nullptr, (int *)nullptr, (int *)nullptr,
                                                (int *)nullptr, (int)na, 0, std::max(1, ceil_log2(std::max(K, 2))),
                                                st));
    OPS_CUDA(h, cub::DeviceScan::ExclusiveSum(nullptr, scan_tmp, (long long *)nullptr, (long long *)nullptr,
                                              (int)na + 1, st));
    const size_t tmp_bytes = align_up(8 * (na + 1), 256) + align_up(4 * na, 256) * 2 + align_up(sort_tmp, 256) +
                             align_up(scan_tmp, 256);
    void *tp = nullptr;
    OPS_CUDA(h, cudaMallocFromPoolAsync(&tp, tmp_bytes, h->pool, st));
    unsigned char *t = static_cast<unsigned char *>(tp);
    long long *blen = reinterpret_cast<long long *>(t);
    t += align_up(8 * (na + 1), 256);
    int *sorted_cols = reinterpret_cast<int *>(t);
    t += align_up(4 * na, 256);
    int *iota = reinterpret_cast<int *>(t);
    t += align_up(4 * na, 256);
    void *sort_scratch = t;
    t += align_up(sort_tmp, 256);
    void *scan_scratch = t;

    // persistent plan arrays (map added below once the product count is known)
    const size_t nb = (size_t)std::max<long long>(nnz_b, 1);
    const size_t list_b = na / kGradShortMax + nb / 32 + 1;  // a chunk a listed row, and one per 32 entries
    const size_t base_bytes = align_up(8 * (na + 1), 256) + align_up(4 * ((size_t)K + 1), 256) +
                              align_up(4 * na, 256) * 3 + align_up(4 * nb, 256) + align_up(4 * list_b, 256);
    void *pp = nullptr;
    OPS_CUDA(h, cudaMallocFromPoolAsync(&pp, base_bytes, h->pool, st));
    unsigned char *m = static_cast<unsigned char *>(pp);
    pl.mem = m;
    pl.bytes = base_bytes;
    pl.pos_base = reinterpret_cast<long long *>(m);
    m += align_up(8 * (na + 1), 256);
    pl.at_ptr = reinterpret_cast<int *>(m);
    m += align_up(4 * ((size_t)K + 1), 256);
    pl.at_ent = reinterpret_cast<int *>(m);
    m += align_up(4 * na, 256);
    pl.arow = reinterpret_cast<int *>(m);
    m += align_up(4 * na, 256);
    pl.at_src = reinterpret_cast<int *>(m);
    m += align_up(4 * na, 256);
    pl.brow = reinterpret_cast<int *>(m);
    m += align_up(4 * nb, 256);
    pl.long_b = reinterpret_cast<int *>(m);

    OPS_CUDA(h, cudaMemsetAsync(blen + na, 0, sizeof(long long), st));
    if (nnz_a > 0) {
        k_blen_of_a<<<grid_of(nnz_a, 256, sms * 16), 256, 0, st>>>(a_col, b_rpt, nnz_a, blen);
        k_iota<<<grid_of(nnz_a, 256, sms * 16), 256, 0, st>>>(iota, nnz_a);
        OPS_CUDA(h, cudaGetLastError());
    }
    OPS_CUDA(h, cub::DeviceScan::ExclusiveSum(scan_scratch, scan_tmp, blen, pl.pos_base, (int)na + 1, st));
    k_expand_rows<<<grid_of((long long)M + K, 8, sms * 8), 256, 0, st>>>(a_rpt, M, nnz_a, pl.arow, b_rpt, K, nnz_b,
                                                                         pl.brow, &h->info->d_cursor);
    OPS_CUDA(h, cudaGetLastError());
    if (nnz_a > 0)
        OPS_CUDA(h, cub::DeviceRadixSort::SortPairs(sort_scratch, sort_tmp, a_col, sorted_cols, iota, pl.at_ent,
                                                    (int)nnz_a, 0, std::max(1, ceil_log2(std::max(K, 2))), st));
    k_col_starts<<<grid_of(nnz_a + 1, 256, sms * 16), 256, 0, st>>>(sorted_cols, nnz_a, K, pl.at_ptr);
    OPS_CUDA(h, cudaGetLastError());
    if (nnz_b > 0) {
        k_list_long_b<<<grid_of(nnz_b, 256, sms * 16), 256, 0, st>>>(nnz_b, pl.brow, b_rpt, pl.at_ptr, pl.long_b,
                                                                     &h->info->d_cursor);
        OPS_CUDA(h, cudaGetLastError());
    }
    // one round trip for the three sizes (through pinned memory: a copy to pageable memory
    // waits for the stream)
    struct Sizes {
        long long products;
        int long_b_count, c_nnz;
    };
    static_assert(sizeof(Sizes) <= sizeof(DevInfo), "the handle's pinned record holds the sizes");
    Sizes *sizes = reinterpret_cast<Sizes *>(h->h_info);
    if (M > 0) OPS_CUDA(h, cudaMemcpyAsync(&sizes->c_nnz, c_rpt + M, sizeof(int), cudaMemcpyDeviceToHost, st));
    OPS_CUDA(h, cudaMemcpyAsync(&sizes->long_b_count, &h->info->d_cursor, sizeof(int), cudaMemcpyDeviceToHost, st));
    OPS_CUDA(h, cudaMemcpyAsync(&sizes->products, pl.pos_base + na - (nnz_a > 0 ? 0 : 1), sizeof(long long),
                                cudaMemcpyDeviceToHost, st));
    OPS_CUDA(h, cudaStreamSynchronize(st));
    const int c_nnz = M > 0 ? sizes->c_nnz : 0;
    const long long products = nnz_a > 0 ? sizes->products : 0;
    pl.long_b_count = sizes->long_b_count;
    pl.products = products;
    // blocks of rows for dB's gathers
    pl.blocks = (int)std::min<long long>(std::min<long long>(((long long)c_nnz + kGradBlock - 1) / kGradBlock, kGradBlocksMax),
                                         nnz_a / ((long long)std::max(K, 1) * kGradBlockMean));
    if (pl.blocks > 1 && nnz_b > 0) {
        const size_t pitch = align_up(4 * (size_t)K, 256);
        void *bp = nullptr;
        if (cudaMallocFromPoolAsync(&bp, pitch * (size_t)(pl.blocks - 1), h->pool, st) == cudaSuccess) {
            pl.at_blk = static_cast<int *>(bp);
            for (int b = 1; b < pl.blocks; ++b)
                k_column_block<<<grid_of(K, 256, sms * 8), 256, 0, st>>>(
                    K, pl.at_ptr, pl.at_ent, pl.arow, c_rpt, M, (int)((long long)c_nnz * b / pl.blocks),
                    pl.at_blk + (b - 1) * (pitch / 4));
            OPS_CUDA(h, cudaGetLastError());
        } else {
            (void)cudaGetLastError();  // no room: one block
            pl.blocks = 1;
        }
    }
    pl.with_map = products > 0 && products <= INT_MAX && (size_t)products * 4 <= h->map_budget;
    if (pl.with_map) {
        void *mp = nullptr;
        cudaError_t e = cudaMallocFromPoolAsync(&mp, (size_t)products * 4, h->pool, st);
        if (e == cudaSuccess) {
            pl.pmap = static_cast<int *>(mp);
            OPS_CUDA(h, cudaMemsetAsync(&h->info->flags, 0, sizeof(int), st));
            k_build_pmap<<<grid_of(M, 8, sms * 8), 256, 0, st>>>(a_rpt, a_col, b_rpt, b_col, M, c_rpt, c_col,
                                                                 pl.pos_base, pl.pmap, &h->info->flags);
            OPS_CUDA(h, cudaGetLastError());
        } else {
            (void)cudaGetLastError();
            pl.with_map = false;  // no room: search positions on every call instead
        }
    }
    if (nnz_a > 0) {
        const int g = grid_of(nnz_a, 256, sms * 16);
        if (pl.with_map) k_column_sources<true><<<g, 256, 0, st>>>(pl.at_ent, nnz_a, pl.pos_base, pl.arow, pl.at_src);
        else k_column_sources<false><<<g, 256, 0, st>>>(pl.at_ent, nnz_a, pl.pos_base, pl.arow, pl.at_src);
        OPS_CUDA(h, cudaGetLastError());
    }
    OPS_CUDA(h, cudaFreeAsync(tp, st));
    // a call on another stream waits for the plan first (settle_plan)
    if (!pl.ready) OPS_CUDA(h, cudaEventCreateWithFlags(&pl.ready, cudaEventDisableTiming));
    OPS_CUDA(h, cudaEventRecord(pl.ready, st));
    OPS_CUDA(h, cudaStreamGetId(st, &pl.stream));
    pl.settled = false;
    pl.M = M;
    pl.K = K;
    pl.N = N;
    pl.nnz_a = nnz_a;
    pl.nnz_b = nnz_b;
    pl.a_rpt = a_rpt;
    pl.a_col = a_col;
    pl.b_rpt = b_rpt;
    pl.b_col = b_col;
    pl.c_rpt = c_rpt;
    pl.c_col = c_col;
    pl.valid = true;
    return OPS_OK;
}

// Waits, once per plan, until the plan is complete where st does not run behind its kernels:
// another stream than theirs, or a captured one, whose graph may run on any.  The wait is
// allowed while st is captured, as the event lies outside the capture.
int settle_plan(ops_handle_s *h, cudaStream_t st)
{
    BackwardPlan &pl = h->bwd;
    if (pl.settled) return OPS_OK;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    OPS_CUDA(h, cudaStreamIsCapturing(st, &capture));
    if (capture == cudaStreamCaptureStatusNone) {
        unsigned long long id = 0;
        OPS_CUDA(h, cudaStreamGetId(st, &id));
        if (id == pl.stream) return OPS_OK;
    }
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    OPS_CUDA(h, cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t waited = cudaEventSynchronize(pl.ready);
    OPS_CUDA(h, cudaThreadExchangeStreamCaptureMode(&mode));
    OPS_CUDA(h, waited);
    pl.settled = true;
    return OPS_OK;
}

template <typename T>
int run_backward(ops_handle_s *h, int M, int K, const int *a_rpt, const int *a_col, const T *a_val,
                 const int *b_rpt, const int *b_col, const T *b_val, const int *c_rpt, const int *c_col, const T *dc,
                 T *da, T *db, cudaStream_t st)
{
    const BackwardPlan &pl = h->bwd;
    const int sms = h->num_sms;
    int *flags = &h->info->flags;
    if (da && pl.nnz_a > 0) {
        // thread per A entry for short chains; the long ones are listed and get a warp each.
        // The list and its length belong to the call: calls may overlap on several streams
        int *long_list = nullptr;
        OPS_CUDA(h, cudaMallocFromPoolAsync(reinterpret_cast<void **>(&long_list), sizeof(int) * (pl.nnz_a + 1),
                                            h->pool, st));
        int *long_count = long_list + pl.nnz_a;
        OPS_CUDA(h, cudaMemsetAsync(long_count, 0, sizeof(int), st));
        const int g1 = grid_of(pl.nnz_a, 256, sms * 16);
        if (pl.with_map) {
            k_grad_a_short<T, true><<<g1, 256, 0, st>>>(a_col, pl.nnz_a, pl.arow, b_rpt, b_col, b_val, c_rpt, c_col, dc,
                                                        pl.pos_base, pl.pmap, da, long_list, long_count, flags);
            k_grad_a_long<T, true><<<sms * 8, 256, 0, st>>>(a_col, pl.arow, b_rpt, b_col, b_val, c_rpt, c_col, dc,
                                                            pl.pos_base, pl.pmap, da, long_list, long_count, flags);
        } else {
            k_grad_a_short<T, false><<<g1, 256, 0, st>>>(a_col, pl.nnz_a, pl.arow, b_rpt, b_col, b_val, c_rpt, c_col,
                                                         dc, pl.pos_base, pl.pmap, da, long_list, long_count, flags);
            k_grad_a_long<T, false><<<sms * 8, 256, 0, st>>>(a_col, pl.arow, b_rpt, b_col, b_val, c_rpt, c_col, dc,
                                                             pl.pos_base, pl.pmap, da, long_list, long_count, flags);
        }
        OPS_CUDA(h, cudaGetLastError());
        OPS_CUDA(h, cudaFreeAsync(long_list, st));
    }
    if (db && pl.nnz_b > 0) {
        const int g1 = grid_of(pl.nnz_b, 256, sms * 16), g2 = grid_of(pl.long_b_count, 8, sms * 8);
        // dB's folds between blocks belong to the call as well; a captured call walks one
        // block, as its graph would keep them
        int blocks = pl.blocks;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        OPS_CUDA(h, cudaStreamIsCapturing(st, &capture));
        if (capture != cudaStreamCaptureStatusNone) blocks = 1;
        typename Acc<T>::S *state = nullptr;
        if (blocks > 1 && cudaMallocFromPoolAsync(reinterpret_cast<void **>(&state), sizeof(*state) * pl.nnz_b,
                                                  h->pool, st) != cudaSuccess) {
            (void)cudaGetLastError();  // no room: one block
            blocks = 1;
        }
        auto launch = [&](auto map) {
            constexpr bool kMap = decltype(map)::value;
            if (blocks <= 1)
                k_grad_b_short<T, kMap, false><<<g1, 256, 0, st>>>(pl.nnz_b, pl.brow, b_rpt, b_col, a_val, pl.at_ptr,
                                                                   pl.at_ent, pl.at_src, c_rpt, c_col, dc, pl.pmap, db,
                                                                   flags, nullptr, nullptr, state, true, true);
            for (int b = 0; b < blocks && blocks > 1; ++b) {
                const size_t pitch = align_up(4 * (size_t)K, 256) / 4;
                const bool first = b == 0, last = b == blocks - 1;
                k_grad_b_short<T, kMap, true><<<g1, 256, 0, st>>>(
                    pl.nnz_b, pl.brow, b_rpt, b_col, a_val, pl.at_ptr, pl.at_ent, pl.at_src, c_rpt, c_col, dc, pl.pmap,
                    db, flags, first ? pl.at_ptr : pl.at_blk + (b - 1) * pitch,
                    last ? pl.at_ptr + 1 : pl.at_blk + b * pitch, state, first, last);
            }
            if (pl.long_b_count > 0)
                k_grad_b_long<T, kMap><<<g2, 256, 0, st>>>(pl.long_b, pl.long_b_count, pl.nnz_b, pl.brow, b_rpt, b_col,
                                                           a_val, pl.at_ptr, pl.at_ent, pl.at_src, c_rpt, c_col, dc,
                                                           pl.pmap, db, flags);
        };
        if (pl.with_map) launch(std::true_type{});
        else launch(std::false_type{});
        const cudaError_t launched = cudaGetLastError();
        if (blocks > 1) OPS_CUDA(h, cudaFreeAsync(state, st));
        OPS_CUDA(h, launched);
    }
    return OPS_OK;
}

}  // namespace

extern "C" int ops_spgemm_backward(ops_handle_t h, int dtype, int32_t rows_a, int32_t cols_a, int32_t cols_b,
                                   const int32_t *a_rpt, const int32_t *a_col, const void *a_val, int64_t a_nnz,
                                   const int32_t *b_rpt, const int32_t *b_col, const void *b_val, int64_t b_nnz,
                                   const int32_t *c_rpt, const int32_t *c_col, const void *dc_val, void *da_val,
                                   void *db_val, void *stream)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    if (dtype != OPS_F64 && dtype != OPS_F32) return fail(h, OPS_INVALID_ARGUMENT, "unknown dtype");
    if (rows_a < 0 || cols_a < 0 || cols_b < 0 || a_nnz < 0 || b_nnz < 0 || a_nnz > INT_MAX || b_nnz > INT_MAX)
        return fail(h, OPS_INVALID_ARGUMENT, "bad matrix sizes");
    if ((rows_a > 0 && (!a_rpt || !c_rpt)) || (cols_a > 0 && !b_rpt) || (a_nnz > 0 && (!a_col || !a_val)) ||
        (b_nnz > 0 && (!b_col || !b_val)) || !dc_val)
        return fail(h, OPS_INVALID_ARGUMENT, "null input");
    try {
        h->last_error.clear();
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        if (!h->info) {  // the handle has not run a forward yet: create its workspace
            void *p = nullptr;
            OPS_CUDA(h, cudaMallocFromPoolAsync(&p, 256, h->pool, st));
            h->ws = static_cast<unsigned char *>(p);
            h->ws_M = 0;
            h->info = reinterpret_cast<DevInfo *>(h->ws);
        }
        OPS_CHECK(build_plan(h, rows_a, cols_a, cols_b, a_rpt, a_col, a_nnz, b_rpt, b_col, b_nnz, c_rpt, c_col, st));
        OPS_CHECK(settle_plan(h, st));
        OPS_CUDA(h, cudaMemsetAsync(&h->info->flags, 0, sizeof(int), st));
        int s;
        if (dtype == OPS_F64)
            s = run_backward<double>(h, rows_a, cols_a, a_rpt, a_col, static_cast<const double *>(a_val), b_rpt, b_col,
                                     static_cast<const double *>(b_val), c_rpt, c_col,
                                     static_cast<const double *>(dc_val), static_cast<double *>(da_val),
                                     static_cast<double *>(db_val), st);
        else
            s = run_backward<float>(h, rows_a, cols_a, a_rpt, a_col, static_cast<const float *>(a_val), b_rpt, b_col,
                                    static_cast<const float *>(b_val), c_rpt, c_col, static_cast<const float *>(dc_val),
                                    static_cast<float *>(da_val), static_cast<float *>(db_val), st);
        return s;
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm_backward");
    }
}

extern "C" int ops_handle_set_map_budget(ops_handle_t h, size_t bytes)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    h->map_budget = bytes;
    h->bwd.valid = false;
    return OPS_OK;
}

extern "C" int ops_backward_plan_info(ops_handle_t h, int64_t *products, int *with_map)
{
    if (!h || !products || !with_map) return OPS_INVALID_ARGUMENT;
    *products = h->bwd.valid ? h->bwd.products : 0;
    *with_map = h->bwd.valid && h->bwd.with_map ? 1 : 0;
    return OPS_OK;
}
