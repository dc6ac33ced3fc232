// spgemm.cu — handle, pipeline and C ABI of the GB300 SpGEMM library.
//
// Pipeline of one C = A*B (compare src/opsparse/core_algo/spgemm/spgemm.cu:16-62 and
// spgemm_phases.cu:12-206 of OpSparse):
//   1. k_setup: product count per row + class lists             (one kernel, no host sync
//      between count and scatter, unlike h_symbolic_binning's D2H/H2D round trip)
//   2. read back class sizes and max products                   (host sync #1)
//   3. symbolic kernels, one stream per non-empty class, joined back onto the caller's
//      stream with events                                       (multi-stream bin dispatch)
//   4. exclusive scan of row nnz into C.row_ptr (one CTA for few rows, else CUB)
//   5. read back nnz(C)                                         (host sync #2)
//   6. C allocated from the handle's stream-ordered pool
//   7. numeric kernels on the same per-class streams, reusing step 1's classes
// Small problems take one kernel per phase instead of step 3's and 7's classes (small_problem);
// rows on structured grids are grouped by pattern between steps 2 and 3 (form_groups).
// Workspace (class lists, counters, scan scratch, dense-row scratch) lives in a
// cudaMemPool owned by the handle and is reused across calls; streams and events are
// created once per handle, never per call.
#include <cub/cub.cuh>

#include <algorithm>
#include <array>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>

#include "regular.cuh"
#include "internal.hpp"
#include "opsparse_gb300.h"

using namespace opsg;
using namespace opsg_internal;

namespace {

const char *kVersion = "opsparse_gb300 0.2 (sm_103a)";
constexpr int kBatchWarpMaxLo = 128;   // range of ops_tuning.batch_warp_max
constexpr int kBatchWarpMaxHi = 512;

struct Mat {
    int rows, cols;
    const int *rpt, *col;
    const void *val;
    long long nnz = -1;  // -1: not known
};

template <typename Sh, typename T>
void set_rank_attrs()
{
    cudaFuncSetAttribute(k_rank_rows<Sh, true, T, Sh::kCap == RankE1::kCap>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Sh::template smem<true>());
    cudaFuncSetAttribute(k_rank_rows<Sh, false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Sh::template smem<false>());
}

// Launch the rank kernel of shape Sh for at most n listed rows (the exact count is on the
// device).  The E1 shape counts its rows by late products.
template <typename Sh, bool kNum, typename T>
void launch_rank(ops_handle_s *h, const SpgemmArgs<T> &g, const int *list, const int *count_ptr, int *cursor, int n,
                 cudaStream_t s)
{
    if (n <= 0) return;
    // one wave of CTAs that stay until the list is empty, or beside D rows as many as take
    // rank_rows_per_group rows each
    constexpr int by_smem = (int)(227 * 1024 / (Sh::template smem<kNum>() + 1024));
    constexpr int ctas = by_smem < Sh::kMinBlocks ? by_smem : Sh::kMinBlocks;
    static_assert(ctas >= 1, "a CTA fits an SM");
    constexpr int per_cta = Sh::kGroups * rank_rows_per_group<Sh>();
    const int wave = std::min((n + Sh::kGroups - 1) / Sh::kGroups, h->num_sms * ctas);
    const bool beside_d = h->counts[kClsD] > 0;
    const int grid = beside_d ? std::max(wave, (n + per_cta - 1) / per_cta) : wave;
    k_rank_rows<Sh, kNum, T, kNum && Sh::kCap == RankE1::kCap><<<grid, Sh::kThreads, Sh::template smem<kNum>(), s>>>(
        g, list, count_ptr, cursor, beside_d ? rank_rows_per_group<Sh>() : INT_MAX);
    ++h->launches;
}

template <typename T>
void set_smem_attrs()
{
    cudaFuncSetAttribute(k_warp_rows<true, T, 2 * kSplitNnz>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_rows_smem<true, T, 2 * kSplitNnz>());
    cudaFuncSetAttribute(k_warp_rows<false, T, 2 * kEsc1FlopMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_rows_smem<false, T, 2 * kEsc1FlopMax>());
    set_rank_attrs<RankW, T>();
    set_rank_attrs<RankS, T>();
    set_rank_attrs<RankM, T>();
    set_rank_attrs<RankE1, T>();
    set_rank_attrs<RankMid, T>();
    set_rank_attrs<RankLarge, T>();
    cudaFuncSetAttribute(k_rank_all<true, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RankS::smem<true>());
    cudaFuncSetAttribute(k_rank_all<false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RankS::smem<false>());
    cudaFuncSetAttribute(k_group_rows<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmem<T>));
}

int ensure_ws(ops_handle_s *h, int M, cudaStream_t st)
{
    if (h->ws && h->ws_M >= M) return OPS_OK;
    size_t cub_bytes = 0;
    OPS_CUDA(h, cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, (int *)nullptr, (int *)nullptr, M + 1, st));
    // one list per class and the extra lists of re-binned classes
    const size_t lists_b = align_up(sizeof(int) * (size_t)(kNumLists) * (size_t)M, 256);
    const size_t flop_b = align_up(sizeof(int) * (size_t)M, 256);
    const size_t soff_b = align_up(sizeof(int) * ((size_t)M + 1), 256);
    const size_t info_b = align_up(sizeof(DevInfo), 256);
    const size_t link_b = align_up((size_t)M, 256);
    const size_t groups_b = align_up(sizeof(int2) * ((size_t)M / kGroupMin + 64), 256);
    const size_t total = lists_b + flop_b + soff_b + info_b + link_b + groups_b + align_up(cub_bytes, 256);
    if (h->ws) {
        OPS_CUDA(h, cudaFreeAsync(h->ws, st));
        h->ws = nullptr;
    }
    void *p = nullptr;
    OPS_CUDA(h, cudaMallocFromPoolAsync(&p, total, h->pool, st));
    h->ws = static_cast<unsigned char *>(p);
    h->ws_bytes = total;
    h->ws_M = M;
    h->lists = reinterpret_cast<int *>(h->ws);
    h->row_flop = reinterpret_cast<int *>(h->ws + lists_b);
    h->soff = reinterpret_cast<int *>(h->ws + lists_b + flop_b);
    h->info = reinterpret_cast<DevInfo *>(h->ws + lists_b + flop_b + soff_b);
    h->link = h->ws + lists_b + flop_b + soff_b + info_b;
    h->groups = reinterpret_cast<int2 *>(h->ws + lists_b + flop_b + soff_b + info_b + link_b);
    h->cub_tmp = h->ws + lists_b + flop_b + soff_b + info_b + link_b + groups_b;
    h->cub_bytes = cub_bytes;
    h->plan_valid = false;
    return OPS_OK;
}

// Region ends of the dense-row scratch for `ctas` CTAs: [vals | bits | tot | cnt | pos],
// each region 256-byte aligned.
std::array<size_t, 5> dense_offsets(int N, int ctas)
{
    const size_t n = (size_t)N * (size_t)ctas, words = (size_t)(N + 31) / 32 * (size_t)ctas;
    std::array<size_t, 5> o{};
    o[0] = align_up(n * 8, 256);
    o[1] = o[0] + align_up(words * 4, 256);
    o[2] = o[1] + align_up(n * 8, 256);
    o[3] = o[2] + align_up(n * 4, 256);
    o[4] = o[3] + align_up(n * 4, 256);
    return o;
}

// Dense-row scratch: per CTA, N accumulator slots (8 bytes), ceil(N/32) bitmap words, and
// for entries folded in blocks N merged-block slots (8 bytes), N product counts and N
// positions (4 bytes each).
int ensure_dense(ops_handle_s *h, int N, int rows, cudaStream_t st)
{
    const size_t words = (size_t)(N + 31) / 32;
    const size_t per_cta = (size_t)N * 24 + words * 4;
    int ctas = std::min(rows, 2 * h->num_sms);
    const size_t by_budget = per_cta ? h->dense_budget / per_cta : (size_t)ctas;
    ctas = (int)std::max<size_t>(1, std::min<size_t>((size_t)ctas, by_budget));
    const size_t need = dense_offsets(N, ctas)[4] + 256;
    if (need > h->dense_bytes) {
        if (h->dense) {
            OPS_CUDA(h, cudaFreeAsync(h->dense, st));
            h->dense = nullptr;
            h->dense_bytes = 0;
        }
        void *p = nullptr;
        OPS_CUDA(h, cudaMallocFromPoolAsync(&p, need, h->pool, st));
        OPS_CUDA(h, cudaMemsetAsync(p, 0, need, st));
        h->dense = static_cast<unsigned char *>(p);
        h->dense_bytes = need;
    }
    h->dense_ctas = ctas;
    return OPS_OK;
}

template <typename T>
DenseScratch<T> dense_view(ops_handle_s *h, int N)
{
    const std::array<size_t, 5> o = dense_offsets(N, h->dense_ctas);
    DenseScratch<T> d;
    d.words = (N + 31) / 32;
    d.vals = reinterpret_cast<typename Acc<T>::S *>(h->dense);
    d.bits = reinterpret_cast<unsigned *>(h->dense + o[0]);
    d.tot = reinterpret_cast<typename Acc<T>::S *>(h->dense + o[1]);
    d.cnt = reinterpret_cast<int *>(h->dense + o[2]);
    d.pos = reinterpret_cast<int *>(h->dense + o[3]);
    return d;
}

int grid_for(long long work_items, int per_block, int cap)
{
    long long b = (work_items + per_block - 1) / per_block;
    return (int)std::max<long long>(1, std::min<long long>(b, cap));
}

// Row pointers of C (or staging offsets) from counts, in place: x[0, M] -> exclusive prefix.
// small: the counts of a small problem, complete only if no row is beyond it.
int scan_rows(ops_handle_s *h, int *x, int M, cudaStream_t st, bool small = false)
{
    if (M + 1 <= kScanMax) {
        k_scan_rows<<<1, 1024, 0, st>>>(x, M + 1, small ? h->info : nullptr);
        OPS_CUDA(h, cudaGetLastError());
    } else {
        size_t cb = h->cub_bytes;
        OPS_CUDA(h, cub::DeviceScan::ExclusiveSum(h->cub_tmp, cb, x, x, M + 1, st));
    }
    ++h->launches;
    return OPS_OK;
}

// Classes whose rows a one-pass call computes in the counting phase: all but R8 (counted
// by k_setup; their numeric writes C directly in the second phase, next to the copy of the
// staged rows), D only if its whole-GPU sort fits the scratch budget, and E1 only if some
// E1 row is staged (not a column-window row; the split is made on the device, and without
// such rows the E1 class keeps its own list and two passes).
bool staged_class(const ops_handle_s *h, int c)
{
    return c != kClsR8 && (c != kClsD || h->stage_d) && (c != kClsE1 || h->stage_e1);
}

// Below this many staged products the set-up of a one-pass call (the offset scan, the
// copy into C) costs more than the counting kernels it saves.
constexpr unsigned long long kMinStageFlop = 1ull << 20;

// Values region of the staging area (after the columns of staged_flop entries).
template <typename T>
T *stage_vals(ops_handle_s *h)
{
    return reinterpret_cast<T *>(h->stage + align_up(sizeof(int) * (size_t)h->stage_entries, 256));
}

// Counting phase of a one-pass call: class c's numeric kernels write its rows' entries
// to the staging area at soff[r] and their counts to c_rpt, in place of the counting
// kernels.  The E1 rows it does not stage are counted as usual.
template <typename T, typename GA>
int launch_staged_class(ops_handle_s *h, const GA &gs, int c, const int *list, const int *count, int n, cudaStream_t s)
{
    SpgemmArgs<T> g{};
    g.arpt = gs.arpt;
    g.acol = gs.acol;
    g.aval = static_cast<const T *>(h->op_aval);
    g.brpt = gs.brpt;
    g.bcol = gs.bcol;
    g.bval = static_cast<const T *>(h->op_bval);
    g.M = gs.M;
    g.K = gs.K;
    g.N = gs.N;
    g.row_flop = gs.row_flop;
    g.c_rpt = gs.c_rpt;
    g.info = gs.info;
    g.soff = h->soff;
    g.c_col = reinterpret_cast<int *>(h->stage);
    g.c_val = stage_vals<T>(h);
    const int sms = h->num_sms;
    const size_t M = (size_t)h->plan_M;
    int *xl = h->lists + (size_t)kNumClasses * M;
    switch (c) {
        case kClsR16:
            k_reg_rows<16, true, T><<<grid_for((n + 1) / 2, 8, sms * 8), 256, 0, s>>>(g, list, n);
            break;
        case kClsR32:
            k_reg_rows<32, true, T><<<grid_for(n, 8, sms * 8), 256, 0, s>>>(g, list, n);
            break;
        case kClsW:
            launch_rank<RankW, true, T>(h, g, list, &h->info->counts[c], nullptr, n, s);
            break;
        case kClsE1: {
            // the staged rows (not column-window rows) into the staging area by rank shape,
            // the larger shapes on an extra stream; the rest counted by the warp hash
            int *one = xl + kXlE1One * M;
            int *two = xl + kXlE1Two * M;
            int *one_large = xl + kXlE1OneLarge * M;
            int *one_half = xl + kXlE1OneHalf * M;
            k_split_list<4, PickStaged><<<grid_for(n, 256, sms * 4), 256, 0, s>>>(
                list, count, PickStaged{h->soff, g.row_flop, g.arpt}, one, (int)M, h->info->split1);
            OPS_CUDA(h, cudaGetLastError());
            ++h->launches;
            OPS_CUDA(h, cudaEventRecord(h->ev_x_fork[0], s));
            OPS_CUDA(h, cudaStreamWaitEvent(h->side_x[0], h->ev_x_fork[0], 0));
            launch_rank<RankE1, true, T>(h, g, one_large, &h->info->split1[2], &h->info->next_sym.e1, h->e1_size[2],
                                         h->side_x[0]);
            launch_rank<RankM, true, T>(h, g, one_half, &h->info->split1[3], &h->info->next_sym.e1_half, h->e1_size[1],
                                        h->side_x[0]);
            OPS_CUDA(h, cudaGetLastError());
            SpgemmArgs<double> gc{};
            gc.arpt = g.arpt;
            gc.acol = g.acol;
            gc.brpt = g.brpt;
            gc.bcol = g.bcol;
            gc.M = g.M;
            gc.K = g.K;
            gc.N = g.N;
            gc.row_flop = g.row_flop;
            gc.c_rpt = g.c_rpt;
            gc.info = g.info;
            if (!h->stage_e1_all) {
                k_warp_rows<false, double, 2 * kEsc1FlopMax>
                    <<<grid_for(n, kWarpRowsThreads / 32, sms * 3), kWarpRowsThreads,
                       warp_rows_smem<false, double, 2 * kEsc1FlopMax>(), h->side_x[0]>>>(gc, two, &h->info->split1[1]);
                OPS_CUDA(h, cudaGetLastError());
                ++h->launches;
            }
            OPS_CUDA(h, cudaEventRecord(h->ev_x_join[0], h->side_x[0]));
            launch_rank<RankS, true, T>(h, g, one, &h->info->split1[0], nullptr, h->e1_size[0], s);
            OPS_CUDA(h, cudaGetLastError());
            OPS_CUDA(h, cudaStreamWaitEvent(s, h->ev_x_join[0], 0));
            break;
        }
        case kClsE2: {
            // the counting phase's split and longest-first orders, then both numeric shapes
            int *mid_list = xl + kXlE2Mid * M;
            int *large_list = xl + kXlE2Large * M;
            k_split_list<2, PickE2><<<grid_for(n, 256, sms * 4), 256, 0, s>>>(
                list, &h->info->counts[c], PickE2{g.arpt, g.row_flop}, mid_list, (int)M, h->info->split2);
            OPS_CUDA(h, cudaGetLastError());
            ++h->launches;
            OPS_CUDA(h, cudaEventRecord(h->ev_x_fork[1], s));
            OPS_CUDA(h, cudaStreamWaitEvent(h->side_x[1], h->ev_x_fork[1], 0));
            if (h->e2_size[1] > 1) {
                k_sort_heavy_first<<<1, 1024, 0, h->side_x[1]>>>(large_list, &h->info->split2[1], h->row_flop);
                OPS_CUDA(h, cudaGetLastError());
                ++h->launches;
            }
            launch_rank<RankLarge, true, T>(h, g, large_list, &h->info->split2[1], &h->info->next_sym.large,
                                            h->e2_size[1], h->side_x[1]);
            OPS_CUDA(h, cudaGetLastError());
            OPS_CUDA(h, cudaEventRecord(h->ev_x_join[1], h->side_x[1]));
            if (h->e2_size[0] > 1) {
                k_sort_heavy_first<<<1, 1024, 0, s>>>(mid_list, &h->info->split2[0], h->row_flop);
                OPS_CUDA(h, cudaGetLastError());
                ++h->launches;
            }
            launch_rank<RankMid, true, T>(h, g, mid_list, &h->info->split2[0], &h->info->next_sym.mid, h->e2_size[0], s);
            OPS_CUDA(h, cudaGetLastError());
            OPS_CUDA(h, cudaStreamWaitEvent(s, h->ev_x_join[1], 0));
            break;
        }
        case kClsD: {  // whole-GPU expand/sort/compress, counts from its head scan
            const int st_d = run_d_rows<T>(h, g, list, n, true, s);
            if (st_d != OPS_OK) return st_d == OPS_NOT_SUPPORTED ? fail(h, OPS_CUDA_ERROR, "D-row scratch changed") : st_d;
            h->d_rows_path[0] = n;
            h->d_rows_path[1] = 0;
            break;
        }
        default:
            return fail(h, OPS_NOT_SUPPORTED, "class without a one-pass kernel");
    }
    return OPS_OK;
}

// Rows that the next row of A repeats from which the groups' five extra launches (about 35 us
// of a two-phase call) pay: 27-point operators of a 27^3 grid (17,000 such rows) 255 us
// grouped against 242, of 30^3 (25,000) 276 against 345.  Short runs do not: k_setup counts
// them cut at every 32 rows, where runs of 28 rows average 14 and of 17 rows 11.
constexpr int kMinChainRows = 20480;
constexpr int kMinChainRun = 14;

// Groups of rows of one pattern (regular.cuh), where k_setup found enough E1 rows that A's
// next row repeats: links from B, groups, and the E1 rows outside them (h->regular).  In a
// call that may stage (want_stage), hi's staged rows and products are those outside the groups
// afterwards: rows of a wider span than the column window would have been staged, and their
// number decides whether the E1 class still has a numeric phase.  They are read back where
// there may be any (one round trip, about 10 us of calls of a millisecond and more).
int form_groups(ops_handle_s *h, DevInfo &hi, const Mat &A, const Mat &B, bool want_stage, cudaStream_t st)
{
    h->regular = false;
    if (hi.e1_chain < kMinChainRows || hi.e1_chain < kMinChainRun * hi.e1_runs) return OPS_OK;
    const int M = A.rows, K = A.cols;
    if (h->b_link_rows < K) {
        if (h->b_link) OPS_CUDA(h, cudaFreeAsync(h->b_link, st));
        h->b_link = nullptr;
        h->b_link_rows = 0;
        void *p = nullptr;
        OPS_CUDA(h, cudaMallocFromPoolAsync(&p, (size_t)K, h->pool, st));
        h->b_link = static_cast<unsigned char *>(p);
        h->b_link_rows = K;
    }
    const int sms = h->num_sms;
    const bool unstage = want_stage && hi.e1_one > 0;  // else no row stages: no sizes to look at
    k_shift_links<<<grid_for(K, 32, sms * 16), 256, 0, st>>>(B.rpt, B.col, K, B.cols, h->b_link);
    k_row_links<<<grid_for(M, 32, sms * 16), 256, 0, st>>>(A.rpt, A.col, B.rpt, M, h->b_link, h->link);
    k_form_groups<<<(M + 4 * kGroupWindow - 1) / (4 * kGroupWindow), 128, 0, st>>>(
        M, h->link, h->groups, unstage ? h->soff : nullptr, h->info);
    OPS_CUDA(h, cudaGetLastError());
    h->launches += 3;
    h->regular = true;
    if (unstage) {
        OPS_CUDA(h, cudaMemcpyAsync(h->h_info, h->info, sizeof(DevInfo), cudaMemcpyDeviceToHost, st));
        OPS_CUDA(h, cudaStreamSynchronize(st));
        hi.staged_flop = h->h_info->staged_flop;
        hi.e1_one = h->h_info->e1_one;
    }
    return OPS_OK;
}

// One-pass set-up, once the class sizes are known: when the call has its values, one
// pass is on and the staged products fit the handle's staging budget, grows the staging
// area and turns the per-row product counts (k_setup's sflop) into staging offsets.
// Otherwise leaves h->staged false: two passes.
int prepare_stage(ops_handle_s *h, const DevInfo &hi, int M, cudaStream_t st)
{
    h->staged = false;
    const int vs = h->op_dtype == OPS_F64 ? 8 : (h->op_dtype == OPS_F32 ? 4 : 0);
    if (!h->one_pass || vs == 0 || M == 0 || hi.staged_flop == 0) return OPS_OK;
    if (h->one_pass == 1 && hi.staged_flop < kMinStageFlop) return OPS_OK;
    const unsigned long long entries = hi.staged_flop;
    const size_t total = align_up(sizeof(int) * (size_t)entries, 256) + align_up((size_t)vs * (size_t)entries, 256);
    if (entries > (unsigned long long)INT_MAX || total > h->stage_budget) return OPS_OK;
    if (total > h->stage_bytes) {
        if (h->stage) OPS_CUDA(h, cudaFreeAsync(h->stage, st));
        h->stage = nullptr;
        h->stage_bytes = 0;
        void *p = nullptr;
        if (cudaMallocFromPoolAsync(&p, total, h->pool, st) != cudaSuccess) {  // two passes instead
            (void)cudaGetLastError();
            return OPS_OK;
        }
        h->stage = static_cast<unsigned char *>(p);
        h->stage_bytes = total;
    }
    h->stage_entries = (long long)entries;
    // D rows are staged only if their whole-GPU sort fits the scratch budget (else they keep
    // two passes and the dense-row kernel may take them)
    h->stage_d = false;
    if (hi.counts[kClsD] > 0) {
        SpgemmArgs<double> gd{};
        gd.N = h->plan_N;
        gd.soff = h->soff;
        h->stage_d = run_d_rows<double>(h, gd, nullptr, hi.counts[kClsD], true, st, true) == OPS_OK;
        h->last_error.clear();
        if (!h->stage_d) {
            k_unstage_rows<<<grid_for(hi.counts[kClsD], 256, h->num_sms * 4), 256, 0, st>>>(
                h->lists + (size_t)kClsD * M, &h->info->counts[kClsD], h->soff);
            OPS_CUDA(h, cudaGetLastError());
            ++h->launches;
        }
    }
    OPS_CHECK(scan_rows(h, h->soff, M, st));
    h->staged = true;
    h->stage_e1 = hi.e1_one > 0;
    h->stage_e1_all = hi.e1_one == hi.counts[kClsE1];
    return OPS_OK;
}

// The groups' counts (symbolic; one row of each is counted) or entries (numeric).
template <bool kNum, typename T>
int launch_groups(ops_handle_s *h, const SpgemmArgs<T> &g, int rows, cudaStream_t s)
{
    const int most = rows / kGroupMin + 1;
    if constexpr (kNum) {
        k_group_rows<T><<<std::min(most, h->num_sms * kGroupCtas), kGroupThreads, sizeof(GroupSmem<T>), s>>>(
            g, h->groups, &h->info->next_num.group);
    } else {
        SpgemmArgs<double> gc{};
        gc.arpt = g.arpt;
        gc.acol = g.acol;
        gc.brpt = g.brpt;
        gc.bcol = g.bcol;
        gc.M = g.M;
        gc.K = g.K;
        gc.N = g.N;
        gc.row_flop = g.row_flop;
        gc.c_rpt = g.c_rpt;
        gc.info = g.info;
        k_group_count<<<std::min(most, h->num_sms * RankE1::kMinBlocks), RankE1::kThreads, RankE1::smem<false>(), s>>>(
            gc, h->groups);
    }
    OPS_CUDA(h, cudaGetLastError());
    ++h->launches;
    return OPS_OK;
}

// Launch the kernels of every non-empty class, each on its own stream forked from `st`
// and joined back into it.  A re-binned class (E1 numeric, E2) first splits its list on
// the device and runs its second kernel on an extra stream forked from the class stream;
// the class stream joins it again, so the class's events span both kernels.
template <bool kNum, typename T>
int launch_classes(ops_handle_s *h, const SpgemmArgs<T> &g, cudaStream_t st)
{
    OPS_CUDA(h, cudaEventRecord(h->ev_fork, st));
    const int sms = h->num_sms;
    const size_t M = (size_t)h->plan_M;
    int *xl = h->lists + (size_t)kNumClasses * M;  // extra lists
    auto fork_x = [&](int x, cudaStream_t from) -> cudaStream_t {
        if (cudaEventRecord(h->ev_x_fork[x], from) != cudaSuccess) return nullptr;
        if (cudaStreamWaitEvent(h->side_x[x], h->ev_x_fork[x], 0) != cudaSuccess) return nullptr;
        return h->side_x[x];
    };
    auto join_x = [&](int x, cudaStream_t into) -> bool {
        return cudaEventRecord(h->ev_x_join[x], h->side_x[x]) == cudaSuccess &&
               cudaStreamWaitEvent(into, h->ev_x_join[x], 0) == cudaSuccess;
    };
    // heaviest classes first: their long kernels then overlap the light classes instead
    // of forming the tail of the phase
    constexpr int kOrder[kNumClasses] = {kClsE2, kClsD, kClsE1, kClsW, kClsR32, kClsR16, kClsR8};
    if (kNum && h->staged) {
        // one-pass call: the rows computed in the counting phase move from the staging
        // area into C, on the caller's stream while the remaining classes run on theirs
        const long long ranges = (h->plan_nnz + kPlaceRange - 1) / kPlaceRange;
        k_place_staged<T><<<grid_for(ranges, 8, sms * 8), 256, 0, st>>>(
            g.M, h->soff, g.c_rpt, reinterpret_cast<const int *>(h->stage), stage_vals<T>(h), g.c_col, g.c_val);
        OPS_CUDA(h, cudaGetLastError());
        ++h->launches;
    }
    for (int oi = 0; oi < kNumClasses; ++oi) {
        const int c = kOrder[oi];
        const int n = h->counts[c];
        if (n <= 0) continue;
        const bool staged = h->staged && staged_class(h, c);
        // R8 rows are counted inside k_setup; staged classes are done after the counting
        // phase, except the E1 rows left to two passes
        if (!kNum && c == kClsR8) continue;
        if (kNum && staged && (c != kClsE1 || h->stage_e1_all)) continue;
        cudaStream_t s = h->side[c];
        OPS_CUDA(h, cudaStreamWaitEvent(s, h->ev_fork, 0));
        const int *list = h->lists + (size_t)c * M;
        if (!kNum && c == kClsD && n > 1 && n <= kLptMax) {
            // longest rows first; the numeric phase reuses the ordered list
            k_sort_heavy_first<<<1, 1024, 0, s>>>(h->lists + (size_t)c * M, &h->info->counts[c], h->row_flop);
            OPS_CUDA(h, cudaGetLastError());
            ++h->launches;
        }
        if (h->timing >= 2) OPS_CUDA(h, cudaEventRecord(h->ev_k[kNum][c][0], s));
        const int *count = &h->info->counts[c];
        if (c == kClsE1 && h->regular) {
            // the groups of one pattern, then the other rows: a list of their own, made while
            // counting and kept for every numeric phase of the plan, whatever was staged
            if (!(kNum && h->no_groups)) OPS_CHECK((launch_groups<kNum, T>(h, g, n, s)));
            int *rest = xl + kXlE1Rest * M;
            if (!kNum) {
                k_split_list<1, PickUngrouped><<<grid_for(n, 256, sms * 4), 256, 0, s>>>(
                    list, count, PickUngrouped{h->link}, rest, (int)M, &h->info->e1_rest);
                OPS_CUDA(h, cudaGetLastError());
                ++h->launches;
            }
            list = rest;
            count = &h->info->e1_rest;
        }
        if (staged && !kNum) {  // one-pass call: numeric into the staging area
            OPS_CHECK(h->op_dtype == OPS_F64 ? launch_staged_class<double>(h, g, c, list, count, n, s)
                                             : launch_staged_class<float>(h, g, c, list, count, n, s));
        } else
        switch (c) {
            case kClsR8:  // numeric only: walks the rows in order
                k_small_rows<T><<<grid_for(g.M, kSmallThreads, sms * 8), kSmallThreads, 0, s>>>(g, h->plan_th.r8);
                break;
            case kClsR16:
                k_reg_rows<16, kNum, T><<<grid_for((n + 1) / 2, 8, sms * 8), 256, 0, s>>>(g, list, n);
                break;
            case kClsR32:
                k_reg_rows<32, kNum, T><<<grid_for(n, 8, sms * 8), 256, 0, s>>>(g, list, n);
                break;
            case kClsW:
                launch_rank<RankW, kNum, T>(h, g, list, &h->info->counts[c], nullptr, n, s);
                break;
            case kClsE1: {
                if (!kNum) {  // distinct-column count: one warp per row, table of 2*flop slots
                    k_warp_rows<false, T, 2 * kEsc1FlopMax>
                        <<<grid_for(n, kWarpRowsThreads / 32, sms * 3), kWarpRowsThreads,
                           warp_rows_smem<false, T, 2 * kEsc1FlopMax>(), s>>>(g, list, count);
                    break;
                }
                // re-bin by output size: the warp's rank shape and warp hash on this stream,
                // the larger rank shapes on an extra stream (a one-pass call re-bins only
                // the rows it left to two passes)
                int *small_list = xl + kXlE1Small * M;
                int *half_list = xl + kXlE1Half * M;
                int *hash_list = xl + kXlE1Hash * M;
                int *rank_list = xl + kXlE1Rank * M;
                const int *e1_list = staged ? xl + kXlE1Two * M : list;
                const int *e1_count = staged ? &h->info->split1[1] : count;
                k_split_list<4, PickE1><<<grid_for(n, 256, sms * 4), 256, 0, s>>>(
                    e1_list, e1_count, PickE1{g.c_rpt, g.row_flop, g.arpt}, small_list, (int)M, h->info->split);
                OPS_CUDA(h, cudaGetLastError());
                ++h->launches;
                cudaStream_t sx = fork_x(0, s);
                if (!sx) return fail(h, OPS_CUDA_ERROR, "stream fork failed");
                launch_rank<RankE1, true, T>(h, g, rank_list, &h->info->split[2], &h->info->next_num.e1, h->e1_size[2],
                                             sx);
                launch_rank<RankM, true, T>(h, g, half_list, &h->info->split[3], &h->info->next_num.e1_half,
                                            h->e1_size[1], sx);
                OPS_CUDA(h, cudaGetLastError());
                if (!join_x(0, s)) return fail(h, OPS_CUDA_ERROR, "stream join failed");
                launch_rank<RankS, true, T>(h, g, small_list, &h->info->split[0], nullptr, h->e1_size[0], s);
                OPS_CUDA(h, cudaGetLastError());
                k_warp_rows<true, T, 2 * kSplitNnz>
                    <<<grid_for(n, kWarpRowsThreads / 32, sms * 4), kWarpRowsThreads,
                       warp_rows_smem<true, T, 2 * kSplitNnz>(), s>>>(g, hash_list, &h->info->split[1]);
                break;
            }
            case kClsE2: {
                // mid shape on this stream, large shape (one CTA per SM) on an extra stream;
                // the split and the longest-first order are made once, by the symbolic
                // phase, and reused by numeric
                int *mid_list = xl + kXlE2Mid * M;
                int *large_list = xl + kXlE2Large * M;
                if (!kNum) {
                    k_split_list<2, PickE2><<<grid_for(n, 256, sms * 4), 256, 0, s>>>(
                        list, &h->info->counts[c], PickE2{g.arpt, g.row_flop}, mid_list, (int)M, h->info->split2);
                    OPS_CUDA(h, cudaGetLastError());
                    ++h->launches;
                }
                cudaStream_t sx = fork_x(1, s);
                if (!sx) return fail(h, OPS_CUDA_ERROR, "stream fork failed");
                if (!kNum && h->e2_size[1] > 1) {
                    k_sort_heavy_first<<<1, 1024, 0, sx>>>(large_list, &h->info->split2[1], h->row_flop);
                    OPS_CUDA(h, cudaGetLastError());
                    ++h->launches;
                }
                RowCursors &next = kNum ? h->info->next_num : h->info->next_sym;
                launch_rank<RankLarge, kNum, T>(h, g, large_list, &h->info->split2[1], &next.large, h->e2_size[1], sx);
                OPS_CUDA(h, cudaGetLastError());
                if (!join_x(1, s)) return fail(h, OPS_CUDA_ERROR, "stream join failed");
                if (!kNum && h->e2_size[0] > 1) {
                    k_sort_heavy_first<<<1, 1024, 0, s>>>(mid_list, &h->info->split2[0], h->row_flop);
                    OPS_CUDA(h, cudaGetLastError());
                    ++h->launches;
                }
                launch_rank<RankMid, kNum, T>(h, g, mid_list, &h->info->split2[0], &next.mid, h->e2_size[0], s);
                break;
            }
            case kClsD: {
                // whole-GPU expand/sort/compress; the CTA-per-row dense kernel when the
                // packed keys or the scratch do not fit
                const int st_d = run_d_rows<T>(h, g, list, n, kNum, s);
                h->d_rows_path[0] = st_d == OPS_OK ? n : 0;
                h->d_rows_path[1] = st_d == OPS_NOT_SUPPORTED ? n : 0;
                if (st_d == OPS_NOT_SUPPORTED) {
                    OPS_CHECK(ensure_dense(h, g.N, n, s));
                    k_dense_rows<kNum, T><<<std::min(n, h->dense_ctas), kDenseRowsThreads, 0, s>>>(
                        g, list, n, dense_view<T>(h, g.N));
                } else if (st_d != OPS_OK) {
                    return st_d;
                }
                break;
            }
        }
        OPS_CUDA(h, cudaGetLastError());
        ++h->launches;
        if (h->timing >= 2) {
            OPS_CUDA(h, cudaEventRecord(h->ev_k[kNum][c][1], s));
            h->kmeasured[kNum][c] = true;
        }
        OPS_CUDA(h, cudaEventRecord(h->ev_join[c], s));
        OPS_CUDA(h, cudaStreamWaitEvent(st, h->ev_join[c], 0));
    }
    return OPS_OK;
}

int check_mat_args(ops_handle_s *h, int rows, int cols, const int *rpt, const int *col, long long nnz)
{
    if (rows < 0 || cols < 0 || nnz < 0) return fail(h, OPS_INVALID_ARGUMENT, "negative matrix size");
    if (nnz > INT_MAX) return fail(h, OPS_INT32_OVERFLOW, "input nnz exceeds INT32_MAX");
    if (!rpt && rows > 0) return fail(h, OPS_INVALID_ARGUMENT, "null row_ptr");
    if (!col && nnz > 0) return fail(h, OPS_INVALID_ARGUMENT, "null col_idx");
    return OPS_OK;
}

float ev_ms(cudaEvent_t a, cudaEvent_t b)
{
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, a, b) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0.f;
    }
    return ms;
}

int dtype_size(int dtype) { return dtype == OPS_F64 ? 8 : (dtype == OPS_F32 ? 4 : 0); }

// Largest C (at one entry per product) that a one-pass ops_spgemm allocates before its
// entry count is known.
constexpr long long kEarlyAllocBytes = 256ll << 20;

// Status of the counting phase from its device results.
int count_status(ops_handle_s *h, const DevInfo &d)
{
    if (d.flags & kErrBadColumn) return fail(h, OPS_INVALID_CSR, "B has a column index outside [0, cols)");
    if (d.flags & kErrProbeLimit) return fail(h, OPS_PROBE_LIMIT, "symbolic hash table overflow");
    if (d.total_nnz > (unsigned long long)INT_MAX) return fail(h, OPS_INT32_OVERFLOW, "nnz(C) exceeds INT32_MAX");
    return OPS_OK;
}

// Whether a problem is launched as a small one: few rows, short ones on average.  One kernel
// against the classes' (FP64, two phases, a 5-point grid of 128 columns): 4,096 rows 81 us
// against 106, 8,192 96 against 107, 16,384 106 against 115, 24,576 126 against 133, 32,640 131
// against 133, all of them scanned by one CTA, which stops paying at 16,384.  Rows of 96, 140 and 224 products each:
// 8,000 of them 101, 105 and 114 us against 112, 135 and 142; 32,000 150, 181 and 204 against
// 158, 208 and 230.  The mean decides for want of the largest row, which must not pass 256
// products: above it the two launches were for nothing (500 rows 176 us against 168).
constexpr int kSmallRows = 16384;
constexpr double kSmallMeanProducts = 96;

bool small_problem(const ops_handle_s *h, const Mat &A, const Mat &B)
{
    if (A.rows == 0 || A.rows > kSmallRows || A.nnz < 0 || B.nnz < 0 || h->timing >= 2) return false;
    if (h->op_dtype >= 0 && h->one_pass == 2) return false;  // staged at any size
    return (double)A.nnz * (double)B.nnz <= kSmallMeanProducts * (double)A.rows * (double)A.cols;
}

template <bool kNum, typename T>
int launch_all(ops_handle_s *h, const SpgemmArgs<T> &g, cudaStream_t st)
{
    const int ctas = std::min((g.M + RankS::kGroups - 1) / RankS::kGroups, h->num_sms * RankS::kMinBlocks);
    k_rank_all<kNum, T><<<ctas, RankS::kThreads, RankS::smem<kNum>(), st>>>(g, h->th.r8);
    OPS_CUDA(h, cudaGetLastError());
    ++h->launches;
    return OPS_OK;
}

// Counting phase: class sizes (one host sync), the classes' kernels, the row_ptr scan and
// nnz(C) (a second sync).  early_alloc (ops_spgemm): where C at one entry per product fits
// kEarlyAllocBytes and no row is a D row, the second sync is left out; *c_nnz is then -1,
// plan_nnz holds the product count (an upper bound of nnz(C)) and the phase's results
// reach h_info_count when the stream gets there, for the caller to read after its own
// sync.  No D row means no kernel indexes memory by a column of B, so the numeric phase
// may run before a bad column is reported, writing at most one entry per product.
int run_symbolic(ops_handle_s *h, const Mat &A, const Mat &B, int *c_rpt, long long *c_nnz, cudaStream_t st,
                 bool early_alloc = false)
{
    const int M = A.rows;
    OPS_CHECK(ensure_ws(h, std::max(M, 1), st));
    h->plan_valid = false;
    h->begun = false;
    h->staged = false;
    h->launches = 0;
    std::memset(h->kmeasured, 0, sizeof(h->kmeasured));
    if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[0], st));
    // a one-pass call also gets the per-row products it may stage (made into offsets once
    // the staging area is known to fit)
    const bool want_stage = h->one_pass != 0 && h->op_dtype >= 0;
    SpgemmArgs<double> g{};
    g.arpt = A.rpt;
    g.acol = A.col;
    g.brpt = B.rpt;
    g.bcol = B.col;
    g.M = M;
    g.K = A.cols;
    g.N = B.cols;
    g.row_flop = h->row_flop;
    g.c_rpt = c_rpt;
    g.info = h->info;
    // small problems: every row by one kernel, the scan behind it, one host sync for all of
    // it.  They are launched before the row sizes are known, where their mean is small; if some
    // row is too large they do nothing, and the usual pipeline goes on from the classes.
    static_assert(kSmallRows + 1 <= kScanMax, "a small problem's counts are scanned by one CTA");
    bool small = small_problem(h, A, B);
    OPS_CUDA(h, cudaMemsetAsync(h->info, 0, sizeof(DevInfo), st));
    if (M == 0) OPS_CUDA(h, cudaMemsetAsync(c_rpt, 0, sizeof(int), st));
    if (M == 0 && want_stage) OPS_CUDA(h, cudaMemsetAsync(h->soff, 0, sizeof(int), st));
    if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[1], st));
    if (M > 0) {
        k_setup<<<(M + kSetupThreads - 1) / kSetupThreads, kSetupThreads, 0, st>>>(
            A.rpt, A.col, B.rpt, B.col, M, A.cols, B.cols, h->row_flop, h->lists, c_rpt,
            want_stage ? h->soff : nullptr, h->link, h->info, h->th);
        OPS_CUDA(h, cudaGetLastError());
        ++h->launches;
    }
    if (small) {
        if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[2], st));
        OPS_CHECK((launch_all<false, double>(h, g, st)));
        if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[3], st));
        OPS_CHECK(scan_rows(h, c_rpt, M, st, true));
        if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[4], st));
    }
    OPS_CUDA(h, cudaMemcpyAsync(h->h_info, h->info, sizeof(DevInfo), cudaMemcpyDeviceToHost, st));
    if (h->timing && !small) OPS_CUDA(h, cudaEventRecord(h->ev_t[2], st));
    OPS_CUDA(h, cudaStreamSynchronize(st));
    DevInfo hi = *h->h_info;
    if (beyond_small(hi)) small = false;
    if (hi.flags & kErrBadColumn)
        return fail(h, OPS_INVALID_CSR, small ? "A or B has a column index outside [0, cols)"
                                              : "A has a column index outside [0, cols)");
    if (hi.flags & kErrRowFlopOverflow)
        return fail(h, OPS_INT32_OVERFLOW, "a row of C has more than INT32_MAX intermediate products");
    std::memcpy(h->counts, hi.counts, sizeof(h->counts));
    std::memcpy(h->e1_size, hi.e1_size, sizeof(h->e1_size));
    std::memcpy(h->e2_size, hi.e2_size, sizeof(h->e2_size));
    h->plan_th = h->th;
    h->plan_M = M;
    h->plan_K = A.cols;
    h->plan_N = B.cols;
    h->plan_flop = (long long)hi.total_flop;
    h->plan_d_flop = (long long)hi.d_flop;
    h->plan_d_len_a = (long long)hi.d_len_a;
    h->staged = false;
    h->small = small;
    h->regular = false;
    h->no_groups = false;
    h->plan_arpt = A.rpt;
    h->plan_acol = A.col;
    h->plan_brpt = B.rpt;
    h->plan_bcol = B.col;
    if (small) {
        OPS_CHECK(count_status(h, hi));
        *c_nnz = (long long)hi.total_nnz;
        h->plan_nnz = (long long)hi.total_nnz;
        h->plan_valid = true;
        return OPS_OK;
    }
    OPS_CHECK(form_groups(h, hi, A, B, want_stage, st));
    if (want_stage) OPS_CHECK(prepare_stage(h, hi, M, st));
    OPS_CHECK((launch_classes<false, double>(h, g, st)));
    if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[3], st));
    OPS_CHECK(scan_rows(h, c_rpt, M, st));
    if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[4], st));
    const int vs = h->op_dtype >= 0 ? dtype_size(h->op_dtype) : 0;
    if (early_alloc && vs > 0 && hi.counts[kClsD] == 0 &&
        (long long)hi.total_flop * (long long)(4 + vs) <= kEarlyAllocBytes) {
        OPS_CUDA(h, cudaMemcpyAsync(h->h_info_count, h->info, sizeof(DevInfo), cudaMemcpyDeviceToHost, st));
        *c_nnz = -1;
        h->plan_nnz = (long long)hi.total_flop;
    } else {
        OPS_CUDA(h, cudaMemcpyAsync(h->h_info, h->info, sizeof(DevInfo), cudaMemcpyDeviceToHost, st));
        OPS_CUDA(h, cudaStreamSynchronize(st));
        const DevInfo h2 = *h->h_info;
        OPS_CHECK(count_status(h, h2));
        *c_nnz = (long long)h2.total_nnz;
        h->plan_nnz = (long long)h2.total_nnz;
        h->no_groups = h2.groups == 0;
    }
    h->plan_valid = true;
    return OPS_OK;
}

template <typename T>
int run_numeric(ops_handle_s *h, const Mat &A, const Mat &B, const int *c_rpt, int *c_col, T *c_val, cudaStream_t st)
{
    if (!h->plan_valid || h->plan_M != A.rows || h->plan_K != A.cols || h->plan_N != B.cols ||
        h->plan_arpt != A.rpt || h->plan_acol != A.col || h->plan_brpt != B.rpt || h->plan_bcol != B.col)
        return fail(h, OPS_NOT_SUPPORTED, "numeric phase without a matching symbolic phase on this handle");
    OPS_CUDA(h, cudaMemsetAsync(h->info, 0, offsetof(DevInfo, next_sym), st));
    SpgemmArgs<T> g{};
    g.arpt = A.rpt;
    g.acol = A.col;
    g.aval = static_cast<const T *>(A.val);
    g.brpt = B.rpt;
    g.bcol = B.col;
    g.bval = static_cast<const T *>(B.val);
    g.M = A.rows;
    g.K = A.cols;
    g.N = B.cols;
    g.row_flop = h->row_flop;
    g.c_rpt = const_cast<int *>(c_rpt);
    g.c_col = c_col;
    g.c_val = c_val;
    g.info = h->info;
    g.hash_slots = h->hash_slots;
    if (h->small) return launch_all<true, T>(h, g, st);
    return launch_classes<true, T>(h, g, st);
}

int check_flags(ops_handle_s *h, cudaStream_t st)
{
    OPS_CUDA(h, cudaMemcpyAsync(&h->h_info->flags, &h->info->flags, sizeof(int), cudaMemcpyDeviceToHost, st));
    OPS_CUDA(h, cudaStreamSynchronize(st));
    const int f = h->h_info->flags;
    if (f & kErrCountMismatch) return fail(h, OPS_COUNT_MISMATCH, "numeric nnz differs from symbolic nnz");
    if (f & kErrProbeLimit) return fail(h, OPS_PROBE_LIMIT, "numeric hash table overflow");
    if (f & kErrBadColumn) return fail(h, OPS_INVALID_CSR, "column index outside [0, cols)");
    return OPS_OK;
}

void fill_timings(ops_handle_s *h, bool with_numeric)
{
    ops_timings &t = h->last_t;
    std::memset(&t, 0, sizeof(t));
    t.flop = h->plan_flop;
    t.nnz = h->plan_nnz;
    for (int c = 0; c < kNumClasses; ++c) t.class_rows[c] = h->counts[c];
    t.launches = h->launches;
    for (int ph = 0; ph < 2; ++ph)
        for (int c = 0; c < kNumClasses; ++c)
            t.kernel_ms[ph][c] = h->kmeasured[ph][c] ? ev_ms(h->ev_k[ph][c][0], h->ev_k[ph][c][1]) : 0.f;
    if (!h->timing) return;
    t.setup = ev_ms(h->ev_t[0], h->ev_t[1]) * 1e-3;
    t.symbolic_binning = ev_ms(h->ev_t[1], h->ev_t[2]) * 1e-3;
    t.symbolic = ev_ms(h->ev_t[2], h->ev_t[3]) * 1e-3;
    t.prefix = ev_ms(h->ev_t[3], h->ev_t[4]) * 1e-3;
    if (with_numeric) {
        t.allocate = ev_ms(h->ev_t[4], h->ev_t[5]) * 1e-3;
        t.numeric = ev_ms(h->ev_t[5], h->ev_t[6]) * 1e-3;
        t.total = ev_ms(h->ev_t[0], h->ev_t[6]) * 1e-3;
    } else {
        t.total = ev_ms(h->ev_t[0], h->ev_t[4]) * 1e-3;
    }
}

// Output arrays of ops_spgemm: the handle's pool (stream-ordered) or plain cudaMalloc.
cudaError_t out_alloc(ops_handle_s *h, void **p, size_t bytes, cudaStream_t st)
{
    if (h->out_malloc) return cudaMalloc(p, bytes);
    return cudaMallocFromPoolAsync(p, bytes, h->pool, st);
}

void out_free(ops_handle_s *h, void *p, cudaStream_t st)
{
    if (!p) return;
    if (h->out_malloc) {
        cudaStreamSynchronize(st);
        cudaFree(p);
    } else {
        cudaFreeAsync(p, st);
    }
}

}  // namespace

// ================================================================== C ABI ==========
extern "C" {

const char *ops_version(void) { return kVersion; }

const char *ops_status_string(int s)
{
    switch (s) {
        case OPS_OK: return "ok";
        case OPS_NONSQUARE: return "nonsquare";
        case OPS_INT32_OVERFLOW: return "int32_overflow";
        case OPS_OOM: return "oom";
        case OPS_CUDA_ERROR: return "cuda_error";
        case OPS_EXCEPTION: return "exception";
        case OPS_INVALID_ARGUMENT: return "invalid_argument";
        case OPS_INVALID_CSR: return "invalid_csr";
        case OPS_PROBE_LIMIT: return "probe_limit";
        case OPS_TIMEOUT: return "timeout";
        case OPS_NOT_SUPPORTED: return "not_supported";
        case OPS_COUNT_MISMATCH: return "count_mismatch";
    }
    return "unknown";
}

int ops_handle_create(ops_handle_t *out)
{
    if (!out) return OPS_INVALID_ARGUMENT;
    *out = nullptr;
    ops_handle_s *h = new (std::nothrow) ops_handle_s();
    if (!h) return OPS_EXCEPTION;
    cudaError_t e = cudaGetDevice(&h->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->device);
    if (e == cudaSuccess) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = h->device;
        e = cudaMemPoolCreate(&h->pool, &props);
    }
    if (e == cudaSuccess) {
        uint64_t thr = UINT64_MAX;
        e = cudaMemPoolSetAttribute(h->pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    // the D rows' whole-GPU sort is a chain of about twenty short launches, the longest
    // path of a call that has D rows: its stream gets the highest priority, so its blocks
    // are scheduled ahead of the other classes' waiting blocks
    int prio_low = 0, prio_high = 0;
    if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
    for (int c = 0; c < kNumClasses && e == cudaSuccess; ++c) {
        e = cudaStreamCreateWithPriority(&h->side[c], cudaStreamNonBlocking, c == kClsD ? prio_high : prio_low);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_join[c], cudaEventDisableTiming);
    }
    for (int x = 0; x < ops_handle_s::kNumExtra && e == cudaSuccess; ++x) {
        e = cudaStreamCreateWithFlags(&h->side_x[x], cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_x_fork[x], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_x_join[x], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming);
    for (int i = 0; i < ops_handle_s::kNumEv && e == cudaSuccess; ++i) e = cudaEventCreate(&h->ev_t[i]);
    for (int ph = 0; ph < 2 && e == cudaSuccess; ++ph)
        for (int c = 0; c < kNumClasses && e == cudaSuccess; ++c)
            for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreate(&h->ev_k[ph][c][k]);
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&h->h_info), sizeof(DevInfo));
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&h->h_info_count), sizeof(DevInfo));
    if (e == cudaSuccess) {
        set_smem_attrs<double>();
        set_smem_attrs<float>();
        cudaFuncSetAttribute(k_group_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RankE1::smem<false>());
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        ops_handle_destroy(h);
        return status_of(e);
    }
    *out = h;
    return OPS_OK;
}

int ops_handle_destroy(ops_handle_t h)
{
    if (!h) return OPS_OK;
    cudaDeviceSynchronize();
    for (ops_handle_s *s : h->spare) ops_handle_destroy(s);
    if (h->ws) cudaFree(h->ws);
    if (h->b_link) cudaFree(h->b_link);
    if (h->dense) cudaFree(h->dense);
    if (h->stage) cudaFree(h->stage);
    if (h->bwd.mem) cudaFree(h->bwd.mem);
    if (h->bwd.pmap) cudaFree(h->bwd.pmap);
    if (h->bwd.at_blk) cudaFree(h->bwd.at_blk);
    if (h->bwd.ready) cudaEventDestroy(h->bwd.ready);
    for (int c = 0; c < kNumClasses; ++c) {
        if (h->side[c]) cudaStreamDestroy(h->side[c]);
        if (h->ev_join[c]) cudaEventDestroy(h->ev_join[c]);
    }
    for (int x = 0; x < ops_handle_s::kNumExtra; ++x) {
        if (h->side_x[x]) cudaStreamDestroy(h->side_x[x]);
        if (h->ev_x_fork[x]) cudaEventDestroy(h->ev_x_fork[x]);
        if (h->ev_x_join[x]) cudaEventDestroy(h->ev_x_join[x]);
    }
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
    for (int i = 0; i < ops_handle_s::kNumEv; ++i)
        if (h->ev_t[i]) cudaEventDestroy(h->ev_t[i]);
    for (int ph = 0; ph < 2; ++ph)
        for (int c = 0; c < kNumClasses; ++c)
            for (int k = 0; k < 2; ++k)
                if (h->ev_k[ph][c][k]) cudaEventDestroy(h->ev_k[ph][c][k]);
    if (h->h_info) cudaFreeHost(h->h_info);
    if (h->h_info_count) cudaFreeHost(h->h_info_count);
    if (h->pool) cudaMemPoolDestroy(h->pool);
    (void)cudaGetLastError();
    delete h;
    return OPS_OK;
}

int ops_handle_set_timing(ops_handle_t h, int enable)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    h->timing = enable < 0 ? 0 : (enable > 2 ? 2 : enable);
    return OPS_OK;
}

int ops_handle_get_timings(ops_handle_t h, ops_timings *out)
{
    if (!h || !out) return OPS_INVALID_ARGUMENT;
    *out = h->last_t;
    return OPS_OK;
}

int ops_handle_set_dense_budget(ops_handle_t h, size_t bytes)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    h->dense_budget = bytes;
    return OPS_OK;
}

int ops_handle_set_thresholds(ops_handle_t h, const int32_t *th, int n)
{
    if (!h || !th || n != 6) return OPS_INVALID_ARGUMENT;
    const Thresholds cap = default_thresholds();
    Thresholds t{th[0], th[1], th[2], th[3], th[4], th[5]};
    if (t.r8 < 0 || t.r8 > cap.r8 || t.r16 < 0 || t.r16 > cap.r16 || t.r32 < 0 || t.r32 > cap.r32 || t.w < 0 ||
        t.w > cap.w || t.e1 < 0 || t.e1 > cap.e1 || t.e2 < 0 || t.e2 > cap.e2)
        return fail(h, OPS_INVALID_ARGUMENT, "threshold above the compiled capacity of its class");
    h->th = t;
    h->plan_valid = false;
    return OPS_OK;
}

int ops_handle_get_thresholds(ops_handle_t h, int32_t *th, int n)
{
    if (!h || !th || n != 6) return OPS_INVALID_ARGUMENT;
    const Thresholds t = h->th;
    const int32_t v[6] = {t.r8, t.r16, t.r32, t.w, t.e1, t.e2};
    std::memcpy(th, v, sizeof(v));
    return OPS_OK;
}

int ops_handle_set_one_pass(ops_handle_t h, int mode)
{
    if (!h || mode < 0 || mode > 2) return OPS_INVALID_ARGUMENT;
    h->one_pass = mode;
    return OPS_OK;
}

int ops_handle_set_tuning(ops_handle_t h, const ops_tuning *t)
{
    if (!h || !t) return OPS_INVALID_ARGUMENT;
    if ((t->hash_slots != 2 && t->hash_slots != 4) || (t->batch_persistent != 0 && t->batch_persistent != 1) ||
        t->batch_warp_max < kBatchWarpMaxLo || t->batch_warp_max > kBatchWarpMaxHi)
        return fail(h, OPS_INVALID_ARGUMENT, "tuning value out of range");
    OPS_CHECK(ops_handle_set_thresholds(h, t->thresholds, 6));
    h->hash_slots = t->hash_slots;
    h->batch_persistent = t->batch_persistent;
    h->batch_warp_max = t->batch_warp_max;
    return OPS_OK;
}

int ops_handle_get_tuning(ops_handle_t h, ops_tuning *t)
{
    if (!h || !t) return OPS_INVALID_ARGUMENT;
    OPS_CHECK(ops_handle_get_thresholds(h, t->thresholds, 6));
    t->hash_slots = h->hash_slots;
    t->batch_persistent = h->batch_persistent;
    t->batch_warp_max = h->batch_warp_max;
    return OPS_OK;
}

int ops_handle_set_stage_budget(ops_handle_t h, size_t bytes)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    h->stage_budget = bytes;
    return OPS_OK;
}

int ops_handle_set_output_malloc(ops_handle_t h, int use_cuda_malloc)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    h->out_malloc = use_cuda_malloc != 0;
    return OPS_OK;
}

const char *ops_handle_last_error(ops_handle_t h) { return h ? h->last_error.c_str() : "null handle"; }

int ops_handle_subclass_rows(ops_handle_t h, int32_t *out, int n)
{
    if (!h || !out || n < 0) return OPS_INVALID_ARGUMENT;
    int v[10] = {};
    v[5] = h->d_rows_path[0];
    v[6] = h->d_rows_path[1];
    if (h->info) {
        DevInfo d{};
        OPS_CUDA(h, cudaMemcpy(&d, h->info, sizeof(DevInfo), cudaMemcpyDeviceToHost));
        // a one-pass call computes its staged E1 rows while counting (split1)
        v[0] = d.split[0] + d.split[3] + d.split1[0] + d.split1[3] + (h->small ? h->e1_size[0] : 0);
        v[1] = d.split[1];
        v[2] = d.split[2] + d.split1[2];
        v[3] = d.split2[0];
        v[4] = d.split2[1];
        for (int i = 0; i < 3; ++i) v[7 + i] = d.rank_rows[i];
    }
    for (int i = 0; i < n && i < 10; ++i) out[i] = v[i];
    return OPS_OK;
}

int ops_spgemm_symbolic(ops_handle_t h, int32_t rows_a, int32_t cols_a, int32_t cols_b, const int32_t *a_rpt,
                        const int32_t *a_col, int64_t a_nnz, const int32_t *b_rpt, const int32_t *b_col, int64_t b_nnz,
                        int32_t *c_rpt, int64_t *c_nnz, void *stream)
{
    if (!h || !c_rpt || !c_nnz) return fail(h, OPS_INVALID_ARGUMENT, "null handle or output");
    try {
        h->last_error.clear();
        OPS_CHECK(check_mat_args(h, rows_a, cols_a, a_rpt, a_col, a_nnz));
        OPS_CHECK(check_mat_args(h, cols_a, cols_b, b_rpt, b_col, b_nnz));
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const Mat A{rows_a, cols_a, a_rpt, a_col, nullptr, a_nnz};
        const Mat B{cols_a, cols_b, b_rpt, b_col, nullptr, b_nnz};
        h->op_dtype = -1;  // no values: two passes
        long long nnz = 0;
        OPS_CHECK(run_symbolic(h, A, B, c_rpt, &nnz, st));
        *c_nnz = nnz;
        fill_timings(h, false);
        return OPS_OK;
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm_symbolic");
    }
}

int ops_spgemm_numeric(ops_handle_t h, int dtype, int32_t rows_a, int32_t cols_a, int32_t cols_b,
                       const int32_t *a_rpt, const int32_t *a_col, const void *a_val, const int32_t *b_rpt,
                       const int32_t *b_col, const void *b_val, const int32_t *c_rpt, int32_t *c_col, void *c_val,
                       void *stream)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    if (dtype_size(dtype) == 0) return fail(h, OPS_INVALID_ARGUMENT, "unknown dtype");
    try {
        h->last_error.clear();
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const Mat A{rows_a, cols_a, a_rpt, a_col, a_val};
        const Mat B{cols_a, cols_b, b_rpt, b_col, b_val};
        if (h->plan_nnz > 0 && (!c_col || !c_val || !a_val || !b_val))
            return fail(h, OPS_INVALID_ARGUMENT, "null values or output");
        h->begun = false;
        h->staged = false;  // rows that a begun call staged
        if (dtype == OPS_F64)
            return run_numeric<double>(h, A, B, c_rpt, c_col, static_cast<double *>(c_val), st);
        return run_numeric<float>(h, A, B, c_rpt, c_col, static_cast<float *>(c_val), st);
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm_numeric");
    }
}

int ops_spgemm_check(ops_handle_t h, void *stream)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    return check_flags(h, static_cast<cudaStream_t>(stream));
}

int ops_spgemm(ops_handle_t h, int dtype, int32_t rows_a, int32_t cols_a, int32_t cols_b, const int32_t *a_rpt,
               const int32_t *a_col, const void *a_val, int64_t a_nnz, const int32_t *b_rpt, const int32_t *b_col,
               const void *b_val, int64_t b_nnz, int32_t **c_rpt, int32_t **c_col, void **c_val, int64_t *c_nnz,
               void *stream)
{
    if (!h || !c_rpt || !c_col || !c_val || !c_nnz) return fail(h, OPS_INVALID_ARGUMENT, "null handle or output");
    const int vs = dtype_size(dtype);
    if (vs == 0) return fail(h, OPS_INVALID_ARGUMENT, "unknown dtype");
    *c_rpt = nullptr;
    *c_col = nullptr;
    *c_val = nullptr;
    *c_nnz = 0;
    try {
        h->last_error.clear();
        OPS_CHECK(check_mat_args(h, rows_a, cols_a, a_rpt, a_col, a_nnz));
        OPS_CHECK(check_mat_args(h, cols_a, cols_b, b_rpt, b_col, b_nnz));
        if ((a_nnz > 0 && !a_val) || (b_nnz > 0 && !b_val)) return fail(h, OPS_INVALID_ARGUMENT, "null values");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const Mat A{rows_a, cols_a, a_rpt, a_col, a_val, a_nnz};
        const Mat B{cols_a, cols_b, b_rpt, b_col, b_val, b_nnz};
        // the values are known before the counting phase: the R16, R32 and W rows may run
        // their numeric kernels there (one pass); reset whichever way the call returns
        struct OnePassScope {
            ops_handle_s *h;
            ~OnePassScope()
            {
                h->op_dtype = -1;
                h->op_aval = h->op_bval = nullptr;
                h->staged = false;
            }
        } one_pass_scope{h};
        h->op_dtype = dtype;
        h->op_aval = a_val;
        h->op_bval = b_val;
        void *p = nullptr;
        OPS_CUDA(h, out_alloc(h, &p, sizeof(int) * ((size_t)rows_a + 1), st));
        int *rpt = static_cast<int *>(p);
        long long nnz = 0;
        int s = run_symbolic(h, A, B, rpt, &nnz, st, true);
        if (s != OPS_OK) {
            out_free(h, rpt, st);
            return s;
        }
        // nnz < 0: C allocated at one entry per product, its count read after the numeric
        // phase, with no host round trip between the two phases
        const bool early = nnz < 0;
        const long long cap = early ? h->plan_nnz : nnz;
        void *col = nullptr, *val = nullptr;
        cudaError_t e = out_alloc(h, &col, sizeof(int) * (size_t)std::max(cap, 1LL), st);
        if (e == cudaSuccess) e = out_alloc(h, &val, (size_t)vs * (size_t)std::max(cap, 1LL), st);
        if (h->timing && e == cudaSuccess) e = cudaEventRecord(h->ev_t[5], st);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            out_free(h, col, st);
            out_free(h, rpt, st);
            return fail(h, status_of(e), std::string("allocating C: ") + cudaGetErrorString(e));
        }
        s = dtype == OPS_F64 ? run_numeric<double>(h, A, B, rpt, static_cast<int *>(col), static_cast<double *>(val), st)
                             : run_numeric<float>(h, A, B, rpt, static_cast<int *>(col), static_cast<float *>(val), st);
        if (s == OPS_OK && h->timing) {
            e = cudaEventRecord(h->ev_t[6], st);
            if (e != cudaSuccess) s = fail(h, status_of(e), "event record");
        }
        if (s == OPS_OK) s = check_flags(h, st);
        if (early) {  // the stream has passed the counting phase's results (a sync above or
                      // on the error path below); they take precedence over the numeric's
            if (s != OPS_OK) cudaStreamSynchronize(st);
            const int sc = count_status(h, *h->h_info_count);
            if (sc != OPS_OK) s = sc;
            nnz = (long long)h->h_info_count->total_nnz;
            h->plan_nnz = nnz;
        }
        if (s != OPS_OK) {
            out_free(h, val, st);
            out_free(h, col, st);
            out_free(h, rpt, st);
            cudaStreamSynchronize(st);
            return s;
        }
        fill_timings(h, true);
        *c_rpt = rpt;
        *c_col = static_cast<int *>(col);
        *c_val = val;
        *c_nnz = nnz;
        return OPS_OK;
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm");
    }
}

int ops_spgemm_begin(ops_handle_t h, int dtype, int32_t rows_a, int32_t cols_a, int32_t cols_b,
                     const int32_t *a_rpt, const int32_t *a_col, const void *a_val, int64_t a_nnz,
                     const int32_t *b_rpt, const int32_t *b_col, const void *b_val, int64_t b_nnz, int32_t *c_rpt,
                     int64_t *c_nnz, void *stream)
{
    if (!h || !c_rpt || !c_nnz) return fail(h, OPS_INVALID_ARGUMENT, "null handle or output");
    if (dtype_size(dtype) == 0) return fail(h, OPS_INVALID_ARGUMENT, "unknown dtype");
    try {
        h->last_error.clear();
        h->begun = false;
        OPS_CHECK(check_mat_args(h, rows_a, cols_a, a_rpt, a_col, a_nnz));
        OPS_CHECK(check_mat_args(h, cols_a, cols_b, b_rpt, b_col, b_nnz));
        if ((a_nnz > 0 && !a_val) || (b_nnz > 0 && !b_val)) return fail(h, OPS_INVALID_ARGUMENT, "null values");
        const Mat A{rows_a, cols_a, a_rpt, a_col, a_val, a_nnz};
        const Mat B{cols_a, cols_b, b_rpt, b_col, b_val, b_nnz};
        long long nnz = 0;
        h->op_dtype = dtype;
        h->op_aval = a_val;
        h->op_bval = b_val;
        const int s = run_symbolic(h, A, B, c_rpt, &nnz, static_cast<cudaStream_t>(stream));
        h->op_dtype = -1;
        h->op_aval = h->op_bval = nullptr;
        if (s != OPS_OK) {
            h->staged = false;
            return s;
        }
        h->begun = true;
        h->begun_dtype = dtype;
        h->begun_rpt = c_rpt;
        h->begun_aval = a_val;
        h->begun_bval = b_val;
        *c_nnz = nnz;
        return OPS_OK;
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm_begin");
    }
}

int ops_spgemm_finish(ops_handle_t h, int32_t *c_col, void *c_val, void *stream)
{
    if (!h) return OPS_INVALID_ARGUMENT;
    if (!h->begun || !h->plan_valid) return fail(h, OPS_NOT_SUPPORTED, "ops_spgemm_finish without ops_spgemm_begin");
    h->begun = false;
    try {
        h->last_error.clear();
        struct StagedScope {  // staged rows belong to this call alone
            ops_handle_s *h;
            ~StagedScope() { h->staged = false; }
        } staged_scope{h};
        if (h->plan_nnz > 0 && (!c_col || !c_val)) return fail(h, OPS_INVALID_ARGUMENT, "null output");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const Mat A{h->plan_M, h->plan_K, h->plan_arpt, h->plan_acol, h->begun_aval};
        const Mat B{h->plan_K, h->plan_N, h->plan_brpt, h->plan_bcol, h->begun_bval};
        if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[5], st));
        OPS_CHECK(h->begun_dtype == OPS_F64
                      ? run_numeric<double>(h, A, B, h->begun_rpt, c_col, static_cast<double *>(c_val), st)
                      : run_numeric<float>(h, A, B, h->begun_rpt, c_col, static_cast<float *>(c_val), st));
        if (h->timing) OPS_CUDA(h, cudaEventRecord(h->ev_t[6], st));
        OPS_CHECK(check_flags(h, st));
        fill_timings(h, true);
        return OPS_OK;
    } catch (...) {
        return fail(h, OPS_EXCEPTION, "exception in ops_spgemm_finish");
    }
}

int ops_free(void *dptr, void *stream)
{
    if (!dptr) return OPS_OK;
    cudaError_t e = cudaFreeAsync(dptr, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return status_of(e);
    }
    return OPS_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ ops_flop -------
namespace {
__global__ void __launch_bounds__(256) k_flop64(const int *__restrict__ arpt, const int *__restrict__ acol,
                                                const int *__restrict__ brpt, int M, int K, long long *row_flop,
                                                unsigned long long *total, int *bad)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long s = 0;
    if (r < M) {
        for (int p = arpt[r]; p < arpt[r + 1]; ++p) {
            const int j = acol[p];
            if ((unsigned)j < (unsigned)K) s += (unsigned long long)(brpt[j + 1] - brpt[j]);
            else atomicOr(bad, 1);
        }
        if (row_flop) row_flop[r] = (long long)s;
    }
    block_add_u64(s, total);
}
}  // namespace

extern "C" int ops_flop(int32_t rows_a, int32_t cols_a, const int32_t *a_rpt, const int32_t *a_col,
                        const int32_t *b_rpt, int64_t *row_flop, int64_t *total, void *stream)
{
    if (rows_a < 0 || !total || (rows_a > 0 && (!a_rpt || !b_rpt))) return OPS_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    void *p = nullptr;
    cudaError_t e = cudaMallocAsync(&p, 16, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, 16, st);
    unsigned long long *d_total = static_cast<unsigned long long *>(p);
    int *d_bad = reinterpret_cast<int *>(d_total + 1);
    if (e == cudaSuccess && rows_a > 0) {
        k_flop64<<<(rows_a + 255) / 256, 256, 0, st>>>(a_rpt, a_col, b_rpt, rows_a, cols_a,
                                                      reinterpret_cast<long long *>(row_flop), d_total, d_bad);
        e = cudaGetLastError();
    }
    unsigned long long h_res[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_res, p, 16, cudaMemcpyDeviceToHost, st);
    if (p) cudaFreeAsync(p, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return status_of(e);
    }
    if (h_res[1] & 1ull) return OPS_INVALID_CSR;
    *total = (int64_t)h_res[0];
    return OPS_OK;
}
