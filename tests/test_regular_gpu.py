"""Groups of consecutive rows of one pattern (regular.cuh): banded operators whose rows move
on by one column, cut by rows that miss an entry of A or whose B rows miss one, so that runs
of every length up to a few hundred rows occur (remainders of 6 to 32 rows, shorter runs
left to their class).  Two passes, one pass and a second numeric call with new values, FP64
and FP32, against the oracle bit for bit; and the same patterns where the rule leaves them
to their class (too many separate B rows to stage; too few rows).
"""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops

pytestmark = pytest.mark.gpu

BANDS = {
    # A offsets (relative to 100), B offsets: products per row, pencils
    "stencil25": ([0, 1, 2, 3, 4, 50, 51, 52, 53, 54, 100, 101, 102, 103, 104, 150, 151, 152, 153, 154, 200, 201, 202,
                   203, 204], [0, 1, 2, 3, 4, 50, 51, 52, 53, 54, 100, 101, 102, 103, 104, 150, 151, 152, 153, 154, 200,
                               201, 202, 203, 204]),
    "one_pencil": (list(range(32)), list(range(32))),         # 1,024 products, one run of B rows
    "short": ([3, 4, 9, 20, 21, 22, 40, 41, 77], list(range(16, 64, 3))),  # 144 products, B rows of 16
    # runs of B rows that start at every offset of 16 bytes, rows of 17
    "odd_pencils": ([0, 1, 2, 30, 31, 32, 63, 64, 65], list(range(0, 34, 2))),
    # 16 runs of one B row each: staged for 32 rows together, not for 64
    "single_rows": (list(range(0, 48, 3)), list(range(0, 51, 3))),
    "pencils": (list(range(0, 96, 3)), list(range(0, 62, 2))),  # 992 products, 32 B rows apart: not staged
}


def banded(name, rows, cuts, seed):
    rng = np.random.default_rng(seed)
    offs_a, offs_b = BANDS[name]
    k = rows + max(offs_a) + 1
    ncols = k + max(offs_b) + 1

    def build(n, offs, cut):
        rows_ = [np.array(offs) + i for i in range(n)]
        for i in cut:
            rows_[i] = np.delete(rows_[i], rng.integers(len(offs)))
        rpt = np.concatenate([[0], np.cumsum([len(r) for r in rows_])]).astype(np.int32)
        col = np.concatenate(rows_).astype(np.int32)
        return rpt, col, rng.standard_normal(len(col))

    cut_a = rng.choice(rows, cuts, replace=False) if cuts else []
    cut_b = rng.choice(k, max(1, cuts // 8), replace=False) if cuts else []
    return build(rows, offs_a, cut_a), build(k, offs_b, cut_b), ncols


@pytest.mark.parametrize("name,rows,cuts,groups", [("stencil25", 25000, 0, True), ("stencil25", 30000, 350, True),
                                                   ("one_pencil", 25001, 300, True), ("short", 60000, 1000, True),
                                                   ("odd_pencils", 30001, 40, True), ("odd_pencils", 33003, 600, True),
                                                   ("single_rows", 25003, 200, True),
                                                   ("pencils", 25000, 20, False), ("short", 1000, 10, False),
                                                   ("short", 40000, 6000, False)])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_groups_of_one_pattern(cuda, dtype, name, rows, cuts, groups):
    torch = cuda
    npdt = np.float64 if dtype == "f64" else np.float32
    tdt = torch.float64 if dtype == "f64" else torch.float32
    a, b, ncols = banded(name, rows, cuts, 11)
    a = (a[0], a[1], a[2].astype(npdt))
    b = (b[0], b[1], b[2].astype(npdt))
    A = ops.csr_to_device(*a, rows, len(b[0]) - 1, dtype=tdt)
    B = ops.csr_to_device(*b, len(b[0]) - 1, ncols, dtype=tdt)
    bits = np.uint64 if dtype == "f64" else np.uint32
    orpt, ocol, oval = oracle.spgemm(*a, *b, ncols, dtype=npdt)

    def same(rpt, col, val, oval):
        assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
        assert np.array_equal(val.view(bits), oval.view(bits))

    with ops.Handle() as h:
        c_rpt, nnz = h.symbolic(A, B)
        c_col, c_val = h.numeric(A, B, c_rpt, nnz)
        same(c_rpt.cpu().numpy(), c_col.cpu().numpy(), c_val.cpu().numpy(), oval)
        grouped = rows - sum(h.subclass_rows()[k] for k in ("e1_sort", "e1_hash", "e1_esc"))
        assert (grouped > rows // 4) == groups, grouped
        h.set_one_pass(2)
        same(*h.spgemm_oneshot(A, B).to_host(), oval)
        rng = np.random.default_rng(5)
        a2, b2 = rng.standard_normal(len(a[1])).astype(npdt), rng.standard_normal(len(b[1])).astype(npdt)
        A.val.copy_(torch.as_tensor(a2))
        B.val.copy_(torch.as_tensor(b2))
        c_rpt, nnz = h.symbolic(A, B)
        for _ in range(2):  # the plan's groups are used again
            c_col, c_val = h.numeric(A, B, c_rpt, nnz)
        same(c_rpt.cpu().numpy(), c_col.cpu().numpy(), c_val.cpu().numpy(),
             oracle.spgemm(a[0], a[1], a2, b[0], b[1], b2, ncols, dtype=npdt)[2])
