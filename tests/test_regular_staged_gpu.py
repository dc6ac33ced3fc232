"""Groups of rows of one pattern (regular.cuh) in calls that compute rows while they count:
grouped rows whose products span more columns than the column window (32,768) would be staged
as well, and must not be; a numeric call with new values on the plan of such a call computes every row.
Grids of a wide cross-section and bands of two distant clusters,
alone, cut by rows that miss an entry, and beside narrow bands, irregular and short rows; both
ways to call, every mode, FP64 and FP32, against the oracle bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import opsparse_gb300 as ops

pytestmark = pytest.mark.gpu

NEAR = np.arange(5)
FAR = 40000  # columns between the clusters of a wide row
B_OFFS = np.arange(0, 40, 2)


def grid27(nx, ny, nz, seed=1):
    rng = np.random.default_rng(seed)
    tri = [sp.diags([np.ones(n - 1), np.ones(n), np.ones(n - 1)], [-1, 0, 1], format="csr") for n in (nx, ny, nz)]
    m = sp.csr_matrix(sp.kron(sp.kron(tri[0], tri[1]), tri[2]))
    m.sort_indices()
    a = (m.indptr.astype(np.int32), m.indices.astype(np.int32), rng.standard_normal(m.nnz))
    return a, a, m.shape[1]


def bands(kind, seed=3):
    """A's rows: wide ones (ten entries in two clusters FAR apart, 200 products), narrow ones
    (ten entries together), irregular ones (12 entries anywhere) and short ones (three)."""
    rng = np.random.default_rng(seed)
    wide = np.concatenate([NEAR, NEAR + FAR])
    narrow = np.arange(10)
    blocks = {"wide": [("w", 25000)], "cut": [("w", 30000), ("i", 6000)],
              "mixed": [("w", 9000), ("n", 9000), ("s", 3000), ("w", 9000), ("i", 6000), ("n", 5000)]}[kind]
    rows = sum(n for _, n in blocks)
    k = rows + FAR + 10
    cols = []
    for what, n in blocks:
        for _ in range(n):
            i = len(cols)
            if what == "i":
                cols.append(np.sort(rng.choice(k, 12, replace=False)))
            else:
                cols.append({"w": wide, "n": narrow, "s": NEAR[:3]}[what] + i)
                if kind != "wide" and what != "s" and rng.random() < 0.02:  # the row misses an entry
                    cols[-1] = np.delete(cols[-1], rng.integers(len(cols[-1])))
    a_rpt = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    a_col = np.concatenate(cols).astype(np.int32)
    b_rpt = (np.arange(k + 1) * len(B_OFFS)).astype(np.int32)
    b_col = (np.arange(k)[:, None] + B_OFFS[None, :]).astype(np.int32).ravel()
    return ((a_rpt, a_col, rng.standard_normal(len(a_col))), (b_rpt, b_col, rng.standard_normal(len(b_col))),
            k + int(B_OFFS[-1]) + 1)


CASES = {"grid8x92x92": lambda: grid27(8, 92, 92), "grid25x100x100": lambda: grid27(25, 100, 100),
         "wide": lambda: bands("wide"), "cut": lambda: bands("cut"), "mixed": lambda: bands("mixed")}


def on_device(cuda, name, dtype):
    npdt = np.float64 if dtype == "f64" else np.float32
    a, b, ncols = CASES[name]()
    same = b is a
    a = (a[0], a[1], a[2].astype(npdt))
    b = a if same else (b[0], b[1], b[2].astype(npdt))
    k = len(b[0]) - 1
    A = ops.csr_to_device(*a, len(a[0]) - 1, k, dtype=cuda.float64 if dtype == "f64" else cuda.float32)
    B = A if same else ops.csr_to_device(*b, k, ncols, dtype=A.val.dtype)
    return a, b, A, B, oracle.spgemm(*a, *b, ncols, dtype=npdt)


def check(got, want):
    rpt, col, val = got
    assert np.array_equal(rpt.astype(np.int64), want[0]) and np.array_equal(col, want[1])
    assert np.array_equal(val.view(np.uint8), want[2].view(np.uint8))


def grouped_rows(h):
    sub = h.subclass_rows()
    return h.timings()["class_rows"][4] - sum(sub[key] for key in ("e1_sort", "e1_hash", "e1_esc"))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("name", list(CASES))
def test_grouped_rows_are_not_staged(cuda, name, dtype):
    a, b, A, B, want = on_device(cuda, name, dtype)
    other = cuda.cuda.Stream()
    for mode, budget in ((1, None), (2, None), (2, 0), (0, None)):
        with ops.Handle() as h:
            h.set_one_pass(mode)
            if budget is not None:  # what is left to stage does not fit: two passes after all
                h.set_stage_budget(budget)
            for stream in (None, other):
                check(h.spgemm_oneshot(A, B, stream=stream).to_host(), want)
                assert grouped_rows(h) > A.rows // 4


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("name", [n for n in CASES if n != "grid25x100x100"])
def test_numeric_on_a_one_pass_plan(cuda, name, dtype):
    a, b, A, B, want = on_device(cuda, name, dtype)
    rng = np.random.default_rng(9)
    c_rpt = cuda.as_tensor(want[0].astype(np.int32)).cuda()
    nnz = len(want[1])
    other = cuda.cuda.Stream()
    for mode in (1, 2):
        with ops.Handle() as h:
            h.set_one_pass(mode)
            for stream in (None, other):  # two halves; ops_spgemm
                h.spgemm_oneshot(A, B, stream=stream)
                new = [rng.standard_normal(len(m[1])).astype(m[2].dtype) for m in (a, b)]
                if B is A:
                    new[1] = new[0]
                A2, B2 = (ops.CsrMatrix(m.rows, m.cols, m.rpt, m.col, cuda.as_tensor(v).cuda())
                          for m, v in zip((A, B), new))
                expect = oracle.spgemm(a[0], a[1], new[0], b[0], b[1], new[1], B.cols, dtype=a[2].dtype)
                for _ in range(2):
                    c_col = cuda.full((nnz,), -1, dtype=cuda.int32, device="cuda")
                    c_val = cuda.full((nnz,), 7.0, dtype=A.val.dtype, device="cuda")
                    h.numeric(A2, B2, c_rpt, nnz, c_col=c_col, c_val=c_val)
                    check((want[0], c_col.cpu().numpy(), c_val.cpu().numpy()), expect)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_repeated_columns_of_b_are_not_grouped(cuda, dtype):
    """B rows that hold a column twice are outside the library's contract: the values are then
    undefined, but C's pattern is the product's, as it is for rows of every other class."""
    rows, offs_a, offs_b = 25000, np.arange(10), np.array([0, 1, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 13, 14, 15])
    k = rows + 10
    tdt = cuda.float64 if dtype == "f64" else cuda.float32

    def band(n, offs):
        return ((np.arange(n + 1) * len(offs)).astype(np.int32),
                (np.arange(n)[:, None] + offs[None, :]).astype(np.int32).ravel(), np.ones(n * len(offs)))

    A = ops.csr_to_device(*band(rows, offs_a), rows, k, dtype=tdt)
    B = ops.csr_to_device(*band(k, offs_b), k, k + 16, dtype=tdt)
    want = band(rows, np.arange(25))
    for mode in (0, 1, 2):
        with ops.Handle() as h:
            h.set_one_pass(mode)
            for multiply in (h.spgemm, h.spgemm_oneshot):
                rpt, col, _ = multiply(A, B).to_host()
                assert np.array_equal(rpt, want[0]) and np.array_equal(col, want[1])
                assert grouped_rows(h) == 0


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("which", ["a", "b"])
def test_changed_matrices_are_refused(cuda, dtype, which):
    """Row pointers that changed behind the plan's back (still those of a CSR matrix): the group
    that they belong to raises the mismatch that the other classes' rows raise, and the same call
    on the matrices of the plan is right again."""
    offs_a, offs_b = np.arange(25), np.arange(0, 40, 2)
    rows = 25000  # 24 windows of 1,024 rows and 424 rows: all of them in groups
    k = rows + 25
    rng = np.random.default_rng(2)
    npdt = np.float64 if dtype == "f64" else np.float32

    def band(n, offs):
        return ((np.arange(n + 1) * len(offs)).astype(np.int32),
                (np.arange(n)[:, None] + offs[None, :]).astype(np.int32).ravel(),
                rng.standard_normal(n * len(offs)).astype(npdt))

    a, b, ncols = band(rows, offs_a), band(k, offs_b), k + 40
    tdt = cuda.float64 if dtype == "f64" else cuda.float32
    A, B = ops.csr_to_device(*a, rows, k, dtype=tdt), ops.csr_to_device(*b, k, ncols, dtype=tdt)
    want = oracle.spgemm(*a, *b, ncols, dtype=npdt)
    with ops.Handle() as h:
        c_rpt, nnz = h.symbolic(A, B)
        changed = (A if which == "a" else B).rpt
        before = changed[1:2].clone()
        # row 0 takes entries of row 1: 40 entries of A, more than a group's rows may have; 35 of B
        changed[1] = 40 if which == "a" else 35
        with pytest.raises(ops.OpsError) as e:
            h.numeric(A, B, c_rpt, nnz)
        assert e.value.status == ops.capi.OPS_COUNT_MISMATCH
        changed[1:2] = before
        c_col, c_val = h.numeric(A, B, c_rpt, nnz)
        check((c_rpt.cpu().numpy(), c_col.cpu().numpy(), c_val.cpu().numpy()), want)
        assert grouped_rows(h) == rows
