"""Small problems (k_rank_all, k_scan_rows): every row by one kernel, launched before the row
sizes are known, and the usual pipeline where some row turns out too large for it.  Rows
either side of the kernel's capacity, row counts either side of the limits, empty rows and
long rows of few products, thresholds that leave its classes out, bad columns; FP64 and FP32,
both calls, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops
from opsparse_gb300 import gen

pytestmark = pytest.mark.gpu


def with_row(products, len_a, rows=50, seed=2):
    """`rows` light rows and one row of `products` products over `len_a` A entries."""
    rng = np.random.default_rng(seed)
    k, ncols = 2000, 5000
    b_len = rng.integers(0, 6, k)
    own = np.sort(rng.choice(k, len_a, replace=False))
    share = np.full(len_a, products // len_a)
    share[:products % len_a] += 1
    b_len[own] = share  # entries without products where len_a > products
    lens = np.r_[rng.integers(0, 8, rows), len_a]
    a_col = np.concatenate([np.sort(rng.choice(k, n, replace=False)) for n in lens[:-1]] + [own]).astype(np.int32)
    a_rpt = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    b_rpt = np.concatenate([[0], np.cumsum(b_len)]).astype(np.int32)
    b_col = np.concatenate([np.sort(rng.choice(ncols, n, replace=False)) for n in b_len]).astype(np.int32)
    return (a_rpt, a_col, rng.standard_normal(len(a_col))), (b_rpt, b_col, rng.standard_normal(len(b_col))), k, ncols


def check(cuda, a, b, k, ncols, dtype, thresholds=None):
    torch = cuda
    npdt = np.float64 if dtype == "f64" else np.float32
    a = (a[0], a[1], a[2].astype(npdt))
    b = (b[0], b[1], b[2].astype(npdt))
    A = ops.csr_to_device(*a, len(a[0]) - 1, k, dtype=torch.float64 if dtype == "f64" else torch.float32)
    B = ops.csr_to_device(*b, k, ncols, dtype=A.val.dtype)
    orpt, ocol, oval = oracle.spgemm(*a, *b, ncols, dtype=npdt)
    with ops.Handle() as h:
        if thresholds:
            h.set_thresholds(thresholds)
        for multiply in (h.spgemm, h.spgemm_oneshot, h.spgemm):
            rpt, col, val = multiply(A, B).to_host()
            assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
            assert np.array_equal(val.view(np.uint8), oval.view(np.uint8))


@pytest.mark.parametrize("products,len_a", [(8, 8), (9, 3), (128, 128), (128, 700), (129, 129), (200, 128), (200, 130),
                                            (256, 100), (257, 100), (1024, 64), (14000, 900)])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_one_row_at_the_capacity(cuda, dtype, products, len_a):
    check(cuda, *with_row(products, len_a), dtype)


@pytest.mark.parametrize("rows", [1, 2, 4095, 4096, 16383, 16384, 16385, 32768, 32769])
def test_row_counts_at_the_limits(cuda, rows):
    a = gen.erdos_renyi(rows, 3.0, seed=rows, ncols=500)
    b = gen.erdos_renyi(500, 4.0, seed=1, ncols=700)
    check(cuda, a, b, 500, 700, "f64")


@pytest.mark.parametrize("thresholds", [[0, 0, 0, 0, 0, 0], [8, 0, 0, 0, 1024, 13312], [0, 16, 32, 128, 1024, 13312],
                                        [4, 0, 32, 64, 128, 13312]])
def test_thresholds(cuda, thresholds):
    check(cuda, *with_row(150, 40), "f64", thresholds)


@pytest.mark.parametrize("which", ["a", "b"])
def test_bad_columns(cuda, which):
    a, b, k, ncols = with_row(100, 20)
    m = a if which == "a" else b
    m[1][len(m[1]) - 1] = k if which == "a" else ncols  # the long row's last entry; B's last
    if which == "b":
        a[1][a[0][-1] - 1] = k - 1  # the long row reaches B's last row
        b[0][-2] = min(b[0][-2], b[0][-1] - 1)
    with ops.Handle() as h:
        A, B = ops.csr_to_device(*a, len(a[0]) - 1, k), ops.csr_to_device(*b, k, ncols)
        for multiply in (h.spgemm, h.spgemm_oneshot):
            with pytest.raises(ops.OpsError):
                multiply(A, B)
