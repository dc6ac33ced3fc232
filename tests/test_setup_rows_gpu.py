"""The setup kernel's ways to sum a row of A (a thread, eight lanes, a warp, the whole CTA), at
the edges of their ranges and with more of the longest rows in one CTA than its list holds:
product counts and results against the oracle, and a column outside B reported by each."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 31, 32, 33, 64, 127, 128, 129, 255, 257, 1023, 1024, 1025, 2600, 5000]


def rows_of(lengths, seed=3):
    rng = np.random.default_rng(seed)
    k, ncols = 6000, 300
    a_rpt = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    a_col = np.concatenate([np.sort(rng.choice(k, n, replace=False)) for n in lengths]).astype(np.int32)
    b_len = rng.integers(0, 4, k)
    b_rpt = np.concatenate([[0], np.cumsum(b_len)]).astype(np.int32)
    b_col = np.concatenate([np.sort(rng.choice(ncols, n, replace=False)) for n in b_len]).astype(np.int32)
    return (a_rpt, a_col, rng.standard_normal(len(a_col))), (b_rpt, b_col, rng.standard_normal(len(b_col))), k, ncols


@pytest.mark.parametrize("lengths", [LENGTHS, LENGTHS[::-1] * 3, [1100] * 40 + [5, 20, 200]],
                         ids=["each", "mixed", "many_long"])
def test_rows_of_every_length(cuda, lengths):
    a, b, k, ncols = rows_of(lengths)
    A = ops.csr_to_device(*a, len(lengths), k)
    B = ops.csr_to_device(*b, k, ncols)
    total, _ = oracle.flop(a[0], a[1], b[0])
    orpt, ocol, oval = oracle.spgemm(*a, *b, ncols)
    with ops.Handle() as h:
        rpt, col, val = h.spgemm(A, B).to_host()
        assert h.timings()["flop"] == total
    assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
    assert np.array_equal(val.view(np.uint64), oval.view(np.uint64))


@pytest.mark.parametrize("length", [8, 9, 128, 129, 1024, 1025, 5000])
def test_bad_column_in_every_length(cuda, length):
    a, b, k, ncols = rows_of([3, length, 40])
    for where in (3, 3 + length // 2, 3 + length - 1):
        col = a[1].copy()
        col[where] = k
        with ops.Handle() as h, pytest.raises(ops.OpsError):
            h.spgemm(ops.csr_to_device(a[0], col, a[2], 3, k), ops.csr_to_device(*b, k, ncols))
