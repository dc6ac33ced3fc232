"""Backward gradients at the edges of their kernels: rows of B and columns of A around a warp
and around the 64 entries up to which one thread folds a chain, empty ones and one long one
of each, with and without the stored position map, bit for bit against the oracle in FP64."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops
from opsparse_gb300.autograd import FixedPatternSpGEMM

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 66, 96, 97, 128, 129, 300]


def factors(rng, m, n):
    """A whose column j has LENGTHS[j // L] entries and B whose row j has LENGTHS[j % L]."""
    L = len(LENGTHS)
    k = L * L
    rows = [np.sort(rng.choice(m, LENGTHS[j // L], replace=False)) for j in range(k)]
    r = np.concatenate(rows)
    c = np.repeat(np.arange(k), [len(x) for x in rows])
    o = np.lexsort((c, r))
    a_rpt = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
    b_len = np.array([LENGTHS[j % L] for j in range(k)])
    b_col = np.concatenate([np.sort(rng.choice(n, x, replace=False)) for x in b_len]).astype(np.int32)
    b_rpt = np.concatenate([[0], np.cumsum(b_len)]).astype(np.int32)
    return ((a_rpt, c[o].astype(np.int32), rng.standard_normal(len(r))),
            (b_rpt, b_col, rng.standard_normal(len(b_col))), k)


@pytest.mark.parametrize("budget", [None, 0], ids=["map", "search"])
@pytest.mark.parametrize("need", [(True, True), (True, False), (False, True)], ids=["both", "a", "b"])
def test_chain_lengths(cuda, budget, need):
    rng = np.random.default_rng(17)
    m, n = 700, 900
    a, b, k = factors(rng, m, n)
    A, B = ops.csr_to_device(*a, m, k), ops.csr_to_device(*b, k, n)
    h = ops.Handle()
    if budget is not None:
        ops.capi.check(h.lib.ops_handle_set_map_budget(h.h, budget))
    op = FixedPatternSpGEMM(A, B, h)
    op.forward_values(A.val, B.val)  # fills C's columns
    w = rng.standard_normal(op.nnz)
    da, db = op.backward_values(A.val, B.val, cuda.as_tensor(w).cuda(), *need)
    assert op.plan_info()[1] == (budget is None)
    oda, odb = oracle.backward(*a, *b, n, op.c_rpt.cpu().numpy().astype(np.int64), op.c_col.cpu().numpy(), w)
    for got, want, asked in ((da, oda, need[0]), (db, odb, need[1])):
        assert (got is not None) == asked
        if asked:
            assert np.array_equal(got.cpu().numpy().view(np.uint64), want.view(np.uint64))
    h.close()


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("budget", [None, 0], ids=["map", "search"])
def test_rows_in_blocks(cuda, budget, dtype):
    """C of more than 14,680,064 entries: dB walks A's rows in blocks, its folds' states kept in
    between (FP64 bit for bit; FP32 within 1e-5 of the FP64 oracle on the same inputs, the
    tolerance of every FP32 gradient)."""
    rng = np.random.default_rng(23)
    m, k, n, da_, db_ = 5000, 6000, 5000, 36, 140

    def random(rows, cols, deg):
        rpt = np.arange(rows + 1, dtype=np.int32) * deg
        col = np.concatenate([np.sort(rng.choice(cols, deg, replace=False)) for _ in range(rows)]).astype(np.int32)
        return rpt, col, rng.standard_normal(rows * deg).astype(np.float32).astype(np.float64)

    a, b = random(m, k, da_), random(k, n, db_)
    tdt = cuda.float64 if dtype == "f64" else cuda.float32
    h = ops.Handle()
    if budget is not None:
        ops.capi.check(h.lib.ops_handle_set_map_budget(h.h, budget))
    A, B = ops.csr_to_device(*a, m, k, dtype=tdt), ops.csr_to_device(*b, k, n, dtype=tdt)
    op = FixedPatternSpGEMM(A, B, h)
    assert op.nnz > 14 << 20
    op.forward_values(A.val, B.val)
    w = rng.standard_normal(op.nnz).astype(np.float32).astype(np.float64)
    for _ in range(2):
        da, db = op.backward_values(A.val, B.val, cuda.as_tensor(w).to(tdt).cuda())
    oda, odb = oracle.backward(*a, *b, n, op.c_rpt.cpu().numpy().astype(np.int64), op.c_col.cpu().numpy(), w)
    for got, want in ((da, oda), (db, odb)):
        got = got.cpu().numpy()
        if dtype == "f64":
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
        else:
            assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1.0)) <= 1e-5
    h.close()
