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
