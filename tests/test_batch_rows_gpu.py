"""Batches whose rows of A are longer than the queues' shapes hold entries, most of them over
empty B rows: the shapes count entries with products, so the batch keeps its persistent kernels.
Rows either side of the bounds, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops

pytestmark = pytest.mark.gpu


def problem(products, len_a, dtype, seed):
    """30 rows of len_a entries over `products` products: B's rows have at most a few entries."""
    rng = np.random.default_rng(seed)
    k, n, rows = 4000, 3000, 30
    own = np.sort(rng.choice(k, len_a, replace=False))
    b_len = np.zeros(k, np.int64)
    np.add.at(b_len, rng.choice(own, products), 1)
    a_rpt = (np.arange(rows + 1) * len_a).astype(np.int32)
    b_rpt = np.concatenate([[0], np.cumsum(b_len)]).astype(np.int32)
    b_col = np.concatenate([np.sort(rng.choice(n, x, replace=False)) for x in b_len]).astype(np.int32)
    return ((a_rpt, np.tile(own, rows).astype(np.int32), rng.standard_normal(rows * len_a).astype(dtype)),
            (b_rpt, b_col, rng.standard_normal(len(b_col)).astype(dtype)), rows, k, n)


@pytest.mark.parametrize("warp_max", [128, 512])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_long_rows_of_few_products(cuda, dtype, warp_max):
    npdt, tdt = (np.float64, cuda.float64) if dtype == "f64" else (np.float32, cuda.float32)
    problems = [problem(f, n, npdt, f + n) for f in (128, 129, 256, 300, 512, 513, 1024, 1280)
                for n in (128, 193, 513, 1280, 1281, 3900)]
    pairs = [(ops.csr_to_device(*a, m, k, dtype=tdt), ops.csr_to_device(*b, k, n, dtype=tdt))
             for a, b, m, k, n in problems]
    with ops.Handle() as h:
        h.set_tuning(batch_warp_max=warp_max)
        batch = ops.Batch(h, pairs)
        assert batch.queues()[0] is True
        batch.execute(False)
        batch.check()
        for i, (a, b, _, _, n) in enumerate(problems):
            rpt, col, val = batch.result(i)[:3]
            orpt, ocol, oval = oracle.spgemm(*a, *b, n, dtype=npdt)
            assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
            assert np.array_equal(val.view(np.uint8), oval.view(np.uint8))
        batch.close()
