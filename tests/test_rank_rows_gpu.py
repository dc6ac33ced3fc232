"""The rank row kernels (rank.cuh) at the edges of their shapes: rows of 1 to 13,312 products
either side of each shape's capacity, B widths either side of each trie depth, columns that
never, sometimes and mostly repeat, A entries with empty B rows between them; two passes
and one pass, FP64 and FP32.  The results are the oracle's fold in the same order, so they
are compared bit for bit.
"""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops

pytestmark = pytest.mark.gpu

SIZES = [9, 17, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 4095, 4096, 4097, 13311,
         13312]


def edge_case(ncols, seed):
    """Per size and kind one A row over B rows of its own (1 to 40 entries, every fifth one
    empty); kinds: distinct columns, one column in 20 repeated, a quarter of the columns."""
    rng = np.random.default_rng(seed)
    b_rows, a_len = [], []
    for n in SIZES:
        for pool in (n, max(1, n - max(1, n // 20)), max(1, n // 4)):
            cols = np.unique(rng.integers(0, ncols, 2 * pool + 8))
            cols = rng.permutation(cols)[:pool]
            left, rows = n, 0
            queue = np.concatenate([rng.permutation(cols) for _ in range(-(-n // max(1, len(cols))) + 1)])
            at = 0
            while left > 0:
                if rows % 5 == 4:
                    b_rows.append(np.zeros(0, np.int64))
                else:
                    take = min(left, int(rng.integers(1, 41)), len(cols))
                    row = np.unique(queue[at:at + take])  # a B row holds a column once
                    at = (at + take) % (len(queue) - len(cols))
                    b_rows.append(row)
                    left -= len(row)
                rows += 1
            a_len.append(rows)
    a_rpt = np.concatenate([[0], np.cumsum(a_len)]).astype(np.int32)
    a_col = np.arange(a_rpt[-1], dtype=np.int32)
    b_rpt = np.concatenate([[0], np.cumsum([len(r) for r in b_rows])]).astype(np.int32)
    b_col = np.concatenate(b_rows).astype(np.int32)
    return (a_rpt, a_col, rng.standard_normal(len(a_col))), (b_rpt, b_col, rng.standard_normal(len(b_col)))


# one, two, three and more trie levels, and the widths either side of the warp shapes' depths
@pytest.mark.parametrize("ncols", [40000, 8192 * 32, 8192 * 32 + 1, (1 << 20) + 1, (1 << 23) + 1, (1 << 30) + 5])
@pytest.mark.parametrize("oneshot", [False, True], ids=["two_phase", "one_pass"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_rank_rows_at_their_edges(cuda, dtype, oneshot, ncols):
    torch = cuda
    npdt = np.float64 if dtype == "f64" else np.float32
    a, b = edge_case(ncols, 7)
    a = (a[0], a[1], a[2].astype(npdt))
    b = (b[0], b[1], b[2].astype(npdt))
    A = ops.csr_to_device(*a, len(a[0]) - 1, len(b[0]) - 1, dtype=torch.float64 if dtype == "f64" else torch.float32)
    B = ops.csr_to_device(*b, len(b[0]) - 1, ncols, dtype=A.val.dtype)
    with ops.Handle() as h:
        h.set_one_pass(2)
        C = h.spgemm_oneshot(A, B) if oneshot else h.spgemm(A, B)
        rpt, col, val = C.to_host()
    orpt, ocol, oval = oracle.spgemm(*a, *b, ncols, dtype=npdt)
    assert np.array_equal(rpt.astype(np.int64), orpt)
    assert np.array_equal(col, ocol)
    bits = np.uint64 if dtype == "f64" else np.uint32
    assert np.array_equal(val.view(bits), oval.view(bits))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_rank_rows_in_a_batch(cuda, dtype):
    """The same rows through the batch's queues (up to 4,096 products), with a problem of
    narrow B beside one of wide B."""
    torch = cuda
    tdt = torch.float64 if dtype == "f64" else torch.float32
    pairs, refs = [], []
    for ncols, seed in ((40000, 3), ((1 << 21) + 3, 4)):
        a, b = edge_case(ncols, seed)
        m = 3 * SIZES.index(4097)
        nnz = a[0][m]
        a = (a[0][:m + 1], a[1][:nnz], a[2][:nnz].astype(np.float64 if dtype == "f64" else np.float32))
        b = (b[0], b[1], b[2].astype(a[2].dtype))
        pairs.append((ops.csr_to_device(*a, m, len(b[0]) - 1, dtype=tdt),
                      ops.csr_to_device(*b, len(b[0]) - 1, ncols, dtype=tdt)))
        refs.append(oracle.spgemm(*a, *b, ncols, dtype=a[2].dtype.type))
    h = ops.Handle()
    batch = ops.Batch(h, pairs)
    assert batch.queues()[0] is True
    batch.execute(False)
    batch.check()
    for i, (orpt, ocol, oval) in enumerate(refs):
        rpt, col, val = batch.result(i)
        assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
        assert np.array_equal(val.view(np.uint8), oval.view(np.uint8))
    batch.close()
    h.close()
