"""Backward calls beside one another and by other routes than one call at a time: two of one
handle at once on two streams, a captured one, and one whose B no longer has an entry of the
plan.  FP64, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops
from opsparse_gb300 import capi
from opsparse_gb300.autograd import FixedPatternSpGEMM

pytestmark = pytest.mark.gpu


def regular_degrees(rows, cols, deg, rng):
    col = np.concatenate([np.sort(rng.choice(cols, deg, replace=False)) for _ in range(rows)]).astype(np.int32)
    return np.arange(rows + 1, dtype=np.int32) * deg, col, rng.standard_normal(rows * deg)


class Product:
    """A fixed product on a handle, its gradients from the library and from the oracle."""

    def __init__(self, cuda, m, k, n, deg_a, deg_b, seed=31):
        self.cuda, self.rng = cuda, np.random.default_rng(seed)
        self.a, self.b = regular_degrees(m, k, deg_a, self.rng), regular_degrees(k, n, deg_b, self.rng)
        self.A, self.B = ops.csr_to_device(*self.a, m, k), ops.csr_to_device(*self.b, k, n)
        self.h = ops.Handle()
        self.op = FixedPatternSpGEMM(self.A, self.B, self.h)
        self.op.forward_values(self.A.val, self.B.val)  # fills C's columns

    def dc(self):
        return self.cuda.as_tensor(self.rng.standard_normal(self.op.nnz)).cuda()

    def outputs(self):
        return self.cuda.full_like(self.A.val, np.nan), self.cuda.full_like(self.B.val, np.nan)

    def call(self, dc, da, db, stream):
        A, B, op = self.A, self.B, self.op
        capi.check(self.h.lib.ops_spgemm_backward(
            self.h.h, capi.OPS_F64, A.rows, A.cols, B.cols, A.rpt.data_ptr(), A.col.data_ptr(), A.val.data_ptr(), A.nnz,
            B.rpt.data_ptr(), B.col.data_ptr(), B.val.data_ptr(), B.nnz, op.c_rpt.data_ptr(), op.c_col.data_ptr(),
            dc.data_ptr(), da.data_ptr() if da is not None else None, db.data_ptr(), ops._stream_ptr(stream)), self.h.h)

    def check(self, dc, da, db):
        want = oracle.backward(*self.a, *self.b, self.B.cols, self.op.c_rpt.cpu().numpy().astype(np.int64),
                               self.op.c_col.cpu().numpy(), dc.cpu().numpy())
        for got, w in zip((da, db), want):
            assert np.array_equal(got.cpu().numpy().view(np.uint64), w.view(np.uint64))


@pytest.mark.parametrize("blocks", [False, True], ids=["one_block", "blocks"])
def test_two_streams_at_once(cuda, blocks):
    """Chains of dA longer than 64 (listed), with dB in one block and in two."""
    p = Product(cuda, *((5000, 6000, 5000, 36, 140) if blocks else (3000, 800, 4000, 20, 90)))
    assert (p.op.nnz > 14 << 20) == blocks
    first, streams = p.outputs(), [cuda.cuda.Stream(), cuda.cuda.Stream()]
    p.call(p.dc(), *first, None)  # the plan
    cuda.cuda.synchronize()
    dcs = [p.dc(), p.dc()]
    rounds = [[p.outputs(), p.outputs()] for _ in range(4)]
    cuda.cuda.synchronize()
    for outs in rounds:
        for i in (0, 1):
            p.call(dcs[i], *outs[i], streams[i])
    cuda.cuda.synchronize()
    capi.check(p.h.lib.ops_spgemm_check(p.h.h, ops._stream_ptr()), p.h.h)
    for i in (0, 1):
        p.check(dcs[i], *rounds[0][i])
        for outs in rounds[1:]:
            assert all(bool((x == y).all()) for x, y in zip(outs[i], rounds[0][i]))
    p.h.close()


@pytest.mark.parametrize("how", ["stream", "graph"])
def test_new_plan_on_another_stream(cuda, how):
    """A plan that was just built, used at once on another stream, or by a graph that was captured
    on its own stream and runs on another."""
    p = Product(cuda, 6000, 800, 4000, 30, 90)
    own, other = cuda.cuda.Stream(), cuda.cuda.Stream()
    dc, outs = p.dc(), [p.outputs(), p.outputs()]
    cuda.cuda.synchronize()
    for _ in range(4):
        capi.check(p.h.lib.ops_handle_set_map_budget(p.h.h, 8 << 30))  # drops the plan
        for t in outs[1]:
            t.fill_(np.nan)
        cuda.cuda.synchronize()
        p.call(dc, *outs[0], own)
        if how == "stream":
            p.call(dc, *outs[1], other)
        else:
            graph = cuda.cuda.CUDAGraph()
            with cuda.cuda.stream(own):
                graph.capture_begin()
                p.call(dc, *outs[1], own)
                graph.capture_end()
            with cuda.cuda.stream(other):
                graph.replay()
        cuda.cuda.synchronize()
        capi.check(p.h.lib.ops_spgemm_check(p.h.h, ops._stream_ptr()), p.h.h)
        p.check(dc, *outs[1])
        graph = None
    p.h.close()


def test_captured_call(cuda):
    """A built plan's call in a graph, replayed with new dC; C of more entries than one block."""
    p = Product(cuda, 5000, 6000, 5000, 36, 140)
    dc, (da, db) = p.dc(), p.outputs()
    p.call(dc, da, db, None)
    cuda.cuda.synchronize()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        p.call(dc, da, db, cuda.cuda.current_stream())
    for _ in range(2):
        dc.copy_(p.dc())
        da.fill_(np.nan)
        db.fill_(np.nan)
        graph.replay()
    cuda.cuda.synchronize()
    p.check(dc, da, db)
    del graph
    p.h.close()


@pytest.mark.parametrize("rows", [1000, 3000], ids=["short_column", "long_column"])
def test_entry_off_the_plan_is_refused(cuda, rows):
    """B's last row loses its last entry behind the plan's back: no gradient for it, an error.
    Columns of A of about 25 entries (a thread per entry of B) and of about 75 (a warp)."""
    p = Product(cuda, rows, 800, 4000, 20, 30)
    dc, (da, db) = p.dc(), p.outputs()
    p.call(dc, None, db, None)
    capi.check(p.h.lib.ops_spgemm_check(p.h.h, ops._stream_ptr()), p.h.h)
    last = float(db[-1])
    assert np.isfinite(last)
    p.B.rpt[-1] -= 1
    db.fill_(np.nan)
    p.call(dc, None, db, None)
    assert p.h.lib.ops_spgemm_check(p.h.h, ops._stream_ptr()) == capi.OPS_COUNT_MISMATCH
    assert bool(cuda.isnan(db[-1])) and bool(cuda.isfinite(db[:-1]).all())
    p.B.rpt[-1] += 1  # the handle and its plan stay usable
    p.call(dc, None, db, None)
    capi.check(p.h.lib.ops_spgemm_check(p.h.h, ops._stream_ptr()), p.h.h)
    assert float(db[-1]) == last
    p.h.close()


def used(cuda):
    cuda.cuda.synchronize()
    free, total = cuda.cuda.mem_get_info()
    return total - free


def test_replaced_plans_are_given_back(cuda):
    """Each plan of a fixed product of 16.2 million products holds a map of 65 MB; twelve more of
    them on one handle, and on handles of their own, take no more memory than the first two did."""
    p = Product(cuda, 6000, 800, 4000, 30, 90)
    dc, (da, db) = p.dc(), p.outputs()

    def build(h):
        for budget in (8 << 30, 8 << 30):  # setting the budget drops the plan
            capi.check(h.lib.ops_handle_set_map_budget(h.h, budget))
            p.h = h
            p.call(dc, da, db, None)
            assert p.op.plan_info() == (16_200_000, True)

    own = p.h
    build(own)
    before = used(cuda)
    for _ in range(6):
        build(own)
    assert used(cuda) - before < 64 << 20
    p.check(dc, da, db)
    with ops.Handle() as h:
        p.op.h = h
        build(h)
    before = used(cuda)
    for _ in range(6):
        with ops.Handle() as h:
            p.op.h = h
            build(h)
    assert used(cuda) - before < 64 << 20
    own.close()
