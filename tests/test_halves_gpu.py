"""ops_spgemm in two halves (ops_spgemm_begin / ops_spgemm_finish), which Handle.spgemm_oneshot
calls, and the batch's results in one call: the same results as ops_spgemm and result(), the
misuses reported, the other calls of a handle between the halves."""
import ctypes as C

import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops
from opsparse_gb300 import capi, gen

pytestmark = pytest.mark.gpu


def begin(h, A, B, c_rpt):
    a, b, nnz = A.ptrs(), B.ptrs(), C.c_int64(0)
    st = h.lib.ops_spgemm_begin(h.h, ops._dtype_code(A.val), A.rows, A.cols, B.cols, a[0], a[1], a[2], A.nnz, b[0],
                                b[1], b[2], B.nnz, c_rpt.data_ptr(), C.byref(nnz), ops._stream_ptr())
    return st, int(nnz.value)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_halves_equal_the_whole(cuda, dtype, mode):
    torch = cuda
    tdt = torch.float64 if dtype == "f64" else torch.float32
    rpt, col, val = gen.web_powerlaw(20000, lmax=2000)
    A = ops.csr_to_device(rpt, col, val, 20000, 20000, dtype=tdt)
    ref = ops.Handle().spgemm(A, A).to_host()
    other = torch.cuda.Stream()
    with ops.Handle() as h:
        h.set_one_pass(mode)
        for stream in (None, torch.cuda.current_stream(), other, None):
            got = h.spgemm_oneshot(A, A, stream=stream).to_host()
            assert all(np.array_equal(x.view(np.uint8), y.view(np.uint8)) for x, y in zip(got, ref))


def test_misuse_and_calls_between(cuda):
    torch = cuda
    a = gen.erdos_renyi(3000, 12.0)
    A = ops.csr_to_device(*a, 3000, 3000)
    o = oracle.spgemm(*a, *a, 3000)
    c_rpt = torch.empty(3001, dtype=torch.int32, device="cuda")
    with ops.Handle() as h:
        h.set_one_pass(2)
        st = ops._stream_ptr()
        assert h.lib.ops_spgemm_finish(h.h, None, None, st) == capi.OPS_NOT_SUPPORTED
        s, nnz = begin(h, A, A, c_rpt)
        assert s == capi.OPS_OK and nnz == len(o[1])
        # a plain numeric call between the halves ends the begun one and computes every row
        c_col, c_val = h.numeric(A, A, c_rpt, nnz)
        assert np.array_equal(c_val.cpu().numpy().view(np.uint64), o[2].view(np.uint64))
        assert h.lib.ops_spgemm_finish(h.h, c_col.data_ptr(), c_val.data_ptr(), st) == capi.OPS_NOT_SUPPORTED
        begin(h, A, A, c_rpt)
        h.symbolic(A, A)
        assert h.lib.ops_spgemm_finish(h.h, c_col.data_ptr(), c_val.data_ptr(), st) == capi.OPS_NOT_SUPPORTED
        begin(h, A, A, c_rpt)
        assert h.lib.ops_spgemm_finish(h.h, None, None, st) == capi.OPS_INVALID_ARGUMENT
        begin(h, A, A, c_rpt)
        c_col.zero_()
        c_val.zero_()
        assert h.lib.ops_spgemm_finish(h.h, c_col.data_ptr(), c_val.data_ptr(), st) == capi.OPS_OK
        assert np.array_equal(c_col.cpu().numpy(), o[1])
        assert np.array_equal(c_val.cpu().numpy().view(np.uint64), o[2].view(np.uint64))


def test_batch_views_equal_results(cuda):
    torch = cuda
    pairs = []
    for i, n in enumerate((300, 64, 500, 1, 900)):
        m = gen.erdos_renyi(n, 0.0 if n == 64 else 6.0, seed=i)  # one problem without entries
        pairs.append((ops.csr_to_device(*m, n, n), ops.csr_to_device(*m, n, n)))
    h = ops.Handle()
    batch = ops.Batch(h, pairs)
    batch.execute(False)
    batch.check()
    for i in range(len(pairs)):
        rpt, col, val, nnz = batch.result_device(i)
        r = batch.result(i)
        assert nnz == len(r[1]) and np.array_equal(rpt.cpu().numpy(), r[0])
        assert np.array_equal(col.cpu().numpy(), r[1]) and np.array_equal(val.cpu().numpy(), r[2])
    batch.close()
    h.close()
