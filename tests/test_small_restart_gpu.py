"""Problems that look small by their entry counts but have rows beyond the small problems' one
kernel (hub graphs): the usual pipeline goes on from the row classes that are there, and no row
is set up or counted twice.  Launch counts, and both calls against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import opsparse_gb300 as ops
from opsparse_gb300 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,degree", [(500, 4), (8000, 6), (16384, 5)])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_the_pipeline_goes_on(cuda, dtype, rows, degree):
    npdt = np.float64 if dtype == "f64" else np.float32
    a = gen.powerlaw_square(rows, degree, 2.2, seed=rows)
    a = (a[0], a[1], a[2].astype(npdt))
    products = gen.row_flop(a[0], a[1], a[0])
    assert products.max() > 256 and products.mean() < 96
    A = ops.csr_to_device(*a, rows, rows, dtype=cuda.float64 if dtype == "f64" else cuda.float32)
    orpt, ocol, oval = oracle.spgemm(*a, *a, rows, dtype=npdt)
    launches = []
    for timing in (0, 2):  # at level 2 no problem is a small one
        with ops.Handle(timing=timing) as h:
            for multiply in (h.spgemm_oneshot, h.spgemm, h.spgemm_oneshot):
                rpt, col, val = multiply(A, A).to_host()
                assert np.array_equal(rpt.astype(np.int64), orpt) and np.array_equal(col, ocol)
                assert np.array_equal(val.view(np.uint8), oval.view(np.uint8))
            h.symbolic(A, A)
            launches.append(h.timings()["launches"])
    assert launches[0] == launches[1] + 2  # the kernel that takes every row, and its scan
