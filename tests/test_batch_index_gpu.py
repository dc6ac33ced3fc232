"""Batch results by an index that the batch does not have: refused, by either way to read them."""
import pytest

import opsparse_gb300 as ops
from opsparse_gb300 import capi, gen

pytestmark = pytest.mark.gpu


def test_index_outside_the_batch_is_refused(cuda):
    pairs = []
    for i, n in enumerate((300, 64, 500)):
        A = ops.csr_to_device(*gen.erdos_renyi(n, 4.0, seed=i), n, n)
        pairs.append((A, A))
    with ops.Handle() as h:
        batch = ops.Batch(h, pairs)
        batch.execute(False)
        batch.check()
        for read in (batch.result, batch.result_device):
            for i in (-1, -3, 3, 1 << 20):
                with pytest.raises(ops.OpsError) as e:
                    read(i)
                assert e.value.status == capi.OPS_INVALID_ARGUMENT
            read(2)
        batch.close()
        with pytest.raises(ops.OpsError):
            batch.result_device(0)
