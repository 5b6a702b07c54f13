"""Recorded kernel times describe one kernel each: recording runs the kernels apart that other flushes
run as one (row groups, tails), also where a plan of the flush was built before it was switched on."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


def test_rows_are_of_single_kernels(gpu_executor):
    ex = gpu_executor
    rt = bh.Runtime(ex)
    x = bh.array(rt, np.random.default_rng(0).standard_normal((300, 700)))
    rt.flush()
    e = bh.exp(x - x.max(1).reshape(300, 1))
    y = e / e.sum(1).reshape(300, 1)
    ir = ex.compile(rt.take())

    def launches():
        n = int(ex.message("CUDA: launches"))
        ir.execute()
        return int(ex.message("CUDA: launches")) - n

    want = None
    try:
        assert launches() == 1  # one row group
        want = ex.peek(y.base)
        ex.message("CUDA: record on")
        count = int(ex.message("CUDA: records count"))
        assert launches() == 3  # maximum; exponential and sum; division
        assert int(ex.message("CUDA: records count")) - count == 3
        # lanes of a row group and of the kernels alone may differ: a sum of 700 terms either way
        np.testing.assert_allclose(ex.peek(y.base), want, rtol=2 * 30 * 1.2e-16, atol=0)
    finally:
        ex.message("CUDA: record off")
    assert launches() == 1
    assert ex.peek(y.base).tobytes() == want.tobytes()
