"""Reductions and accumulates over axes of length zero: a reduction gives its identity, an accumulate an
empty array, and nothing writes to an array that has no memory. Plans on the CPU; values on a GPU."""
import re

import numpy as np
import pytest

import bohrium_b200 as bh


def accumulates(x, axis):
    return [x.cumsum(axis), x.cumprod(axis), (x + 1).cumsum(axis)]


EMPTY = [((0,), 0), ((0, 5, 7), 0), ((200, 0), 1), ((0, 200), 0), ((5, 0, 3), 1), ((5, 0), 0), ((0, 5), 1)]


@pytest.mark.parametrize("shape,axis", EMPTY)
def test_nothing_writes_to_an_empty_array(shape, axis):
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = accumulates(bh.empty(rt, shape, np.float64), axis)
    plan = bh.dry_run(rt.take(), compile=True)["kernels"]
    written = [m for k in plan for m in re.findall(r"BH_IDENTITY a\d+\[([^\]]*)\]", k["block"])]
    for view in written:  # "first:count:stride" per dimension
        assert any(int(d.split(":")[1]) == 0 for d in view.split(",")), (view, plan)
    assert len(keep) == 3 and not any(u["compile_error"] for k in plan for u in k["units"])


def test_a_reduction_of_nothing_is_launched():
    for prog in (lambda x: [x.sum()], lambda x: [(x * 2 + 1).sum() + 3], lambda x: [x.max(), x.sum()]):
        rt = bh.Runtime(bh.DryRunExecutor())
        keep = prog(bh.empty(rt, (0,), np.float64))
        units = [u for k in bh.dry_run(rt.take(), compile=True)["kernels"] for u in k["units"]]
        assert len(keep) and units and all(u["work"] > 0 and not u["compile_error"] for u in units)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,axis", EMPTY)
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
def test_values(gpu_rt, shape, axis, dtype):
    x = np.zeros(shape, dtype)
    filler = bh.array(gpu_rt, np.full(4096, 77.0))  # memory that has held something else
    gpu_rt.flush()
    del filler
    a = bh.array(gpu_rt, x)
    gpu_rt.flush()
    got = accumulates(a, axis) + [a.sum(axis), a.sum(axis) * 2 + 3, a.prod(axis)]
    gpu_rt.flush()
    total = x.sum(axis, dtype=dtype)
    for g, w in zip(got, [x, x, x, total, total * 2 + 3, x.prod(axis, dtype=dtype)]):
        assert g.numpy().shape == np.shape(w)
        np.testing.assert_array_equal(g.numpy(), w)
