"""Infinities and NaN in rows that run as one kernel (row fusion) and as kernels of their own: an in-place
normalisation of a view, against NumPy and against each other."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


@pytest.fixture
def executors(monkeypatch):
    """An engine that fuses rows and one that does not."""
    both = []
    for value in ("true", "false"):
        monkeypatch.setenv("BH_CUDA_FUSE_ROWS", value)
        both.append(bh.NativeExecutor(stack="cuda"))
    yield both
    for ex in both:
        ex.close()


def inputs(dtype):
    x = np.random.default_rng(2).integers(-9, 9, (300, 200)).astype(dtype)
    x[:, 5] = 20  # every row's maximum is positive: a floating-point maximum starts from the smallest normal number
    x[6, 4], x[7, 60], x[8, 4], x[8, 100] = np.inf, -np.inf, np.inf, -np.inf
    return x


def in_place(a, n, maximum, total):
    v = a[:, 3:190]
    m = maximum(v).reshape(n, 1)
    if isinstance(a, np.ndarray):
        v -= m
        v += total(v).reshape(n, 1)
    else:
        bh.binary("SUBTRACT", v, m, out=v)
        bh.binary("ADD", v, total(v).reshape(n, 1), out=v)
    return a


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_infinities(executors, dtype):
    x = inputs(dtype)
    with np.errstate(invalid="ignore"):
        want = in_place(x.copy(), 300, lambda v: v.max(1), lambda v: v.sum(1))
    assert np.isnan(want[6]).any() and np.isinf(want[7]).any() and np.isnan(want[8]).any()
    for k, ex in enumerate(executors):
        rt = bh.Runtime(ex)
        a = bh.array(rt, x)
        rt.flush()
        launches = int(ex.message("CUDA: launches"))
        in_place(a, 300, lambda v: v.max(1), lambda v: v.sum(1))
        rt.flush()
        launches = int(ex.message("CUDA: launches")) - launches
        assert launches == 1 if k == 0 else launches > 1
        np.testing.assert_array_equal(a.numpy(), want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_nan_reaches_the_sums_of_its_row_only(executors, dtype):
    x = inputs(dtype)
    x[5, 7], x[9, 0] = np.nan, np.nan  # inside and outside the view
    with np.errstate(invalid="ignore"):
        v = x[:, 3:190]
        s = v.sum(1)
        want = [v * 2 - s[:, None], s, (v * 2 - s[:, None]).sum(1)]
    assert np.isnan(want[1][5]) and not np.isnan(want[1][9])
    for ex in executors:
        rt = bh.Runtime(ex)
        a = bh.array(rt, x)
        rt.flush()
        w = a[:, 3:190]
        t = w.sum(1)
        y = w * 2 - t.reshape(300, 1)
        got = [y, t, y.sum(1)]
        rt.flush()
        for g, q in zip(got, want):
            np.testing.assert_array_equal(g.numpy(), q)
