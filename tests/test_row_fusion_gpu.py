"""Row-wise kernels of one flush that run as one (ROWS): softmax and normalisation at the edges of
lanes and registers, kept and dropped intermediate arrays, in-place updates, views, broadcasts of
other arrays, and programs whose rows depend on one another, which must stay apart."""
import numpy as np
import pytest

import bohrium_b200 as bh
from bohrium_b200.inspect import DryRunExecutor, dry_run

pytestmark = pytest.mark.gpu

# lanes 2..256, one and several rows per CTA, a ragged last CTA, the last sizes that fit registers
SHAPES = [(148, 3), (149, 8), (300, 31), (5000, 33), (151, 257), (2000, 1000), (160, 1536), (150, 1537), (149, 3072)]


def scheds(prog, shape, dtype):
    rt = bh.Runtime(DryRunExecutor())
    keep = prog(rt, bh.empty(rt, shape, dtype))
    return [u["sched"] for k in dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]], keep


def softmax(rt, x):
    n = x.shape[0]
    e = bh.exp(x - x.max(1).reshape(n, 1))
    return [e / e.sum(1).reshape(n, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_softmax(gpu_rt, shape, dtype):
    x = (np.random.default_rng(0).standard_normal(shape) * 3).astype(dtype)
    (got,) = softmax(gpu_rt, bh.array(gpu_rt, x))
    e = np.exp(x.astype(np.float64) - x.max(1, keepdims=True))
    want = e / e.sum(1, keepdims=True)
    # exp within 2 ulp, the subtraction and division half an ulp each, the argument's rounding (an
    # error of u |x - max| <= 30 u in the exponent) and a sum of n terms in at most 60 + 8 roundings
    u = np.finfo(dtype).eps / 2
    np.testing.assert_allclose(got.numpy().astype(np.float64), want, rtol=(2 * 2 + 1 + 30 * 2 + 68) * u, atol=0)


def program(rt, x):
    """Integers only, so exact: kept and dropped arrays, values per row with instructions after the
    reduction, a row vector and a column of other arrays, a map after the last reduction."""
    n, c = x.shape
    row = bh.arange(rt, c).astype(x.dtype) % 3
    col = (bh.arange(rt, n).astype(x.dtype) % 5).reshape(n, 1)
    a = x * 2 + row
    m = a.max(1) + 1
    b = a - m.reshape(n, 1) * col
    s = b.sum(1)
    return [b + s.reshape(n, 1), a, m, s]


@pytest.mark.parametrize("shape", SHAPES[:8])
@pytest.mark.parametrize("dtype", [np.int64, np.float64, np.int32])
def test_kept_arrays_and_row_values(gpu_rt, shape, dtype):
    x = np.random.default_rng(1).integers(-9, 9, shape).astype(dtype)
    got = program(gpu_rt, bh.array(gpu_rt, x))
    n, c = shape
    a = x * 2 + (np.arange(c) % 3).astype(dtype)
    m = a.max(1)
    if np.dtype(dtype).kind == "f":  # a floating-point maximum starts from the smallest positive normal number
        m = np.maximum(m, np.finfo(dtype).tiny)
    m = m + 1
    b = (a - m[:, None] * (np.arange(n) % 5).astype(dtype)[:, None]).astype(dtype)
    s = b.sum(1).astype(dtype)
    for g, w in zip(got, [b + s[:, None], a, m, s]):
        np.testing.assert_array_equal(g.numpy(), w)


def test_in_place_views_and_nan(gpu_rt):
    x = np.random.default_rng(2).integers(-9, 9, (300, 200)).astype(np.float64)
    x[5, 7], x[6, 0], x[7, 3] = np.nan, np.inf, -np.inf
    a = bh.array(gpu_rt, x)
    v = a[:, 3:190]
    bh.binary("SUBTRACT", v, v.max(1).reshape(300, 1), out=v)
    s = v.sum(1)
    bh.binary("ADD", v, s.reshape(300, 1), out=v)
    w = x.copy()
    with np.errstate(invalid="ignore"):
        # the engine's maximum keeps x when the comparison with it is false, NumPy's returns NaN
        mx = np.array([np.nan if np.isnan(r).any() else r.max() for r in w[:, 3:190]])
        w[:, 3:190] -= mx[:, None]
        w[:, 3:190] += w[:, 3:190].sum(1)[:, None]
    rows = np.array([r for r in range(300) if r not in (5, 6, 7)])
    np.testing.assert_array_equal(a.numpy()[rows], w[rows])


def test_rows_that_depend_on_one_another_stay_apart(gpu_rt):
    x = np.random.default_rng(3).integers(-9, 9, (400, 64)).astype(np.float64)

    def prog(rt, a):
        n = a.shape[0]
        b = a - a.max(1).reshape(n, 1)      # row by row
        c = b[::-1, :] + b.sum(1).reshape(n, 1)  # but this reads another row of b
        return [b, c]

    got = prog(gpu_rt, bh.array(gpu_rt, x))
    b = x - x.max(1, keepdims=True)
    np.testing.assert_array_equal(got[1].numpy(), b[::-1] + b.sum(1, keepdims=True))
    np.testing.assert_array_equal(got[0].numpy(), b)


def test_which_programs_fuse():
    assert scheds(softmax, (20000, 1500), np.float32)[0] == ["rows"]
    assert scheds(softmax, (149, 3072), np.float32)[0] == ["rows"]
    assert "rows" not in scheds(softmax, (149, 3073), np.float32)[0]
    assert "rows" not in scheds(softmax, (100, 1000), np.float32)[0]  # too few rows for a lane schedule


def test_grouped_launches_are_bit_identical(gpu_executor):
    x = np.random.default_rng(4).standard_normal((200, 700)).astype(np.float32)
    got = {}
    for mode in ("off", "grouped", "graph"):
        gpu_executor.message("CUDA: batch " + mode)
        try:
            rt = bh.Runtime(gpu_executor)
            arrays = [bh.array(rt, x + k) for k in range(3)]
            rt.flush()
            got[mode] = [softmax(rt, a)[0].numpy().tobytes() for a in arrays]
        finally:
            gpu_executor.message("CUDA: batch off")
    assert got["off"] == got["grouped"] == got["graph"]
