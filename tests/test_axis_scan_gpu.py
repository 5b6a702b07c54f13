"""Accumulates along one axis of arrays of two or more dimensions (AXIS_SCAN): both layouts, one and
several chunks, the edges of strips and chunks, maps around the accumulate, strided views, and the
forms that keep the thread-per-point schedule. Values are small integers, so every sum is exact in
every type and order and the results must equal NumPy's."""
import numpy as np
import pytest

import bohrium_b200 as bh
from tests.harness import U32, assert_cumsum_within_bound

pytestmark = pytest.mark.gpu


def ints(shape, dtype, seed=0):
    return np.random.default_rng(seed).integers(-3, 4, shape).astype(dtype)


# contiguous axis: below a warp, strip and block edges (32, 256), chunk edges (1024, several chunks)
# other axes: below the unroll, its edges, several chunks and a ragged last one
SHAPES = [((5, 31), 1), ((5, 32), 1), ((9, 33), 1), ((3, 255), 1), ((3, 257), 1), ((2, 1025), 1), ((2, 100_003), 1),
          ((6000, 40), 1), ((1, 7), 0), ((7, 300), 0), ((8, 300), 0), ((9, 257), 0), ((1000, 3), 0), ((100_003, 2), 0),
          ((33, 5, 40), 0), ((5, 70, 40), 1), ((4, 5, 300), 2)]


@pytest.mark.parametrize("shape,axis", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int8, np.complex64])
def test_cumulative_sums(gpu_rt, shape, axis, dtype):
    x = ints(shape, dtype)
    got = bh.accumulate("ADD_ACCUMULATE", bh.array(gpu_rt, x), axis).numpy()
    np.testing.assert_array_equal(got, np.cumsum(x, axis, dtype=dtype))


@pytest.mark.parametrize("shape,axis", [((3, 2100), 1), ((3000, 7), 0)])
def test_maps_around_the_accumulate(gpu_rt, shape, axis):
    """Temporaries and kept arrays before and after the accumulate, and an array read by both."""
    x = ints(shape, np.float64)
    a = bh.array(gpu_rt, x)
    kept = a * 2.0 + 1.0
    c = bh.accumulate("ADD_ACCUMULATE", kept, axis)
    out = c * 3.0 + kept - a
    want_kept = x * 2 + 1
    want_c = np.cumsum(want_kept, axis)
    for got, want in [(out, want_c * 3 + want_kept - x), (c, want_c), (kept, want_kept)]:
        np.testing.assert_array_equal(got.numpy(), want)


@pytest.mark.parametrize("axis", [0, 1])
def test_views_and_arrays_changed_in_place(gpu_rt, axis):
    x = ints((300, 700), np.int64)
    a = bh.array(gpu_rt, x)
    views = [(a[::-1, :], x[::-1, :]), (a[:, ::-1], x[:, ::-1]), (a[3:, 5:650:3], x[3:, 5:650:3]), (a.T, x.T)]
    outs = [bh.accumulate("ADD_ACCUMULATE", v, axis) for v, _ in views]
    for o, (_, w) in zip(outs, views):
        np.testing.assert_array_equal(o.numpy(), np.cumsum(w, axis))
    # the input is changed in the same flush, before and after the accumulate reads it
    b = bh.array(gpu_rt, x)
    bh.binary("ADD", b, 1, out=b)
    c = bh.accumulate("ADD_ACCUMULATE", b, axis)
    bh.binary("MULTIPLY", c, 2, out=b)
    np.testing.assert_array_equal(c.numpy(), np.cumsum(x + 1, axis))
    np.testing.assert_array_equal(b.numpy(), 2 * np.cumsum(x + 1, axis))


def test_products_and_special_values(gpu_rt):
    """Integer products wrap as NumPy's; float products keep one running product per point; NaN and
    infinity reach exactly the elements after them."""
    x = ints((4, 3000), np.int32)
    x[x == 0] = 5
    np.testing.assert_array_equal(bh.array(gpu_rt, x).cumprod(1).numpy(), np.cumprod(x, 1, dtype=np.int32))
    f = np.full((2, 4000), 0.5)
    f[:, 1000:] = 2.0
    np.testing.assert_array_equal(bh.array(gpu_rt, f).cumprod(1).numpy(), np.cumprod(f, 1))
    s = ints((3, 5000), np.float64)
    s[0, 2500], s[1, 70], s[1, 4000], s[2, 0] = np.inf, np.inf, -np.inf, np.nan
    for y, ax in [(s, 1), (np.ascontiguousarray(s.T), 0)]:
        np.testing.assert_array_equal(bh.array(gpu_rt, y).cumsum(ax).numpy(), np.cumsum(y, ax))


@pytest.mark.parametrize("shape,axis", [((3, 50_001), 1), ((50_001, 3), 0)])
def test_rounding_stays_within_the_sequential_bound(gpu_rt, shape, axis):
    """Any order of n additions errs by at most gamma_n sum|x|; chunks keep far fewer roundings: at
    most the strips or elements of a chunk, the chunks, and 8 for the shuffles and the last sum."""
    x = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    got = bh.array(gpu_rt, x).cumsum(axis).numpy()
    g, w = np.moveaxis(got, axis, -1), np.moveaxis(x, axis, -1)
    for r in range(g.shape[0]):
        assert_cumsum_within_bound(g[r], w[r], 2100, U32, f"row {r}")


def test_grouped_launches_are_bit_identical(gpu_executor):
    x = np.random.default_rng(2).standard_normal((6, 3000)).astype(np.float32)
    got = {}
    for mode in ("off", "grouped"):
        gpu_executor.message("CUDA: batch " + mode)
        try:
            rt = bh.Runtime(gpu_executor)
            arrays = [bh.array(rt, x + k) for k in range(4)]
            rt.flush()
            outs = [a.cumsum(1) for a in arrays] + [a.cumsum(0) for a in arrays]
            got[mode] = [o.numpy().tobytes() for o in outs]
        finally:
            gpu_executor.message("CUDA: batch off")
    assert got["off"] == got["grouped"]
