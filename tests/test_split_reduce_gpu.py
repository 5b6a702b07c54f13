"""Reductions of one axis over few points (SPLIT_REDUCE): points side by side in a CTA with several
groups along the axis, one point per CTA when the axis is contiguous, one and many chunks, ragged
last blocks. Values are small integers, so sums are exact and must equal NumPy's in every type."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


def ints(shape, dtype, seed=0):
    return np.random.default_rng(seed).integers(-3, 4, shape).astype(dtype)


@pytest.mark.parametrize("points", [1, 2, 3, 50, 85, 86, 127, 128, 129, 255, 256, 257, 1000])
@pytest.mark.parametrize("rows", [32, 127, 4099])
@pytest.mark.parametrize("dtype", [np.float32, np.int64, np.complex128])
def test_sums_over_the_outer_axis(gpu_rt, points, rows, dtype):
    x = ints((rows, points), dtype)
    np.testing.assert_array_equal(bh.array(gpu_rt, x).sum(0).numpy(), x.sum(0, dtype=dtype))


@pytest.mark.parametrize("points,n", [(2, 33), (3, 4096), (5, 100_003), (147, 255), (147, 257), (147, 70_001)])
@pytest.mark.parametrize("op", ["ADD", "MAXIMUM"])
def test_few_points_along_the_contiguous_axis(gpu_rt, points, n, op):
    x = ints((points, n), np.float64)
    got = bh.reduce(op + "_REDUCE", bh.array(gpu_rt, x), 1).numpy()
    np.testing.assert_array_equal(got, x.sum(1) if op == "ADD" else x.max(1))


@pytest.mark.parametrize("shape,axis", [((3, 5000, 7), 1), ((300, 4, 5), 0), ((2, 3, 9000), 2)])
def test_three_dimensions_views_and_kept_maps(gpu_rt, shape, axis):
    """A kept map, two reductions of it in one nest, a reversed view, and NaN."""
    x = ints(shape, np.float64)
    a = bh.array(gpu_rt, x)
    y = a * 2.0 + 1.0
    s, m, r = y.sum(axis), y.max(axis), a[::-1].sum(axis)
    want = x * 2 + 1
    for got, w in [(s, want.sum(axis)), (m, want.max(axis)), (y, want), (r, x[::-1].sum(axis))]:
        np.testing.assert_array_equal(got.numpy(), w)
    x[(0,) * 3] = np.nan
    np.testing.assert_array_equal(bh.array(gpu_rt, x).sum(axis).numpy(), x.sum(axis))
