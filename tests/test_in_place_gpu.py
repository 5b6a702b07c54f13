"""Arrays updated in place: the generated code keeps the element in a register between the load and
the store, and units that run the instructions more than once must not repeat the update."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5,), (1024,), (100_003,), (40, 2048), (300, 700)])
@pytest.mark.parametrize("dtype", [np.int8, np.float32, np.float64, np.complex128])
def test_maps(gpu_rt, shape, dtype):
    x = np.random.default_rng(0).integers(-3, 4, shape).astype(dtype)
    a = bh.array(gpu_rt, x)
    bh.binary("ADD", a, 1, out=a)
    b = a * 2
    bh.binary("MULTIPLY", a, a, out=a)
    np.testing.assert_array_equal(a.numpy(), (x + dtype(1)) ** 2)
    np.testing.assert_array_equal(b.numpy(), (x + dtype(1)) * dtype(2))
    # a view that starts off the word boundary
    v = bh.array(gpu_rt, x)
    bh.binary("ADD", v[..., 1:], 1, out=v[..., 1:])
    w = x.copy()
    w[..., 1:] += dtype(1)
    np.testing.assert_array_equal(v.numpy(), w)


@pytest.mark.parametrize("n", [1000, 2048, 50_001, 3_000_017])
def test_maps_fused_with_a_full_reduction(gpu_rt, n):
    x = np.random.default_rng(1).integers(-3, 4, n).astype(np.float64)
    a = bh.array(gpu_rt, x)
    bh.binary("ADD", a, 1, out=a)
    s = a.sum()
    assert float(s.numpy()) == (x + 1).sum()
    np.testing.assert_array_equal(a.numpy(), x + 1)


@pytest.mark.parametrize("n", [1000, 2048, 50_001, 3_000_017])
def test_maps_before_a_one_dimensional_accumulate(gpu_rt, n):
    x = np.random.default_rng(2).integers(-3, 4, n).astype(np.float64)
    a = bh.array(gpu_rt, x)
    bh.binary("ADD", a, 1, out=a)
    c = a.cumsum(0)
    d = c + a
    np.testing.assert_array_equal(d.numpy(), np.cumsum(x + 1) + x + 1)
    np.testing.assert_array_equal(c.numpy(), np.cumsum(x + 1))
    np.testing.assert_array_equal(a.numpy(), x + 1)
