"""Full reductions at the edges of GRID_REDUCE's tiles, items and CTA walks: one and many tiles per
CTA, more tiles than the shared memory of a CTA holds, a ragged last item, heavy and light bodies,
several reductions of several types at once, kept maps -- against the exact order model for sums and
NumPy for order-free ones."""
import numpy as np
import pytest

import bohrium_b200 as bh
from tests.harness import grid_reduce_sum

pytestmark = pytest.mark.gpu

# 2048-element tiles; 4 tiles per item from 9472 tiles on (light bodies)
SIZES = [1, 2047, 2049, 4096, 2048 * 593 + 1, 2048 * 9472 + 5, 2048 * 148 * 5 * 66 + 77]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_sum_keeps_its_order(gpu_rt, n, dtype):
    if n > 50_000_000 and dtype == np.float64:
        n //= 2
    x = np.random.default_rng(n).standard_normal(n).astype(dtype)
    assert bh.array(gpu_rt, x).sum().numpy().tobytes() == grid_reduce_sum(x).tobytes()


@pytest.mark.parametrize("n", SIZES[:-1])
def test_heavy_body_with_a_kept_map_and_three_reductions(gpu_rt, n):
    x = np.random.default_rng(n).integers(1, 50, n).astype(np.float64)
    a = bh.array(gpu_rt, x)
    y = bh.sqrt(a * a) / a + a  # a division makes the body heavy; x + 1 exactly
    s, m, c = y.sum(), y.max(), (y > 20.0).any()
    assert float(s.numpy()) == (x + 1).sum()
    assert float(m.numpy()) == (x + 1).max()
    assert bool(c.numpy()) == bool((x + 1 > 20).any())
    np.testing.assert_array_equal(y.numpy(), x + 1)
