"""TILE2D without TMA: rows and starts off the 16-byte boundary and grouped launches, whose tiles go
through shared memory by plain loads. Ragged edges of the tiles, one and two transposed views and a
row-wise view beside them; single additions, so bit-exact against NumPy."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.int64])
@pytest.mark.parametrize("shape", [(33, 65), (32, 64), (97, 127), (517, 301), (1001, 64), (2050, 1999)])
@pytest.mark.parametrize("mode", ["off", "grouped"])
def test_transposed_operands(gpu_executor, shape, dtype, mode):
    rng = np.random.default_rng(0)
    A = rng.integers(-99, 99, shape).astype(dtype)
    B, C = (rng.integers(-99, 99, shape[::-1]).astype(dtype) for _ in range(2))
    gpu_executor.message("CUDA: batch " + mode)
    try:
        rt = bh.Runtime(gpu_executor)
        a, b, c = (bh.array(rt, x) for x in (A, B, C))
        rt.flush()
        outs = [a + b.T, a - c.T, b.T + c.T, a[1:, 1:] + b[1:, 1:].T]
        got = [o.numpy() for o in outs]
    finally:
        gpu_executor.message("CUDA: batch off")
    for g, w in zip(got, [A + B.T, A - C.T, B.T + C.T, A[1:, 1:] + B[1:, 1:].T]):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("types", [(np.float32, np.int32), (np.int32, np.float32), (np.uint32, np.float32),
                                   (np.float64, np.int64), (np.int64, np.float64)])
@pytest.mark.parametrize("shape", [(65, 99), (256, 320), (517, 301)])
@pytest.mark.parametrize("mode", ["off", "grouped"])
def test_operands_of_two_types(gpu_executor, types, shape, mode):
    """One element size, two types, on every way into the tile (256 x 320: tensor maps)."""
    ta, tb = types
    to = ta if np.issubdtype(ta, np.floating) else tb
    rng = np.random.default_rng(1)
    A = rng.integers(0, 99, shape).astype(ta)
    B = rng.integers(0, 99, shape[::-1]).astype(tb)
    if np.issubdtype(ta, np.floating):
        A += ta(0.5)
    if np.issubdtype(tb, np.floating):
        B += tb(0.5)
    gpu_executor.message("CUDA: batch " + mode)
    try:
        rt = bh.Runtime(gpu_executor)
        a, b = bh.array(rt, A), bh.array(rt, B)
        rt.flush()
        out = a.astype(to) + b.T.astype(to)
        got = out.numpy()
    finally:
        gpu_executor.message("CUDA: batch off")
    np.testing.assert_array_equal(got, A.astype(to) + B.T.astype(to))
