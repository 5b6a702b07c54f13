"""Maps whose two innermost ranks are walked as one: row lengths around the chunk and word edges,
views with and without gaps between their rows, broadcasts, an outer rank and generated values that
depend on the element's index, against the CPU oracle (bit-exact: integers,
and sums and products of small integers in floating point)."""
import numpy as np
import pytest

import bohrium_b200 as bh
from tests.harness import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int8, np.float32, np.float64, np.complex128])
@pytest.mark.parametrize("shape", [(1, 5), (700, 1), (3, 2), (257, 3), (100, 7), (1000, 50), (33, 257), (11, 700),
                                   (5, 1025), (1100, 1000), (3, 17, 5), (2, 3, 9, 4)])
def test_maps_over_narrow_rows(gpu_rt, oracle_rt, shape, dtype):
    x = np.random.default_rng(0).integers(-3, 4, shape).astype(dtype)

    def prog(rt):
        a = bh.array(rt, x)
        row = bh.array(rt, np.arange(shape[-1]) % 5 + 1).astype(dtype)
        col = bh.array(rt, (np.arange(int(np.prod(shape[:-1]))) % 7).reshape(shape[:-1] + (1,))).astype(dtype)
        rt.flush()
        out = [a * row + col, a[..., ::-1] * col, a[..., 1:] - a[..., :-1]]
        b = a.copy()
        b[..., 1:] = a[..., :-1] * row[1:] + col  # a view with gaps is written
        return out + [b]

    gpu, cpu = run(gpu_rt, prog), run(oracle_rt, prog)
    for g, c in zip(gpu, cpu):
        np.testing.assert_array_equal(g, c)


def test_generated_values_use_the_elements_index(gpu_rt, oracle_rt):
    def prog(rt):
        r = bh.random123(rt, (300, 11), 5, 7)
        w = bh.arange(rt, 11, np.uint64)
        rt.flush()
        return [bh.random123(rt, (300, 11), 5, 7) + w, r]

    gpu, cpu = run(gpu_rt, prog), run(oracle_rt, prog)
    for g, c in zip(gpu, cpu):
        np.testing.assert_array_equal(g, c)
