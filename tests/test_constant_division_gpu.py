"""Division by a constant (a multiplication for powers of two) and the conversion of unsigned 64-bit
integers to float64: bit for bit NumPy's, for ordinary and extreme values, and with the constants of
a replayed plan changed."""
import numpy as np
import pytest

import bohrium_b200 as bh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_quotients_are_correctly_rounded(gpu_rt, dtype):
    fi = np.finfo(dtype)
    rng = np.random.default_rng(0)
    x = (rng.standard_normal(3000) * 10.0 ** rng.integers(-30, 30, 3000)).astype(dtype)
    x[:12] = [0.0, -0.0, np.inf, -np.inf, np.nan, fi.max, -fi.max, fi.tiny, fi.smallest_subnormal, -fi.smallest_subnormal, 1, 3]
    a = bh.array(gpu_rt, x)
    big = 2.0 ** (fi.maxexp - 1)
    for c in [1.0, -2.0, 0.5, 2.0 ** 20, big, 1 / big, float(fi.tiny), float(fi.smallest_subnormal), 3.0, 0.1, np.inf, 0.0]:
        c = float(dtype(c))
        with np.errstate(all="ignore"):
            want = x / dtype(c)
        got = (a / c).numpy()
        np.testing.assert_array_equal(got, want, err_msg=str(c))
        number = ~np.isnan(want)  # IEEE 754 leaves the sign of a NaN open
        np.testing.assert_array_equal(np.signbit(got)[number], np.signbit(want)[number], err_msg=str(c))


def test_plans_are_not_shared_between_kinds_of_divisor(gpu_rt):
    """The same flush with another constant: a power of two, another one, and none."""
    x = np.random.default_rng(2).standard_normal(5000)
    for c in [8.0, 0.25, 3.0, 16.0, 7.0]:
        a = bh.array(gpu_rt, x)
        np.testing.assert_array_equal((a / c + 1.0).numpy(), x / c + 1.0, err_msg=str(c))


def test_uint64_to_float64(gpu_rt):
    rng = np.random.default_rng(1)
    x = rng.integers(0, 2 ** 64, 5000, dtype=np.uint64) >> rng.integers(0, 64, 5000).astype(np.uint64)
    edge = [0, 1, 2 ** 52, 2 ** 53 - 1, 2 ** 53, 2 ** 53 + 1, 2 ** 53 + 3, 2 ** 63, 2 ** 63 + 1024, 2 ** 63 + 1025, 2 ** 64 - 1,
            2 ** 64 - 1024, 2 ** 64 - 1025, 2 ** 32 - 1, 2 ** 32, 2 ** 54 + 2, 2 ** 54 + 6]
    x[:len(edge)] = np.array(edge, dtype=np.uint64)
    np.testing.assert_array_equal(bh.array(gpu_rt, x).astype(np.float64).numpy(), x.astype(np.float64))
