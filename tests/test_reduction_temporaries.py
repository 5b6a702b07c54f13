"""Reductions along an axis whose result only the next instructions read: the schedule's accumulator is
the temporary. Every schedule of axis reductions, one and several reductions, chains after them."""
import re

import numpy as np
import pytest

import bohrium_b200 as bh

# rows on lanes, rows split over CTAs, a serial loop per point; two and three dimensions
SHAPES = [(200, 31), (149, 8), (300, 4000), (3, 70_000), (40, 50, 400), (3, 5, 4000), (5, 7, 3)]


def one(x, axis):
    return [x.sum(axis) * 2]


def twice(x, axis):
    s = x.sum(axis)
    return [s + s]


def two_reductions(x, axis):
    s, m = x.sum(axis), x.max(axis)
    return [s * 3 - m, s]


def chain(x, axis):
    s = x.sum(axis) * 2 + 1
    return [s * s - s]


PROGRAMS = [one, twice, two_reductions, chain]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_no_register_is_read_before_it_is_set(prog, shape):
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = prog(bh.empty(rt, shape, np.int64), len(shape) - 1)
    units = [u for k in bh.dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]]
    assert len(keep)
    for u in units:
        body = u["source"].split("struct P {")[1].split('extern "C" __global__')[0]
        for t in set(re.findall(r"\b(t\d+);\n", body)):
            uses = [line.strip() for line in body.splitlines() if re.search(rf"\b{t}\b", line) and not re.search(rf"\w {t};$", line)]
            # the first use in the text is a plain assignment
            assert not uses or re.match(rf"{t} = (?!.*\b{t}\b)", uses[0]), (u["sched"], t, uses)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
@pytest.mark.parametrize("dtype", [np.int64, np.float64, np.float32])
def test_values(gpu_rt, prog, shape, dtype):
    x = np.random.default_rng(0).integers(0, 3, shape).astype(dtype)  # small: every step exact in every type
    x[..., 0] = 1
    a = bh.array(gpu_rt, x)
    gpu_rt.flush()
    got = prog(a, len(shape) - 1)
    gpu_rt.flush()
    for g, w in zip(got, prog(x.astype(np.int64), len(shape) - 1)):
        if dtype == np.float32 and np.abs(w).max() > 1 << 24:
            np.testing.assert_allclose(g.numpy(), w, rtol=3 * 2.0 ** -24)  # up to three rounded steps after an exact sum
        else:
            np.testing.assert_array_equal(g.numpy(), w.astype(dtype))
