"""Full reductions of several types in one kernel: each reduction's part of the shared memory that
holds the warps' trees lies on its type's alignment, apart from the others, and within the array."""
import itertools
import re

import numpy as np
import pytest

import bohrium_b200 as bh

TYPES = [np.bool_, np.int8, np.uint16, np.int32, np.float64, np.complex64, np.complex128]


def reduced(a):
    return a.any() if a.dtype == np.bool_ else a.sum()


def slots(dtypes, n=3_000_000):
    """(offset, bytes per element, elements) of every reduction's slots, and the array's size."""
    rt = bh.Runtime(bh.DryRunExecutor())
    arrays = [bh.empty(rt, (n,), t) for t in dtypes]
    keep = [reduced(a) for a in arrays]
    (unit,) = [u for k in bh.dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]]
    assert unit["sched"] == "grid_reduce" and len(keep) == len(dtypes)
    src = unit["source"]
    (size,) = re.findall(r"unsigned char warp_sm\[(\d+)\]", src)
    (held,) = re.findall(r"if \(held < (\d+) &&", src)
    at = [(int(k), int(off)) for k, off in re.findall(r"\* ws(\d+) = \([^)]*\)\(warp_sm \+ (\d+)\)", src)]
    assert [k for k, _ in at] == list(range(len(dtypes)))
    # one slot per warp (8) and held tile
    return [(off, np.dtype(t).itemsize, 8 * int(held)) for (_, off), t in zip(at, dtypes)], int(size)


@pytest.mark.parametrize("count", [2, 3, 5])
def test_every_reduction_has_aligned_slots_of_its_own(count):
    if count == 5:  # the smallest types first, several of the largest after them
        combinations = [(t,) + (np.complex128,) * 4 for t in TYPES]
    else:
        combinations = itertools.product(TYPES, repeat=count)
    for dtypes in combinations:
        regions, size = slots(dtypes)
        end = 0
        for off, itemsize, elements in regions:
            assert off % itemsize == 0, (dtypes, regions)
            assert off >= end, (dtypes, regions)
            end = off + itemsize * elements
        assert end <= size, (dtypes, regions, size)


@pytest.mark.parametrize("dtype,count", [(np.float64, 400), (np.complex128, 200), (np.float64, 3)])
def test_shared_memory_of_many_reductions(dtype, count):
    """A plain launch's shared memory grows by one set of slots a reduction: what it needs beside the
    warps' slots lies in the same array, so a kernel of many reductions stays below 48 KB."""
    rt = bh.Runtime(bh.DryRunExecutor())
    arrays = [bh.empty(rt, (5000,), dtype) for _ in range(count)]
    keep = [a.sum() for a in arrays]
    (unit,) = [u for k in bh.dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]]
    assert len(keep) == count
    main = unit["source"].split("void bh_main(const P &p)")[1].split("\n}\n")[0]
    declared = [(t, int(n)) for t, n in re.findall(r"__shared__ (?:alignas\(\d+\) )?([\w ]+?) \w+\[(\d+)\]", main)]
    size = {"unsigned char": 1, "unsigned long long": 8}
    assert sum(size[t] * n for t, n in declared) <= 48 * 1024 - 64


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [2, 4])
@pytest.mark.parametrize("narrow", [np.int8, np.bool_])
def test_narrow_and_wide_sums_in_one_kernel(gpu_rt, narrow, wide):
    n = 3_000_017  # more tiles than one CTA holds at a time would need, and a ragged last one
    rng = np.random.default_rng(wide)
    m = (rng.random(n) < 1e-6).astype(narrow)
    z = [(rng.integers(-9, 9, n) + 1j * rng.integers(-9, 9, n)).astype(np.complex128) for _ in range(wide)]
    a, zs = bh.array(gpu_rt, m), [bh.array(gpu_rt, v) for v in z]
    gpu_rt.flush()
    outs = [reduced(a)] + [reduced(v) for v in zs]
    gpu_rt.flush()
    assert outs[0].numpy() == (m.any() if narrow == np.bool_ else m.sum(dtype=narrow))
    for o, v in zip(outs[1:], z):  # sums of integers: exact in any order
        assert o.numpy() == v.sum()
