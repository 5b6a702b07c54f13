"""Generated integer-valued programs of maps, reductions, accumulates, slices, reversed and transposed
views, broadcasts, in-place updates and assignments, in one to three dimensions, against NumPy, exactly;
and the invariants of their plans: every array that a flush frees is freed once, by the last kernel
that accesses it."""
import random
import re

import numpy as np
import pytest

import bohrium_b200 as bh
from bohrium_b200 import ir

NUMPY = {"ADD": np.add, "SUBTRACT": np.subtract, "MULTIPLY": np.multiply, "MAXIMUM": np.maximum, "MINIMUM": np.minimum}


def binary(name, a, b, out=None):
    return NUMPY[name](a, b, out=out) if isinstance(a, np.ndarray) else bh.binary(name, a, b, out=out)


def reduction(a, name, axis):
    return a.sum(axis, dtype=a.dtype) if name == "sum" and isinstance(a, np.ndarray) else getattr(a, name)(axis)


def accumulated(a, axis):
    return np.cumsum(a, axis, dtype=a.dtype) if isinstance(a, np.ndarray) else a.cumsum(axis)


def program(seed, make):
    rng = random.Random(seed)
    shape = rng.choice([
        [(1,), (7,), (255,), (1024,), (2049,), (5000,), (100_003,)],
        [(5, 7), (33, 65), (150, 20), (149, 300), (300, 150), (256, 256), (1000, 3), (3, 5000), (200, 1025), (64, 64)],
        [(5, 7), (33, 65), (150, 20), (149, 300), (300, 150), (256, 256), (1000, 3), (3, 5000), (200, 1025), (64, 64)],
        [(3, 4, 5), (20, 30, 40), (2, 3, 1000), (160, 3, 7), (7, 150, 33)]][rng.randrange(4)])
    types = rng.choice([[np.int64], [np.int32], [np.int64, np.int32], [np.float64]])
    arrays = {shape: [make(shape, rng.choice(types), i) for i in range(rng.randint(1, 3))]}
    if len(shape) > 1:
        for axis in range(len(shape)):
            s = shape[:axis] + shape[axis + 1:]
            arrays.setdefault(s, []).append(make(s, rng.choice(types), 10 + axis))
    products = 0

    def pick(s=None):
        return rng.choice(arrays[s or rng.choice([k for k in arrays if arrays[k]])])

    def add(x):
        arrays.setdefault(tuple(x.shape), []).append(x)

    def view(a, least, *choices):
        return a[tuple(rng.choice(choices) if n > least else slice(None) for n in a.shape)]

    for _ in range(rng.randint(3, 15)):
        kind = rng.choice(["map", "map", "constant", "broadcast", "broadcast", "reduce", "reduce", "reduce", "accumulate", "in place",
                           "view in place", "slice", "reversed", "transposed", "cast", "compare", "step", "assign", "fill"])
        a = pick()
        op = rng.choice(list(NUMPY))
        if op == "MULTIPLY" and types == [np.float64]:
            products += 1
            op = "MULTIPLY" if products <= 2 else "ADD"  # float64 values stay exact
        if kind == "map":
            add(binary(op, a, pick(tuple(a.shape))))
        elif kind == "constant":
            add(a * 2 + 1)
        elif kind == "broadcast" and len(shape) > 1:
            axis = rng.randrange(len(shape))
            r = pick(shape[:axis] + shape[axis + 1:]).reshape(shape[:axis] + (1,) + shape[axis + 1:])
            add(binary(op, pick(shape), r))
        elif kind == "reduce" and len(a.shape) > 1:
            name = rng.choice(["sum", "max", "min"])
            # (a floating-point maximum starts from the smallest positive normal number, NumPy's does not)
            add(reduction(a, "min" if name == "max" and types == [np.float64] else name, rng.randrange(len(a.shape))))
        elif kind == "accumulate":
            add(accumulated(a, rng.randrange(len(a.shape))))
        elif kind == "in place":
            binary("ADD", a, rng.choice([1, 2]), out=a)
        elif kind == "view in place":
            v = view(a, 2, slice(0, None), slice(1, None))
            binary(rng.choice(["MAXIMUM", "ADD"]), v, 1, out=v)
        elif kind == "slice":
            add(view(a, 5, slice(0, -1), slice(1, None), slice(2, -1)) + 1)
        elif kind == "step":
            add(view(a, 0, slice(None), slice(None, None, 2)) * 3)
        elif kind == "reversed":
            add(binary("ADD", view(a, 0, slice(None), slice(None, None, -1)), a))
        elif kind == "transposed" and len(a.shape) == 2:
            add(binary("ADD", a.T, a) if a.shape[0] == a.shape[1] else a.T + 1)
        elif kind == "cast" and types != [np.float64]:
            add(a.astype(np.int32 if a.dtype == np.int64 else np.int64))
        elif kind == "compare":
            add((a > pick(tuple(a.shape))).astype(a.dtype) + a)
        elif kind == "assign":
            b = pick(tuple(a.shape))
            if b is not a and a.dtype == b.dtype:
                a[...] = b
        elif kind == "fill":
            a[...] = 3
        if sum(map(len, arrays.values())) > 8:
            s = rng.choice([k for k in arrays if len(arrays[k]) > 1] or list(arrays))
            if len(arrays[s]) > 1:
                arrays[s].pop(rng.randrange(len(arrays[s])))
    return [x for s in arrays for x in arrays[s] if rng.random() < 0.6] or [pick()]


def values(shape, dtype, i):
    return np.random.default_rng(i).integers(-4, 5, shape).astype(dtype)


DEFAULT = "greedy,push_reductions_inwards,collapse_redundant_axes"
FUSERS = [DEFAULT, "greedy,push_reductions_inwards,split_for_threading,collapse_redundant_axes",
          "breadth_first,push_reductions_inwards,collapse_redundant_axes", "serial,push_reductions_inwards,collapse_redundant_axes",
          "greedy", "collapse_redundant_axes"]


@pytest.mark.parametrize("fusers", FUSERS)
def test_every_freed_array_is_freed_once_after_its_last_access(fusers):
    free = ir.OPCODES["FREE"]
    for seed in range(150):
        rt = bh.Runtime(bh.DryRunExecutor())
        keep = program(seed, lambda shape, dtype, i: bh.empty(rt, shape, dtype))
        flush = rt.take()
        blocks = [k["block"] for k in bh.dry_run(flush, compile=False, fuser_list=fusers)["kernels"]]
        named = set(re.findall(r"\ba\d+\b", " ".join(blocks)))  # (contraction takes temporaries out of a program)
        want = {f"a{op.base.handle}" for i in flush.instrs if i.opcode == free for op in i.operands if op is not None} & named
        freed = []
        for k, block in enumerate(blocks):
            here = {a for names in re.findall(r"frees: \{([^}]*)\}", block) for a in names.split(",") if a}
            for a in here:
                assert not any(re.search(rf"\b{a}\b", later) for later in blocks[k + 1:]), (seed, a)
            freed += here
        assert sorted(freed) == sorted(want), (seed, set(freed) ^ want)
        assert len(keep)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,fusers,seeds", [("off", DEFAULT, 200), ("grouped", DEFAULT, 200), ("off", FUSERS[1], 40),
                                                ("off", FUSERS[2], 40), ("grouped", FUSERS[3], 40), ("off", FUSERS[5], 40)])
def test_generated_programs_equal_numpy(gpu_executor, batch, fusers, seeds):
    gpu_executor.message("CUDA: batch " + batch)
    gpu_executor.message("CUDA: fuser " + fusers)
    try:
        rt = bh.Runtime(gpu_executor)
        for seed in range(seeds):
            got = program(seed, lambda shape, dtype, i: bh.array(rt, values(shape, dtype, i)))
            rt.flush()
            for k, (g, w) in enumerate(zip(got, program(seed, values))):
                np.testing.assert_array_equal(g.numpy(), w, err_msg=f"program {seed}, output {k}")
    finally:
        gpu_executor.message("CUDA: batch off")
        gpu_executor.message("CUDA: fuser " + DEFAULT)


def dropped_reduction(x):
    """A reduction whose result nothing reads: it is computed all the same, in an array of its own."""
    x.max(0)
    return [x * 2 + 1]


@pytest.mark.parametrize("fusers", FUSERS)
@pytest.mark.parametrize("shape", [(160, 3, 7), (2, 3, 1000), (300, 31), (5, 4000)])
def test_dropped_reductions_lower(shape, fusers):
    rt = bh.Runtime(bh.DryRunExecutor())
    x = bh.empty(rt, shape, np.int64)
    rt.flush()
    keep = [dropped_reduction(x), reduction(binary("MINIMUM", x, x) + 1, "min", 0).shape]
    units = [u for k in bh.dry_run(rt.take(), compile=False, fuser_list=fusers)["kernels"] for u in k["units"]]
    assert len(keep) and units
