"""Which kernels of a flush run as one row-wise unit: those that share rows, in bounded groups;
independent work of one shape stays apart, although the fuser merges it into common kernels. Plans on
the CPU; values of generated integer programs on a GPU against NumPy, exactly."""
import random

import numpy as np
import pytest

import bohrium_b200 as bh


def softmax(x):
    n = x.shape[0]
    e = bh.exp(x - x.max(1).reshape(n, 1))
    return e / e.sum(1).reshape(n, 1)


def units_of(prog):
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = prog(rt)
    units = [u for k in bh.dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]]
    return units, keep


@pytest.mark.parametrize("count", [1, 2, 5, 24])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_independent_softmaxes_are_units_of_one_source(count, dtype):
    units, _ = units_of(lambda rt: [softmax(bh.empty(rt, (2000, 1500), dtype)) for _ in range(count)])
    assert [u["sched"] for u in units] == ["rows"] * count
    assert len({u["source"] for u in units}) == 1


def test_independent_work_without_rows_in_common_keeps_its_kernels():
    """A maximum and a map of other arrays of the same shape share nothing with the softmax."""
    def prog(rt):
        x, y, z = (bh.empty(rt, (2000, 700), np.float64) for _ in range(3))
        return [softmax(x), y.max(1), z * 2.0 + 1.0]
    units, _ = units_of(prog)
    assert sorted(u["sched"] for u in units).count("rows") == 1
    (rows,) = [u for u in units if u["sched"] == "rows"]
    assert rows["source"] == units_of(lambda rt: [softmax(bh.empty(rt, (2000, 700), np.float64))])[0][0]["source"]


@pytest.mark.parametrize("dtype,cols", [(np.float32, 300), (np.float64, 1500), (np.float64, 3072)])
def test_long_chains_are_cut(dtype, cols):
    """Forty normalisations one after another: several units, none of them much longer than the others."""
    def prog(rt):
        x = bh.empty(rt, (2000, cols), dtype)
        for _ in range(40):
            x = x / x.sum(1).reshape(2000, 1)
        return [x]
    units, _ = units_of(prog)
    rows = [u for u in units if u["sched"] == "rows"]
    assert len(rows) > 1 and max(len(u["source"]) for u in rows) < 40_000


NUMPY = {"ADD": np.add, "SUBTRACT": np.subtract, "MULTIPLY": np.multiply, "MAXIMUM": np.maximum}


def binary(name, a, b, out=None):
    return NUMPY[name](a, b, out=out) if isinstance(a, np.ndarray) else bh.binary(name, a, b, out=out)


def total(a):
    return a.sum(1, dtype=a.dtype) if isinstance(a, np.ndarray) else a.sum(1)


def program(seed, make):
    """Maps, reductions, chains of row values, in-place updates and broadcasts over matrices of one
    shape: several independent and dependent threads of work interleaved. Integers: exact."""
    rng = random.Random(seed)
    n, c = rng.choice([(148, 3), (200, 31), (300, 100), (151, 257), (2000, 600)])
    dt = rng.choice([np.int64, np.int32])
    mats = [make((n, c), dt, i) for i in range(rng.choice([1, 2, 3, 4]))]
    vals, cols = [make((n,), dt, 10)], [make((c,), dt, 20)]
    for _ in range(rng.randint(4, 16)):
        kind = rng.choice(["map", "map", "column", "column", "reduce", "reduce", "reduce", "value", "value", "in place", "row",
                           "constant", "slice", "other axis", "reversed"])
        a = rng.choice(mats)
        if kind == "map":
            mats.append(binary(rng.choice(["ADD", "SUBTRACT", "MULTIPLY", "MAXIMUM"]), a, rng.choice(mats)))
        elif kind == "column":
            mats.append(binary(rng.choice(["ADD", "SUBTRACT", "MULTIPLY"]), a, rng.choice(vals).reshape(n, 1)))
        elif kind == "row":
            mats.append(a + rng.choice(cols))
        elif kind == "constant":
            mats.append(a * 3 + 1)
        elif kind == "reduce":
            vals.append(total(a) if rng.random() < 0.5 else a.max(1))
        elif kind == "value":
            r, q = rng.choice(vals), rng.choice(vals)
            vals.append(rng.choice([lambda: r + q, lambda: r * 2 + 1, lambda: r - q * q])())
        elif kind == "in place":
            if rng.random() < 0.5:
                binary("ADD", a, 1, out=a)
            else:
                binary("SUBTRACT", a, rng.choice(vals).reshape(n, 1), out=a)
        elif kind == "slice" and c > 4:
            vals.append(total(a[:, 1:c - 1]))
        elif kind == "other axis" and rng.random() < 0.3:
            cols.append(a.max(0))
        elif kind == "reversed" and rng.random() < 0.3:
            mats.append(a[::-1, :] + rng.choice(mats))
        if len(mats) > 6:
            mats.pop(rng.randrange(len(mats)))
        if len(vals) > 5:
            vals.pop(rng.randrange(len(vals)))
    return [x for x in mats + vals + cols if rng.random() < 0.6] or [mats[-1]]


def values(shape, dtype, i):
    return np.random.default_rng(i).integers(-5, 6, shape).astype(dtype)


def test_generated_programs_lower():
    """Every generated program lowers, with and without row fusion the same arrays being written."""
    fused = 0
    for seed in range(200):
        units, _ = units_of(lambda rt: program(seed, lambda shape, dtype, i: bh.empty(rt, shape, dtype)))
        fused += sum(u["sched"] == "rows" for u in units)
    assert fused >= 20  # the generator does reach row fusion


@pytest.mark.gpu
@pytest.mark.parametrize("batch", ["off", "grouped"])
def test_generated_programs_equal_numpy(gpu_executor, batch):
    gpu_executor.message("CUDA: batch " + batch)
    try:
        rt = bh.Runtime(gpu_executor)
        for seed in range(100):
            got = program(seed, lambda shape, dtype, i: bh.array(rt, values(shape, dtype, i)))
            rt.flush()
            want = program(seed, values)
            for k, (g, w) in enumerate(zip(got, want)):
                np.testing.assert_array_equal(g.numpy(), w, err_msg=f"program {seed}, output {k}")
    finally:
        gpu_executor.message("CUDA: batch off")


@pytest.mark.gpu
@pytest.mark.parametrize("batch", ["off", "grouped", "graph"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_softmaxes_of_one_flush(gpu_executor, dtype, batch):
    """Several softmaxes recorded before the first is read: units side by side, in one grouped launch
    (or one graph level), bit for bit what each gives alone."""
    rng = np.random.default_rng(5)
    xs = [rng.standard_normal((200, 700)).astype(dtype) for _ in range(5)]
    rt = bh.Runtime(gpu_executor)
    alone = [softmax(bh.array(rt, x)).numpy().tobytes() for x in xs]
    gpu_executor.message("CUDA: batch " + batch)
    try:
        for _ in range(3):  # the plan's first run, its replay, a graph's launch
            arrays = [bh.array(rt, x) for x in xs]
            rt.flush()
            launches = int(gpu_executor.message("CUDA: launches"))
            outs = [softmax(a) for a in arrays]
            rt.flush()
            launches = int(gpu_executor.message("CUDA: launches")) - launches
            assert [o.numpy().tobytes() for o in outs] == alone
            if batch != "graph":
                assert launches == (len(xs) if batch == "off" else 1)
            del arrays, outs
    finally:
        gpu_executor.message("CUDA: batch off")
