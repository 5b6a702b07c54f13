"""One-dimensional accumulates whose inputs are computed beside arrays that the same loop updates: the
update runs once, in a map before the scan, and the scan keeps its own schedule. Plans on the CPU; values
on a GPU against NumPy (integers and integer-valued floats, so exact)."""
import numpy as np
import pytest

import bohrium_b200 as bh


def add(a, b, out):
    if isinstance(a, np.ndarray):
        np.add(a, b, out=out)
    else:
        bh.binary("ADD", a, b, out=out)


def multiply(a, b, out):
    if isinstance(a, np.ndarray):
        np.multiply(a, b, out=out)
    else:
        bh.binary("MULTIPLY", a, b, out=out)


def fill(a, value):
    if isinstance(a, np.ndarray):
        a[...] = value
    else:
        a.assign(value)


def scan_of_a_map(x, y):
    add(x, 1, x)
    return [(x * 2 + 1).cumsum(), x]


def scan_of_a_product(x, y):
    add(x, 1, x)
    return [(x * y).cumsum(), x]


def scan_of_the_old_values(x, y):
    t = x * 3
    add(x, 1, x)
    return [t.cumsum(), x]


def scan_of_old_and_new_values(x, y):
    t = x * 3
    add(x, 1, x)
    return [(t + x).cumsum(), x]


def two_updates(x, y):
    t = x * 2
    add(x, t, x)
    add(t, 1, t)
    return [(x + t).cumsum(), x, t]


def independent_temporary(x, y):
    t = y * 3
    add(x, 1, x)
    return [(t + x).cumsum(), x]


def temporary_of_both(x, y):
    t = y * 2
    add(x, t, x)
    return [(t - x).cumsum(), x]


def update_after_the_scan(x, y):
    add(x, 1, x)
    c = (x * 2).cumsum()
    out = c + x
    add(x, out, x)
    return [c, out, x]


def overwritten_after_it_was_read(x, y):
    t = x + y
    fill(x, 5)
    return [(t * 2).cumsum() + x, x]


def kept_map_and_two_arrays(x, y):
    k = x - y
    add(x, 1, x)
    multiply(y, 2, y)
    return [(k + x + y).cumsum() * 2, k, x, y]


PROGRAMS = [scan_of_a_map, scan_of_a_product, scan_of_the_old_values, scan_of_old_and_new_values, two_updates,
            independent_temporary, temporary_of_both, update_after_the_scan, overwritten_after_it_was_read, kept_map_and_two_arrays]


@pytest.mark.parametrize("dtype", [np.float64, np.int32])
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_updates_run_as_maps_before_the_scan(prog, dtype):
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = prog(bh.empty(rt, (3_000_000,), dtype), bh.empty(rt, (3_000_000,), dtype))
    units = [u for k in bh.dry_run(rt.take(), compile=True)["kernels"] for u in k["units"]]
    scheds = [u["sched"] for u in units]
    after = prog in (scan_of_the_old_values, overwritten_after_it_was_read)  # the update comes last in the loop
    assert scheds[-3:] == ["scan1d"] * 3 and set(scheds[:-3]) == (set() if after else {"flat"}), scheds
    assert len(keep) and not any(u["compile_error"] for u in units)


def test_a_map_that_the_scan_can_compute_stays_with_it():
    """x += 1, then the scan of x * 2 + 1: the map moves x twice, and the scan is that of x * 2 + 1 alone."""
    n = 3_000_000

    def units(prog):
        rt = bh.Runtime(bh.DryRunExecutor())
        keep = prog(bh.empty(rt, (n,), np.float64))
        assert keep
        return [u for k in bh.dry_run(rt.take(), compile=False)["kernels"] for u in k["units"]]

    got, alone = units(lambda x: scan_of_a_map(x, None)), units(lambda x: [(x * 2 + 1).cumsum(), x])
    assert [u["sched"] for u in got] == ["flat", "scan1d", "scan1d", "scan1d"] and got[0]["bytes"] == 2 * 8 * n
    assert [u["bytes"] for u in got[1:]] == [u["bytes"] for u in alone]


def test_the_single_pass_does_not_take_scans_whose_inputs_change(monkeypatch):
    """Its fallback would read the changed input: the update after the accumulate keeps the three units."""
    monkeypatch.setenv("BH_CUDA_SCAN_SINGLE_PASS", "true")
    for prog, want in [(scan_of_the_old_values, 3), (scan_of_a_map, 1)]:
        rt = bh.Runtime(bh.DryRunExecutor())
        keep = prog(bh.empty(rt, (3_000_000,), np.float64), None)
        scheds = [u["sched"] for k in bh.dry_run(rt.take(), compile=True)["kernels"] for u in k["units"]]
        assert scheds.count("scan1d") == want and len(keep)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 2048, 50_001, 3_000_017])
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_values(gpu_rt, prog, dtype, n):
    rng = np.random.default_rng(3)
    x, y = rng.integers(-3, 4, n).astype(dtype), rng.integers(-3, 4, n).astype(dtype)
    a, b = bh.array(gpu_rt, x), bh.array(gpu_rt, y)
    gpu_rt.flush()
    got = prog(a, b)
    gpu_rt.flush()
    want = [w.astype(dtype) for w in prog(x.copy(), y.copy())]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.numpy(), w)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", ["off", "grouped", "graph"])
def test_repeated_flushes(gpu_executor, batch):
    """The plan's replays update the array once more each time. The values grow with every replay, past
    what float64 holds exactly: 64-bit integers, whose sums are exact modulo 2^64 in any order."""
    gpu_executor.message("CUDA: batch " + batch)
    try:
        rt = bh.Runtime(gpu_executor)
        rng = np.random.default_rng(4)
        x, y = rng.integers(-3, 4, 50_001), rng.integers(-3, 4, 50_001)
        for prog in PROGRAMS:
            a, b = bh.array(rt, x), bh.array(rt, y)
            rt.flush()
            outs = prog(a, b)
            ir = gpu_executor.compile(rt.take())
            wx, wy = x.copy(), y.copy()
            for _ in range(4):
                ir.execute()
                want = prog(wx, wy)
                for o, w in zip(outs, want):
                    np.testing.assert_array_equal(gpu_executor.peek(o.base), w, err_msg=prog.__name__)
            del ir, outs, a, b
            rt.flush()
    finally:
        gpu_executor.message("CUDA: batch off")


@pytest.mark.gpu
@pytest.mark.parametrize("prog", [scan_of_the_old_values, overwritten_after_it_was_read, scan_of_a_map], ids=lambda f: f.__name__)
def test_single_pass_that_gives_up(monkeypatch, prog):
    """The single-pass scan with a negative wait cap redoes what the update may have changed."""
    for key, value in [("SCAN_SINGLE_PASS", "true"), ("SCAN_SPIN_CAP", "-1"), ("CACHE_DIR", "NONE")]:
        monkeypatch.setenv("BH_CUDA_" + key, value)
    ex = bh.NativeExecutor(stack="cuda")
    try:
        rng = np.random.default_rng(5)
        x, y = rng.integers(-3, 4, 300_001), rng.integers(-3, 4, 300_001)
        rt = bh.Runtime(ex)
        a, b = bh.array(rt, x), bh.array(rt, y)
        rt.flush()
        got = prog(a, b)
        rt.flush()
        for g, w in zip(got, prog(x, y)):
            np.testing.assert_array_equal(g.numpy(), w)
    finally:
        ex.close()
