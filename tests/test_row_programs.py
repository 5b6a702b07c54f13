"""Row-wise programs with several instructions after a reduction: temporaries of one kernel beside
arrays and values that the fused kernels share. Lowering and compilation on the CPU, values on a GPU
against NumPy in 64 bits."""
import numpy as np
import pytest

import bohrium_b200 as bh

SHAPES = [(2000, 1000), (300, 31), (149, 3072), (150, 257)]
EPS = 1e-5


def layer_norm(rt, x):
    n, c = x.shape
    mean = x.sum(1) / float(c)
    d = x - mean.reshape(n, 1)
    var = (d * d).sum(1) / float(c)
    return [d / bh.sqrt(var + EPS).reshape(n, 1)]


def rms_norm(rt, x):
    n, c = x.shape
    s = bh.sqrt((x * x).sum(1) / float(c) + EPS) * 2.0 + 1.0
    return [x / s.reshape(n, 1)]


def log_softmax(rt, x):
    n = x.shape[0]
    m = x.max(1)
    return [x - (bh.log(bh.exp(x - m.reshape(n, 1)).sum(1)) + m).reshape(n, 1)]


def chains(rt, x):
    """Integers, so exact: chains of row values of which some are kept, some read by the next stage
    only and some by the next instruction only."""
    n = x.shape[0]
    m = x.max(1) * 3 - 2
    k = m * m + m
    y = x + (k - 1).reshape(n, 1)
    t = (y.sum(1) + k) * 2 + 5
    return [y * (t - k).reshape(n, 1), t]


PROGRAMS = [layer_norm, rms_norm, log_softmax, chains]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_programs_are_one_kernel_that_compiles(prog, shape, dtype):
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = prog(rt, bh.empty(rt, shape, dtype))
    units = [u for k in bh.dry_run(rt.take(), compile=True)["kernels"] for u in k["units"]]
    # (149, 3072) holds 12 elements a lane: too many for programs that carry more than a softmax does
    assert [u["sched"] for u in units] == ["rows"] or shape == (149, 3072)
    assert len(keep) and not any(u["compile_error"] for u in units)


def expected(prog, x, u):
    """The result in 64 bits and a bound on the error of a computation whose roundings are u: sums of a
    row in at most 70 roundings, exp and log within 2 ulp (4 u), division and square root rounded once."""
    x = x.astype(np.float64)
    c, terms = x.shape[1], 70 * u
    big = np.abs(x).max(1, keepdims=True)
    if prog is layer_norm:
        d = x - x.mean(1, keepdims=True)
        var = (d * d).mean(1, keepdims=True)
        s = np.sqrt(var + EPS)
        err_d = (terms + 3 * u) * big
        err_var = 2 * np.sqrt(var) * err_d + err_d ** 2 + (terms + 3 * u) * (var + err_d ** 2)
        return d / s, err_d / s + np.abs(d) * err_var / (2 * s ** 3) * 1.1 + 6 * u * np.abs(d / s)
    if prog is rms_norm:
        s = np.sqrt((x * x).sum(1, keepdims=True) / c + EPS) * 2 + 1
        return x / s, (terms + 8 * u) * np.abs(x / s)
    m = x.max(1, keepdims=True)
    log = np.log(np.exp(x - m).sum(1, keepdims=True))
    spread = np.abs(x - m).max(1, keepdims=True)
    out = x - (log + m)
    return out, terms + 4 * u + u * spread + 4 * u * np.abs(log) + 2 * u * (np.abs(log) + np.abs(m)) + 2 * u * np.abs(out)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("prog", [layer_norm, rms_norm, log_softmax], ids=lambda f: f.__name__)
def test_values(gpu_rt, prog, shape, dtype):
    x = (np.random.default_rng(0).standard_normal(shape) * 2 + 1).astype(dtype)
    a = bh.array(gpu_rt, x)
    gpu_rt.flush()
    (got,) = prog(gpu_rt, a)
    want, bound = expected(prog, x, np.finfo(dtype).eps / 2)
    assert np.all(np.abs(got.numpy().astype(np.float64) - want) <= bound)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [np.int64, np.float64])
def test_chains_of_row_values(gpu_rt, shape, dtype):
    x = np.random.default_rng(1).integers(1, 9, shape).astype(dtype)
    a = bh.array(gpu_rt, x)
    gpu_rt.flush()
    got = chains(gpu_rt, a)
    m = x.max(1) * 3 - 2
    k = m * m + m
    y = x + (k - 1)[:, None]
    t = (y.sum(1) + k) * 2 + 5
    np.testing.assert_array_equal(got[0].numpy(), y * (t - k)[:, None])
    np.testing.assert_array_equal(got[1].numpy(), t)
