"""Accumulates whose output the same flush updates in place: an accumulate reads the element that it wrote
before, so the update belongs to a later kernel. Plans on the CPU, values on a GPU against NumPy."""
import re

import numpy as np
import pytest

import bohrium_b200 as bh
from tests.test_generated_programs import accumulated, binary, values


def accumulate_then_update(x):
    c = accumulated(x, 0)
    binary("ADD", c, 2, out=c)
    return [c, c * 2]


def accumulate_then_update_along_rows(x):
    c = accumulated(x, len(x.shape) - 1)
    binary("MULTIPLY", c, 3, out=c)
    return [c + x, c]


UPDATES = [accumulate_then_update, accumulate_then_update_along_rows]


@pytest.mark.parametrize("shape", [(100_003,), (300, 700), (700, 3)])
@pytest.mark.parametrize("prog", UPDATES, ids=lambda f: f.__name__)
def test_an_accumulates_output_is_updated_by_another_kernel(prog, shape):
    """The accumulate reads the element it wrote before: its loop may not hold the update."""
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = prog(bh.empty(rt, shape, np.int64))
    plan = bh.dry_run(rt.take(), compile=False)["kernels"]
    for block in (k["block"] for k in plan):
        for out in re.findall(r"BH_ADD_ACCUMULATE (a\d+)\[", block):
            assert not re.findall(rf"BH_(?:ADD|MULTIPLY|IDENTITY) {out}\[(?!\S* 0\n)", block.replace(f"BH_IDENTITY {out}", "")), block
    assert len(keep) and not any(u["sched"] == "serial" for k in plan for u in k["units"])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1,), (2049,), (100_003,), (300, 700), (700, 3)])
@pytest.mark.parametrize("prog", UPDATES, ids=lambda f: f.__name__)
def test_values_of_an_updated_accumulate(gpu_rt, prog, shape):
    x = values(shape, np.int64, 1)
    a = bh.array(gpu_rt, x)
    gpu_rt.flush()
    got = prog(a)
    gpu_rt.flush()
    for g, w in zip(got, prog(x)):
        np.testing.assert_array_equal(g.numpy(), w)


def accumulate_of_an_accumulate(x):
    c = accumulated(x, 0)
    return [accumulated(c, 0) + x, c]


def test_sweeps_apart_from_maps_are_seeded_too(monkeypatch):
    """With avoid_rank0_sweep the sweeping loops are kernels of their own: the accumulates of a loop that
    no schedule takes start from the identity that an instruction before the loop writes."""
    monkeypatch.setenv("BH_CUDA_AVOID_RANK0_SWEEP", "true")
    rt = bh.Runtime(bh.DryRunExecutor())
    keep = accumulate_of_an_accumulate(bh.empty(rt, (5000,), np.int64))
    blocks = [k["block"] for k in bh.dry_run(rt.take(), compile=True)["kernels"]]
    outs = re.findall(r"BH_ADD_ACCUMULATE (a\d+)\[", "".join(b.split("block list:", 1)[1] for b in blocks))
    assert len(keep) and len(set(outs)) == 2
    for out in set(outs):
        assert any(re.search(rf"BH_IDENTITY {out}\[0:1:1\] 0\n", b) for b in blocks)


@pytest.mark.gpu
def test_values_of_sweeps_apart_from_maps(monkeypatch):
    monkeypatch.setenv("BH_CUDA_AVOID_RANK0_SWEEP", "true")
    ex = bh.NativeExecutor(stack="cuda")
    try:
        rt = bh.Runtime(ex)
        for seed in range(5):
            x = values((5000,), np.int64, seed)
            a = bh.array(rt, x)
            rt.flush()
            got = accumulate_of_an_accumulate(a)
            rt.flush()
            for g, w in zip(got, accumulate_of_an_accumulate(x)):
                np.testing.assert_array_equal(g.numpy(), w)
    finally:
        ex.close()
