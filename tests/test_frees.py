"""Arrays that a flush frees while loops are taken apart (a reduction pushed inwards, loops split for
threads): each is freed by the last kernel that reads or writes it, and is a register of no other."""
import re

import numpy as np
import pytest

import bohrium_b200 as bh


def column_maximum_beside_row_values(args):
    """The maxima over the rows run with the axes swapped, apart from the chain of row values. The
    program holds the only references to its inputs, so they are freed too."""
    x, r = args.pop(), args.pop()
    c = x.max(0)
    u = r * 2 + 1
    v = x * x
    m = v - r.reshape(r.shape[0], 1)
    return [c, m, u]


def row_values_dropped_before_their_array(args):
    x, r = args.pop(), args.pop()
    u = r * 2 + 1
    del u
    c = x.max(0)
    v = np.maximum(x, x) if isinstance(x, np.ndarray) else bh.binary("MAXIMUM", x, x)
    m = v - r.reshape(r.shape[0], 1)
    return [c, m, v]


def scan_beside_nested_maps(args):
    """The accumulate's nest is built anew with its axes swapped; the arrays that the maps inside it read
    last are freed in them."""
    x, r = args.pop(), args.pop()
    y = x.reshape(40, 5, 31)
    s = r.reshape(40, 5)
    c = np.cumsum(s, 0) if isinstance(s, np.ndarray) else s.cumsum(0)
    t = s * 3
    m = np.minimum(y, t.reshape(40, 5, 1)) if isinstance(y, np.ndarray) else bh.binary("MINIMUM", y, t.reshape(40, 5, 1))
    d = y + s.reshape(40, 5, 1)
    return [c, m, d]


PROGRAMS = [column_maximum_beside_row_values, row_values_dropped_before_their_array, scan_beside_nested_maps]
FUSERS = [None, "greedy,push_reductions_inwards,split_for_threading,collapse_redundant_axes"]


@pytest.mark.parametrize("fusers", FUSERS)
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_frees_follow_the_last_access(prog, fusers):
    rt = bh.Runtime(bh.DryRunExecutor())
    args = [bh.empty(rt, (200,), np.int64), bh.empty(rt, (200, 31), np.int64)]
    rt.flush()
    keep = prog(args)
    flush = rt.take()
    blocks = [k["block"] for k in bh.dry_run(flush, compile=False, fuser_list=fusers)["kernels"]]
    named = set(re.findall(r"\ba\d+\b", " ".join(blocks)))  # (contraction takes temporaries out of a program)
    want = {f"a{op.base.handle}" for i in flush.instrs if i.opcode == bh.ir.OPCODES["FREE"] for op in i.operands if op is not None}
    assert len(keep)
    freed = []
    for i, block in enumerate(blocks):
        here = {a for names in re.findall(r"frees: \{([^}]*)\}", block) for a in names.split(",") if a}
        for a in here:
            assert not any(re.search(rf"\b{a}\b", later) for later in blocks[i + 1:]), (a, blocks)
        freed += here
    assert sorted(freed) == sorted(want & named) and freed


@pytest.mark.gpu
@pytest.mark.parametrize("batch", ["off", "grouped"])
@pytest.mark.parametrize("prog", PROGRAMS, ids=lambda f: f.__name__)
def test_values(gpu_executor, prog, batch):
    rng = np.random.default_rng(0)
    x, r = rng.integers(-9, 9, (200, 31)), rng.integers(-9, 9, 200)
    gpu_executor.message("CUDA: batch " + batch)
    try:
        rt = bh.Runtime(gpu_executor)
        for _ in range(3):  # other arrays have held other values by then
            args = [bh.array(rt, r), bh.array(rt, x)]
            rt.flush()
            got = prog(args)
            rt.flush()
            for g, w in zip(got, prog([r, x])):
                np.testing.assert_array_equal(g.numpy(), w)
            x, r = x + 1, r - 1
    finally:
        gpu_executor.message("CUDA: batch off")
