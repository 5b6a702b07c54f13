"""The front end's quick paths give the same bytecode as the general ones: constants of every type and
extreme value, views, empty flushes, and result types and shapes of mixed operands."""
import numpy as np
import pytest

import bohrium_b200 as bh
from bohrium_b200 import ir


@pytest.mark.parametrize("dtype,values", [
    (np.float64, [0.0, -0.0, 1.5, float("inf"), float("-inf"), float("nan"), 5e-324, 1.7976931348623157e308, np.float64(2.5), 3, True]),
    (np.int64, [0, -1, 2 ** 63 - 1, -2 ** 63, np.int64(7), True]), (np.uint64, [0, 2 ** 64 - 1]), (np.float32, [1.5, -0.0]),
    (np.int8, [-128, 127]), (np.bool_, [True, False]), (np.complex128, [1 + 2j]), (np.complex64, [1 - 2j])])
def test_constant_words_are_the_values_bytes(dtype, values):
    for v in values:
        words = ir.Constant(v, ir.bh_type(dtype)).words()
        raw = np.array([v], dtype=dtype).tobytes().ljust(16, b"\0")
        assert all(type(w) is int for w in words)
        assert np.array(words, dtype=np.int64).tobytes() == raw, (dtype, v)


def test_encoding_of_views_and_flushes():
    assert ir.encode([]).dtype == np.int64 and ir.encode([]).size == 0
    base = ir.Base(np.float64, 12)
    base.handle = 77
    ins = ir.Instr(ir.OPCODES["ADD"], [ir.View(base, 1, (2, 3), (6, -1)), None, ir.View(base, np.int64(0), (np.int64(2), 3), (6, 1))],
                   ir.Constant(2.0, ir.FLOAT64))
    one = int(np.float64(2.0).view(np.int64))
    assert ir.encode([ins]).tolist() == [1, 3, ir.FLOAT64, one, 0, 77, 1, 2, 2, 3, 6, -1, 0, 77, 0, 2, 2, 3, 6, 1]
    base.handle = 0
    with pytest.raises(RuntimeError):
        ir.encode([ins])
    assert ir.View(base, 1, (2,), (1,)) == ir.View(base, 1, (2,), (1,)) and hash(ir.View(base, 1, (2,), (1,))) is not None
    assert ir.View.whole(base).ndim == 1 and ir.View(base, 0, (2, 3), (3, 1)).ndim == 2


@pytest.mark.parametrize("sa,sb", [((3,), (3,)), ((2, 3), (3,)), ((3,), (2, 3)), ((2, 1), (1, 3)), ((), (3,)), ((3,), ()), ((), ())])
def test_broadcast_shapes_and_result_types(sa, sb):
    rt = bh.Runtime(bh.DryRunExecutor())
    for ta in (np.float32, np.float64, np.int32, np.int64, np.bool_):
        for tb in (np.float32, np.float64, np.int64):
            c = bh.binary("ADD", bh.empty(rt, sa, ta), bh.empty(rt, sb, tb))
            assert c.shape == np.broadcast_shapes(sa, sb) and c.dtype == np.result_type(ta, tb)
    with pytest.raises(ValueError):
        bh.binary("ADD", bh.empty(rt, (2,), np.float32), bh.empty(rt, (3,), np.float32))
    for t, k, want in [(np.int32, 2.5, np.float64), (np.float32, 2.5, np.float32), (np.int64, True, np.int64), (np.float32, 1j, np.complex64)]:
        assert bh.binary("ADD", bh.empty(rt, (4,), t), k).dtype == want
    assert bh.empty(rt, (0, 5)).size == 0 and bh.empty(rt, ()).size == 1


@pytest.mark.parametrize("t", [np.int8, np.int16, np.int32, np.uint8, np.int64])
def test_shapes_of_narrow_integers(t):
    """Element counts and strides of shapes given in NumPy integers do not wrap in their type."""
    rt = bh.Runtime(bh.DryRunExecutor())
    side = {1: 100, 2: 30_000, 4: 70_000, 8: 70_000}[np.dtype(t).itemsize]
    a = bh.empty(rt, (t(side), t(side), t(3)), np.int8)
    assert a.base.nelem == side * side * 3 and a.strides == (side * 3, 3, 1) and a.size == a.base.nelem
    assert bh.empty(rt, t(5)).shape == (5,) and bh.empty(rt, np.array([3, 4], dtype=t)).base.nelem == 12


def test_views_given_in_whole_floats_still_encode():
    base = ir.Base(np.float64, 12)
    base.handle = 77
    ins = ir.Instr(ir.OPCODES["IDENTITY"], [ir.View(base, 2.0, (4.0,), (1,)), None], ir.Constant(1.0, ir.FLOAT64))
    assert ir.encode([ins]).tolist()[-6:] == [77, 2, 1, 4, 1, 0]
