"""The binding's logits arrays: memory is reused only when nothing refers to it."""
import sys
import types

import numpy as np
import pytest

from nano_b200 import engine
from nano_b200.engine import RowPool


def test_rows_in_use_are_never_given_out_again():
    pool = RowPool(20000)
    held = [pool.take() for _ in range(9)]
    for i, a in enumerate(held):
        a[:] = i
    tails = [a[100:200].reshape(10, 10) for a in held]          # views of views hold their buffer too
    del held, a
    for _ in range(30):
        pool.take()[:] = -1.0
    assert all((t == i).all() for i, t in enumerate(tails))


def test_rows_that_nobody_holds_are_used_again_and_bounded():
    pool = RowPool(20000)
    seen = set()
    for _ in range(50):
        seen.add(pool.take().ctypes.data)
    assert len(seen) == 1
    many = [pool.take() for _ in range(500)]
    assert len({a.ctypes.data for a in many}) == 500
    assert sum(b.nbytes for b in pool.kept) <= 32 << 20
    small = RowPool(100)
    assert small.take().shape == (100,) and not small.kept


def test_changing_an_array_does_not_change_the_next_one():
    pool = RowPool(20000)
    a = pool.take()
    a.shape = (2, 10000)
    a.flags.writeable = False
    del a
    b = pool.take()
    assert b.shape == (20000,) and b.dtype == np.float32 and b.flags.writeable


# what an interpreter's count of a free buffer and of one with a view may be, beside CPython 3.12's 2 and 3: 1 and 2 where a call's argument is lent, more where frames hold
# their own; a count that says nothing
@pytest.mark.parametrize("count", [lambda real: real - 1, lambda real: real + 3, lambda real: 2, lambda real: 1 << 30])
def test_the_interpreters_way_of_counting_does_not_matter(monkeypatch, count):
    def real(buf):
        return sys.getrefcount(buf)
    probe = np.empty(1)
    own = real(probe) - sys.getrefcount(probe)          # what the call in between adds
    monkeypatch.setattr(engine, "sys", types.SimpleNamespace(getrefcount=lambda buf: count(real(buf) - own - 1)))
    pool = RowPool(20000)
    held = [pool.take() for _ in range(9)]
    for i, a in enumerate(held):
        a[:] = i
    for _ in range(30):
        pool.take()[:] = -1.0
    assert all((a == i).all() for i, a in enumerate(held))


def test_memory_is_used_again_here():
    """The page faults that the pool is there to save."""
    pool = RowPool(20000)
    assert pool.reuse and len({pool.take().ctypes.data for _ in range(50)}) == 1
