"""The binding's logits arrays: memory is reused only when nothing refers to it."""
import numpy as np

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
