"""Page-locked memory of results: parts are given back when the last view is gone and used again, what does not fit is pageable, the region outlives its
pool for as long as an array lives, and threads may take and drop at once."""
import ctypes as C
import gc
import threading

import numpy as np

from jacobiforcing_b200.hostmem import ALIGN, SMALLEST, ResultMemory


class Counted:
    def __init__(self):
        self.blocks = {}

    def alloc(self, size):
        b = (C.c_char * size)()
        at = C.addressof(b)
        self.blocks[at] = b
        return at

    def free(self, at):
        del self.blocks[at]


def make(size=8 * SMALLEST):
    c = Counted()
    return c, ResultMemory(c.alloc, c.free, size)


def inside(c, a):
    at = a.__array_interface__["data"][0]
    return any(b <= at and at + a.nbytes <= b + len(m) for b, m in c.blocks.items())


def test_parts_are_used_again_and_do_not_overlap():
    c, m = make()
    rows = [m.empty((SMALLEST // 16, 4)) for _ in range(8)]
    assert all(inside(c, r) and r.dtype == np.float32 and r.flags.writeable and r.flags.c_contiguous for r in rows)
    for i, r in enumerate(rows):
        r.fill(i)
    assert [r.min() for r in rows] == [r.max() for r in rows] == list(range(8))
    assert not inside(c, m.empty((SMALLEST // 4,)))                        # full: pageable
    view = rows[3][5:7]
    rows[3] = rows[4] = None
    gc.collect()
    a = m.empty((SMALLEST // 4,))
    assert inside(c, a) and not inside(c, m.empty((SMALLEST // 4,)))       # the view still holds its part
    assert (view == 3).all()
    del view, a, rows, r
    gc.collect()
    assert inside(c, m.empty((2 * SMALLEST,), np.float32))                 # neighbours have grown together again
    assert len(c.blocks) == 1


def test_small_and_oversized_results_are_pageable():
    c, m = make()
    assert m.empty((3, 5)).shape == (3, 5) and m.empty((0, 7)).shape == (0, 7) and m.empty((16 * SMALLEST,)).shape == (16 * SMALLEST,)
    assert not any(inside(c, m.empty(s)) for s in ((3, 5), (0, 7), (16 * SMALLEST,)))
    m = ResultMemory(lambda size: None, c.free)
    assert m.empty((SMALLEST,)).shape == (SMALLEST,)                       # nothing to be had


def test_an_array_outlives_its_pool():
    c, m = make()
    a = m.empty((SMALLEST + ALIGN // 2 + 4,), np.uint8)
    a.fill(7)
    m.close()
    del m
    gc.collect()
    assert len(c.blocks) == 1 and (a == 7).all()
    del a
    gc.collect()
    assert not c.blocks


def test_threads():
    c, m = make(64 * SMALLEST)
    wrong = []

    def work(k):
        for i in range(300):
            a = m.empty((SMALLEST // 4,), np.int32)
            a.fill(k * 1000 + i)
            b = m.empty((SMALLEST // 2,), np.int32)
            b.fill(-k)
            if not ((a == k * 1000 + i).all() and (b == -k).all()):
                wrong.append(k)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not wrong and len(c.blocks) == 1
