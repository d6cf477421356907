"""Page-locked memory of results: parts are given back when the last view is gone and used again, what does not fit is pageable, the region outlives its
pool for as long as an array lives, and threads may take and drop at once.  Nothing is page-locked before a large result is there, and a forked process
keeps what it saw."""
import ctypes as C
import gc
import mmap
import os
import subprocess
import sys
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


def test_regions_are_made_for_the_results_that_need_them():
    mb = 1 << 20
    c, m = make(64 * mb)
    held = [m.empty((SMALLEST - 1,), np.uint8)]
    assert not c.blocks                                                    # small ones need none

    def sizes():
        return [len(b) // mb for b in c.blocks.values()]
    held += [m.empty((SMALLEST,), np.uint8) for _ in range(64)]
    assert sizes() == [4]
    held += [m.empty((5 * mb,), np.uint8) for _ in range(8)]               # no room: a second region, for eight of these
    assert sizes() == [4, 40]
    held += [m.empty((5 * mb,), np.uint8) for _ in range(5)]               # and one with what is left of the limit
    assert sizes() == [4, 40, 20] and sum(inside(c, a) for a in held) == 64 + 8 + 4
    held += [m.empty((SMALLEST,), np.uint8)]
    assert sizes() == [4, 40, 20]
    m.close()
    del held
    gc.collect()
    assert not c.blocks


def test_a_forked_process_keeps_what_it_saw():
    """Memory as page-locked memory is: shared between the processes."""
    class Shared(Counted):
        def alloc(self, size):
            b = mmap.mmap(-1, size)
            at = C.addressof(C.c_char.from_buffer(b))
            self.blocks[at] = b
            return at

        def free(self, at):
            self.blocks.pop(at)
    c = Shared()
    m = ResultMemory(c.alloc, c.free, 8 * SMALLEST)
    a = m.empty((SMALLEST,), np.uint8)
    assert inside(c, a)
    a.fill(3)
    there = os.pipe()
    pid = os.fork()
    if pid == 0:
        ok = False
        try:
            os.read(there[0], 1)                                           # the parent has dropped its array and made others
            mine = m.empty((SMALLEST,), np.uint8)
            ok = bool((a == 3).all()) and not inside(c, mine)
            mine.fill(9)
        finally:
            os._exit(0 if ok else 1)
    del a
    gc.collect()
    others = [m.empty((SMALLEST,), np.uint8) for _ in range(8)]
    for o in others:
        o.fill(5)
    os.write(there[1], b"x")
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0
    assert all(inside(c, o) and (o == 5).all() for o in others) and len(c.blocks) == 1      # a new region, the old one is gone
    for fd in there:
        os.close(fd)


def test_a_region_at_the_interpreters_end():
    """A pool and an array that a program never lets go of."""
    src = ("import ctypes as C, sys\nfrom jacobiforcing_b200 import hostmem\nkept = {}\n"
           "def alloc(n):\n    b = (C.c_char * n)()\n    kept[C.addressof(b)] = b\n    return C.addressof(b)\n"
           "m = hostmem.ResultMemory(alloc, lambda at: None)\na = m.empty((100000,))\nhostmem.forever = sys.forever = (m, a)\n")
    r = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stderr == ""
