"""Host memory of large results (logits): page-locked, so that the device writes straight into the array that the caller gets.

An array of fresh pageable memory costs its page faults and a second copy through the driver's staging buffer: 4.9 MB of logits (eight rows of 151936) took
0.75 ms behind a forward of 1.3 ms.  A runtime holds up to 64 MB in regions, each made for a result that finds no room in those before it and large enough
for eight like it (page-locking takes about 1 ms per MB; a runtime that returns no large results takes none).  A result takes a part for as long as
the array (or a view of it) lives and gives it back then, from whatever thread.  What finds no room gets pageable memory as before, so a program may keep
as many results as it likes.

A forked process shares page-locked memory with its parent, where pageable memory would be a copy: behind a fork no part of the regions from before it is
used again, so what the child reads stays, and the child itself gets pageable memory."""
from __future__ import annotations

import os
import threading
import weakref
from collections import deque

import numpy as np

REGION_BYTES = 64 << 20
SMALLEST = 64 << 10                                                        # below this an array costs less than the bookkeeping
RESULTS, LEAST = 8, 4 << 20                                                # a region: so many results like its first one, so many bytes
ALIGN = 4096


class _Region:
    """Page-locked memory, released when the pool and every array in it are gone."""

    def __init__(self, at, size, free):
        self.at, self.size, self.free, self.owner = at, size, free, os.getpid()
        self.gaps = [(0, size)]                                            # free parts: (offset, size), by offset
        self.returned = deque()                                            # appended by whoever drops an array, drained by take()

    def __del__(self, getpid=os.getpid):                                   # also when the interpreter ends and modules are empty
        if self.owner == getpid():
            self.free(self.at)

    def take(self, need):
        back = self.returned
        while back:
            self.gaps.append(back.popleft())
            self.gaps.sort()
            merged = [self.gaps[0]]
            for at, size in self.gaps[1:]:
                last, held = merged[-1]
                if last + held == at:
                    merged[-1] = (last, held + size)
                else:
                    merged.append((at, size))
            self.gaps = merged
        for i, (at, size) in enumerate(self.gaps):
            if size >= need:
                if size == need:
                    del self.gaps[i]
                else:
                    self.gaps[i] = (at + need, size - need)
                return at
        return None


class _Part:
    """What an array in a region holds on to."""

    def __init__(self, region, offset, size, shape, dtype):
        self.region, self.offset, self.size = region, offset, size
        self.__array_interface__ = {"shape": shape, "typestr": np.dtype(dtype).str, "data": (region.at + offset, False), "version": 3}

    def __del__(self):
        self.region.returned.append((self.offset, self.size))


class ResultMemory:
    """alloc(bytes) -> address of page-locked memory or None, free(address); up to `size` bytes."""

    def __init__(self, alloc, free, size=REGION_BYTES):
        self._alloc, self._free, self._size = alloc, free, size
        self._regions = []                                                 # in use
        self._alive = weakref.WeakSet()                                    # these, and older ones that arrays still hold
        self._lock = threading.Lock()
        _pools.add(self)

    def empty(self, shape, dtype=np.float32) -> np.ndarray:
        need = int(np.prod(shape, dtype=np.int64)) * np.dtype(dtype).itemsize
        if need < SMALLEST or need > self._size:
            return np.empty(shape, dtype=dtype)
        need = (need + ALIGN - 1) // ALIGN * ALIGN
        with self._lock:
            part = self._take(need)
        if part is None:
            return np.empty(shape, dtype=dtype)
        return np.asarray(_Part(*part, need, tuple(shape), dtype))

    def _take(self, need):
        for i, region in enumerate(self._regions):
            offset = region.take(need)
            if offset is not None:
                if i:                                                      # the next one is tried there first
                    self._regions[0], self._regions[i] = region, self._regions[0]
                return region, offset
        size = min(self._size - sum(r.size for r in self._alive), max(RESULTS * need, LEAST))
        if size < need:
            return None
        at = self._alloc(size)
        if not at:
            self._size = 0                                                 # nothing more to be had
            return None
        region = _Region(at, size, self._free)
        self._regions.insert(0, region)
        self._alive.add(region)
        return region, region.take(need)

    def close(self):
        """Lets the regions go; arrays that are still held keep theirs until they are gone."""
        with self._lock:
            self._regions, self._size = [], 0


_pools = weakref.WeakSet()
_forking = []


def _before_fork():
    _forking[:] = list(_pools)
    for pool in _forking:
        pool._lock.acquire()
        pool._regions = []


def _after_fork_in_parent():
    for pool in _forking:
        pool._lock.release()
    _forking.clear()


def _after_fork_in_child():
    for pool in _forking:
        pool._lock, pool._size = threading.Lock(), 0
    _forking.clear()


os.register_at_fork(before=_before_fork, after_in_parent=_after_fork_in_parent, after_in_child=_after_fork_in_child)


def of_library(alloc_fn, free_fn, device, size=REGION_BYTES) -> ResultMemory:
    """With a library's page-locked allocation: alloc_fn(device, bytes, void**) -> 0, free_fn(void*)."""
    import ctypes as C

    def alloc(size):
        p = C.c_void_p()
        return p.value if alloc_fn(device, C.c_int64(size), C.byref(p)) == 0 else None
    return ResultMemory(alloc, lambda at: free_fn(C.c_void_p(at)), min(size, REGION_BYTES))
