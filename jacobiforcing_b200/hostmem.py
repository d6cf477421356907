"""Host memory of large results (logits): page-locked, so that the device writes straight into the array that the caller gets.

An array of fresh pageable memory costs its page faults and a second copy through the driver's staging buffer: 4.9 MB of logits (eight rows of 151936) took
0.75 ms behind a forward of 1.3 ms.  A runtime holds one region, made with the runtime; a result takes a part of it for as long as the
array (or a view of it) lives and gives it back then, from whatever thread.  What finds no room gets pageable memory as before, so a program may
keep as many results as it likes."""
from __future__ import annotations

import threading
from collections import deque

import numpy as np

REGION_BYTES = 64 << 20
SMALLEST = 64 << 10                                                        # below this an array costs less than the bookkeeping
ALIGN = 4096


class _Region:
    """A page-locked region, released when the pool and every array in it are gone."""

    def __init__(self, size, alloc, free):
        self.free, self.size, self.at = free, 0, None
        at = alloc(size)
        if at:
            self.at, self.size = at, size
        self.returned = deque()                                            # appended by whoever drops an array, drained by take()

    def __del__(self):
        if self.at is not None:
            self.free(self.at)


class _Part:
    """What an array in the region holds on to."""

    def __init__(self, region, offset, size, shape, dtype):
        self.region, self.offset, self.size = region, offset, size
        self.__array_interface__ = {"shape": shape, "typestr": np.dtype(dtype).str, "data": (region.at + offset, False), "version": 3}

    def __del__(self):
        self.region.returned.append((self.offset, self.size))


class ResultMemory:
    """alloc(bytes) -> address of page-locked memory or None, free(address)."""

    def __init__(self, alloc, free, size=REGION_BYTES):
        self._size = size
        self._region = _Region(size, alloc, free)
        self._gaps = [(0, size)] if self._region.size else []              # free parts: (offset, size), by offset
        self._lock = threading.Lock()

    def empty(self, shape, dtype=np.float32) -> np.ndarray:
        need = int(np.prod(shape, dtype=np.int64)) * np.dtype(dtype).itemsize
        if need < SMALLEST or need > self._size:
            return np.empty(shape, dtype=dtype)
        need = (need + ALIGN - 1) // ALIGN * ALIGN
        with self._lock:
            offset = self._take(need)
            region = self._region
        if offset is None:
            return np.empty(shape, dtype=dtype)
        return np.asarray(_Part(region, offset, need, tuple(shape), dtype))

    def _take(self, need):
        if self._region is None:                                           # closed
            return None
        back = self._region.returned
        while back:
            self._gaps.append(back.popleft())
            self._gaps.sort()
            merged = [self._gaps[0]]
            for at, size in self._gaps[1:]:
                last, held = merged[-1]
                if last + held == at:
                    merged[-1] = (last, held + size)
                else:
                    merged.append((at, size))
            self._gaps = merged
        for i, (at, size) in enumerate(self._gaps):
            if size >= need:
                if size == need:
                    del self._gaps[i]
                else:
                    self._gaps[i] = (at + need, size - need)
                return at
        return None

    def close(self):
        """Lets the region go; arrays that are still held keep it until they are gone."""
        with self._lock:
            self._region, self._gaps, self._size = None, [], 0


def of_library(alloc_fn, free_fn, size=REGION_BYTES) -> ResultMemory:
    """With a library's page-locked allocation: alloc_fn(bytes, void**) -> 0, free_fn(void*)."""
    import ctypes as C

    def alloc(size):
        p = C.c_void_p()
        return p.value if alloc_fn(C.c_int64(size), C.byref(p)) == 0 else None
    return ResultMemory(alloc, lambda at: free_fn(C.c_void_p(at)), min(size, REGION_BYTES))
