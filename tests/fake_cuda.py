"""The engines' host code on a CUDA runtime without a GPU (tests/host/fake_cuda.cpp): what is launched, in which order, on which device,
and what happens when a call fails."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jacobiforcing_b200", "csrc")
FAKE = os.path.join(ROOT, "tests", "host", "fake_cuda.cpp")
LAUNCH, ATTRIBUTE, TENSOR_MAP, TO_HOST = 0, 1, 2, 3


def build(engine: str) -> str:
    """The engine's source with device code that nothing loads, linked against the runtime that notes things down."""
    out = os.path.join(ROOT, "build", "lib%s_fake.so" % engine)
    srcs = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", f) for f in os.listdir(os.path.join(ROOT, "include"))] + [FAKE]
    if os.path.exists(out) and all(os.path.getmtime(s) <= os.path.getmtime(out) for s in srcs):
        return out
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    tmp = "%s.%d.tmp" % (out, os.getpid())
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler", "-fPIC,-O1,-fno-gnu-unique", "-w",
                           "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic",
                           os.path.join(CSRC, engine + "_engine.cu"), FAKE, "-o", tmp])
    os.replace(tmp, out)
    return out


class Fake:
    def __init__(self, path):
        self.lib = C.CDLL(path)
        self.lib.fake_launch_name.restype = C.c_char_p
        self.lib.fake_count.restype = C.c_long
        self.lib.fake_fail.argtypes = [C.c_int, C.c_long]
        self.lib.fake_room.argtypes = [C.c_longlong]
        self.lib.fake_used.restype = C.c_longlong
        self.lib.fake_cleared.restype, self.lib.fake_cleared.argtypes = C.c_long, [C.c_long]
        self.lib.fake_plant.argtypes = [C.c_long, C.c_long, C.c_int, C.c_long]
        self.reset()

    def reset(self):
        self.lib.fake_reset()

    def fail(self, what, at):
        """The call number `at` from here on (0: the next one) of this kind fails."""
        self.lib.fake_fail(what, at)

    def count(self, what):
        return self.lib.fake_count(what)

    def room(self, size=1 << 40):
        """The device has this many bytes."""
        self.lib.fake_room(size)

    def used(self):
        return self.lib.fake_used()

    def pinned(self):
        """The device of every page-locked region that was made for results since the last reset."""
        return [self.lib.fake_pinned_device(i) for i in range(self.lib.fake_pinned())]

    def on_their_way(self):
        """Copies to the host since the last wait for the stream."""
        return self.lib.fake_on_their_way()

    def plant(self, size, at, value, first=0):
        """Copies to the host of `size` bytes bring this int at byte `at`, from copy number `first` of that size on, until the next reset: what kernels that ran would
        have left there."""
        self.lib.fake_plant(size, at, value, first)

    def watch(self, on):
        """From here on, look whether the sources of copies to the device stay as they are until the wait behind them."""
        self.lib.fake_watch(int(on))

    def changed(self):
        """How many did not."""
        return self.lib.fake_changed()

    def cleared(self, size):
        """How often this many bytes were set on the stream since the last reset."""
        return self.lib.fake_cleared(size)

    def launches(self):
        """(kernel, device) of every launch that went through since the last reset."""
        return [(self.lib.fake_launch_name(i).decode(), self.lib.fake_launch_device(i)) for i in range(self.lib.fake_launches())]

    def overlaps(self):
        """Whether each launch may start under the one before it."""
        return [bool(self.lib.fake_launch_overlaps(i)) for i in range(self.lib.fake_launches())]

    def blocks(self, kernel):
        """Blocks along x of every launch of the kernels whose name holds this."""
        return [self.lib.fake_launch_blocks(i) for i in range(self.lib.fake_launches()) if kernel in self.lib.fake_launch_name(i).decode()]
