"""Single kernels of the hybrid engine on torch tensors (tests/cuda/row_ops.cu), for tests of their arithmetic."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jacobiforcing_b200", "csrc")
SOURCE = os.path.join(ROOT, "tests", "cuda", "row_ops.cu")


def build() -> str:
    out = os.path.join(ROOT, "build", "librow_ops.so")
    srcs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")] + [SOURCE]
    if os.path.exists(out) and all(os.path.getmtime(s) <= os.path.getmtime(out) for s in srcs):
        return out
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    os.makedirs(os.path.dirname(out), exist_ok=True)
    tmp = "%s.%d.tmp" % (out, os.getpid())
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-w", "-I",
                           os.path.join(ROOT, "include"), "-I", CSRC, SOURCE, "-o", tmp])
    os.replace(tmp, out)
    return out


def _at(t):
    return C.c_void_p(t.data_ptr())


class RowOps:
    def __init__(self):
        self.lib = C.CDLL(build())
        self.lib.ops_split_tiles.restype = C.c_longlong
        self.err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def _ok(self, rc):
        assert rc == 0, rc

    def exp_rates(self, dt, a):
        """exp(dt a) for dt, a [n] fp32, n even, steps equal in pairs."""
        out = torch.empty_like(dt)
        torch.cuda.synchronize()
        self._ok(self.lib.ops_exp_rates(_at(dt), _at(a), _at(out), dt.numel()))
        return out

    def sigmoid(self, z):
        out = torch.empty_like(z)
        torch.cuda.synchronize()
        self._ok(self.lib.ops_sigmoid(_at(z), _at(out), z.numel()))
        return out

    def swiglu(self, gate, up, divide):
        """bf16(g / (1 + exp(-g))) * u of fp32 vectors of bf16 values, a multiple of eight long; divide: with IEEE division."""
        out = torch.empty_like(up)
        torch.cuda.synchronize()
        self._ok(self.lib.ops_swiglu(_at(gate), _at(up), _at(out), gate.numel(), int(divide)))
        return out

    def few(self, a, w, kernel="few", out=None, wait=True):
        """a [T, K] w [N, K]^T in bf16 -> fp32, by the kernel of few rows ("few") or the one beside it ("rows")."""
        t, k = a.shape
        out = torch.empty(t, w.shape[0], device="cuda") if out is None else out
        if wait:
            torch.cuda.synchronize()
        self._ok(getattr(self.lib, "ops_" + kernel)(_at(a), a.stride(0), _at(w), t, w.shape[0], k, _at(out), int(wait)))
        return out

    def split_rows(self, a):
        """a [T, K] fp32 -> its three parts [T, 3, K up to a multiple of 64], the lowest first."""
        t, k = a.shape
        out = torch.empty(t, 3, (k + 63) // 64 * 64, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        self._ok(self.lib.ops_split_rows(_at(a), a.stride(0), t, k, _at(out)))
        return out

    def split_product(self, a, w):
        """a [T, K] fp32 times w [N, K]^T bf16, in three parts on the tensor cores."""
        (t, k), n = a.shape, w.shape[0]
        host = w.float().cpu().contiguous()
        tiles = torch.empty(self.lib.ops_split_tiles(None, n, k, None), dtype=torch.int16)
        assert self.lib.ops_split_tiles(_at(host), n, k, _at(tiles)) == tiles.numel()
        tiles, parts, out = tiles.cuda(), self.split_rows(a), torch.empty(t, n, device="cuda")
        torch.cuda.synchronize()
        self._ok(self.lib.ops_split_product(_at(parts), t, k, _at(tiles), n, _at(out), _at(self.err)))
        assert int(self.err) == 0
        return out

    def fp32_product(self, a, w):
        (t, k), n = a.shape, w.shape[0]
        out = torch.empty(t, n, device="cuda")
        torch.cuda.synchronize()
        self._ok(self.lib.ops_fp32_product(_at(a), a.stride(0), _at(w), t, n, k, _at(out)))
        return out
