"""tests/cpp/linalg_calls.cpp built with g++ against the product library and loaded."""
import ctypes as C
import os
import subprocess
import tempfile

import numpy as np
import torch

from test_cpp_facade import CUDA_INC, LIB, ROOT

STRIP = np.dtype([("e0", "i4"), ("b0", "i4"), ("nx", "i4"), ("ny", "i4"), ("j0", "i4"), ("nr", "i4"),
                  ("ex", "i8", 2), ("pk", "i8")])
_lib = None


def lib():
    global _lib
    if _lib is None:
        out = os.path.join(tempfile.mkdtemp(), "linalg_calls.so")
        r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", "-I",
                            os.path.join(ROOT, "iceicle_b200", "csrc"), "-I", CUDA_INC,
                            os.path.join(ROOT, "tests", "cpp", "linalg_calls.cpp"), "-o", out, LIB,
                            f"-Wl,-rpath,{os.path.dirname(LIB)}"], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-4000:]
        _lib = C.CDLL(out)
        _lib.strip_bytes.restype = C.c_longlong
    return _lib


def ptr(t):
    return C.c_void_p(t.data_ptr())


class StripGrid:
    """an nx x ny grid with random factors in natural order, cut into strips and packed"""

    def __init__(self, bs, nx, ny, f32, seed=0):
        self.bs, self.f32, S = bs, int(f32), lib().strip_rows(bs)
        rng = np.random.default_rng(seed)
        nnz = 5 * nx * ny - 2 * nx - 2 * ny
        rand = lambda *s: torch.from_numpy(rng.standard_normal(s) * (0.3 / bs ** 0.5)).cuda()
        self.lu, self.uinv = rand(nnz, bs, bs), rand(nx * ny, bs, bs)
        self.x = torch.from_numpy(rng.standard_normal(nx * ny * bs)).cuda()
        self.f = torch.empty_like(self.x)
        self.err = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.strips, nex, pk = [], 0, 0
        for j in range(0, ny, S):
            nr = min(S, ny - j)
            self.strips.append((0, 0, nx, ny, j, nr, (nex, nex + nx * bs), pk))
            nex += 2 * nx * bs
            pk += lib().strip_bytes(bs, nx, nr, self.f32)
        self.shape = (nx + min(S, ny) - 1, nx)
        self.nex = nex
        raw = np.array(self.strips, dtype=STRIP).view(np.uint8).copy()
        self.d_strips = torch.from_numpy(raw).cuda()
        self.ex = torch.empty(nex, dtype=torch.float64, device="cuda")
        self.ticket = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.pk = torch.empty(pk, dtype=torch.uint8, device="cuda")
        self.pack()

    def _plan(self, first=0):
        return (C.c_int(self.bs), C.c_int(len(self.strips) - first), C.c_int(self.shape[0]), C.c_int(self.shape[1]),
                C.c_void_p(self.d_strips.data_ptr() + first * STRIP.itemsize), ptr(self.ex), C.c_longlong(self.nex),
                ptr(self.ticket))

    def pack(self):
        assert lib().strip_pack(*self._plan(), ptr(self.lu), ptr(self.uinv), ptr(self.pk), self.f32) == 0

    def apply(self, y, side_by_side=False, first=0):
        """the strips from `first` on; returns the error flag"""
        st = lib().strip_apply(*self._plan(first), ptr(self.pk), self.f32, ptr(self.x), ptr(y), ptr(self.f),
                               ptr(self.err), int(side_by_side))
        assert st == 0, st
        torch.cuda.synchronize()
        return int(self.err[0])
