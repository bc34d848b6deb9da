"""The library's host side on a simulated CUDA runtime (fake_cuda.cpp): builds it with
the host compiler and binds the C ABI and the sim_* controls."""
from __future__ import annotations

import ctypes as C
import os
import re
import subprocess

import numpy as np

from ctl_b200 import _lib as L

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
CSRC = os.path.join(ROOT, "ctl_b200", "csrc")
CUDA = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")
UNITS = ("ctlcu", "group", "hostcopy", "den", "nrrd")  # the ones without kernels

# loops (enum class Mode)
GATHER, NEAREST, CELLS, PAIRS, SEGMENTS, CELLS_UP, SEGMENTS_UP = 0, 1, 3, 4, 5, 6, 7


def build(folder: str) -> str:
    flags = ["g++", "-std=c++17", "-O1", "-fPIC", "-pthread", "-I", CUDA, "-I", os.path.join(ROOT, "include"), "-I",
             CSRC, "-include", "cuda_runtime.h"]
    srcs = [(os.path.join(CSRC, u + ".cu"), u + ".o") for u in UNITS]
    srcs.append((os.path.join(HERE, "fake_cuda.cpp"), "fake_cuda.o"))
    jobs = [subprocess.Popen([*flags, "-x", "c++", "-c", src, "-o", os.path.join(folder, obj)]) for src, obj in srcs]
    assert [j.wait() for j in jobs] == [0] * len(jobs)
    lib = os.path.join(folder, "libhostsim.so")
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-pthread", "-o", lib, *(os.path.join(folder, o) for _, o in srcs), "-ldl"],
                   check=True)
    return lib


class Sim:
    """One context of the simulated library."""

    def __init__(self, path: str, free_at_creation: int = 0):
        self.lib = lib = C.CDLL(path)
        for name, res, args in L.SIGNATURES:
            fn = getattr(lib, name, None)  # the geometry encoder is not built
            if fn is not None:
                fn.restype, fn.argtypes = res, args
        lib.sim_record.restype = C.c_char_p
        lib.sim_device_memory.restype = C.c_void_p
        lib.sim_device_memory.argtypes = [C.c_uint64]
        lib.sim_stream.restype = C.c_void_p
        lib.sim_used.restype = C.c_uint64
        lib.sim_capacity.argtypes = [C.c_uint64]
        lib.sim_mode_ms.argtypes = [C.c_int, C.c_float]
        lib.sim_free_of_device.argtypes = [C.c_int, C.c_uint64]
        lib.sim_reset()
        self.free_answers([free_at_creation])
        self.h = C.c_void_p()
        assert lib.ctlcu_create(0, C.byref(self.h)) == L.OK

    def close(self):
        self.lib.ctlcu_destroy(self.h)

    def free_answers(self, values):
        self.lib.sim_free_answers((C.c_uint64 * len(values))(*values), len(values))

    def fail(self, what, nth=1):
        self.lib.sim_fail(what.encode(), nth)

    def device(self, nbytes):
        return self.lib.sim_device_memory(nbytes)

    def settings(self, **kw):
        self.lib.ctlcu_settings_default.restype = L.Settings
        s = self.lib.ctlcu_settings_default()
        for k, v in kw.items():
            if k == "rays_per_pixel":
                s.rays_per_pixel[0], s.rays_per_pixel[1] = v
            else:
                setattr(s, k, v)
        return s

    def desc(self, n):
        d = L.VolumeDesc()
        for k in range(3):
            d.n[k], d.voxel_mm[k], d.offset_mm[k] = n[k], 1.0, 0.0
        return d

    def volume(self, n=(16, 16, 16)):
        data = np.zeros(n[::-1], np.float32)
        h = C.c_uint64()
        rc = self.lib.ctlcu_volume_create(self.h, C.byref(self.desc(n)), data.ctypes.data, 0, C.byref(h))
        return (h.value if rc == L.OK else None), rc

    def project(self, volume, s, views=4, channels=8, rows=8, host=False, stream=None, call="ctlcu_project"):
        """Status of a call with matrices and result in host or device memory."""
        pm_bytes, out_bytes = 96 * views, 4 * views * channels * rows
        if host:
            self._keep = np.zeros(pm_bytes, np.uint8), np.zeros(out_bytes, np.uint8)
            pm, out = (a.ctypes.data for a in self._keep)
        else:
            pm, out = self.device(pm_bytes), self.device(out_bytes)
        return getattr(self.lib, call)(self.h, volume, C.byref(s), pm, views, 1, channels, rows, out, stream)

    def error(self):
        return self.lib.ctlcu_last_error(self.h).decode()

    def memory_used(self):
        n = C.c_uint64()
        assert self.lib.ctlcu_memory_used(self.h, C.byref(n)) == L.OK
        return n.value

    def record(self):
        return self.lib.sim_record().decode().splitlines()

    def clear(self):
        self.lib.sim_clear_record()

    def projections(self):
        """(loop, views, stream, array, its state, sub-rays on lanes) of every projection launch."""
        out = []
        for line in self.record():
            m = re.match(r"project mode=(\d+) views=(\d+) stream=(\d+) array=(\S+) (\S+) sub=(\d),(\d)", line)
            if m:
                out.append((int(m[1]), int(m[2]), int(m[3]), m[4], m[5], (int(m[6]), int(m[7]))))
        return out

    def count(self, what):
        return sum(line.startswith(what) for line in self.record())
