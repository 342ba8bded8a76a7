"""The library's host code without a GPU: its objects linked against the fake
CUDA runtime of host/fake_cudart.cpp (see there), loaded beside the real one."""
import ctypes
import glob
import os
import subprocess

import numpy as np

from hera_gpu_gb300 import _native, build

HERE = os.path.dirname(os.path.abspath(__file__))


def build_library(out_dir):
    """Path of the library with the fake runtime."""
    build.build()
    src = os.path.join(HERE, "host", "fake_cudart.cpp")
    out = os.path.join(str(out_dir), "libheravis_fake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", cuda, "-o", out, src,
                    *sorted(glob.glob(os.path.join(build.BUILD, "*.o")))], check=True)
    return out


class FakeGpu:
    """One device of `capacity` bytes.  Operations are read with log()."""

    def __init__(self, path, capacity):
        self.lib = ctypes.CDLL(path)
        for name, (res, args) in _native.SIGNATURES.items():
            fn = getattr(self.lib, name)
            fn.restype, fn.argtypes = res, args
        self.lib.fake_reset.argtypes = [ctypes.c_size_t]
        self.lib.fake_used.restype = ctypes.c_size_t
        self.lib.fake_log.restype = ctypes.c_size_t
        self.lib.fake_log.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
        self.lib.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
        self.lib.fake_capture.argtypes = [ctypes.c_void_p]
        self.reset(capacity)
        self.contexts = []

    def reset(self, capacity):
        self.lib.fake_reset(capacity)

    def log(self):
        """Lines since the last call: (operation, first value, second value); of a
        launch the stream and the blocks."""
        n = self.lib.fake_log(None, 0) + 1
        buf = ctypes.create_string_buffer(n)
        self.lib.fake_log(buf, n)
        rows = [line.rsplit(" ", 2) for line in buf.value.decode().splitlines()]
        return [(op, int(a), int(b)) for op, a, b in rows]

    def context(self, budget=0):
        h = ctypes.c_void_p()
        assert self.lib.hv_create(ctypes.byref(h), 0, budget) == 0
        self.contexts.append(h)
        self.log()
        return h

    def close(self):
        for h in self.contexts:
            self.lib.hv_destroy(h)

    def call(self, ctx, precision, method, nant, nsrc, ntimes, nfreq=1, px=15, stream=0):
        """hv_vis_multifreq_device on arrays that are never read; its status."""
        freqs = np.full(nfreq, 1.5e8)
        dev = ctypes.c_void_p(1 << 20)
        return self.lib.hv_vis_multifreq_device(
            ctx, precision, _native.METHODS[method], dev, nant,
            ctypes.c_void_p(freqs.ctypes.data), nfreq, dev, ntimes, dev, dev, nsrc, dev, px, dev,
            ctypes.c_void_p(stream))

    def batch(self, ctx, sims, flags=0, px=15):
        """hv_batch_create of (antennas, sources, times, frequencies); its
        status and the batch."""
        freqs = [np.full(nf, 1.5e8) for *_, nf in sims]
        arr = (_native.HvSim * len(sims))(*[
            _native.HvSim(*[1 << 20] * 5, f.ctypes.data, 1 << 20, nant, nt, nsrc, nf, px)
            for (nant, nsrc, nt, nf), f in zip(sims, freqs)])
        h = ctypes.c_void_p()
        return self.lib.hv_batch_create(ctx, arr, len(sims), flags, ctypes.byref(h)), h


def kernels(log):
    """Names of the kernels launched (mangled)."""
    return [op.split(" ", 1)[1] for op, _, _ in log if op.startswith("launch ")]


def launched(log, name):
    return sum(name in k for k in kernels(log))
