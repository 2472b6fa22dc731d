"""The C-ABI over fake_cudart.cpp: the library's own objects linked with a CUDA runtime
whose memory is the host's and whose launches are recorded only.

``run(fn)`` calls the module-level function ``fn`` with a ``FakeCuda`` in a process of its
own, so that the two copies of the library never share one."""
import ctypes as C
import multiprocessing as mp
import os
import subprocess

import numpy as np

from msplat_street_b200 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(build.BUILD, "libmsplat_fake.so")


def _build():
    build.build()
    src = os.path.join(HERE, "fake_cudart.cpp")
    objs = sorted(os.path.join(build.BUILD, os.path.basename(s)[:-3] + ".o") for s in build.sources())
    if build._stale(LIB, [src] + objs):
        inc = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
        # -Bsymbolic: its cudart, not one the process has loaded
        cmd = ["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", inc, "-o", LIB, src, *objs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return LIB


def _call(fn, path, args):
    return fn(FakeCuda(path), *args)


def run(fn, *args):
    path = _build()
    with mp.get_context("spawn").Pool(1) as pool:
        return pool.apply_async(_call, (fn, path, args)).get(timeout=300)


class FakeCuda:
    def __init__(self, path):
        self.lib = C.CDLL(path)
        for name, (res, args) in _lib._SIGS.items():
            fn = getattr(self.lib, name)
            fn.restype, fn.argtypes = res, args
        self.lib.fake_readback.argtypes = [C.c_int64]
        self.lib.fake_launch.restype = C.c_char_p

    def context(self):
        ctx = C.c_void_p()
        assert self.lib.msplat_cuda_ctx_create(C.byref(ctx)) == 0
        return ctx

    def allocs_left(self, n):
        """Only the next n allocations succeed (-1: all)."""
        self.lib.fake_allocs_left(n)

    def readback(self, v):
        """What the library reads where it copies one 64-bit count to the host."""
        self.lib.fake_readback(v)

    def launches(self):
        """(kernel name, grid x, grid y, block x) of every launch since the last call."""
        out = []
        for i in range(self.lib.fake_launches()):
            g, h, b = C.c_uint(), C.c_uint(), C.c_uint()
            name = self.lib.fake_launch(i, C.byref(g), C.byref(h), C.byref(b)).decode()
            out.append((name, g.value, h.value, b.value))
        self.lib.fake_clear_launches()
        return out

    def render(self, ctx, n, w, h, degree=0):
        """msplat_cuda_render of n Gaussians (addresses only: nothing reads them)."""
        return self.lib.msplat_cuda_render(ctx, *self._view(n, w, h, degree), 64, 64, 64, _BG.ctypes.data,
                                           C.byref(C.c_void_p()))

    def render_backward(self, ctx, n, w, h, degree=0):
        return self.lib.msplat_cuda_render_backward(ctx, *self._view(n, w, h, degree), _BG.ctypes.data, *[64] * 7)

    def render_batch(self, ctx, views, n, w, h):
        vs = (_lib.View * views)()
        for v in vs:
            v.num_points, v.img_width, v.img_height = n, w, h
            v.means3d = v.scales = v.quats = v.features_dc = v.opacities = v.out_img = 64
            v.glob_scale = v.fx = v.fy = 1.0
        return self.lib.msplat_cuda_render_batch(ctx, views, vs)

    def pair_counts(self, ctx):
        out = (C.c_int64 * 2)()
        return self.lib.msplat_cuda_frame_pair_counts(ctx, out)

    @staticmethod
    def _view(n, w, h, degree):
        return (n, 64, 64, 1.0, 64, _EYE.ctypes.data, _EYE.ctypes.data, 100.0, 100.0, w / 2, h / 2, h, w,
                (w + 15) // 16, (h + 15) // 16, 0.01, degree, degree, _BG.ctypes.data)


_EYE = np.eye(4, dtype=np.float32)
_BG = np.zeros(3, np.float32)
