"""The library on a CUDA runtime without a device (tests/fake_runtime.cpp): its host side --
allocations, accounting, choice of routes -- runs and is checked on the CPU."""
import contextlib
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from bskit_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
MESH = ctypes.c_void_p(1 << 20)   # a device address; kernels are not run
OUT = ctypes.c_void_p(1 << 21)


def link(tmp):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    build.build()
    objs = [os.path.join(build.BUILD, f[:-3] + ".o") for f in sorted(os.listdir(build.CSRC))
            if f.endswith(".cu")]
    fake, so = os.path.join(tmp, "fake.o"), os.path.join(tmp, "libfake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-c", "-I",
                    os.path.join(build.cuda_home(), "include"),
                    os.path.join(HERE, "fake_runtime.cpp"), "-o", fake], check=True)
    # the fake's names stay inside the library: its objects bind to them, nothing else does
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", so] + objs + [fake],
                   check=True)
    return so


class Engine(object):
    def __init__(self, so):
        self.lib = ctypes.CDLL(so)
        for name, res, args in _lib.SIGNATURES:
            fn = getattr(self.lib, name)
            fn.restype, fn.argtypes = res, args
        self.lib.fake_live_bytes.restype = ctypes.c_longlong
        self.lib.fake_set_limit.argtypes = [ctypes.c_longlong]
        self.lib.fake_launches.argtypes = [ctypes.c_char_p]

    def error(self):
        buf = ctypes.create_string_buffer(512)
        self.lib.bsk_last_error(buf, 512)
        return buf.value.decode()

    def ok(self, rc):
        assert rc == _lib.BSK_OK, self.error()

    def live(self):
        return int(self.lib.fake_live_bytes())

    def launches(self, part=""):
        return self.lib.fake_launches(part.encode())

    @contextlib.contextmanager
    def capture(self):
        self.lib.fake_set_capturing(1)
        try:
            yield
            assert not self.lib.fake_capture_broken()
        finally:
            self.lib.fake_set_capturing(0)

    def plan(self, n, box, edges, budget=0, grid=_lib.GRID_REDUCED):
        e = np.ascontiguousarray(edges, dtype=np.float64)
        h = ctypes.c_void_p()
        self.ok(self.lib.bsk_plan_create(n, box, len(e), e.ctypes.data, grid, budget,
                                         ctypes.byref(h)))
        return h

    def close(self, plan, *sets):
        for s in sets:
            self.ok(self.lib.bsk_triset_destroy(s))
        self.ok(self.lib.bsk_plan_destroy(plan))

    def triangles(self, plan, tri):
        t = np.ascontiguousarray(tri, dtype=np.int32)
        h = ctypes.c_void_p()
        self.ok(self.lib.bsk_triset_create(plan, len(t), t.ctypes.data, ctypes.byref(h)))
        return h

    def levels(self, ts):
        out = (ctypes.c_int64 * 60)()
        n = self.lib.bsk_triset_levels(ts, out, 10)
        return [int(out[6 * k]) for k in range(n)]

    def info(self, plan, which):
        out = (ctypes.c_int64 * _lib.INFO_COUNT)()
        self.ok(self.lib.bsk_plan_query(plan, out))
        return int(out[which])

    def footprint(self, plan):
        return self.info(plan, _lib.INFO_FOOTPRINT)

    def paint(self, plan, slot=0):
        self.ok(self.lib.bsk_paint(plan, slot, MESH, None))

    def measure(self, plan, ts, slots=(0, 0, 0), precision=_lib.PREC_BF16X3, stream=None):
        self.ok(self.lib.bsk_measure_b(plan, ts, *slots, precision, OUT, stream))
