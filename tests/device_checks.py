"""tests/device_checks.cu compiled against the library's headers and linked to ``libhpgpu.so``."""

import ctypes
import functools
import os
import subprocess
import tempfile

import numpy as np

from horton_part_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache(maxsize=None)
def load():
    lib = build.build()
    out = os.path.join(tempfile.mkdtemp(prefix="hp_device_checks_"), "libchecks.so")
    cmd = [build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-shared", os.path.join(HERE, "device_checks.cu"), "-o", out,
           "-cudart", "shared", lib, "-Xlinker", "-rpath=" + os.path.dirname(lib)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    return ctypes.CDLL(out)


WHAT = {name: i for i, name in enumerate(
    ("exp64", "div64", "rsqrt64", "clip01", "below", "exp_ff512", "exp_ff", "rcp_seed", "rsqrt_seed"))}


def evaluate(what, x, y=None):
    """(value, low part) of a device function; the low part is 0 but for the float pairs."""
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.ascontiguousarray(np.zeros_like(x) if y is None else y, dtype=np.float64)
    out, lo = np.empty_like(x), np.empty_like(x)
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (x, y, out, lo)]
    assert load().dc_eval(WHAT[what], len(x), *ptr) == 0
    return out, lo
