"""tests/device_checks.cu compiled against the library's headers and linked to ``libhpgpu.so``."""

import ctypes
import functools
import os
import subprocess
import tempfile

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
