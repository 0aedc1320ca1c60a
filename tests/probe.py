"""Builds a .cu file of this folder, which includes kernels' sources, into a
shared library and loads it: for tests of what the C ABI does not show."""
import ctypes
import glob
import os
import subprocess

from multigrid_meshless_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, defines=()):
    src = os.path.join(HERE, name + ".cu")
    tag = "".join("_" + d.replace("=", "_") for d in defines)
    out = os.path.join(HERE, "build", f"{name}{tag}.so")
    inputs = [src] + [f for e in ("cu", "cuh", "h") for f in glob.glob(os.path.join(build.CSRC, "*." + e))]
    if not os.path.exists(out) or any(os.path.getmtime(f) > os.path.getmtime(out) for f in inputs):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        cmd = [build.NVCC] + build.NVCC_FLAGS + ["-Xcompiler", "-fvisibility=default"] + \
            ["-D" + d for d in defines] + ["-I", os.path.join(build.ROOT, "include"), "-o", out, src]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    return ctypes.CDLL(out)
