"""Compiles the hooks that see the library's internal headers."""
import ctypes as C
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "soil_b200", "csrc")


def build_internal(out_dir, name):
    """tests/hooks/<name>.cu (nvcc) or .cpp (g++: host-only headers), loaded."""
    out = os.path.join(str(out_dir), f"lib{name}.so")
    src = os.path.join(ROOT, "tests", "hooks", name)
    if os.path.exists(src + ".cu"):
        cmd = ["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a",
               "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", src + ".cu"]
    else:
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", src + ".cpp"]
    subprocess.check_call(cmd + ["-shared", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                                 "-o", out])
    return C.CDLL(out)
