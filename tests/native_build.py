"""Builds the helper libraries of tests/native that need nvcc; a test that uses one is skipped where nvcc is missing."""
import ctypes
import glob
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "litenn_b200", "csrc")


def load(name, device_code, link_library=None):
    """tests/native/<name>.cu as a shared library; with link_library it resolves that library's functions."""
    src, out = (os.path.join(HERE, "native", f) for f in (name + ".cu", "lib" + name + ".so"))
    deps = [src, *glob.glob(os.path.join(CSRC, "*.cuh")), *glob.glob(os.path.join(CSRC, "*.h")),
            *(glob.glob(os.path.join(CSRC, "llama_kernels.cu")) if device_code else [])]
    if not os.path.exists(out) or any(os.path.getmtime(d) > os.path.getmtime(out) for d in deps):
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not os.path.exists(nvcc):
            pytest.skip("nvcc not available")
        cmd = [nvcc, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", out, src,
               "-gencode", "arch=compute_100a,code=sm_100a"]
        if os.path.exists("/usr/bin/g++"):
            cmd[1:1] = ["-ccbin", "/usr/bin/g++"]
        env = dict(os.environ)
        if link_library:
            d, f = os.path.split(os.path.abspath(link_library))
            cmd += ["-L", d, "-l:" + f]
            env["LD_RUN_PATH"] = "$ORIGIN/" + os.path.relpath(d, os.path.dirname(out))
        subprocess.run(cmd, check=True, env=env)
    return ctypes.CDLL(out)
