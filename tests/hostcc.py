"""Device functions of csrc/*.cuh compiled for the host, so that their arithmetic (only IEEE operations and
library calls) can be checked without a GPU."""
import ctypes
import os
import shutil
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "quickcbc_b200", "csrc")


def compile_host(tmp_path, code, *flags):
    """Shared library of `code` (C++) with the device headers on the include path and __ldg defined."""
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, out = os.path.join(tmp_path, "host.cpp"), os.path.join(tmp_path, "host.so")
    with open(src, "w") as f:
        f.write("#include <cmath>\n#include <cstring>\n#include <cstdint>\n"
                "template <class T> static inline T __ldg(const T* p) { return *p; }\n" + code)
    subprocess.run(["g++", "-std=c++17", "-O1", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I", inc,
                    "-I", CSRC, *flags, src, "-o", out], check=True)
    return ctypes.CDLL(out)
