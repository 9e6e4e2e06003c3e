"""Device functions of csrc/*.cuh compiled for the host, so that their arithmetic (only IEEE operations and
library calls) can be checked without a GPU."""
import ctypes
import os
import shutil
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "quickcbc_b200", "csrc")


HELPERS = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
using std::fma;
using std::rint;
template <class T> static inline T __ldg(const T* p) { return *p; }
static inline uint64_t bits_(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static inline int __double2hiint(double x) { return (int)(bits_(x) >> 32); }
static inline int __double2loint(double x) { return (int)bits_(x); }
static inline double __hiloint2double(int hi, int lo) {
  const uint64_t b = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
}
"""


def compile_host(tmp_path, code, *flags):
    """Shared library of `code` (C++) with the device headers on the include path and the device's helpers defined."""
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    src, out = os.path.join(tmp_path, "host.cpp"), os.path.join(tmp_path, "host.so")
    with open(src, "w") as f:
        f.write(HELPERS + code)
    subprocess.run(["g++", "-std=c++17", "-O1", "-mfma", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I", inc,
                    "-I", CSRC, *flags, src, "-o", out], check=True)
    return ctypes.CDLL(out)
