"""Device headers of parrelray_b200/csrc compiled for the host with g++, so that a CPU test calls the very functions that
the kernels inline (those without warp or memory intrinsics).  The SFU approximations, which are PTX, become
their exact counterparts."""
import ctypes as C
import hashlib
import shutil
import subprocess
import tempfile
from pathlib import Path

import pytest

from parrelray_b200 import build

SHIM = r"""
#include <algorithm>
#include <cmath>
#include <cstring>
#include <cuda_runtime.h>
using std::acos; using std::atan2; using std::fabs; using std::floor; using std::fmax; using std::fmin; using std::isnan;
using std::max; using std::min; using std::sqrt;
#undef __noinline__
#define __noinline__  // a macro of nvcc's
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __powf(float a, float b) { return std::pow(a, b); }
template <class T> inline T __ldg(const T *p) { return *p; }
#include "prr_device.cuh"
#define sfu_rcp(v) (1.0f / (v))
#define sfu_rsqrt(v) (1.0f / sqrtf(v))
"""


def library(source: str) -> C.CDLL:
    """A library of the shim and `source` (extern "C" functions over the csrc headers it includes)."""
    gxx, inc = shutil.which("g++"), Path(build.nvcc()).resolve().parents[1] / "include"
    if not gxx or not (inc / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = Path(tempfile.gettempdir()) / f"prr_host_{hashlib.sha1(source.encode()).hexdigest()[:12]}"
    d.mkdir(exist_ok=True)
    (d / "t.cpp").write_text(SHIM + source)
    subprocess.run([gxx, "-std=c++17", "-O1", "-w", "-fpermissive", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(inc), "-I",
                    str(build.INCLUDE), "-I", str(build.CSRC), str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    return C.CDLL(str(d / "t.so"))
