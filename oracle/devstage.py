"""ctypes binding of oracle/devstage.cc: the library's per-site code compiled
for the host.

TEST INFRASTRUCTURE ONLY: the tests use it to check the kernels' own code on
the CPU; the product library never links it.
"""
from __future__ import annotations

import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "ewpt-gpu_gb300", "csrc")
LIB = os.path.join(HERE, "build", "libdevstage.so")
SRC = os.path.join(HERE, "devstage.cc")


def _cuda_include():
    nvcc = next((c for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc")
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        raise RuntimeError("nvcc not found")
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def build(force: bool = False) -> str:
    deps = [SRC, os.path.join(HERE, "host_device.h"), os.path.join(ROOT, "include", "ewpt.h"),
            *glob.glob(os.path.join(CSRC, "*.cuh"))]
    if not force and os.path.exists(LIB) and all(os.path.getmtime(d) <= os.path.getmtime(LIB) for d in deps):
        return LIB
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    tmp = f"{LIB}.{os.getpid()}"
    subprocess.check_call([os.environ.get("CXX", "g++"), "-shared", "-fPIC", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread",
                           "-I", HERE, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", _cuda_include(), SRC,
                           "-o", tmp])
    os.replace(tmp, LIB)
    return LIB


_lib = None


def lib():
    global _lib
    if _lib is None:
        build()
        L = C.CDLL(LIB)
        dp = C.POINTER(C.c_double)
        for f in (L.ds_stencils, L.ds_diffs):
            f.argtypes = [C.c_int, C.c_int, C.c_int, dp, C.c_int, dp]
            f.restype = None
        L.ds_rates.argtypes = [C.c_int, C.c_int, C.c_int, dp, dp, dp, C.c_double, C.c_double, C.c_int]
        L.ds_rates.restype = None
        _lib = L
    return _lib


def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _call(f, rows, shape, y, a):
    y = np.ascontiguousarray(y, dtype=np.float64)
    out = np.empty((rows, int(np.prod(shape))))
    f(*shape, _ptr(y), a, _ptr(out))
    return out


def stencils(shape, y, a):
    """Rows: grad (3) and Laplacian of array a by grad_lap, grad (3) by grad,
    divergence of a, a + 1, a + 2 (times 60 dx, the Laplacian 180 dx^2)."""
    return _call(lib().ds_stencils, 8, shape, y, a)


def diffs(shape, y, a):
    """The diagnostics' rows: grad (3) of array a, divergence and curl (3) of a, a + 1, a + 2."""
    return _call(lib().ds_diffs, 7, shape, y, a)


FORMS = {"fp64": 0, "fp32": 1, "orders": 2}


def rates(shape, coef, y, Jex=0.0, gamma=0.0, form="fp64"):
    """Rates of every site.  coef: (gw, gy, gp2, lambda, vev, beta_w, beta_y, dx);
    form: the code of the FP64 stages, the equations of the FP32 forms, or those
    of the DF64 form and the alternative stencil orders."""
    y = np.ascontiguousarray(y, dtype=np.float64)
    cp = np.ascontiguousarray(coef, dtype=np.float64)
    r = np.full_like(y, np.nan)
    lib().ds_rates(*shape, _ptr(cp), _ptr(y), _ptr(r), Jex, gamma, FORMS[form])
    return r
