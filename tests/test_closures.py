"""The boundary closures of the device code (ocfd_face.cuh), compiled for the
host: the value of a face that a closure replaces comes from the cells
between the closed faces alone (OCFD_bound_scheme_kernel_{p,m},
src/OCFD_bound_Scheme.cu:554-944)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opencfd-scu_b200", "csrc")

HOST = r"""
#include <cmath>
#define __device__
#define __forceinline__ inline
using std::fma; using std::fabs; using std::sqrt; using std::fmin; using std::fmax;
#include "ocfd_face.cuh"
#define CLOSURE(name, R) extern "C" int name(int sign, int lo, int hi, int KA, int KB, int F, int n, \
    const R *v, R *out) { return ocfd::closure<R>(sign, lo, hi, KA, KB, F, n, v, *out); }
CLOSURE(closure_f64, double)
CLOSURE(closure_f32, float)
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("closures")
    (d / "host.cpp").write_text(HOST)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I", CSRC, str(d / "host.cpp"),
                    "-o", str(d / "host.so")], check=True)
    return ctypes.CDLL(str(d / "host.so"))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("extents", [((2, 2), (2, 2)), ((3, 3), (3, 3)), ((3, 4), (4, 3))])
def test_closures_read_no_ghost(host, dtype, extents):
    """Every closed face and sign, of the extents of each scheme: the same
    value whatever stands in the ghosts, not-a-number included."""
    n = 12
    fn = host.closure_f64 if dtype == np.float64 else host.closure_f32
    f = np.random.default_rng(4).uniform(0.5, 2.0, n).astype(dtype)
    replaced = 0
    for sign in (0, 1):
        for lo, hi in ((1, 0), (0, 1), (1, 1)):
            for F in range(-1, n):
                got = []
                for ghost in (0.0, 1.0, np.nan, np.inf):
                    line = np.concatenate([np.full(4, ghost, dtype), f, np.full(5, ghost, dtype)])
                    v = np.ascontiguousarray(line[F - 3 + 4:F + 5 + 4])
                    out = np.full(1, -7.0, dtype)
                    hit = fn(sign, lo, hi, *extents[sign], F, n, v.ctypes.data_as(ctypes.c_void_p),
                             out.ctypes.data_as(ctypes.c_void_p))
                    if hit:
                        got.append(out[0])
                replaced += bool(got)
                assert all(np.isfinite(g) and g == got[0] for g in got), (sign, lo, hi, F, got)
    assert replaced >= 20
