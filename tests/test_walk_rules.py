"""The host-side rules that choose and split the inviscid walks
(ocfd_walk.cuh), compiled for the host: at the sizes where both sides were
measured they take the faster one."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "opencfd-scu_b200", "csrc")

HOST = r"""
#include <cmath>
#define __device__
#define __forceinline__ inline
#define __noinline__
#define __ldg(x) (*(x))
using std::fma; using std::fabs; using std::sqrt; using std::fmin; using std::fmax;
#include "ocfd_walk.cuh"
extern "C" int march(int nx, long long cells, int uniform, int fp32) {
    return ocfd::walk::march_is_faster(nx, cells, uniform, fp32);
}
extern "C" int lanes(int nx, long long rows, long long slots) { return ocfd::walk::row_lanes(nx, rows, slots); }
extern "C" int segment(long long groups, int n, int LY, long long slots, int fp32) {
    using namespace ocfd::walk;
    return segment_cells(groups, n, LY, slots, 3, fp32 ? segment_tail<float>() : segment_tail<double>());
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "host.cpp").write_text(HOST)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I", CSRC, str(d / "host.cpp"),
                    "-o", str(d / "host.so")], check=True)
    h = ctypes.CDLL(str(d / "host.so"))
    h.segment.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    h.lanes.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong]
    h.march.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return h


# (grid, FP64 uniform, FP64 metric fields, FP32): 1 where the marches measured faster, 0 the ring
MARCH = [((12, 12, 12), 0, 0, 0), ((32, 32, 32), 0, 0, 0), ((48, 48, 48), 0, 0, 0), ((56, 56, 56), 0, 0, 0),
         ((64, 64, 64), 1, 0, 0), ((65, 64, 64), 0, 0, 0), ((33, 90, 70), 0, 0, 0), ((33, 200, 200), 0, 0, 0),
         ((70, 120, 100), 0, 0, 0), ((72, 256, 256), 0, 0, 0), ((64, 80, 80), 1, 1, 0), ((84, 84, 84), 1, 1, 0),
         ((96, 96, 96), 1, 1, 1), ((112, 112, 112), 1, 1, 1), ((256, 256, 256), 1, 1, 1)]


@pytest.mark.parametrize("dims,uniform,fields,fp32", MARCH)
def test_up7_walk_choice(host, dims, uniform, fields, fp32):
    n = dims[0] * dims[1] * dims[2]
    assert (host.march(dims[0], n, 1, 0), host.march(dims[0], n, 0, 0), host.march(dims[0], n, 1, 1)) == \
        (uniform, fields, fp32)


def test_segments_of_fp32_lines(host):
    """WENO7 lines in FP32 take more segments than in FP64 where one round of
    warps would walk long ones beside idle schedulers (both measured, see
    segment_cells): the z lines of 160x33x65 and the x lines of 400x40x40,
    five blocks an SM.  Every line is covered whatever the size."""
    slots = 148 * 5 * 4
    assert (host.segment(20 * 33, 65, 4, slots, 1), host.segment(20 * 33, 65, 4, slots, 0)) == (11, 22)
    assert (host.segment(1600, 400, 32, slots, 1), host.segment(1600, 400, 32, slots, 0)) == (58, 400)
    for n in (8, 9, 31, 65, 250, 4099):
        for groups in (1, 30, 4096, 300000):
            for fp32 in (0, 1):
                assert 1 <= host.segment(groups, n, 4, slots, fp32) <= n


@pytest.mark.parametrize("nx,rows,lanes", [(93, 836, 32), (74, 1456, 32), (65, 4096, 32), (130, 1600, 32),
                                           (160, 2145, 32), (80, 6400, 32), (96, 9216, 8), (64, 4096, 16), (60, 2000, 16),
                                           (32, 1024, 8), (60, 6000, 16), (12, 90000, 8), (160, 25600, 8),
                                           (256, 65536, 32)])
def test_row_lanes(host, nx, rows, lanes):
    """Lanes a row of the UP7 x walk in FP64 (four blocks an SM): short
    chains of passes on small grids, the fewest wasted cells on large ones."""
    assert host.lanes(nx, rows, 148 * 4 * 4) == lanes
