"""What the multi-level CUDA kernels run -- plane and colour indices by one multiplication, mask classes,
lists of cells in extra planes, stencils at constant offsets -- executed on the host for every thread of
every launch and compared with the general cell and face functions (tests/csrc/amr_planes.cpp).  With
MAESTRO_HOST_ASAN=1 (see test_amr_host_exec.py) every access is bounds-checked."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER
from tests.test_amr_host_exec import ROOT, _opt_flags


@pytest.fixture(scope="module")
def planes_lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("amrp") / "libamr_planes.so")
    subprocess.run([cxx, *_opt_flags(), "-std=c++17", "-fPIC", "-fopenmp", "-shared",
                    "-I", os.path.join(ROOT, "maestro_gb300", "csrc"), "-I", os.path.join(ROOT, "oracle"),
                    os.path.join(ROOT, "tests", "csrc", "amr_planes.cpp"),
                    os.path.join(ROOT, "oracle", "mac_oracle.cpp"), "-o", out],
                   check=True, capture_output=True)
    return ctypes.CDLL(out)


P, N, D = BC_PER, BC_NEU, BC_DIR
LAYOUTS = {
    # name: (level-0 cells, bc low, bc high, boxes of the finer levels)
    "middle": ((24, 20, 28), (P, P, N), (P, P, N), [[((12, 12, 12), (35, 27, 43))]]),
    "several_blocks_a_plane": ((96, 80), (P, N), (P, D), [[((4, 8), (119, 131)), ((120, 8), (179, 67))]]),
    "corner": ((16, 16, 16), (N, D, N), (D, N, D), [[((0, 0, 0), (19, 15, 31))]]),
    "wrap": ((20, 12, 16), (P, P, N), (P, P, N), [[((0, 4, 8), (7, 19, 23)), ((32, 4, 8), (39, 19, 23))]]),
    "covered": ((12, 10, 14), (P, N, D), (P, D, N), [[((0, 0, 0), (23, 19, 27))]]),
    "covered_twice": ((10, 8), (N, P), (D, P), [[((0, 0), (19, 15))], [((0, 0), (39, 31))]]),
    "three_levels": ((16, 12, 12), (P, N, D), (P, N, N),
                     [[((4, 0, 4), (27, 19, 19))], [((12, 0, 12), (35, 27, 27)), ((36, 0, 12), (47, 11, 27))]]),
    "thin": ((8, 8, 64), (P, P, N), (P, P, N), [[((4, 4, 4), (7, 11, 119))]]),
    "l_shape": ((28, 36), (P, N), (P, N), [[((0, 8), (51, 31)), ((0, 32), (15, 63))]]),
}


@pytest.mark.parametrize("name", list(LAYOUTS))
def test_kernel_planes_match_the_general_functions(planes_lib, name):
    n, lo, hi, fine = LAYOUTS[name]
    dx = tuple(1.0 / (v * (1 + 0.1 * d)) for d, v in enumerate(n))
    o = O._opts(n, dx, lo, hi, 1, 0, 0, 0, 0, 0, 0, 0, 0, False, 0)
    boxes = [[]] + fine
    nb, bx = O._ml_layout(n, boxes)
    ip = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))  # noqa: E731
    out = (ctypes.c_double * 2)()
    planes_lib.amrp_check(ctypes.byref(o), len(boxes), ip(nb), ip(bx), 5, out)
    assert out[1] == 0
    # tolerances 1e-13 (FP64) and 1e-5 (FP32) of an output's largest value: sums of at most 13
    # products of numbers of order one, some in another order
    assert out[0] <= 1.0
