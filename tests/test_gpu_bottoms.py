"""Bottoms of the cell-centred V-cycle where the solver's split changes: 65 to 128 cells belong to one CTA of
the cluster, more are spread over all of them (64 and fewer have an inverse, switched off here)."""
import importlib
import os
import subprocess

import numpy as np
import pytest

import oracle as O
from maestro_gb300 import capi
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER, make_case
from maestro_gb300.macproject import BcTower, Layout, MacError, MacProjector
from tests._util import phi_rel_err, u_rel_err
from tests.test_gpu_parity import gpu_project

pytestmark = pytest.mark.gpu

BOTTOMS = {
    # name: (cells of a two-level hierarchy unless it stops by itself, top face)
    "64": ((16, 16), BC_NEU),
    "65_odd": ((10, 26), BC_NEU),
    "125_odd": ((10, 10, 10), BC_NEU),
    "126_odd": ((18, 28), BC_DIR),
    "128": ((8, 64), BC_NEU),
    "129_odd": ((6, 86), BC_DIR),
    "195_odd": ((26, 30), BC_NEU),
}


@pytest.mark.parametrize("name", list(BOTTOMS))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bottom_split_matches_oracle(cuda_lib, name, precision):
    n, top = BOTTOMS[name]
    dm = len(n)
    c = make_case(name=name, dm=dm, n=n, box=n, H_frac=0.25, noise=0.02, kmax=1, seed=41)
    c.dx = (1.0 / max(n),) * dm
    c.bc_lo = (BC_PER,) * (dm - 1) + (BC_NEU,)
    c.bc_hi = (BC_PER,) * (dm - 1) + (top,)
    u_o, phi_o, st_o = O.macproject(c.umac, c.phi0, c.rho, c.dx, c.bc_lo, c.bc_hi,
                                    macrhs=c.macrhs, beta0=c.beta0, beta0_edge=c.beta0_edge,
                                    nlevels=2, rel_eps=1e-12)
    assert st_o["status"] == 0
    got = [gpu_project(c, precision, rel_eps=1e-12, max_levels=2, inner_exact_bottom=0, coarse_tail=t)
           for t in (1, 0)]
    for u, phi, st in got:
        assert st["status"] == 0 and st["nlevels"] == 2 and st["bottom_iters"] > 0
        if precision == "fp64":
            # both bottoms are solved to 1e-3: the contraction is that of the two-level cycle
            assert abs(st["vcycles"] - st_o["vcycles"]) <= 1
        # conditioning below 1e3 under rel_eps = 1e-12
        assert phi_rel_err(phi, phi_o, top != BC_DIR) <= 1e-9
        assert u_rel_err(u, u_o) <= 1e-9
    np.testing.assert_array_equal(got[0][1], got[1][1])


@pytest.fixture(scope="module")
def bottom_check(cuda_lib, tmp_path_factory):
    """tests/csrc/bottom_check.cu, linked with the library."""
    B = importlib.import_module("maestro_gb300.build")
    exe = str(tmp_path_factory.mktemp("bottom") / "bottom_check")
    lib = os.path.dirname(B.LIB)
    cmd = [B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "-I", os.path.join(B.ROOT, "include"), "-I", B.CSRC,
           os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc", "bottom_check.cu"),
           B.LIB, "-Xlinker", "-rpath", "-Xlinker", lib, "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return exe


# cells, dimensions, Dirichlet top, periodic vertical: edges of the split over CTAs and colours
SOLVES = [((4, 4, 4), 3, 0, 0), ((3, 7, 3), 3, 1, 0), ((5, 13, 1), 2, 0, 0), ((5, 5, 5), 3, 0, 0),
          ((127, 1, 1), 2, 1, 0), ((8, 16, 1), 2, 0, 1), ((3, 43, 1), 2, 1, 0), ((10, 10, 10), 3, 0, 0),
          ((9, 7, 13), 3, 0, 1), ((25, 325, 1), 2, 1, 0), ((32, 16, 16), 3, 0, 0)]


@pytest.mark.parametrize("n,dm,top,per", SOLVES)
def test_cluster_bottom_matches_the_one_cta_solver(bottom_check, n, dm, top, per):
    r = subprocess.run([bottom_check, *map(str, (*n, dm, top, per, 3))], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    w = r.stdout.split()
    its, res, dist = [int(v) for v in w[1:3]], [float(v) for v in w[4:7]], [float(v) for v in w[8:10]]
    # both reduce the residual left by the first sweeps by 1e-10 (the recursive residual may part from
    # the true one by two decades); a condition number of 1e4, for 25 x 325 cells 1e5, separates the
    # solutions
    assert max(res) <= 1e-8, r.stdout
    assert max(dist) <= (1e-3 if max(n) > 128 else 1e-4), r.stdout
    assert its[0] > 0 and its[1] > 0
    if not per and all(v % 2 == 0 for v in n[:dm - 1]):
        # no cells of one colour side by side: the same iteration up to the order of its sums
        assert abs(its[0] - its[1]) <= 3 + its[0] // 5, r.stdout


@pytest.mark.parametrize("n,box", [((25, 325), (25, 325)), ((45, 90), (45, 45)), ((9, 7, 6), (9, 7, 6))])
def test_one_level_contexts_are_refused(cuda_lib, n, box):
    # the cluster's bottom solver relies on it: a bottom always starts from a zero correction
    with pytest.raises(MacError) as e:
        MacProjector(Layout.tiled(n, box), (1.0 / max(n),) * len(n),
                     BcTower((BC_PER,) * len(n), (BC_PER,) * len(n)))
    assert e.value.code == capi.MAC_ERR_UNSUPPORTED
