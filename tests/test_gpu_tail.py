"""The cluster tail of the V-cycle (small levels and the bottom in one kernel) where its split can
go wrong: rows that do not divide over the CTAs, levels held by every CTA next to spread ones, one
and two pairs of cells a thread, 2-D levels, bottoms from a few cells to thousands, bottoms with odd
periodic extents (same-colour neighbours) and one too large for the cluster.

With the same bottom solver the tail runs the arithmetic of the per-level kernels, so the results
are bitwise those of coarse_tail = 0; both are within 1e-9 of the oracle, every solver driven to
1e-12 (the conditioning of these cases, below 1e3, leaves two orders of margin)."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER, make_case
from tests._util import phi_rel_err, u_rel_err
from tests.test_gpu_parity import gpu_project

pytestmark = pytest.mark.gpu

SHAPES = {
    # name: (cells, box, top face)
    "one_pair": ((32, 32, 32), (16, 16, 16), BC_NEU),
    "two_pairs": ((64, 64, 64), (32, 32, 32), BC_NEU),
    "flat_rows": ((64, 32, 16), (16, 16, 16), BC_DIR),
    "bottom_840": ((40, 24, 56), (20, 12, 28), BC_DIR),
    "bottom_315_odd": ((36, 20, 28), (36, 20, 28), BC_NEU),
    "bottom_3360": ((80, 48, 56), (10, 6, 14), BC_NEU),
    "bottom_13824": ((48, 48, 48), (4, 4, 4), BC_NEU),
    "2d_square": ((128, 128), (128, 128), BC_NEU),
    "2d_ragged": ((96, 40), (48, 20), BC_DIR),
    "2d_odd": ((72, 88), (72, 88), BC_NEU),
}


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tail_matches_levels_and_oracle(cuda_lib, name, precision):
    n, box, top = SHAPES[name]
    dm = len(n)
    c = make_case(name=name, dm=dm, n=n, box=box, H_frac=0.25, noise=0.02, kmax=4, seed=17)
    c.bc_lo = (BC_PER,) * (dm - 1) + (BC_NEU,)
    c.bc_hi = (BC_PER,) * (dm - 1) + (top,)
    u1, phi1, st1 = gpu_project(c, precision, rel_eps=1e-12, coarse_tail=1, inner_exact_bottom=0)
    u0, phi0, st0 = gpu_project(c, precision, rel_eps=1e-12, coarse_tail=0, inner_exact_bottom=0)
    assert st1["status"] == 0 and st0["status"] == 0
    np.testing.assert_array_equal(phi1, phi0)
    for a, b in zip(u1, u0):
        np.testing.assert_array_equal(a, b)
    u2, phi2, st2 = gpu_project(c, precision, rel_eps=1e-12)     # the default bottom
    assert st2["status"] == 0
    u_o, phi_o, st_o = O.macproject(c.umac, c.phi0, c.rho, c.dx, c.bc_lo, c.bc_hi,
                                    macrhs=c.macrhs, beta0=c.beta0, beta0_edge=c.beta0_edge,
                                    nlevels=O.nlevels_for_boxes([box]), rel_eps=1e-12)
    assert st_o["status"] == 0
    for u, phi in ((u1, phi1), (u2, phi2)):
        assert phi_rel_err(phi, phi_o, top != BC_DIR) <= 1e-9
        assert u_rel_err(u, u_o) <= 1e-9


NODAL = {
    # name: (cells, top face, precision): the cluster tail's slab split, the blocked inverse, and the
    # tiled levels (tiles off the faces, slab pairs of an odd number of slabs, restriction at faces)
    "two_slabs_a_cta": ((32, 32, 32), BC_NEU, "mixed"),      # 17 slabs over 16 CTAs: two a CTA
    "three_slabs_a_cta": ((64, 64, 64), BC_NEU, "mixed"),   # 33 slabs, isotropic
    "uneven_extents": ((24, 20, 36), BC_DIR, "fp64"),       # bottom 6 x 5 x 9: odd periodic extent
    "periodic_vertical": ((32, 16, 48), BC_PER, "fp64"),
    "bottom_one_block": ((16, 16, 16), BC_NEU, "fp64"),     # 12 unknowns: less than one block
    "bottom_576": ((32, 24, 44), BC_NEU, "mixed"),          # 8 x 6 x 12 nodes: 36 whole blocks
    "tiles_odd_slabs": ((96, 112, 32), BC_NEU, "mixed"),    # 33 slabs, tiles off the faces
    "tiles_periodic": ((96, 96, 48), BC_PER, "mixed"),
    "tiles_outflow": ((96, 80, 48), BC_DIR, "fp64"),
}


@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("name", list(NODAL))
def test_nodal_tail_and_bottom_match_oracle(cuda_lib, name, dense):
    from tests.test_gpu_zz_hg import _run
    n, top, precision = NODAL[name]
    rng = np.random.default_rng(29)
    dx = tuple(1.0 / v for v in n)
    lo, hi = (BC_PER, BC_PER, BC_NEU), (BC_PER, BC_PER, top)
    if top == BC_PER:
        lo = hi
    z = np.exp(-np.arange(n[2]) / n[2])
    unew = rng.standard_normal(n + (3,))
    gpi = rng.standard_normal(n + (3,))
    rho = z * np.exp(0.2 * rng.standard_normal(n))
    pi = np.zeros(tuple(v + 1 for v in n))
    u, g, p, st = _run(n, dx, lo, hi, O.HG_REGULAR, 0.01, unew, unew, gpi, rho, pi, dense=dense,
                       rel_eps=O.EPS_HG, precision=precision)
    assert st["status"] == 0 and st["rel_resid"] <= O.EPS_HG
    uo, go, po, pho, so = O.hgproject(unew, unew, gpi, rho, pi, dx, lo, hi, proj_type=O.HG_REGULAR,
                                      dt=0.01, dense=dense, rel_eps=O.EPS_HG)
    assert so["status"] == 0
    # eps_hg = 1e-12 on operators of contrast below 20: three orders under the 1e-9 bar
    assert np.max(np.abs(u - uo)) <= 1e-9 * np.max(np.abs(uo))
    assert np.max(np.abs(g - go)) <= 1e-9 * np.max(np.abs(go))


@pytest.mark.parametrize("n,top", [((128, 128, 128), BC_NEU), ((160, 128, 112), BC_DIR),
                                   ((192, 112, 128), BC_NEU)])
def test_finest_level_paths_match_oracle(cuda_lib, n, top):
    # 2^21 cells (one thread a cell) and just above it (staged planes, rows that are no power of
    # two, plane chunks that do not divide the extent)
    box = tuple(v // 2 for v in n)
    c = make_case(name="paths", dm=3, n=n, box=box, H_frac=0.25, noise=0.02, kmax=8, seed=23)
    c.bc_hi = (BC_PER, BC_PER, top)
    u, phi, st = gpu_project(c, "mixed", rel_eps=1e-12)
    assert st["status"] == 0 and st["rel_resid"] <= 1e-12
    u_o, phi_o, st_o = O.macproject(c.umac, c.phi0, c.rho, c.dx, c.bc_lo, c.bc_hi,
                                    macrhs=c.macrhs, beta0=c.beta0, beta0_edge=c.beta0_edge,
                                    nlevels=O.nlevels_for_boxes([box]), rel_eps=1e-12)
    assert st_o["status"] == 0
    assert phi_rel_err(phi, phi_o, top != BC_DIR) <= 1e-9
    assert u_rel_err(u, u_o) <= 1e-9
