"""Bottoms of the cell-centred V-cycle where the solver's split changes: 65 to 128 cells belong to one CTA of
the cluster, more are spread over all of them (64 and fewer have an inverse, switched off here)."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER, make_case
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
