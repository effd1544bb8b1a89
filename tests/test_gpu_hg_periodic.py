"""Nodal projection with every direction periodic on levels swept by tiles: the tiles that are staged
without folding must not reach the image slab above the last one, whose values the sweeps leave
stale (the solve then needs many times the cycles, or never converges)."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_PER

pytestmark = pytest.mark.gpu


# 72: the smallest extent of 3-D boxes with a tile off the faces.  (Bottoms of at most 640 unknowns, which
# are solved exactly.)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(72, 72, 16), (72, 104, 24), (112, 72, 24)])
def test_periodic_vertical_tiles(cuda_lib, n, precision):
    from tests.test_gpu_zz_hg import _run
    rng = np.random.default_rng(31)
    dx = tuple(1.0 / max(n) for _ in n)
    bc = (BC_PER,) * 3
    z = 1.5 + np.cos(2 * np.pi * (np.arange(n[2]) + 0.5) / n[2])
    unew = rng.standard_normal(n + (3,))
    gpi = rng.standard_normal(n + (3,))
    rho = z * np.exp(0.2 * rng.standard_normal(n))
    pi = np.zeros(tuple(v + 1 for v in n))
    u, g, p, st = _run(n, dx, bc, bc, O.HG_REGULAR, 0.01, unew, unew, gpi, rho, pi, rel_eps=O.EPS_HG,
                       precision=precision)
    assert st["status"] == 0 and st["rel_resid"] <= O.EPS_HG
    uo, go, po, pho, so = O.hgproject(unew, unew, gpi, rho, pi, dx, bc, bc, proj_type=O.HG_REGULAR,
                                      dt=0.01, rel_eps=O.EPS_HG)
    assert so["status"] == 0
    # the same V-cycle in FP64 (its bottom is solved exactly); mixed: steps of three FP32 cycles, one
    # step of slack
    assert st["vcycles"] <= so["vcycles"] + (1 if precision == "fp64" else 6)
    assert np.max(np.abs(u - uo)) <= 1e-9 * np.max(np.abs(uo))
    assert np.max(np.abs(g - go)) <= 1e-9 * np.max(np.abs(go))
