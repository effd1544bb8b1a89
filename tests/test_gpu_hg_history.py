"""The nodal V-cycle's residual history against the oracle's, cycle by cycle: the cluster tail, the slabs and the
tiles keep the oracle's update order, so every cycle contracts by the same factor (another order of colours or
slabs converges as well, to the same answer, but not by the same steps)."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER

pytestmark = pytest.mark.gpu

SHAPES = {
    # name: (cells, low, high): the tail with one to three slabs a CTA, slabs and tiles above it
    "tail_16": ((16, 16, 16), (BC_PER, BC_PER, BC_NEU), (BC_PER, BC_PER, BC_NEU)),
    "tail_uneven": ((32, 16, 48), (BC_PER, BC_NEU, BC_NEU), (BC_PER, BC_DIR, BC_DIR)),
    "tail_walls": ((64, 32, 32), (BC_NEU, BC_NEU, BC_NEU), (BC_NEU, BC_NEU, BC_DIR)),
    "tail_periodic": ((32, 32, 64), (BC_PER, BC_PER, BC_PER), (BC_PER, BC_PER, BC_PER)),
    "tiles": ((96, 80, 32), (BC_PER, BC_NEU, BC_NEU), (BC_PER, BC_NEU, BC_DIR)),
}


@pytest.mark.parametrize("name", list(SHAPES))
def test_residual_history_matches_oracle(cuda_lib, name):
    from tests.test_gpu_zz_hg import _run
    n, lo, hi = SHAPES[name]
    rng = np.random.default_rng(37)
    dx = tuple(1.0 / max(n) for _ in n)
    unew = rng.standard_normal(n + (3,))
    gpi = rng.standard_normal(n + (3,))
    rho = np.exp(0.2 * rng.standard_normal(n))
    pi = np.zeros(tuple(v + 1 for v in n))
    *_, st = _run(n, dx, lo, hi, O.HG_REGULAR, 0.01, unew, unew, gpi, rho, pi, rel_eps=O.EPS_HG)
    *_, so = O.hgproject(unew, unew, gpi, rho, pi, dx, lo, hi, proj_type=O.HG_REGULAR, dt=0.01, rel_eps=O.EPS_HG)
    assert st["status"] == 0 and so["status"] == 0
    # the bottom (exact here, 60 sweeps there) leaves the first cycles equal to a part in a thousand
    k = 4
    a, b = np.array(st["hist"][:k]), np.array(so["hist"][:k])
    assert np.max(np.abs(a - b) / b) <= 1e-3, (a, b)
