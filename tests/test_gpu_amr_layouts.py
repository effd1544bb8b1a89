"""Multi-level projection on the GPU against the oracle on layouts the fixtures leave out: planes of several
blocks, levels that cover their whole parent (no reflux), thin planes, boxes at corners and across the
periodic wrap (the layouts whose cell functions tests/test_amr_planes.py checks on the host)."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_DIR, BC_NEU, BC_PER, cell_to_edge
from tests.test_amr_planes import LAYOUTS
from tests.test_oracle_amr import G, phi_err, u_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# two planes a thread, lists longer than a block on every SM (the other layouts: one plane, short lists)
LARGE = {"large": ((64, 56, 48), (BC_PER, BC_PER, BC_NEU), (BC_PER, BC_PER, BC_DIR),
                   [[((12, 12, 8), (115, 103, 87))]])}


def make_case(name):
    n0, lo, hi, fine = {**LAYOUTS, **LARGE}[name]
    dm, boxes = len(n0), [[]] + fine
    rng = np.random.default_rng(19)
    c = dict(n0=n0, dm=dm, nlev=len(boxes), boxes=boxes, bc_lo=lo, bc_hi=hi,
             dx0=tuple(1.0 / max(n0) for _ in n0), umac=[], phi=[], rho=[], macrhs=[], beta0=[], beta0_edge=[])
    for l in range(len(boxes)):
        n = tuple(v << l for v in n0)
        z = np.exp(-(np.arange(n[-1]) + 0.5) / n[-1])
        b0 = z ** 0.7
        c["beta0"].append(b0)
        c["beta0_edge"].append(cell_to_edge(b0))
        c["rho"].append(np.asfortranarray(z * np.exp(0.2 * rng.standard_normal(n))))
        c["macrhs"].append(np.asfortranarray(rng.standard_normal(n)))
        c["phi"].append(np.zeros(n, order="F"))
        u = []
        for d in range(dm):
            a = rng.standard_normal([v + (e == d) for e, v in enumerate(n)])
            first, last = [slice(None)] * dm, [slice(None)] * dm
            first[d], last[d] = 0, -1
            if lo[d] == O.BC_PER:
                a[tuple(last)] = a[tuple(first)]
            u.append(np.asfortranarray(a))
        c["umac"].append(u)
    return c


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", [*LAYOUTS, *LARGE])
def test_layouts_match_oracle(cuda_lib, name, precision):
    from tests.test_gpu_zz_amr import _run
    c = make_case(name)
    H = G.Hierarchy(c["n0"], c["dx0"], c["bc_lo"], c["bc_hi"], c["boxes"])
    eps = 1e-13 * 10 ** (c["nlev"] - 1)
    uo, po, so = O.macproject_ml(c["umac"], c["phi"], c["rho"], c["dx0"], c["bc_lo"], c["bc_hi"], c["boxes"],
                                 macrhs=c["macrhs"], beta0=c["beta0"], beta0_edge=c["beta0_edge"], rel_eps=eps)
    assert so["status"] == 0
    u, phi, st = _run(c, rel_eps=1e-13, precision=precision)
    assert st["status"] == 0 and st["rel_resid"] <= eps
    if precision == "fp64":
        assert abs(st["vcycles"] - so["vcycles"]) <= 1
    # conditioning of these grids (at most 128 cells a side) below 1e3 under eps <= 1e-11
    assert phi_err(H, phi, po) <= 1e-8
    assert u_err(H, u, uo) <= 1e-8
