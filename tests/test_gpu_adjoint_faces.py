"""Kernels of the adjoint MAC projection at the edges of their tiles (32 columns x 64 rows of a
layer, 8 planes of the right-hand side), against numpy on the phi and nu that the call returns."""
import numpy as np
import pytest

import oracle as O
from maestro_gb300.inputs import BC_NEU, BC_PER, cell_to_edge, make_case
from maestro_gb300.macproject import BcTower, Layout, MacProjector

pytestmark = pytest.mark.gpu

CASES = {
    # odd tiles: one column and rows past the tile, planes that do not divide
    "ragged": ((64, 72, 28), (BC_PER, BC_PER, BC_NEU), 0),
    "walls": ((32, 64, 24), (BC_NEU, BC_PER, BC_NEU), 1),
    "small": ((4, 4, 4), (BC_PER, BC_NEU, BC_NEU), 0),
    "plane": ((260, 132), (BC_PER, BC_NEU), 1),
    "column": ((16, 40), (BC_NEU, BC_NEU), 0),
}


def layer(a, d, dm):
    return np.asarray(a).reshape([-1 if q == dm - 1 else 1 for q in range(dm)])


@pytest.mark.parametrize("name", sorted(CASES))
def test_adjoint_kernels_at_tile_edges(cuda_lib, name):
    torch = pytest.importorskip("torch")
    n, bc, alt = CASES[name]
    dm = len(n)
    c = make_case(dm=dm, n=n, box=n, H_frac=0.3, noise=0.02, kmax=2, seed=77, with_w=True)
    c.bc_lo = c.bc_hi = bc
    dev = torch.device("cuda", 0)

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(np.asarray(a).transpose())).to(dev)

    def back(x):
        return np.asfortranarray(x.cpu().numpy().transpose())

    u, w = [t(a) for a in c.umac], [t(a) for a in c.w]
    du = [torch.zeros_like(x) for x in u]
    rho, rhs = t(c.rho), t(c.macrhs)
    b0, b0e = torch.from_numpy(c.beta0).to(dev), torch.from_numpy(c.beta0_edge).to(dev)
    drinv, dmac, phi, db0 = (torch.zeros_like(x) for x in (rho, rho, rho, b0))
    P = MacProjector(Layout.tiled(c.n, c.box), c.dx, BcTower(c.bc_lo, c.bc_hi), precision="fp64",
                     rel_eps=1e-12, use_alt_energy_fix=alt,   # (the plane reaches 7e-13 at best)
                     stream=torch.cuda.current_stream().cuda_stream)
    try:
        st = P.adjoint_dense([x.data_ptr() for x in u], rho.data_ptr(), rhs.data_ptr(),
                             b0.data_ptr(), b0e.data_ptr(), [x.data_ptr() for x in w],
                             [x.data_ptr() for x in du], drinv.data_ptr(), db0.data_ptr(),
                             dmac.data_ptr(), phi.data_ptr())
        torch.cuda.synchronize()
        assert st["status"] == 0
        for a, b in zip(u, c.umac):   # the inputs are left alone
            np.testing.assert_array_equal(back(a), b)
    finally:
        P.close()
    nu, phi, p = back(dmac), back(phi), 1 + alt
    lam, lnu, dsig = np.zeros(n), np.zeros(n), np.zeros(n)
    sh, sv = np.zeros(n[-1]), np.zeros(n[-1] + 1)
    for d in range(dm):
        idx = 1.0 / c.dx[d]
        b = layer(c.beta0_edge if d == dm - 1 else c.beta0, d, dm)
        per = bc[d] == BC_PER

        def ends(a, lo, hi):   # cells below and above every face entry
            pad = [(int(q == d), int(q == d)) for q in range(dm)]
            e = np.pad(a, pad, mode="wrap" if (lo, hi) == (1, 1) else "constant")
            return (np.take(e, range(n[d] + 1), axis=d), np.take(e, range(1, n[d] + 2), axis=d))

        ra, rb = ends(c.rho, 1, 1)
        h = 2.0 / (ra + rb)
        face = np.ones(n[d] + 1)          # wall faces carry no coefficient
        once = np.ones(n[d] + 1)          # a periodic face once
        if per:
            once[-1] = 0.0
        else:
            face[[0, -1]] = 0.0
        shp = [-1 if q == d else 1 for q in range(dm)]
        h = h * face.reshape(shp)
        pa, pb = ends(phi, 1, 1)
        na, nb = ends(nu, 1, 1)
        gphi, gnu = (pb - pa) * idx * face.reshape(shp), (nb - na) * idx * face.reshape(shp)
        za, zb = ends(nu, 0, 0)
        dt = (zb - za) * idx
        ref = c.w[d] + b * dt
        # products of a few rounded factors: 1e-12 of the largest entry
        assert np.max(np.abs(back(du[d]) - ref)) <= 1e-12 * np.max(np.abs(ref))
        dbeta, dc = -gnu * gphi * once.reshape(shp), -c.w[d] * gphi
        dh = b ** p * dbeta + b ** (p - 1) * dc
        share = c.umac[d] * dt + p * b ** (p - 1) * h * dbeta + (p - 1) * h * dc
        tot = share.sum(axis=tuple(range(dm - 1)))
        if d == dm - 1:
            sv += tot
        else:
            sh += tot

        def cells(a):          # sum of each cell's two physical faces, entries of one face merged
            a = a.copy()
            if per:
                lo = np.take(a, [0], axis=d) + np.take(a, [n[d]], axis=d)
                a[tuple(slice(0, 1) if q == d else slice(None) for q in range(dm))] = lo
                a[tuple(slice(n[d], None) if q == d else slice(None) for q in range(dm))] = lo
            return np.take(a, range(n[d]), axis=d), np.take(a, range(1, n[d] + 1), axis=d)

        lo, hi = cells(dh * h * h)
        dsig += 0.5 * c.rho ** 2 * (lo + hi)
        lo, hi = cells(b ** (p - 1) * h * c.w[d] * idx)
        lam += hi - lo
        flux = b ** p * h * gnu * idx
        lnu -= np.diff(flux, axis=d)
    assert np.max(np.abs(back(drinv) - dsig)) <= 1e-11 * np.max(np.abs(dsig))
    # the solve stops at 1e-12 of |lambda|; nu is rounded to 1e-16 of itself under the operator
    assert np.max(np.abs(lnu - lam)) <= 1e-9 * np.max(np.abs(lam))
    jac = np.empty((n[-1] + 1, n[-1]))     # cell_to_edge is piecewise linear
    for k in range(n[-1]):
        e = c.beta0.copy()
        e[k] *= 1.0 + 1e-7
        jac[:, k] = (cell_to_edge(e) - c.beta0_edge) / (e[k] - c.beta0[k])
    ref = sh + jac.T @ sv
    scale = np.max(np.abs(sh)) + np.max(np.abs(sv))
    assert np.max(np.abs(db0.cpu().numpy() - ref)) <= 1e-7 * scale
