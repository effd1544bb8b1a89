"""Workloads of the projection library for timing: what a user's program calls, from the smallest
2-D solve to the largest 3-D one, through the public Python and C entry points.

A case is a plain dict; ``kind`` says which entry point it goes through:

* ``mac``      ``MacProjector.macproject_dense``: the MAC projection on whole-domain device arrays;
* ``boxes``    ``mac_macproject`` on per-box device fabs with ghost cells (the drop-in form);
* ``adjoint``  ``MacProjector.adjoint_dense``: forward and adjoint solve, all four gradients;
* ``heat``     ``mac_multigrid`` with alpha on per-box device fabs (implicit thermal diffusion);
* ``amr``      ``MacProjector.macproject_ml_dense``: two or three refinement levels;
* ``hg``       ``MacProjector.hgproject_dense``: the nodal projection.

The inputs are the stratified atmosphere of the library's own configurations: rho0 = 1e7
exp(-z / H), density noise, beta0 = rho0^(1/1.4), random Fourier edge velocities of 1e6 cm/s,
S - Sbar of 1e-3 /s; the horizontal directions are periodic, the vertical one has a slip wall below
and a slip wall or an outlet above.  Arrays are torch tensors indexed [z][y][x] (2-D: [z][x]),
which is the library's Fortran order.

Entry points that work in place get fresh inputs by one copy (and phi's zero guess with it), as the
advection step leaves new edge velocities before every projection.  In a closed domain phi is
determined up to a constant; its mean is taken out, as a program that stores or compares it does.
"""
import ctypes
import itertools
import math

import torch

from maestro_gb300 import capi
from maestro_gb300.macproject import BcTower, Layout, MacProjector

PER, DIR, NEU = capi.MAC_BC_PER, capi.MAC_BC_DIR, capi.MAC_BC_NEU
DEV = "cuda"


def listed():
    return [
        # the smallest production solve: 2-D, one box; launches and host round trips count
        dict(name="mac2d_128_fp64", kind="mac", n0=128, n1=128, n2=0, box=128, precision="fp64",
             H=0.25, noise=0.01, kmax=8, top="wall", alt=0),
        # a small 3-D solve in 32^3 boxes: every level is small
        dict(name="mac3d_64_mixed", kind="mac", n0=64, n1=64, n2=64, box=32, precision="mixed",
             H=0.25, noise=0.01, kmax=8, top="wall", alt=0),
        # the plain FP64 drop-in at the production size
        dict(name="mac3d_256_fp64", kind="mac", n0=256, n1=256, n2=256, box=128, precision="fp64",
             H=0.25, noise=0.01, kmax=16, top="wall", alt=0),
        # the headline: the mixed-precision solve at the same size
        dict(name="mac3d_256_mixed", kind="mac", n0=256, n1=256, n2=256, box=128,
             precision="mixed", H=0.25, noise=0.01, kmax=16, top="wall", alt=0),
        # the stiff stratification (density contrast 1e6, 5% noise)
        dict(name="mac3d_384_stiff_mixed", kind="mac", n0=384, n1=384, n2=384, box=128,
             precision="mixed", H=0.072, noise=0.05, kmax=16, top="wall", alt=0),
        # the largest one-level solve
        dict(name="mac3d_512_mixed", kind="mac", n0=512, n1=512, n2=512, box=128,
             precision="mixed", H=0.15, noise=0.01, kmax=32, top="wall", alt=0),
        # gradients through the projection, FP64 forward and adjoint
        dict(name="adjoint3d_256_fp64", kind="adjoint", n0=256, n1=256, n2=256, box=128,
             precision="fp64", H=0.25, noise=0.01, kmax=16, top="wall", alt=0),
        # the boxed call on a domain of unequal, uneven extents with an outlet above
        dict(name="boxes3d_ragged_fp64", kind="boxes", n0=160, n1=96, n2=112, box=0,
             precision="fp64", H=0.25, noise=0.01, kmax=8, top="outlet", alt=0),
        # implicit thermal diffusion: the Helmholtz form, started from the old field
        dict(name="heat3d_128_mixed", kind="heat", n0=128, n1=128, n2=128, box=64,
             precision="mixed", H=0.25, noise=0.05, kmax=8, top="wall", alt=0),
        # two levels: a 128^3 base with a patch refined twice in its middle
        dict(name="amr3d_128_mixed", kind="amr", n0=128, n1=128, n2=128, box=64, levels=2,
             precision="mixed", H=0.25, noise=0.05, kmax=4, top="wall", alt=0),
        # the nodal projection of a regular time step at the production size
        dict(name="hg3d_256_mixed", kind="hg", n0=256, n1=256, n2=256, box=128, proj=4, dense=1,
             precision="mixed", H=0.25, noise=0.01, kmax=8, top="wall", alt=0),
        # a pressure iteration with a nodal source on a smaller uneven domain, FP64
        dict(name="hg3d_ragged_fp64", kind="hg", n0=96, n1=80, n2=64, box=0, proj=3, dense=1,
             precision="fp64", H=0.25, noise=0.05, kmax=8, top="outlet", alt=0),
    ]


# edge range (cells per direction, 3-D and 2-D) of each kind and how often it is drawn
_DRAWN = {
    "mac": (0.40, (24, 300), (64, 1000)),
    "boxes": (0.15, (24, 200), (64, 800)),
    "adjoint": (0.10, (24, 220), (64, 600)),
    "heat": (0.10, (24, 200), (64, 800)),
    "amr": (0.10, (24, 110), (32, 300)),
    "hg": (0.15, (24, 220), (64, 600)),
}


def draw(rng):
    """Extents m 2^t with m of 3 to 8 a direction (every level but the coarsest has to be even):
    the coarsest level is what box sizes with few factors of two leave."""
    kind = rng.choices(list(_DRAWN), weights=[v[0] for v in _DRAWN.values()])[0]
    dm = 2 if rng.random() < 0.25 else 3
    lo, hi = _DRAWN[kind][1 if dm == 3 else 2]
    edge = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    t = max(2, round(math.log2(edge / 5.0)))
    n = [max(3, min(8, round(edge / 2 ** t * rng.uniform(0.75, 1.3)))) << t for _ in range(dm)]
    H, noise = rng.choice([(0.25, 0.01), (0.25, 0.05), (0.15, 0.01), (0.15, 0.05)])
    c = dict(kind=kind, n0=n[0], n1=n[1], n2=n[2] if dm == 3 else 0,
             box=rng.choice([0, 1]), precision=rng.choice(["fp64", "mixed"]), H=H, noise=noise,
             kmax=rng.choice([4, 8, 12]), top=rng.choice(["wall", "wall", "outlet"]),
             alt=rng.choice([0, 0, 1]))
    if kind in ("adjoint", "amr"):
        c["top"] = "wall"
    if kind in ("boxes", "heat"):
        c["alt"] = 0
        if kind == "boxes":
            c["top"] = "outlet"
    if kind == "amr":
        c["levels"] = rng.choice([2, 2, 3]) if edge < 60 else 2
    if kind == "hg":
        c["proj"] = rng.choice([1, 3, 4, 4])
        c["dense"] = rng.choice([1, 1, 0])
    return c


# ---- shapes ------------------------------------------------------------------------------------

def _n(case):
    return tuple(case[k] for k in ("n0", "n1", "n2") if case[k])


def _shape(n, face=None, nodes=False):
    """Tensor shape of a cell, face or node array: the directions in reverse."""
    return tuple(v + (1 if nodes or d == face else 0) for d, v in reversed(list(enumerate(n))))


def _axis(n, d):
    return len(n) - 1 - d


def _boxes(case):
    """`box` cells a side; 1: one box; 0: two boxes along every direction a multiple of 8 long."""
    n, box = _n(case), case["box"]
    return Layout.tiled(n, [box if box > 1 else v // 2 if box == 0 and v % 8 == 0 else v
                            for v in n])


def _dx(n):
    return tuple(1.0 / v for v in n)


def _bc(case):
    dm = len(_n(case))
    hi = DIR if case["top"] == "outlet" else NEU
    return BcTower((PER,) * (dm - 1) + (NEU,), (PER,) * (dm - 1) + (hi,))


def _projector(case):
    n = _n(case)
    return MacProjector(_boxes(case), _dx(n), _bc(case), precision=case["precision"],
                        stream=torch.cuda.current_stream().cuda_stream,
                        use_alt_energy_fix=case["alt"])


# ---- inputs --------------------------------------------------------------------------------------

def _gen(seed, k):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + k)


def _randn(g, shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _column(a, dm):
    return a.reshape((-1,) + (1,) * (dm - 1))


def _rho0(n, H):
    nz = n[-1]
    z = (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5) / nz
    return 1e7 * torch.exp(-z / H)


def _edges(c):
    """beta0 on the vertical faces: copies at the ends, means one cell in, else the limited
    fourth-order value (MAESTRO's cell_to_edge)."""
    a, b = c[1:], c[:-1]
    e = torch.cat([c[:1], 0.5 * (a + b), c[-1:]])
    if c.numel() > 3:
        t = 7.0 / 12.0 * (a[1:-1] + b[1:-1]) - 1.0 / 12.0 * (c[3:] + c[:-3])
        t = torch.minimum(torch.maximum(t, torch.minimum(a, b)[1:-1]),
                          torch.maximum(a, b)[1:-1])
        e = torch.cat([e[:2], t, e[-2:]])
    return e


def _fourier(g, n, kmax, face=None, amp=1.0):
    """A random real field of modes |k| <= kmax with maximum `amp` (None: as it comes), on faces
    of direction `face` or cells; the wall-normal component vanishes on the walls."""
    dm = len(n)
    kh = torch.arange(-kmax, kmax + 1, device=DEV, dtype=torch.float64)
    kv = torch.arange(0, kmax + 1, device=DEV, dtype=torch.float64)
    ks = [kv] + [kh] * (dm - 1)                      # vertical first, as the tensors are
    r2 = sum(k.reshape([-1 if e == a else 1 for e in range(dm)]) ** 2 for a, k in enumerate(ks))
    C = torch.complex(_randn(g, r2.shape), _randn(g, r2.shape))
    C = torch.where((r2 <= kmax * kmax) & (r2 > 0), C, 0).to(torch.complex64)
    out = C
    for a in range(dm):
        d = dm - 1 - a
        m = n[d] + (1 if face == d else 0)
        x = (torch.arange(m, device=DEV, dtype=torch.float64) + (0.0 if face == d else 0.5)) / n[d]
        ph = torch.outer(ks[a], x)
        if a == 0:
            B = (torch.sin(math.pi * ph) if face == d else torch.cos(math.pi * ph)) + 0j
        else:
            B = torch.polar(torch.ones_like(ph), 2 * math.pi * ph)
        out = torch.tensordot(out, B.to(torch.complex64), dims=([0], [0]))
    u = out.real.to(torch.float64).contiguous()
    return u if amp is None else u * (amp / u.abs().max())


def _atmosphere(case, seed):
    n = _n(case)
    dm = len(n)
    rho0 = _rho0(n, case["H"])
    rho = _column(rho0, dm) * torch.exp(case["noise"] * _randn(_gen(seed, 0), _shape(n)))
    beta0 = rho0 ** (1.0 / 1.4)
    kmax = max(2, min(case["kmax"], min(n) // 4))
    u = [_fourier(_gen(seed, 1 + d), n, kmax, face=d, amp=1e6) for d in range(dm)]
    s = 1e-3 * _randn(_gen(seed, 8), _shape(n))
    s = s - s.mean(dim=tuple(range(1, dm)), keepdim=True)
    return dict(rho=rho, beta0=beta0, beta0e=_edges(beta0), u=u, rhs=_column(beta0, dm) * s)


class _Flat:
    """Several arrays in one buffer (each on a 256-byte boundary): filled again by one copy."""

    def __init__(self, arrays):
        at, places = 0, []
        for a in arrays:
            places.append(at)
            at += -(-a.numel() // 32) * 32
        self.src = torch.zeros(at, device=DEV, dtype=torch.float64)
        for a, p in zip(arrays, places):
            self.src[p:p + a.numel()] = a.reshape(-1)
        self.buf = torch.empty_like(self.src)
        self.views = [self.buf[p:p + a.numel()].view(a.shape) for a, p in zip(arrays, places)]
        self.ptrs = [v.data_ptr() for v in self.views]

    def fill(self):
        self.buf.copy_(self.src)


# ---- per-box fabs ------------------------------------------------------------------------------

def _fab_index(case, box, ng, face):
    """Per direction: the global indices of a fab's entries and whether they are beyond a wall."""
    n = _n(case)
    lo, hi = box
    idx, out = [], []
    for d in range(len(n)):
        ext = 1 if d == face else 0
        r = torch.arange(lo[d] - ng, hi[d] + 1 + ext + ng, device=DEV)
        lim = n[d] + ext
        if d < len(n) - 1:
            r = torch.where(r < 0, r + n[d], r)
            r = torch.where(r >= lim, r - n[d], r)
            out.append(torch.zeros_like(r, dtype=torch.bool))
        else:
            out.append((r < 0) | (r >= lim))
            r = r.clamp(0, lim - 1)
        idx.append(r)
    return idx, out


def _fabs(case, a, ng, face=None):
    got = []
    for box in _boxes(case).boxes:
        idx, _ = _fab_index(case, box, ng, face)
        f = a
        for d, r in enumerate(idx):
            f = f.index_select(_axis(idx, d), r)
        got.append(f.contiguous())
    return got


def _table(ptrs):
    P = ctypes.POINTER(ctypes.c_double)
    return (P * len(ptrs))(*[ctypes.cast(ctypes.c_void_p(p), P) for p in ptrs])


def _dp(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def _heat(case, seed):
    """alpha = rho, beta = rho D on the faces with D dt / h^2 = 5 for the finest spacing, rh =
    alpha x the old field, which is the first guess."""
    n = _n(case)
    dm = len(n)
    a = _atmosphere(case, seed)
    rho = a["rho"]
    D = 5.0 * min(_dx(n)) ** 2
    beta = []
    for d in range(dm):
        lo, hi, _ = _sides(case, rho, d)
        beta.append(D * 0.5 * (lo + hi))
    old = 1e9 * (_column(a["beta0"], dm) / a["beta0"][0] + 0.1 * _fourier(_gen(seed, 9), n, 4)
                 + 0.01 * _randn(_gen(seed, 10), _shape(n)))
    return dict(alpha=rho, beta=beta, rh=rho * old, old=old)


# ---- preparation -----------------------------------------------------------------------------

class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.kind = case, case["kind"]
    s.closed = case["top"] == "wall"
    n = _n(case)
    dm = len(n)
    s.P = _projector(case)
    if s.kind in ("mac", "adjoint"):
        a = _atmosphere(case, seed)
        s.rho, s.rhs, s.beta0, s.beta0e = a["rho"], a["rhs"], a["beta0"], a["beta0e"]
        if s.kind == "mac":
            s.flat = _Flat(a["u"] + [torch.zeros(_shape(n), device=DEV, dtype=torch.float64)])
            s.phi = torch.empty(_shape(n), device=DEV, dtype=torch.float64)
        else:
            s.u = a["u"]
            s.w = [_randn(_gen(seed, 20 + d), _shape(n, face=d)) for d in range(dm)]
            s.du = [torch.empty_like(x) for x in s.u]
            s.drinv, s.dmacrhs = torch.empty_like(s.rho), torch.empty_like(s.rho)
            s.dbeta0 = torch.empty_like(s.beta0)
    elif s.kind == "boxes":
        a = _atmosphere(case, seed)
        zero = torch.zeros(_shape(n), device=DEV, dtype=torch.float64)
        fu = [f for d in range(dm) for f in _fabs(case, a["u"][d], 1, face=d)]
        s.flat = _Flat(fu + _fabs(case, zero, 1))
        s.keep = [_fabs(case, a["rho"], 1), _fabs(case, a["rhs"], 0), a["beta0"], a["beta0e"]]
        s.tu, s.tphi = _table(s.flat.ptrs[:len(fu)]), _table(s.flat.ptrs[len(fu):])
        s.trho, s.trhs = (_table([f.data_ptr() for f in k]) for k in s.keep[:2])
        s.nu = len(fu)
    elif s.kind == "heat":
        h = _heat(case, seed)
        s.flat = _Flat(_fabs(case, h["old"], 1))
        s.keep = [_fabs(case, h["rh"], 0), _fabs(case, h["alpha"], 1),
                  [f for d in range(dm) for f in _fabs(case, h["beta"][d], 1, face=d)]]
        s.trh, s.talpha, s.tbeta = (_table([f.data_ptr() for f in k]) for k in s.keep)
        s.tphi = _table(s.flat.ptrs)
    elif s.kind == "amr":
        _prepare_amr(s, case, seed)
    else:
        f = _nodal(case, seed)
        s.flat = _Flat([f["unew"], f["gpi"], f["pi"]])
        s.f = f
        s.pi = torch.empty_like(f["pi"])
    return s


def _amr_boxes(case):
    """Level l refines the middle half of level l - 1's patch (cells of level l, aligned to 4)."""
    n = _n(case)
    lo, hi = [0] * len(n), list(n)
    got = [[]]
    for l in range(1, case["levels"]):
        w = [b - a for a, b in zip(lo, hi)]
        lo = [2 * (a + max(2, v // 4 // 2 * 2)) for a, v in zip(lo, w)]
        hi = [2 * (b - max(2, v // 4 // 2 * 2)) for b, v in zip(hi, w)]
        got.append([(tuple(lo), tuple(b - 1 for b in hi))])
    return got


def _waves(g, n, kmax):
    """A smooth field of the unit cube sampled at this level's cells: 16 cosine products."""
    dm = len(n)
    k = torch.randint(-kmax, kmax + 1, (16, dm), generator=g, device=DEV).double()
    ph = torch.rand((16, dm), generator=g, device=DEV, dtype=torch.float64) * 2 * math.pi
    amp = _randn(g, (16,)) / (1 + (k * k).sum(1))
    out = 0
    for m in range(16):
        t = amp[m]
        for d in range(dm):
            x = (torch.arange(n[d], device=DEV, dtype=torch.float64) + 0.5) / n[d]
            w = torch.cos((math.pi if d == dm - 1 else 2 * math.pi) * k[m, d] * x + ph[m, d])
            t = t * w.reshape([-1 if e == _axis(n, d) else 1 for e in range(dm)])
        out = out + t
    return out / out.abs().max()


def _prepare_amr(s, case, seed):
    n0 = _n(case)
    dm = len(n0)
    boxes = _amr_boxes(case)
    s.P.set_amr(boxes)
    nl = len(boxes)
    s.rho, s.rhs, s.beta0, s.beta0e, u, phi = [], [], [], [], [], []
    for l in range(nl):
        n = tuple(v << l for v in n0)
        rho0 = _rho0(n, case["H"])
        s.rho.append((_column(rho0, dm) * torch.exp(case["noise"] * _waves(_gen(seed, 0), n, 4)))
                     .contiguous())
        b = rho0 ** (1.0 / 1.4)
        s.beta0.append(b)
        s.beta0e.append(_edges(b))
        kmax = max(2, min(case["kmax"], min(n0) // 4))
        u.append([_fourier(_gen(seed, 1 + d), n, kmax, face=d, amp=None) for d in range(dm)])
        S = 1e-3 * _waves(_gen(seed, 8), n, 4)
        S = S - S.mean(dim=tuple(range(1, dm)), keepdim=True)
        s.rhs.append((_column(b, dm) * S).contiguous())
        phi.append(torch.zeros(_shape(n), device=DEV, dtype=torch.float64))
    top = [x.abs().max() for x in u[0]]              # every level samples the same field
    u = [[x * (1e6 / m) for x, m in zip(ul, top)] for ul in u]
    for l in range(nl - 1, 0, -1):      # the density of covered cells: the mean of their children
        r = s.rho[l]
        for a in range(dm):
            r = 0.5 * (r.index_select(a, torch.arange(0, r.shape[a], 2, device=DEV))
                       + r.index_select(a, torch.arange(1, r.shape[a], 2, device=DEV)))
        lo, hi = boxes[l][0]
        at = tuple(slice(lo[d] // 2, hi[d] // 2 + 1) for d in reversed(range(dm)))
        s.rho[l - 1][at] = r[at]
    s.flat = _Flat([x for ul in u for x in ul] + phi)
    v = s.flat.ptrs
    s.up = [v[l * dm:(l + 1) * dm] for l in range(nl)]
    s.pp = v[nl * dm:]
    s.views = s.flat.views
    s.phi = [torch.empty_like(p) for p in phi]
    s.nl, s.dm = nl, dm


def _nodal(case, seed):
    n = _n(case)
    dm = len(n)
    rho0 = _column(_rho0(n, case["H"]), dm)
    cells, nodes = _shape(n), _shape(n, nodes=True)
    rho = rho0 * torch.exp(case["noise"] * _randn(_gen(seed, 0), cells))
    smooth = [_fourier(_gen(seed, 1 + d), n, case["kmax"], amp=1e6) for d in range(dm)]
    unew = torch.stack(smooth) + 1e4 * _randn(_gen(seed, 5), (dm,) + cells)
    f = dict(rho=rho, unew=unew, beta0=(rho0 ** (1 / 1.4)).expand(cells).contiguous(),
             gpi=1e6 * rho * _randn(_gen(seed, 6), (dm,) + cells), dt=1e-3,
             pi=torch.zeros(nodes, device=DEV, dtype=torch.float64), uold=None, nodalrhs=None)
    if case["proj"] == 3:
        f["uold"] = unew - 1e3 * _randn(_gen(seed, 7), (dm,) + cells)
        src = torch.zeros(nodes, device=DEV, dtype=torch.float64)
        inner = tuple(slice(1, -1) for _ in n)       # away from the faces and their images
        src[inner] = 1e12 * _randn(_gen(seed, 8), src[inner].shape)
        f["nodalrhs"] = src
    return f


# ---- one pass ------------------------------------------------------------------------------------

def run(s):
    P, case = s.P, s.case
    if s.kind == "mac":
        s.flat.fill()
        *u, phi = s.flat.ptrs
        P.macproject_dense(u[0], u[1], u[2] if len(u) == 3 else 0, phi, s.rho.data_ptr(),
                           s.rhs.data_ptr(), s.beta0.data_ptr(), s.beta0e.data_ptr(), strict=True)
        *u, phi = s.flat.views
        if s.closed:
            phi = torch.sub(phi, phi.mean(), out=s.phi)
        return {"u": u, "phi": phi}
    if s.kind == "adjoint":
        p = lambda v: [x.data_ptr() for x in v]  # noqa: E731
        P.adjoint_dense(p(s.u), s.rho.data_ptr(), s.rhs.data_ptr(), s.beta0.data_ptr(),
                        s.beta0e.data_ptr(), p(s.w), p(s.du), s.drinv.data_ptr(),
                        s.dbeta0.data_ptr(), s.dmacrhs.data_ptr())
        return {"du": s.du, "drinv": s.drinv, "dbeta0": s.dbeta0, "dmacrhs": s.dmacrhs}
    if s.kind == "boxes":
        s.flat.fill()
        st = capi.MacStats()
        _ok(capi.lib().mac_macproject(P.ctx, capi.MAC_PTR_DEVICE, s.tu, 1, s.tphi, 1, s.trho, 1,
                                      1, 0, s.trhs, 0, _dp(s.keep[2]), _dp(s.keep[3]),
                                      ctypes.byref(st)))
        k = s.flat.views[s.nu].storage_offset()      # the velocity fabs, then phi's
        return {"u": s.flat.buf[:k], "phi": s.flat.buf[k:]}
    if s.kind == "heat":
        s.flat.fill()
        st = capi.MacStats()
        _ok(capi.lib().mac_multigrid(P.ctx, capi.MAC_PTR_DEVICE, s.trh, 0, s.tphi, 1, s.talpha,
                                     1, s.tbeta, 1, ctypes.byref(st)))
        return {"phi": s.flat.buf}
    if s.kind == "amr":
        s.flat.fill()
        q = lambda v: [x.data_ptr() for x in v]  # noqa: E731
        P.macproject_ml_dense(s.up, s.pp, q(s.rho), macrhs=q(s.rhs), beta0=q(s.beta0),
                              beta0_edge=q(s.beta0e), strict=True)
        phi = s.views[s.nl * s.dm:]
        mean = phi[0].mean()                         # covered cells hold their children's mean
        return {"u": s.views[:s.nl * s.dm],
                "phi": [torch.sub(p, mean, out=o) for p, o in zip(phi, s.phi)]}
    s.flat.fill()
    f, (unew, gpi, pi) = s.f, s.flat.views
    opt = lambda x: 0 if x is None else x.data_ptr()  # noqa: E731
    P.hgproject_dense(case["proj"], f["dt"], unew.data_ptr(), opt(f["uold"]), gpi.data_ptr(),
                      f["rho"].data_ptr(), pi.data_ptr(), beta0_cart=f["beta0"].data_ptr(),
                      nodalrhs=opt(f["nodalrhs"]), dense_stencil=bool(case["dense"]), strict=True)
    if s.closed and case["proj"] != 1:
        pi = torch.sub(pi, pi.mean(), out=s.pi)
    return {"u": unew, "gpi": gpi, "pi": pi}


def _ok(rc):
    if rc != capi.MAC_OK:
        raise capi.MacError(rc, "perf case")


def work(case):
    """Bytes: every input array read once, every output array written once.  Operations: the
    coefficients, right-hand side, one residual and the correction of each cell (a solver's
    iterations are its own choice)."""
    n = _n(case)
    dm, N = len(n), math.prod(n)
    kind = case["kind"]
    if kind == "amr":
        for l, b in enumerate(_amr_boxes(case)):
            N += sum(math.prod(y - x + 1 for x, y in zip(lo, hi)) for lo, hi in b)
    words = {"mac": 2 * dm + 4, "boxes": 2 * dm + 4, "amr": 2 * dm + 4, "adjoint": 3 * dm + 4,
             "heat": dm + 4, "hg": 4 * dm + 3}[kind]
    return {"bytes": 8.0 * words * N, "flops": (30.0 if dm == 2 else 50.0) * N}


# ---- 64-bit values -----------------------------------------------------------------------------
# Conjugate gradients, preconditioned by the exact inverse of the operator with horizontally
# averaged coefficients (Fourier transforms horizontally, a generalised eigenproblem vertically).

def _sides(case, a, d):
    """A cell array on either side of every face of direction d; wall faces get the cell's own
    value on both sides.  Also which faces are interior or periodic (else None: all)."""
    n = _n(case)
    ax = _axis(n, d)
    first, last = a.narrow(ax, 0, 1), a.narrow(ax, n[d] - 1, 1)
    if d < len(n) - 1:
        return torch.cat([last, a], ax), torch.cat([a, first], ax), None
    inner = torch.ones(n[d] + 1, device=DEV, dtype=torch.float64)
    inner[0] = inner[-1] = 0
    return torch.cat([first, a], ax), torch.cat([a, last], ax), _column(inner, len(n))


def _grad(case, phi, d):
    """Difference over h across every face of direction d: zero at a wall, the one-sided
    difference to phi = 0 on an outlet face."""
    n = _n(case)
    lo, hi, inner = _sides(case, phi, d)
    g = (hi - lo) * n[d]
    if inner is not None and case["top"] == "outlet":
        g[-1] = -2.0 * n[d] * phi[-1]
    return g


def _div(case, faces):
    n = _n(case)
    return sum(torch.diff(f, dim=_axis(n, d)) * n[d] for d, f in enumerate(faces))


def _layer(a):
    return a.mean(dim=tuple(range(1, a.dim())))


def _pcg(apply, solve, f, tol=1e-14):
    x, r = torch.zeros_like(f), f.clone()
    top = f.norm()
    z = solve(r)
    p, rz = z, (r * z).sum()
    best, stale = float("inf"), 0
    for _ in range(80):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        now = float(r.norm() / top)
        stale = 0 if now < 0.7 * best else stale + 1
        best = min(best, now)
        if now < tol or stale > 3:
            break
        z = solve(r)
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    r = f - apply(x)                                 # one step from the true residual
    return x + solve(r)


def _separable(lam, A, B):
    """Solves (A + lam B) x = f: A, B vertical (nz x nz, symmetric, B positive definite), lam the
    horizontal symbol (broadcast over the rfft of the horizontal axes)."""
    L = torch.linalg.cholesky(B)
    Li = torch.linalg.inv(L)
    w, V = torch.linalg.eigh(Li @ A @ Li.T)
    V = Li.T @ V
    inv = w.reshape((-1,) + (1,) * lam.dim()) + lam
    small = inv.abs() < 1e-9 * w.abs().max()
    inv = torch.where(small, 0.0, 1.0 / torch.where(small, 1.0, inv))

    def solve(f):
        dims = tuple(range(1, f.dim()))
        h = torch.view_as_real(torch.fft.rfftn(f, dim=dims))
        g = (V.T @ h.reshape(h.shape[0], -1)).reshape((V.shape[1],) + h.shape[1:])
        g = V @ (g * inv.unsqueeze(-1)).reshape(g.shape[0], -1)
        return torch.fft.irfftn(torch.view_as_complex(g.reshape(h.shape).contiguous()),
                                s=f.shape[1:], dim=dims)
    return solve


def _symbols(n):
    """2 - 2 cos(theta) of the horizontal directions on the rfft grid, in tensor order."""
    dm = len(n)
    got = []
    for d in reversed(range(dm - 1)):
        k = torch.arange(n[d] // 2 + 1 if d == 0 else n[d], device=DEV, dtype=torch.float64)
        s = 2 - 2 * torch.cos(2 * math.pi * k / n[d])
        got.append(s.reshape([-1 if e == dm - 2 - d else 1 for e in range(dm - 1)]))
    return got                                       # got[a]: direction dm - 2 - a


def _elliptic(case, beta, f, alpha=None):
    """(alpha - div beta grad) phi = f; the mean of a singular problem's f and phi removed."""
    n = _n(case)
    dm = len(n)
    sing = alpha is None and case["top"] == "wall"
    if sing:
        f = f - f.mean()

    def apply(x):
        y = -_div(case, [beta[d] * _grad(case, x, d) for d in range(dm)])
        return y if alpha is None else y + alpha * x
    bv = _layer(beta[dm - 1]) * n[-1] ** 2
    bv[0] = 0
    bv[-1] = 2 * bv[-1] if case["top"] == "outlet" else 0
    A = torch.diag(bv[:-1] + bv[1:]) - torch.diag(bv[1:-1], 1) - torch.diag(bv[1:-1], -1)
    if alpha is not None:
        A = A + torch.diag(_layer(alpha))
    bh = _layer(beta[0][..., :-1])
    lam = sum(s * n[d] ** 2 for s, d in zip(_symbols(n), reversed(range(dm - 1))))
    x = _pcg(apply, _separable(lam, A, torch.diag(bh)), f)
    return x - x.mean() if sing else x


def _face_beta0(case, a, d):
    dm = len(_n(case))
    return _column(a["beta0e"] if d == dm - 1 else a["beta0"], dm)


def _projection(case, a):
    """phi and the projected velocities."""
    n = _n(case)
    dm = len(n)
    p = 1 + case["alt"]
    beta, b0 = [], []
    for d in range(dm):
        lo, hi, _ = _sides(case, a["rho"], d)
        b0.append(_face_beta0(case, a, d))
        beta.append(b0[d] ** p * 2.0 / (lo + hi))
    f = a["rhs"] - _div(case, [b0[d] * a["u"][d] for d in range(dm)])
    phi = _elliptic(case, beta, f)
    u = [a["u"][d] - beta[d] / b0[d] * _grad(case, phi, d) for d in range(dm)]
    return phi, u


def _gradients(case, a, w):
    """dL/dU, dL/d(1/rho), dL/dbeta0 and dL/dmacrhs of L = sum(w U_proj): the derivative of
    L + nu (f - A phi) at fixed phi and nu, nu the adjoint solution."""
    n = _n(case)
    dm = len(n)
    p = 1 + case["alt"]
    phi, _ = _projection(case, a)
    rinv = (1.0 / a["rho"]).requires_grad_()
    beta0 = a["beta0"].clone().requires_grad_()
    u = [x.clone().requires_grad_() for x in a["u"]]
    rhs = a["rhs"].clone().requires_grad_()
    b = {"beta0": beta0, "beta0e": _edges(beta0)}
    loss, beta = 0, []
    for d in range(dm):
        lo, hi, _ = _sides(case, 1.0 / rinv, d)
        b0 = _face_beta0(case, b, d)
        beta.append(b0 ** p * 2.0 / (lo + hi))
        loss = loss + (w[d] * (u[d] - beta[d] / b0 * _grad(case, phi, d))).sum()
    x = torch.zeros_like(phi).requires_grad_()       # dL/dphi: linear in phi
    c = [(beta[d] / _face_beta0(case, b, d)).detach() for d in range(dm)]
    lam, = torch.autograd.grad(-sum((w[d] * c[d] * _grad(case, x, d)).sum() for d in range(dm)), x)
    nu = _elliptic(case, [t.detach() for t in beta], lam)
    flux = [_face_beta0(case, b, d) * u[d] - beta[d] * _grad(case, phi, d) for d in range(dm)]
    loss = loss + (nu * (rhs - _div(case, flux))).sum()
    return torch.autograd.grad(loss, u + [rinv, beta0, rhs])


def _cells_to_nodes(case, c):
    """Adds per-cell corner values (a dict by corner bits) onto the nodes; periodic images are one
    node (the last horizontal node is left out)."""
    n = _n(case)
    dm = len(n)
    out = 0
    for bits, v in c.items():
        for d in range(dm):
            ax = _axis(n, d)
            if d < dm - 1:
                v = torch.roll(v, 1, ax) if bits[d] else v
            else:
                z = torch.zeros_like(v[:1])
                v = torch.cat([z, v]) if bits[d] else torch.cat([v, z])
        out = out + v
    return out


def _corners(case, x):
    n = _n(case)
    dm = len(n)
    got = {(): x}
    for d in range(dm):
        ax = _axis(n, d)
        new = {}
        for bits, v in got.items():
            if d < dm - 1:
                new[bits + (0,)], new[bits + (1,)] = v, torch.roll(v, -1, ax)
            else:
                new[bits + (0,)], new[bits + (1,)] = v[:-1], v[1:]
        got = new
    return got


def _transform(c, dm, back=False):
    """Corner values to means and differences along every direction; back: its transpose."""
    for d in range(dm):
        new = {}
        for bits in c:
            if bits[d]:
                continue
            hi = bits[:d] + (1,) + bits[d + 1:]
            a, b = c[bits], c[hi]
            new[bits], new[hi] = (0.5 * a - b, 0.5 * a + b) if back else (0.5 * (a + b), b - a)
        c = new
    return c


def _nodal_exact(case, seed):
    f = _nodal(case, seed)
    n = _n(case)
    dm = len(n)
    out, proj, dt = case["top"] == "outlet", case["proj"], f["dt"]
    alt = case["alt"] and proj not in (1, 2)
    rho, b0 = f["rho"], f["beta0"]
    u = f["unew"]
    if proj == 3:
        u = (u - f["uold"]) / dt
    elif proj == 4:
        u = u + dt * f["gpi"] / rho
    sigma = b0 ** (2 if alt else 1) / rho
    third = 1.0 / 12.0 if case["dense"] else 0.25    # square of a difference in the 1-D mass
    weight = {}
    for bits in itertools.product((0, 1), repeat=dm):
        weight[bits] = sum(n[d] ** 2 * math.prod(third if bits[e] else 1.0
                                                 for e in range(dm) if e != d)
                           for d in range(dm) if bits[d])
    free = torch.ones(n[-1] + 1, device=DEV, dtype=torch.float64)
    if out:
        free[-1] = 0
    free = _column(free, dm)

    def apply(x):
        c = _transform(_corners(case, x), dm)
        c = {k: weight[k] * sigma * v for k, v in c.items()}
        return free * _cells_to_nodes(case, _transform(c, dm, back=True))
    bu = b0 * u
    rh = 0
    for d in range(dm):                              # every cell gives to its corners
        rh = rh + _cells_to_nodes(case, {
            bits: (-1.0 if bits[d] else 1.0) * n[d] * bu[d] / 2 ** (dm - 1)
            for bits in itertools.product((0, 1), repeat=dm)})
    if f["nodalrhs"] is not None:
        src = f["nodalrhs"]
        for d in range(dm - 1):
            src = src.narrow(_axis(n, d), 0, n[d])
        rh = rh - src
    rh = free * rh
    if not out:
        rh = rh - rh.mean()
    # horizontally averaged: symbols s n^2 of the stiffness, 1 - c s of the mass
    c = 1.0 / 6.0 if case["dense"] else 0.0
    ratio = sum(s * n[d] ** 2 / (1 - c * s) for s, d in zip(_symbols(n), reversed(range(dm - 1))))
    mass = math.prod(1 - c * s for s in _symbols(n))
    sl = _layer(sigma)
    z = torch.zeros(1, device=DEV, dtype=torch.float64)
    both = torch.cat([sl, z]) + torch.cat([z, sl])
    K = (torch.diag(both) - torch.diag(sl, 1) - torch.diag(sl, -1)) * n[-1] ** 2
    M = torch.diag(both) / 3 + (torch.diag(sl, 1) + torch.diag(sl, -1)) / 6 if case["dense"] \
        else torch.diag(both) / 2
    if out:
        K, M = K[:-1, :-1], M[:-1, :-1]
    inner = _separable(ratio, K, M)

    def solve(r):
        t = r[:-1] if out else r
        dims = tuple(range(1, t.dim()))
        t = torch.fft.irfftn(torch.fft.rfftn(t, dim=dims) / mass, s=t.shape[1:], dim=dims)
        t = inner(t)
        return torch.cat([t, torch.zeros_like(r[:1])]) if out else t
    phi = -_pcg(apply, solve, rh)
    if not out:
        phi = phi - phi.mean()
    corner = _transform(_corners(case, phi), dm)
    g = torch.stack([n[d] * corner[tuple(1 if e == d else 0 for e in range(dm))]
                     for d in range(dm)])
    if alt:
        g = b0 * g
    u = u - g / rho
    for d in range(dm - 1):                          # the images of the periodic nodes
        ax = _axis(n, d)
        phi = torch.cat([phi, phi.narrow(ax, 0, 1)], ax)
    if proj == 1:
        return {"u": u, "gpi": torch.zeros_like(g), "pi": torch.zeros_like(phi)}
    if proj == 3:
        u, g, pi = f["uold"] + dt * u, f["gpi"] + g, f["pi"] + phi
    else:
        g, pi = g / dt, phi / dt
    return {"u": u, "gpi": g, "pi": pi if out else pi - pi.mean()}


def exact(case, seed):
    kind = case["kind"]
    n = _n(case)
    dm = len(n)
    if kind == "amr":                                # no short 64-bit form of the composite solve
        return None
    if kind == "hg":
        return _nodal_exact(case, seed)
    if kind == "heat":
        h = _heat(case, seed)
        phi = _elliptic(case, h["beta"], h["rh"], alpha=h["alpha"])
        return {"phi": _boxed(case, [(None, h["old"], phi)])}
    a = _atmosphere(case, seed)
    if kind == "adjoint":
        w = [_randn(_gen(seed, 20 + d), _shape(n, face=d)) for d in range(dm)]
        g = _gradients(case, a, w)
        return {"du": list(g[:dm]), "drinv": g[dm], "dbeta0": g[dm + 1], "dmacrhs": g[dm + 2]}
    phi, u = _projection(case, a)
    if kind == "boxes":
        return {"u": _boxed(case, [(d, a["u"][d], u[d]) for d in range(dm)]),
                "phi": _boxed(case, [(None, torch.zeros_like(phi), phi)])}
    return {"u": u, "phi": phi}


def _boxed(case, fields):
    """The flat buffer of per-box fabs with one ghost layer: new values where the call writes
    them (the ghosts beyond a wall, and a cell field's ghosts, keep what the caller had)."""
    got = []
    for face, old, new in fields:
        for box, a, b in zip(_boxes(case).boxes, _fabs(case, old, 1, face),
                             _fabs(case, new, 1, face)):
            _, beyond = _fab_index(case, box, 1, face)
            keep = beyond[-1]
            got.append(torch.where(_column(keep, len(_n(case))), a, b))
    return _Flat(got).src
