"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one call chain through the public Python API on a handle that the
program already holds: give it an initial field, run the outer iteration (or
the transient steps, or the adjoint), read the fields back. The sizes are
those of this repository's own decks (``giftbte_b200.decks``): the gray
square, the 300 nm porous cell, the population of porous cells, the 3D
hotspot block and the thermal grating.

Kinds:
  steady     set_initial, ``iters`` outer iterations, all fields
  batch      the same for several geometries in one handle
  adjoint    gradient of k_eff at a converged state, ``iters`` transposed
             iterations
  transient  ``iters`` explicit steps, all fields and the probe's history

The handle (mesh, band table, quadrature, device buffers) is what such a
program builds once per geometry, so ``prepare`` builds it; every pass starts
from an initial field and ends with the fields in host memory. A program
that picks the FP32-mixed form keeps its fields in single precision.

``exact`` restates the solver in 64-bit torch, without the package's solver:
sparse stencils, the sweep level by level over all directions at once, and
conjugate gradients to rounding level for the macro system.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import giftbte_b200 as g
from giftbte_b200 import decks


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the quickstart deck: a gray square, one band. Launches and latency.
        dict(name="gray_square_f64", kind="steady", deck="square", n=40, bands=1, n_phi=8, prec=64, iters=20),
        # a coarse porous cell in the default FP64 form: the everyday call
        dict(name="porous_small_f64", kind="steady", deck="porous", h=8.0, bands=20, n_phi=8, prec=64, iters=20),
        # the 300 nm porous cell at its benchmark size, FP32-mixed
        dict(name="porous_f32", kind="steady", deck="porous", h=3.0, bands=40, n_phi=16, prec=32, iters=20),
        # the same cell in the plain FP64 form that replaces the reference
        dict(name="porous_f64", kind="steady", deck="porous", h=3.0, bands=40, n_phi=16, prec=64, iters=10),
        # a band count that no vector divides and an odd angular grid
        dict(name="porous_ragged_f32", kind="steady", deck="porous", h=5.3, bands=13, n_phi=7, prec=32, iters=10),
        # CONTROL Order=2limit, the limited gradient
        dict(name="porous_limited_f64", kind="steady", deck="porous", h=5.0, bands=20, n_phi=8, prec=64, iters=10,
             order="2limit"),
        # a sweep over structures: several porous cells in one handle
        dict(name="population_f32", kind="batch", n=6, h=5.0, bands=20, n_phi=8, prec=32, iters=10),
        # the 3D hotspot block: a coarse FP64 run, a mid-size and a large FP32 run
        dict(name="block_f64", kind="steady", deck="block", h=5.0, x=50.0, z=100.0, bands=40, n_theta=4, n_phi=4,
             prec=64, iters=5),
        dict(name="block_f32", kind="steady", deck="block", h=5.0, x=100.0, z=100.0, bands=40, n_theta=4, n_phi=4,
             prec=32, iters=8),
        dict(name="block_large_f32", kind="steady", deck="block", h=2.5, x=100.0, z=50.0, bands=40, n_theta=4,
             n_phi=4, prec=32, iters=6),
        # backward: the gradient of k_eff for an optimisation or a fit
        dict(name="adjoint_f64", kind="adjoint", h=5.0, bands=20, n_phi=8, prec=64, iters=40),
        # the explicit transient solver on a thermal grating
        dict(name="transient_f64", kind="transient", n=96, bands=20, n_phi=8, prec=64, iters=40),
    ]


def _spread(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["square", "porous", "porous", "porous", "block", "block", "batch", "adjoint", "transient"])
    bands = int(round(_spread(rng, 4, 44)))
    if rng.random() < 0.6:
        bands = max(4, bands // 4 * 4)
    prec = rng.choice([32, 64])
    iters = rng.randint(5, 12)
    h = round(_spread(rng, 3.5, 12.0), 2)
    n_phi = rng.randint(3, 14)
    if kind == "square":
        return dict(kind="steady", deck="square", n=rng.randint(9, 80), bands=rng.choice([1, bands]), n_phi=n_phi,
                    prec=prec, iters=iters)
    if kind == "porous":
        c = dict(kind="steady", deck="porous", h=h, bands=bands, n_phi=n_phi, prec=prec, iters=iters)
        option = rng.choice(["", "", "", "1", "2limit", "Sequential"])
        if option == "Sequential":
            c["scheme"] = option
        elif option and not (option == "2limit" and prec == 32):
            c["order"] = option
        return c
    if kind == "block":
        hb = rng.choice([4.0, 5.0, 6.25, 10.0])
        x = hb * rng.randint(4, max(5, int(60 / hb)))
        return dict(kind="steady", deck="block", h=hb, x=x, z=hb * rng.randint(max(5, int(30 / hb)), int(100 / hb)),
                    bands=bands, n_theta=rng.randint(2, 4), n_phi=rng.randint(2, 4), prec=prec, iters=rng.randint(3, 6))
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(2, 8), h=round(rng.uniform(5.0, 12.0), 2), bands=bands,
                    n_phi=rng.randint(3, 8), prec=prec, iters=iters)
    if kind == "adjoint":
        return dict(kind="adjoint", h=round(rng.uniform(6.0, 12.0), 2), bands=bands, n_phi=rng.randint(3, 8), prec=64,
                    iters=rng.randint(10, 40))
    return dict(kind="transient", n=4 * rng.randint(6, 30), bands=bands, n_phi=rng.randint(3, 10), prec=64,
                iters=rng.randint(10, 60))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _porous(h, bands, n_phi):
    return decks.config2_deck(h_nm=h, n_bands=bands, n_phi=n_phi)


@functools.lru_cache(maxsize=None)
def _population(n, h, bands, n_phi):
    return [decks.porous_population_member(i, h_nm=(h, 1.5 * h), n_bands=bands, n_phi=n_phi) for i in range(n)]


@functools.lru_cache(maxsize=None)
def _block(h, x, z, bands, n_theta, n_phi):
    return decks.config3_deck(h_nm=h, size_nm=(x, x, z), n_bands=bands, n_theta=n_theta, n_phi=n_phi)


@functools.lru_cache(maxsize=None)
def _square(n, bands, n_phi):
    d = decks.config1_deck(n, n_phi=n_phi)
    if bands > 1:
        d.bands = decks.sine_dispersion_bands(bands)
    return d


def _decks(case):
    """The geometries of a case. A mesh is a file that a user has: it does
    not depend on the seed, and each is made once."""
    if case["kind"] == "batch":
        return _population(case["n"], case["h"], case["bands"], case["n_phi"])
    if case["kind"] == "adjoint":
        return [_specular(case["h"], case["bands"], case["n_phi"])]
    if case["kind"] == "transient":
        return [_grating(case["n"], case["bands"], case["n_phi"])]
    if case["deck"] == "square":
        return [_square(case["n"], case["bands"], case["n_phi"])]
    if case["deck"] == "block":
        return [_block(case["h"], case["x"], case["z"], case["bands"], case["n_theta"], case["n_phi"])]
    return [_porous(case["h"], case["bands"], case["n_phi"])]


@functools.lru_cache(maxsize=None)
def _specular(h, bands, n_phi):
    return decks.config4_deck(h_nm=h, n_bands=bands, n_phi=n_phi)


@functools.lru_cache(maxsize=None)
def _grating(n, bands, n_phi):
    return decks.grating_deck(nx=n, ny=n // 4, n_bands=bands, n_phi=n_phi)


def _centres(deck):
    return deck.mesh.nodes[np.asarray(deck.mesh.cells)].mean(axis=1)


def _initial(deck, rng):
    """A guess of the temperature field: the deck's reference temperature and
    a few smooth modes, as an earlier solution of a neighbouring problem
    would give."""
    x = _centres(deck)
    x = (x - x.min(0)) / (x.max(0) - x.min(0))
    T = np.full(len(x), float(deck.tref))
    for _ in range(4):
        k = rng.integers(0, 4, x.shape[1])
        T += rng.normal(0.0, 0.1) * np.cos(2 * np.pi * (x @ k) + rng.uniform(0, 2 * np.pi))
    return T


def _options(case):
    o = {"precision": g.GBTE_FP32_MIXED if case["prec"] == 32 else g.GBTE_FP64}
    if case["prec"] == 64:
        o["macro_exact"] = 1  # the drop-in form: every macro solve exact, as the reference's LU
    order = case.get("order", "2")
    o["order"] = 1 if order == "1" else 2
    o["use_limiter"] = 1 if order == "2limit" else 0
    o["scheme"] = 1 if case.get("scheme") == "Sequential" else 0
    return o


def _scatter(deck, rng):
    return np.exp(rng.normal(0.0, 0.2, deck.mesh.n_cells))


def prepare(case, seed):
    ds = _decks(case)
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        o = _options(case)
        s = g.StaticBTESynthetic.from_decks(ds, **o)
        return {"case": case, "solver": s, "T0": np.concatenate([_initial(d, rng) for d in ds])}
    if case["kind"] == "adjoint":
        # a sample whose scattering is being fitted, at its converged state
        s = g.StaticBTESynthetic.from_deck(ds[0], precision=g.GBTE_FP64, cell_scatter=_scatter(ds[0], rng))
        s.solve(max_iter=2000, err_temp=1e-9, err_flux=1e-9)
        return {"case": case, "solver": s, "q_bar": s.keff_cotangent(axis=0, length=300e-9, delta_T=1.0)}
    if case["kind"] == "transient":
        s = g.StaticBTESynthetic.from_deck(ds[0], precision=g.GBTE_FP64, cell_scatter=_scatter(ds[0], rng))
        return {"case": case, "solver": s}
    s = g.StaticBTESynthetic.from_deck(ds[0], **_options(case))
    return {"case": case, "solver": s, "T0": _initial(ds[0], rng)}


def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "adjoint":
        r = s.vjp(q_bar=state["q_bar"], max_iter=case["iters"], tol=1e-300)
        return {"tau": r["tau"], "scatter": r["scatter"], "specularity": r["specularity"]}
    if case["kind"] == "transient":
        r = s.transient_solve(1e-13, case["iters"] * 1e-13)
        f = s.fields()
        return {"history": r["history"], "T": f["T"], "q": f["q"]}
    s.set_initial(state["T0"])
    s.solve(max_iter=case["iters"], err_temp=0.0, err_flux=0.0)
    f = s.fields()
    if case["prec"] == 32:
        return {k: v.astype(np.float32) for k, v in f.items()}
    return f


def _directions(case):
    return (8 * case["n_theta"] if "n_theta" in case else 4) * case["n_phi"]


def work(case):
    """Each outer iteration reads and writes every intensity once. The flops
    of an update: the least-squares gradient over the vertex neighbours, the
    second-order face values, the sweep and the ten angular moments."""
    ds = _decks(case)
    nc = sum(d.mesh.n_cells for d in ds)
    dim = ds[0].dimension
    updates = float(nc) * case["bands"] * _directions(case) * case["iters"]
    stencil = 0 if case.get("order") == "1" else (65 if dim == 3 else 12)
    flops = 2 * dim * stencil + 2 * (dim + 1) * (dim + 2) + 12 + 20
    passes = 2 if case["kind"] == "adjoint" else 1  # the transposed iteration and the change of its state
    return {"bytes": updates * 2 * passes * (case["prec"] // 8), "flops": updates * flops}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _angles(case):
    """Unit vectors and weights (summing to one) of the two quadratures."""
    n = case["n_phi"]
    if "n_theta" not in case:  # uniform midpoints in the plane
        phi = (np.arange(4 * n) + 0.5) * (0.5 * np.pi / n)
        return np.stack([np.cos(phi), np.sin(phi), 0 * phi], 1), np.full(4 * n, 1.0 / (4 * n))
    # Gauss-Legendre in cos(theta) on both hemispheres and in phi per quadrant
    x, w = np.polynomial.legendre.leggauss(case["n_theta"])
    mu, wmu = (x - 1) / 2, w / 2
    mu, wmu = np.concatenate([-mu, mu[::-1]]), np.concatenate([wmu, wmu[::-1]])
    x, w = np.polynomial.legendre.leggauss(n)
    ph, wph = (x + 1) * np.pi / 4, w * np.pi / 4
    c, s = np.cos(ph), np.sin(ph)
    cp = np.concatenate([c, -c[::-1], -c, c[::-1]])
    sp = np.concatenate([s, s[::-1], -s, -s[::-1]])
    wp = np.concatenate([wph, wph[::-1], wph, wph[::-1]])
    st = np.sqrt(1 - mu * mu)
    d = np.stack([np.outer(st, cp), np.outer(st, sp), np.outer(mu, np.ones_like(cp))], -1).reshape(-1, 3)
    return d, np.outer(wmu, wp).reshape(-1) / (4 * np.pi)


def _sparse(rows, cols, vals, shape, dev):
    m = torch.sparse_coo_tensor(torch.as_tensor(np.stack([rows, cols])), torch.as_tensor(vals), shape)
    return m.coalesce().to_sparse_csr().to(dev)


class _Exact:
    """One geometry of triangles or tetrahedra, one material."""

    def __init__(self, deck, case, dev):
        m = deck.mesh
        self.dev, self.case = dev, case
        dim = self.dim = deck.dimension
        scale = np.ones(3)
        scale[:dim] = deck.scale[:dim]
        X = np.zeros((len(m.nodes), 3))
        X[:, :dim] = m.nodes
        X *= scale
        Lx = deck.scale[0]
        cells = np.asarray(m.cells)
        nc, nv = cells.shape
        nn = len(X)
        self.nc, self.nn = nc, nn
        cen = X[cells].mean(1)
        # faces: opposite each vertex
        loc = [[(j + 1 + k) % nv for k in range(nv - 1)] for j in range(nv)]
        fv = cells[:, loc]  # [nc, nv, nv - 1]
        P = X[fv]
        fc = P.mean(2)
        if dim == 2:
            t = P[:, :, 1] - P[:, :, 0]
            area = np.linalg.norm(t, axis=2)
            nrm = np.stack([t[..., 1], -t[..., 0], 0 * area], -1) / area[..., None]
            a, b = X[cells[:, 1]] - X[cells[:, 0]], X[cells[:, 2]] - X[cells[:, 0]]
            vol = 0.5 * np.abs(a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0])
        else:
            cr = np.cross(P[:, :, 1] - P[:, :, 0], P[:, :, 2] - P[:, :, 0])
            l = np.linalg.norm(cr, axis=2)
            area, nrm = l / 2, cr / l[..., None]
            e = X[cells[:, 1:]] - X[cells[:, :1]]
            vol = np.abs(np.linalg.det(e)) / 6
        flip = np.einsum("cjk,cjk->cj", cen[:, None] - fc, nrm) > 0
        nrm[flip] *= -1
        # neighbours across faces and boundary elements, by their vertices
        key = np.sort(fv, 2).reshape(nc * nv, nv - 1)
        bkey = np.sort(np.asarray(m.edges), 1)
        uni, inv = np.unique(np.concatenate([key, bkey]), axis=0, return_inverse=True)
        inv = inv.reshape(-1)
        order = np.argsort(inv[:nc * nv], kind="stable")
        ks = inv[order]
        same = np.flatnonzero(ks[1:] == ks[:-1])
        nbr = np.full(nc * nv, -1)
        nbr[order[same]] = order[same + 1] // nv
        nbr[order[same + 1]] = order[same] // nv
        first = np.full(len(uni), -1)
        first[ks[::-1]] = order[::-1]
        side = first[inv[nc * nv:]]  # cell * nv + face of every boundary element
        tag = np.asarray(m.edge_tags)
        self.nb_ = len(side)
        bound = np.full(nc * nv, -1)
        bound[side] = np.arange(len(side))
        nbr, bound = nbr.reshape(nc, nv), bound.reshape(nc, nv)
        bc = {b.tag: b for b in deck.bcs}
        btype = np.array([bc[t].type for t in tag])
        bT = np.array([bc[t].value for t in tag], dtype=np.float64)
        bfc = fc.reshape(-1, 3)[side]
        connect = np.full(len(side), -1)
        for t in {t for t in tag if bc[t].type < 0}:
            mine, other = np.flatnonzero(tag == t), np.flatnonzero(tag == -bc[t].type)
            d = np.linalg.norm(bfc[mine][:, None] - bfc[other][None], axis=2)
            connect[mine] = other[d.argmin(1)]
        # vertex-neighbour least squares
        flat = cells.reshape(-1)
        by = np.argsort(flat, kind="stable")
        cnt = np.bincount(flat, minlength=nn)
        start = np.concatenate([[0], np.cumsum(cnt)])
        width = cnt.max()
        table = np.full((nn, width), -1)
        table[flat[by], np.arange(len(by)) - start[flat[by]]] = by // nv
        cand = table[cells].reshape(nc, -1)
        r, c = np.repeat(np.arange(nc), cand.shape[1]), cand.reshape(-1)
        keep = (c >= 0) & (c != r)
        pair = np.unique(r[keep].astype(np.int64) * nc + c[keep])
        r, c = pair // nc, pair % nc
        d = (cen[c] - cen[r])[:, :dim] / Lx
        M = np.zeros((nc, dim, dim))
        np.add.at(M, r, d[:, :, None] * d[:, None, :])
        ok = np.bincount(r, minlength=nc) > (2 if dim == 2 else 3)
        M[~ok] = np.eye(dim)
        w = np.einsum("pij,pj->pi", np.linalg.inv(M)[r], d) / Lx * ok[r][:, None]
        self.grad = [_sparse(np.concatenate([r, np.arange(nc)]), np.concatenate([c, np.arange(nc)]),
                             np.concatenate([w[:, k], -np.bincount(r, w[:, k], minlength=nc)]), (nc, nc), dev)
                     for k in range(dim)]
        # inverse-distance vertex values: of the cells, and of the cells or,
        # on walls, of the wall faces
        dist = np.linalg.norm(X[cells] - cen[:, None], axis=2)
        wc = 1 / dist.reshape(-1)
        cc = np.repeat(np.arange(nc), nv)
        tot = np.bincount(flat, wc, minlength=nn)
        self.vertT = _sparse(flat, cc, wc / tot[flat], (nn, nc), dev)
        bv = fv.reshape(nc * nv, nv - 1)[side]
        wb = 1 / np.linalg.norm(X[bv] - bfc[:, None], axis=2).reshape(-1)
        totb = np.bincount(bv.reshape(-1), wb, minlength=nn)
        inner = totb[flat] == 0
        self.vertc = _sparse(flat[inner], cc[inner], (wc / tot[flat])[inner], (nn, nc), dev)
        self.vertb = _sparse(bv.reshape(-1), np.repeat(np.arange(len(side)), nv - 1), wb / totb[bv.reshape(-1)],
                             (nn, len(side)), dev)

        def t_(v, dt=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(v), dtype=dt, device=dev)

        i_ = functools.partial(t_, dt=torch.int64)
        self.vol, self.area, self.nrm, self.fc, self.cen = t_(vol), t_(area), t_(nrm), t_(fc), t_(cen)
        self.nbr, self.bound, self.fv = i_(nbr), i_(bound), i_(fv)
        self.bcell, self.bnrm = i_(side // nv), t_(nrm.reshape(-1, 3)[side])
        self.boff = t_(bfc - cen[side // nv])
        self.btype, self.bT, self.connect = btype, t_(bT), i_(connect)
        self.connect_np = connect
        # face tangents: the in-plane gradient that the vertex values give
        p = X[fv]
        if dim == 2:
            mvec = p[:, :, 1] - p[:, :, 0]
            self.tang = t_(mvec / (mvec ** 2).sum(-1, keepdims=True))[:, :, None]  # times (phi1 - phi0)
        else:
            J = np.stack([nrm, p[:, :, 1] - p[:, :, 0], p[:, :, 2] - p[:, :, 1]], 2)
            self.tang = t_(np.swapaxes(np.linalg.inv(J), 2, 3)[:, :, 1:])  # [.., 2, 3] times the two differences
        B = deck.bands
        self.v, self.tau, self.C, self.lat, self.hr = (t_(getattr(B, k)) for k in
                                                       ("v", "tau", "C", "lattice_ratio", "heat_ratio"))
        self.kappa = float((self.C * self.v ** 2 * self.tau).sum() / deck.material_dim)
        heat = deck.cell_heat()
        self.heat = t_(heat if heat is not None else np.zeros(nc))
        s, w = _angles(case)
        self.s, self.w = t_(s), t_(w)
        self.nd, self.nb = len(s), len(B.v)
        # the macro system (negated: symmetric positive definite)
        wall = (bound >= 0)
        spec = wall & (btype[np.maximum(bound, 0)] == 3)
        a = np.where(wall[..., None], fc, cen[np.maximum(nbr, 0)]) - cen[:, None]
        coef = self.kappa * area / np.einsum("cjk,cjk->cj", nrm, a)
        coef[spec] = 0
        rr, jj = np.nonzero(~wall)
        self.K = _sparse(np.concatenate([rr, np.arange(nc)]), np.concatenate([nbr[rr, jj], np.arange(nc)]),
                         np.concatenate([-coef[rr, jj], coef.sum(1)]), (nc, nc), dev)
        self.Kd = t_(coef.sum(1))
        self.mcoef, self.spec, self.wall, self.a = t_(coef), t_(spec, torch.bool), t_(wall, torch.bool), t_(a)

    def levels(self):
        """Upwind levels of all directions at once; False where a direction has a cycle."""
        nd, nc, dev = self.nd, self.nc, self.dev
        nv = self.nbr.shape[1]
        sn = torch.einsum("dk,cjk->dcj", self.s, self.nrm)
        inflow = (sn < 0) & ~self.wall
        base = (torch.arange(nd, device=dev) * nc)[:, None, None]
        up = torch.where(inflow, base + self.nbr.clamp(min=0), torch.full((), nd * nc, device=dev)).reshape(-1, nv)
        cf = torch.where(inflow, sn * (self.area / self.vol[:, None]), torch.zeros((), device=dev,
                                                                                  dtype=sn.dtype)).reshape(-1, nv)
        self.sig = (sn.clamp(min=0) * (self.area / self.vol[:, None])).sum(2).reshape(-1, 1)
        lv = torch.zeros(nd * nc + 1, dtype=torch.int32, device=dev)
        lv[-1] = -1
        for _ in range(4000):
            new = lv[up].amax(1) + 1
            if torch.equal(new, lv[:-1]):
                break
            lv[:-1] = new
        else:
            return False
        order = torch.argsort(lv[:-1], stable=True)
        self.order = torch.split(order, torch.bincount(lv[:-1]).tolist())
        self.up, self.cf = up, cf
        return True

    def gradient(self, e):
        if self.case.get("order") == "1":
            return [torch.zeros_like(e) for _ in range(self.dim)]
        return [m @ e for m in self.grad]

    def limit(self, d, e, eb, gr):
        if self.case.get("order") != "2limit":
            return gr
        mx, mn = e.clone(), e.clone()
        for j in range(self.nbr.shape[1]):
            v = torch.where(self.wall[:, j, None], e, e[self.nbr[:, j].clamp(min=0)])
            inw = self.wall[:, j] & ~self.spec[:, j] & ((self.nrm[:, j] @ self.s[d]) < 0)
            v = torch.where(inw[:, None], eb[d][self.bound[:, j].clamp(min=0)], v)
            mx, mn = torch.maximum(mx, v), torch.minimum(mn, v)
        lim = torch.ones_like(e)
        for j in range(self.nbr.shape[1]):
            r = self.fc[:, j] - self.cen
            dl = sum(gr[k] * r[:, k, None] for k in range(self.dim))
            for sign, end in ((-1, mn), (1, mx)):
                bad = sign * (dl * lim + e - end) > 0
                y = (end - e) / dl
                lim = torch.where(bad, (y * y + 2 * y) / (y * y + y + 2), lim)
        return [x * lim for x in gr]

    def outgoing(self, d, e, gr, eb):
        out = (self.bnrm @ self.s[d]) >= 0
        v = e[self.bcell] + sum(gr[k][self.bcell] * self.boff[:, k, None] for k in range(self.dim))
        eb[d] = torch.where(out[:, None], v, eb[d])

    def incoming(self, eb):
        sn = self.bnrm @ self.s.T  # [walls, directions]
        inw = sn < 0
        for t in sorted({int(x) for x in self.btype}):
            rows = torch.as_tensor(np.flatnonzero(self.btype == t), device=self.dev)
            if t == 1:
                val = (self.C * self.bT[rows, None])[None].expand(self.nd, -1, -1)
            elif t == 2:
                wt = (sn[rows].clamp(min=0) * self.w)
                val = (torch.einsum("rd,drb->rb", wt, eb[:, rows]) / wt.sum(1)[:, None])[None].expand(self.nd, -1, -1)
            elif t == 3:
                n = self.bnrm[rows]
                mir = self.s[None] - 2 * sn[rows][:, :, None] * n[:, None]
                src = torch.cdist(mir.reshape(-1, 3), self.s).argmin(1).reshape(len(rows), self.nd)
                val = eb[src.T, rows[None].expand(self.nd, -1)]
            else:
                val = eb[:, self.connect[rows]] + self.C * (self.bT[rows] - self.bT[self.connect[rows]])[:, None]
            m = inw[rows].T[:, :, None]
            eb[:, rows] = torch.where(m, val, eb[:, rows])

    def residual(self, d, e, gr, eb, Told, fixed):
        acc = torch.zeros_like(e)
        for j in range(self.nbr.shape[1]):
            sn = self.nrm[:, j] @ self.s[d]
            r = self.fc[:, j] - self.cen
            y = e + sum(gr[k] * r[:, k, None] for k in range(self.dim))
            nb = self.nbr[:, j].clamp(min=0)
            rn = self.fc[:, j] - self.cen[nb]
            yn = e[nb] + sum(gr[k][nb] * rn[:, k, None] for k in range(self.dim))
            yn = torch.where(self.wall[:, j, None], eb[d][self.bound[:, j].clamp(min=0)], yn)
            acc += (self.area[:, j] / self.vol * sn)[:, None] * torch.where(sn[:, None] >= 0, y, yn)
        return fixed - e - self.tau * self.v * acc

    def side_fields(self, e):
        """The seven moments whose face gradients form the synthetic source: [rows, 7] of e[d, row, b]."""
        syn = (self.hr > 0).double()
        th = self.kappa * torch.einsum("dnb,d,b->n", e, self.w, self.lat / self.C * syn)
        e2 = torch.einsum("dnb,b->dn", e, self.tau * self.v ** 2 * syn)
        Q = torch.einsum("dn,d,dk,dl->nkl", e2, self.w, self.s, self.s)
        return torch.cat([th[:, None], Q.reshape(-1, 9)], 1)

    def tangent(self, vert, j):
        """The in-plane gradient on face j of every cell of vertex fields [nn, n]: [nc, n, 3]."""
        p = [vert[self.fv[:, j, k]] for k in range(self.fv.shape[2])]
        return sum((p[k + 1] - p[k])[:, :, None] * self.tang[:, j, k, None] for k in range(len(p) - 1))

    def source(self, e, eb):
        fc, fb = self.side_fields(e), self.side_fields(eb)
        vert = self.vertc @ fc + self.vertb @ fb
        out = torch.zeros(self.nc, dtype=torch.float64, device=self.dev)
        for j in range(self.nbr.shape[1]):
            other = torch.where(self.wall[:, j, None], fb[self.bound[:, j].clamp(min=0)], fc[self.nbr[:, j].clamp(min=0)])
            a, n = self.a[:, j], self.nrm[:, j]
            gn = (other - fc) * ((a * n).sum(1) / (a * a).sum(1))[:, None]
            gr = gn[:, :, None] * n[:, None] + self.tangent(vert, j)
            div = (gr[:, 0] * n).sum(1) - torch.einsum("cklk,cl->c", gr[:, 1:].reshape(-1, 3, 3, 3), n)
            out += torch.where(self.spec[:, j], torch.zeros_like(div), self.area[:, j] * div)
        return out

    def cg(self, b, x):
        r = b - (self.K @ x[:, None])[:, 0]
        z = r / self.Kd
        p, rz = z.clone(), r @ z
        stop = 1e-15 * b.norm()
        for it in range(20 * int(math.sqrt(self.nc)) + 2000):
            if it % 16 == 0 and not bool(r.norm() > stop):
                break
            Ap = (self.K @ p[:, None])[:, 0]
            al = rz / (p @ Ap)
            x = x + al * p
            r = r - al * Ap
            z = r / self.Kd
            new = r @ z
            p = z + (new / rz) * p
            rz = new
        return x

    def macro(self, T, src, eb):
        bTm = torch.einsum("dnb,d,b->n", eb, self.w, self.lat / self.C)
        for i in np.flatnonzero(self.btype < 0):
            if float(self.bT[i]) > 0:
                bTm[i] = self.bT[i] / 2
                bTm[self.connect_np[i]] = -self.bT[i] / 2
        for _ in range(1000):
            old = T
            vert = (self.vertT @ T[:, None])
            rhs = src - self.heat * self.vol
            for j in range(self.nbr.shape[1]):
                a, n = self.a[:, j], self.nrm[:, j]
                on = ~self.spec[:, j]
                wl = self.wall[:, j]
                bt = torch.where(wl, bTm[self.bound[:, j].clamp(min=0)], torch.zeros_like(T))
                rhs = rhs - self.mcoef[:, j] * bt
                a2 = n - a / (a * n).sum(1)[:, None]
                gT = self.tangent(vert, j)[:, 0]
                if self.dim == 3:
                    gT = gT + torch.where((wl & ~on)[:, None], torch.zeros_like(a), a)
                rhs = rhs - torch.where(on, self.kappa * self.area[:, j] * (a2 * gT).sum(1), torch.zeros_like(T))
            T = self.cg(-rhs, T)
            if float(((T - old) ** 2).mean()) <= 1e-6:
                break
        return T

    def steady(self, T0):
        case, nd, nc, nb = self.case, self.nd, self.nc, self.nb
        if not self.levels():
            return None
        T = torch.as_tensor(T0, device=self.dev)
        e = (T[:, None] * self.C).expand(nd, nc, nb).clone()
        eb = torch.zeros(nd, self.nb_, nb, dtype=torch.float64, device=self.dev)
        for d in range(nd):
            gr = self.limit(d, e[d], eb, self.gradient(e[d]))
            self.outgoing(d, e[d], gr, eb)
        self.incoming(eb)
        kb = self.tau * self.v
        x = torch.zeros(nd * nc + 1, nb, dtype=torch.float64, device=self.dev)
        for _ in range(case["iters"]):
            fixed = T[:, None] * self.C + self.heat[:, None] * (self.hr * self.tau)
            x.zero_()
            grb = []
            for d in range(nd):
                gr = self.limit(d, e[d], eb, self.gradient(e[d]))
                x[d * nc:(d + 1) * nc] = self.residual(d, e[d], gr, eb, T, fixed)
                grb.append([k[self.bcell] for k in gr])
            for rows in self.order:
                up = (x[self.up[rows]] * self.cf[rows][:, :, None]).sum(1)
                x[rows] = (x[rows] - kb * up) / (1 + kb * self.sig[rows])
            e += x[:-1].reshape(nd, nc, nb)
            for d in range(nd):
                out = (self.bnrm @ self.s[d]) >= 0
                v = e[d][self.bcell] + sum(grb[d][k] * self.boff[:, k, None] for k in range(self.dim))
                eb[d] = torch.where(out[:, None], v, eb[d])
            S0 = torch.einsum("dnb,d->nb", e, self.w)
            S1 = torch.einsum("dnb,d,dk,b->nk", e, self.w, self.s, self.v)
            src = None if case.get("scheme") == "Sequential" else self.source(e, eb)
            self.incoming(eb)
            Tl = (S0 * (self.lat / self.C)).sum(1)
            T = Tl if src is None else self.macro(Tl, src, eb)
        return {"E": (S0.sum(1) / self.C.sum()).cpu().numpy(), "T": T.cpu().numpy(), "q": S1.cpu().numpy(),
                "Tband": (S0 / self.C).T.contiguous().cpu().numpy()}


def exact(case, seed):
    """The fields after the same iterations in 64 bits. None for the adjoint
    (its exact value is the limit of differences of converged solves), the
    transient solver's own start, and the largest block (minutes)."""
    if case["kind"] not in ("steady", "batch"):
        return None
    ds = _decks(case)
    size = sum(d.mesh.n_cells for d in ds) * case["bands"] * _directions(case)
    if size > 3e8 or not (torch.cuda.is_available() or size < 3e6):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    parts = []
    for T0, d in [(_initial(d, rng), d) for d in ds]:
        r = _Exact(d, case, dev).steady(T0)
        if r is None:
            return None
        parts.append(r)
    return {k: np.concatenate([p[k] for p in parts], axis=-1 if k == "Tband" else 0) for k in parts[0]}
