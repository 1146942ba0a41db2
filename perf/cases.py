"""What this framework's speed is measured on: CG2D solves, adjoints and pressure steps as a program makes them.

A case is one call (or the few calls of one model step) through the package's public entry points, on seeded
synthetic fields of an LLC grid made on the GPU: land from smoothed noise (30 % land), depths of 500-6000 m, spacing
from a smooth latitude, ensemble members with depths perturbed by 10 % and right-hand sides of their own.

Kinds of case ("kind"):
  solve   cg2d_solve on one instance (count 0) or a batch
  grad    cg2d_solve and its backward pass: gradients of <w, x> in the right-hand side and the operator
  pair    solve_with_adjoint: forward and adjoint solve of every instance in one launch, coefficient gradients
  graph   solve_groups captured once (GraphedSolve) and replayed on its static inputs
  step    update_cg2d and solve_for_pressure, the free-surface step of a model with nr levels
  groups  solve_groups over a batch of each of two grid sizes
  adjoint exact_adjoint: reverse mode through the iterations
"""

import functools
import math
import types

import numpy as np
import torch
import torch.nn.functional as F

from mit_jax_b200 import cg2d as cg
from mit_jax_b200 import pressure as pr
from mit_jax_b200.graph import GraphedSolve
from mit_jax_b200.topology import LLCTopology

GRAVITY, DELTA_T, OFFDIAG = 9.81, 3600.0, 0.51
DEV, F64 = "cuda", torch.float64
L2_BYTES = 126e6


def listed():
    return [
        # a small regional or test configuration, one model step's solve with the parameters a user gets by default
        # (the reference's sequential sum order) at the production tolerance: the smallest call
        {"name": "llc32_default", "kind": "solve", "n": 32, "ts": 16, "count": 0, "order": "fortran", "tol": 1e-7},
        # one time step of the LLC90 model with 50 levels and the default parameters: what a run does every step
        {"name": "llc90_step_default", "kind": "step", "n": 90, "ts": 90, "count": 0, "order": "fortran",
         "tol": 1e-7, "nr": 50},
        # one LLC90 solve to 1e-12 in double precision, the drop-in call in the GPU's own sum order
        {"name": "llc90_f64", "kind": "solve", "n": 90, "ts": 90, "count": 0, "order": "rowblock", "tol": 1e-12},
        # the same inside an adjoint model: forward, then the implicit derivative by autograd
        {"name": "llc90_grad", "kind": "grad", "n": 90, "ts": 90, "count": 0, "order": "rowblock", "tol": 1e-12},
        # forward and adjoint of one instance in mixed precision
        {"name": "llc90_pair_1", "kind": "pair", "n": 90, "ts": 90, "count": 1, "prec": "mixed", "tol": 1e-12,
         "passive": False},
        # an ensemble of forward + adjoint pairs: the workload of the benchmark
        {"name": "llc90_pair_64", "kind": "pair", "n": 90, "ts": 90, "count": 64, "prec": "mixed", "tol": 1e-12,
         "passive": False},
        # an odd batch on 117 small tiles, operator passive
        {"name": "llc90_tiles30_pair_9", "kind": "pair", "n": 90, "ts": 30, "count": 9, "prec": "mixed",
         "tol": 1e-12, "passive": True},
        # a double-precision ensemble, captured once and replayed
        {"name": "llc90_f64_64_graph", "kind": "graph", "n": 90, "ts": 90, "count": 64, "prec": "f64", "tol": 1e-12},
        # a time step of an ensemble of 16 models with 50 levels
        {"name": "llc90_step_16", "kind": "step", "n": 90, "ts": 90, "count": 16, "order": "rowblock", "tol": 1e-12,
         "nr": 50},
        # one solve on the large grid
        {"name": "llc270_f64", "kind": "solve", "n": 270, "ts": 270, "count": 0, "order": "rowblock", "tol": 1e-12},
        # both grid sizes in one launch
        {"name": "llc270x8_llc90x32", "kind": "groups", "n": 270, "ts": 270, "count": 8, "n2": 90, "ts2": 90,
         "count2": 32, "prec": "mixed", "tol": 1e-12},
        # reverse mode through the iterations for a batch of 16, checkpoints every 30
        {"name": "llc90_adjoint_16", "kind": "adjoint", "n": 90, "ts": 90, "count": 16, "tol": 1e-12, "every": 30},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo, hi):
        """A facet size and a tile size: even, the tiles a half or a third of the facet at times."""
        split = rng.choice((1, 1, 2, 3))
        ts = max(8, 2 * (log(lo, hi) // split // 2))
        return ts * split, ts

    kind = rng.choice(("solve", "solve", "grad", "pair", "pair", "graph", "step", "groups", "adjoint"))
    tol = rng.choice((1e-7, 1e-12, 1e-12))
    if kind == "solve" or kind == "grad":
        order = rng.choice(("fortran", "rowblock", "rowblock"))
        n, ts = size(16, 90 if order == "fortran" else 270)
        most = 1 if order == "fortran" else max(1, min(20, int(12 * (90 / n) ** 3)))
        return {"kind": kind, "n": n, "ts": ts, "count": rng.choice((0, log(1, most))), "order": order, "tol": tol}
    if kind == "pair" or kind == "graph":
        n, ts = size(32, 200)
        most = max(1, min(100, int(64 * (90 / n) ** 3)))
        c = {"kind": kind, "n": n, "ts": ts, "count": log(1, most), "prec": rng.choice(("mixed", "mixed", "f64")),
             "tol": 1e-12}
        return dict(c, passive=rng.random() < 0.3) if kind == "pair" else c
    if kind == "step":
        order = rng.choice(("fortran", "rowblock", "rowblock"))
        n, ts = size(16, 100)
        most = 1 if order == "fortran" else max(1, int(16 * (90 / n) ** 2)) if n > 60 else 32
        return {"kind": kind, "n": n, "ts": ts, "count": rng.choice((0, log(1, most))), "order": order, "tol": tol,
                "nr": rng.choice((1, 15, 23, 50))}
    if kind == "groups":
        n, ts = size(64, 200)
        n2, ts2 = size(32, 90)
        return {"kind": kind, "n": n, "ts": ts, "count": log(1, max(1, min(8, int(8 * (150 / n) ** 3)))), "n2": n2,
                "ts2": ts2, "count2": log(1, 32), "prec": rng.choice(("mixed", "f64")), "tol": 1e-12}
    n, ts = size(16, 90)
    return {"kind": kind, "n": n, "ts": ts, "count": log(1, 16), "tol": 1e-12, "every": rng.choice((0, 7, 30, 30))}


# ---------------------------------------------------------------------------------------------------------------
# grids and seeded fields


class Grid:
    """One LLC layout: exchange maps, index tables and spacing on the GPU, its Exchanger."""

    def __init__(self, n, ts):
        topo = LLCTopology(n, ts)
        L = self.L = topo.L
        self.n, self.dims, self.tiles = n, topo.grid.dims, topo.grid.tiles()
        self.ex = cg.Exchanger(L, topo.maps)
        self.J, self.I = L.interior
        self.maps = {k: (torch.as_tensor(s.astype(np.int64), device=DEV), torch.as_tensor(c, device=DEV))
                     for k, (s, c, _) in topo.maps.items()}
        # smoothing over a facet axis: Gaussian of sigma 5 n / 90, edge values repeated
        sigma = 5.0 * n / 90.0
        R = int(4 * sigma + 0.5)
        k = np.exp(-0.5 * (np.arange(-R, R + 1) / sigma) ** 2)
        k /= k.sum()
        self.smooth_by = {}
        for m in (n, 3 * n):
            G = np.zeros((m, m))
            for o, w in zip(range(-R, R + 1), k):
                np.add.at(G, (np.arange(m), np.clip(np.arange(m) + o, 0, m - 1)), w)
            self.smooth_by[m] = torch.as_tensor(G, device=DEV)
        # the stencil's view of a vector: compact interior index of every point of [T, nj + 2, ni + 2], the value 0
        # (one past the end) where the exchange writes nothing
        T, nj, ni = L.nTiles, L.sNy, L.sNx
        compact = np.full(L.shape2d, T * nj * ni, np.int64)
        compact[:, self.J, self.I] = np.arange(T * nj * ni).reshape(T, nj, ni)
        src, comp, _ = topo.maps["T"]
        ring = np.where(comp == 1, compact.reshape(-1)[src], compact.reshape(-1)).reshape(L.shape2d)
        ring = ring[:, L.OLy - 1:L.OLy + nj + 1, L.OLx - 1:L.OLx + ni + 1]
        self.ring = torch.as_tensor(np.ascontiguousarray(ring).reshape(-1), device=DEV)
        self.ring_shape = ring.shape
        lat = self._latitude()
        scale = 90.0 / n
        self.dx = self.to_tiles({f: (20e3 + 90e3 * v.cos())[None] * scale for f, v in lat.items()}, 1.0)
        self.dy = self.to_tiles({f: (65e3 + 45e3 * v.cos())[None] * scale for f, v in lat.items()}, 1.0)
        self.mask = torch.zeros(L.shape2d, dtype=torch.bool, device=DEV)
        self.mask[:, self.J, self.I] = True

    def _latitude(self):
        lat = {}
        for f, (nx, ny) in self.dims.items():
            jj, ii = np.meshgrid((np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx, indexing="ij")
            if f < 3:
                v = -75.0 + 140.0 * jj
            elif f == 3:
                v = 90.0 - 50.0 * np.hypot(jj - 0.5, ii - 0.5)
            else:
                v = 65.0 - 140.0 * ii
            lat[f] = torch.as_tensor(np.deg2rad(v), device=DEV)
        return lat

    def to_tiles(self, facets, fill=0.0):
        """{facet: [B, ny, nx]} -> padded [B, T, ny, nx]."""
        B, ts = facets[1].shape[0], self.L.sNx
        out = torch.full((B,) + tuple(self.L.shape2d), fill, dtype=F64, device=DEV)
        for t, (f, i0, j0) in enumerate(self.tiles):
            out[:, t, self.J, self.I] = facets[f][:, j0:j0 + ts, i0:i0 + ts]
        return out

    def noise(self, gen, count):
        """Smoothed unit noise per facet, {facet: [count, ny, nx]}."""
        return {f: self.smooth_by[ny] @ torch.randn(count, ny, nx, dtype=F64, device=DEV, generator=gen)
                @ self.smooth_by[nx].T for f, (nx, ny) in self.dims.items()}

    def exch(self, a):
        """exch_xy of [B, T, ny, nx]."""
        src, comp = self.maps["T"]
        f = a.reshape(a.shape[0], -1)
        return torch.where(comp == 1, f[:, src], f).reshape(a.shape)

    def exch_faces(self, u, v):
        """The face exchange of the pair (u, v) of [B, T, (levels,) ny, nx], in place."""
        if u.dim() == 4:
            self.exch_faces(u.unsqueeze(2), v.unsqueeze(2))
            return u, v
        ny, nx = self.L.ny, self.L.nx
        got = []
        for a, key in ((u, "UVn_u"), (v, "UVn_v")):
            src, comp = self.maps[key]
            for c, b in ((1, u), (2, v)):
                p = torch.nonzero(comp == c).flatten()
                s = src[p]
                got.append((a, p, b[:, s // (ny * nx), :, s // nx % ny, s % nx].clone()))
        for a, p, val in got:
            a[:, p // (ny * nx), :, p // nx % ny, p % nx] = val
        return u, v

    def ringed(self, v):
        """[B, T, nj, ni] -> [B, T, nj + 2, ni + 2] with the neighbours' values, as the stencil reads them."""
        B = v.shape[0]
        return F.pad(v.reshape(B, -1), (0, 1))[:, self.ring].reshape((B,) + self.ring_shape)


@functools.lru_cache(maxsize=8)
def grid(n, ts):
    return Grid(n, ts)


def depths(G, gen, count):
    """(ocean [T, ny, nx], depth [count, T, ny, nx]): members perturb one seeded bathymetry by up to 10 %."""
    land = G.noise(gen, 1)
    level = torch.quantile(torch.cat([v.flatten() for v in land.values()])[::max(1, 13 * G.n ** 2 // 100000)], 0.30)
    ocean = G.to_tiles({f: (v >= level).double() for f, v in land.items()})
    H = G.to_tiles({f: 500.0 + 5500.0 * torch.rand(1, ny, nx, dtype=F64, device=DEV, generator=gen)
                    for f, (nx, ny) in G.dims.items()}) * ocean
    e = G.to_tiles(G.noise(gen, count))
    e = e / e.abs().amax(dim=(1, 2, 3), keepdim=True)
    return ocean[0], H * (1.0 + 0.1 * e)


def rhs_of(G, gen, ocean, count):
    """Smoothed noise on the ocean, its mean removed, 0 on land."""
    f = G.to_tiles(G.noise(gen, count)) * ocean
    return (f - f.sum(dim=(1, 2, 3), keepdim=True) / ocean.sum()) * ocean


def operator_of(G, aW, aS, norm, bo_ra):
    """(aW2d, aS2d, aC2d, pW, pS, pC) of the un-normalised faces aW, aS on padded arrays (halo faces 0)."""
    L, J, I = G.L, G.J, G.I
    n4 = norm.view(-1, 1, 1, 1)
    aW, aS = G.exch_faces(aW * n4, aS * n4)
    return finish_operator(G, aW, aS, n4, bo_ra)


def finish_operator(G, aW, aS, n4, bo_ra, pre=None):
    L, J, I = G.L, G.J, G.I
    Ip, Jp = L.is_(2, L.sNx + 1), L.js(2, L.sNy + 1)
    aC = torch.zeros_like(aW)
    aC[:, :, J, I] = -(aW[:, :, J, I] + aW[:, :, J, Ip] + aS[:, :, J, I] + aS[:, :, Jp, I]
                       + (n4 * bo_ra)[:, :, J, I] / DELTA_T / DELTA_T)
    aC = G.exch(aC)
    J1, I1, Im, Jm = L.js(1, L.sNy + 1), L.is_(1, L.sNx + 1), L.is_(0, L.sNx), L.js(0, L.sNy)
    a, zero = aC[:, :, J1, I1], torch.zeros((), dtype=F64, device=DEV)
    pW, pS, pC = (torch.zeros_like(aW) if p is None else p.clone() for p in (pre or (None,) * 3))
    pC[:, :, J1, I1] = torch.where(a == 0, zero + 1, 1.0 / a)
    tw, ts = a + aC[:, :, J1, Im], a + aC[:, :, Jm, I1]
    pW[:, :, J1, I1] = torch.where(tw == 0, zero, -aW[:, :, J1, I1] / (OFFDIAG * tw) ** 2)
    pS[:, :, J1, I1] = torch.where(ts == 0, zero, -aS[:, :, J1, I1] / (OFFDIAG * ts) ** 2)
    return aW, aS, aC, pW, pS, pC


def problem(n, ts, count, gen):
    """(grid, ops, cg2dNorm [count], b, w) of `count` members."""
    G = grid(n, ts)
    J, I, L = G.J, G.I, G.L
    ocean, H = depths(G, gen, count)
    He = G.exch(H)
    aW, aS = torch.zeros_like(H), torch.zeros_like(H)
    aW[:, :, J, I] = (torch.minimum(He[:, :, J, I], He[:, :, J, L.is_(0, L.sNx - 1)]) * (G.dy / G.dx)[:, :, J, I])
    aS[:, :, J, I] = (torch.minimum(He[:, :, J, I], He[:, :, L.js(0, L.sNy - 1), I]) * (G.dx / G.dy)[:, :, J, I])
    norm = 1.0 / torch.maximum(aW.amax(dim=(1, 2, 3)), aS.amax(dim=(1, 2, 3)))
    ops = operator_of(G, aW, aS, norm, G.dx * G.dy / GRAVITY)
    return G, ops, norm, rhs_of(G, gen, ocean, count), rhs_of(G, gen, ocean, count)


def model(case, gen):
    """Fields of a model step, leading dimension `count` (1 for a single model): a namespace."""
    B, Nr = max(1, case["count"]), case["nr"]
    G = grid(case["n"], case["ts"])
    L, J, I = G.L, G.J, G.I
    ocean, H = depths(G, gen, B)
    g = np.geomspace(10.0, 460.0, Nr)
    drF = torch.as_tensor(g * (6000.0 / g.sum()), device=DEV)
    top = F.pad(torch.cumsum(drF, 0), (1, 0))[:-1]
    He = G.exch(H).unsqueeze(2)
    hC = ((He - top.view(-1, 1, 1)) / drF.view(-1, 1, 1)).clamp_(0.0, 1.0)
    hW, hS = torch.zeros_like(hC), torch.zeros_like(hC)
    hW[..., J, I] = torch.minimum(hC[..., J, I], hC[..., J, L.is_(0, L.sNx - 1)])
    hS[..., J, I] = torch.minimum(hC[..., J, I], hC[..., L.js(0, L.sNy - 1), I])
    del hC
    G.exch_faces(hW, hS)
    gU, gV = (torch.randn(hW.shape, dtype=F64, device=DEV, generator=gen).mul_(1e-5).mul_(h > 0) for h in (hW, hS))
    G.exch_faces(gU, gV)

    def inner(a):
        return torch.where(G.mask, a, torch.zeros((), dtype=F64, device=DEV))

    dyG, dxG = G.exch_faces(inner(G.dy), inner(G.dx))
    rdxC, rdyC = G.exch_faces(inner(1.0 / G.dx), inner(1.0 / G.dy))

    def field(scale, mask):
        f = G.to_tiles(G.noise(gen, B))
        return G.exch(inner(scale * f / f.abs().max() * mask))

    Bo = G.exch(inner(GRAVITY * (1.0 + 0.01 * field(1.0, 1.0)[:1])))
    Bo = torch.where(Bo == 0, GRAVITY, Bo)
    J1, I1 = (G.J, G.I)
    aW = (hW * drF.view(-1, 1, 1)).sum(2)[:, :, J1, I1] * (dyG * rdxC)[:, :, J1, I1]
    aS = (hS * drF.view(-1, 1, 1)).sum(2)[:, :, J1, I1] * (dxG * rdyC)[:, :, J1, I1]
    norm = float(1.0 / max(aW.max(), aS.max()))
    m = types.SimpleNamespace(
        G=G, Nr=Nr, hFacW=hW, hFacS=hS, gU=gU, gV=gV, norm=norm, Bo=Bo[0], recip_Bo=(1.0 / Bo)[0],
        EmPmR=field(1e-5, ocean), etaN=field(0.5, ocean), etaH=field(0.5, ocean),
        pre=tuple(torch.zeros((B,) + tuple(L.shape2d), dtype=F64, device=DEV) for _ in range(3)),
        g=types.SimpleNamespace(layout=L, drF=drF, dyG=dyG[0], dxG=dxG[0], recip_dxC=rdxC[0], recip_dyC=rdyC[0],
                                rA=G.exch(inner(G.dx * G.dy))[0], maskInC=inner(ocean)),
        p=pr.FreeSurfParams(deltaTMom=DELTA_T, deltaTFreeSurf=DELTA_T, freeSurfFac=1.0, implicSurfPress=1.0,
                            implicDiv2DFlow=1.0, mass2rUnit=1.0 / 1029.0, rUnit2mass=1029.0, facEmP=1.0,
                            hFacInf=0.2, hFacSup=2.0, rStarAreaWeight=True, pfFacMom=1.0, select_rStar=2,
                            nonlinFreeSurf=4, useRealFreshWaterFlux=True, Nr=Nr))
    return m


def iteration_cap(case, n=None):
    return max(300, 5 * (n or case["n"]))


# ---------------------------------------------------------------------------------------------------------------
# prepare, run


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    kind = case["kind"]
    s = types.SimpleNamespace(case=case, kind=kind)
    if kind == "step":
        m = s.m = model(case, gen)
        if case["count"] == 0:
            for k in ("hFacW", "hFacS", "gU", "gV", "EmPmR", "etaN", "etaH"):
                setattr(m, k, getattr(m, k)[0])
            m.pre = tuple(a[0] for a in m.pre)
        s.p = cg.Cg2dParams(cg2dMaxIters=iteration_cap(case), cg2dTolerance=case["tol"], cg2dNorm=m.norm,
                            cg2dpcOffDFac=OFFDIAG, sum_order=case["order"])
        return s
    B = max(1, case["count"])
    s.G, s.ops, s.norm, s.b, s.w = problem(case["n"], case["ts"], B, gen)
    s.x0 = torch.zeros_like(s.b)
    if kind in ("solve", "grad"):
        # one normalisation for the call, as its parameters hold one: the members' operators share it
        s.norm = float(s.norm[0])
        if case["count"] == 0:
            s.ops, s.b, s.w, s.x0 = tuple(a[0] for a in s.ops), s.b[0], s.w[0], s.x0[0]
        s.p = cg.Cg2dParams(cg2dMaxIters=iteration_cap(case), cg2dTolerance=case["tol"], cg2dNorm=s.norm,
                            sum_order=case["order"], adj_tolerance=case["tol"] / 10)
    elif kind in ("graph", "groups"):
        cap = iteration_cap(case)
        s.groups = [cg.GroupSpec(s.G.ex, s.ops, [s.b, s.w], [s.x0, s.x0], [case["tol"]] * 2, [cap] * 2, s.norm)
                    if kind == "groups" else
                    cg.GroupSpec(s.G.ex, s.ops, [s.b], [s.x0], [case["tol"]], [cap], s.norm)]
        if kind == "groups":
            s.G2, ops, norm, b, w = problem(case["n2"], case["ts2"], case["count2"], gen)
            cap = iteration_cap(case, case["n2"])
            s.groups.append(cg.GroupSpec(s.G2.ex, ops, [b, w], [torch.zeros_like(b)] * 2, [case["tol"]] * 2,
                                         [cap] * 2, norm))
        else:
            s.graph = GraphedSolve(s.groups, precision=case["prec"])
    return s


def run(s):
    case, kind = s.case, s.kind
    if kind == "solve":
        x, diag = cg.cg2d_solve(s.p, s.G.ex, s.ops, s.b, s.x0)
        return {"x": x}
    if kind == "grad":
        b = s.b.detach().requires_grad_()
        aW, aS, aC = (a.detach().requires_grad_() for a in s.ops[:3])
        x, _ = cg.cg2d_solve(s.p, s.G.ex, (aW, aS, aC) + tuple(s.ops[3:]), b, s.x0)
        grads = torch.autograd.grad(x, (b, aW, aS, aC), s.w)
        return {"x": x.detach(), "grads": grads}
    if kind == "pair":
        r = cg.solve_with_adjoint(s.G.ex, s.ops, s.b, s.w, s.x0, cg2dNorm=s.norm, tolerance=case["tol"],
                                  max_iters=iteration_cap(case), adj_tolerance=case["tol"],
                                  adj_max_iters=iteration_cap(case), precision=case["prec"],
                                  coeff_grad="passive" if case["passive"] else "implicit")
        return {k: r[k] for k in ("x", "lam", "gW", "gS", "gC") if r[k] is not None}
    if kind == "graph":
        (slots,), _ = s.graph.replay()
        return {"x": slots[0][0]}
    if kind == "groups":
        return [[slot[0] for slot in slots] for slots in cg.solve_groups(s.groups, precision=case["prec"])]
    if kind == "adjoint":
        x, _, grads = cg.exact_adjoint(s.G.ex, s.ops, s.b, s.x0, s.w, cg2dNorm=s.norm, tolerance=case["tol"],
                                       max_iters=iteration_cap(case), checkpoint_every=case["every"])
        return {"x": x, "grads": grads}
    m = s.m
    ops = pr.update_cg2d(m.p, s.p, m.g, m.G.ex, m.hFacW, m.hFacS, m.recip_Bo, *m.pre)
    eta, info = pr.solve_for_pressure(m.p, s.p, m.g, m.G.ex, ops, m.gU, m.gV, m.hFacW, m.hFacS, m.EmPmR, m.etaN,
                                      m.etaH, m.Bo, m.recip_Bo)
    return {"ops": ops, "etaN": eta, "b": info["cg2d_b"]}


# ---------------------------------------------------------------------------------------------------------------
# work and tolerance


def points(case, second=False):
    return 13 * (case["n2"] if second else case["n"]) ** 2


def iterations(n, tol):
    """Iterations of one solve on these fields: they grow with the grid's diameter and the digits asked for."""
    return 2.6 * n * (0.6 if tol > 1e-9 else 1.0)


def solves(case):
    """[(points, instances, right-hand sides, iterations each, mixed)]: the CG work of one pass."""
    kind, mixed = case["kind"], case.get("prec") == "mixed"
    k, B = iterations(case["n"], case["tol"]), max(1, case["count"])
    nrhs = 2 if kind in ("pair", "groups", "grad") else 1
    got = [(points(case), B, nrhs, k, mixed)]
    if kind == "groups":
        got.append((points(case, True), case["count2"], nrhs, iterations(case["n2"], case["tol"]), mixed))
    return got


def work(case):
    """One pass: every input read once and every output written once; where the solves' state (six coefficients and
    r, s, x of each right-hand side) exceeds the L2 cache, each iteration reads it and writes r, s, x again. An
    iteration takes two stencils, three vector updates and three dot products: 30 operations a point."""
    kind = case["kind"]
    state = io = loop = flops = 0.0
    for n, B, nrhs, k, mixed in solves(case):
        v = 4 if mixed else 8
        state += n * B * (6 * v + nrhs * (2 * v + 8))
        loop += n * B * k * (6 * v + nrhs * 2 * (2 * v + 8))
        io += n * B * 8 * (6 + 3 * nrhs)
        flops += 30.0 * n * B * nrhs * k
        if kind in ("grad", "pair") and not case.get("passive"):
            io += n * B * 8 * 3
    if kind == "step":
        n, B = points(case), max(1, case["count"])
        io += n * B * 8 * (4 * case["nr"] + 6 + 3 + 3) + n * 8 * 8
        flops += n * B * 26.0 * case["nr"]
    if kind == "adjoint":
        # the reverse of an iteration reads the coefficients, xbar and the iteration's r and s, updates the cotangents
        # of r and s and of the six coefficients: twice the forward's stencils and their edge products
        n, B, _, k, _ = solves(case)[0]
        state, loop, flops = state + n * B * 9 * 8, loop + n * B * k * 8 * (6 + 1 + 2 + 4), flops * 4
        io += n * B * 8 * 7
    return {"bytes": io + (loop if state > L2_BYTES else 0.0), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    # the reference's sum order gives its results bit for bit; the derivative through the iterations has entries (of the
    # preconditioner, which a converged solution does not depend on) that are nothing but the rounding of the forward's
    # sums, so only the documented order of those sums, bit for bit, gives the same ones
    if kind == "adjoint" or (case.get("order") == "fortran" and kind != "grad"):
        return "exact"
    if case["tol"] > 1e-9:      # other sum orders: 7e-11 seen against the plain solve with the same stop
        return {"rel": 1e-9, "max": 1e-7}
    if case.get("prec") == "mixed":     # 5e-14 seen on LLC90, 2e-13 on LLC32
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 1e-13, "max": 1e-11}     # 1e-15 to 3e-15 seen


# ---------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, by plain torch


class Plain:
    """A batch's stencils and CG solve on interior arrays [B, T, nj, ni]."""

    def __init__(self, G, ops, norm):
        L, J, I = G.L, G.J, G.I
        self.G = G
        Ip, Jp = L.is_(2, L.sNx + 1), L.js(2, L.sNy + 1)
        ops = [a.reshape((-1,) + tuple(L.shape2d)) for a in ops]
        self.A = [ops[0][:, :, J, I], ops[0][:, :, J, Ip], ops[1][:, :, J, I], ops[1][:, :, Jp, I],
                  ops[2][:, :, J, I]]
        self.M = [ops[3][:, :, J, I], ops[3][:, :, J, Ip], ops[4][:, :, J, I], ops[4][:, :, Jp, I],
                  ops[5][:, :, J, I]]
        n = norm if torch.is_tensor(norm) else torch.full((ops[0].shape[0],), float(norm), dtype=F64, device=DEV)
        self.norm = n.view(-1, 1, 1, 1)

    def apply(self, C, v):
        V = self.G.ringed(v)
        return (C[0] * V[:, :, 1:-1, :-2] + C[1] * V[:, :, 1:-1, 2:] + C[2] * V[:, :, :-2, 1:-1]
                + C[3] * V[:, :, 2:, 1:-1] + C[4] * v)

    @staticmethod
    def dot(a, b):
        return (a * b).sum(dim=(1, 2, 3), keepdim=True)

    def solve(self, b, x0, tol, cap, keep=None):
        """(x, rhsNorm, iterations [B]) of the preconditioned CG iteration on padded b, x0."""
        G = self.G
        bn = b[..., G.J, G.I] * self.norm
        big = bn.abs().amax(dim=(1, 2, 3), keepdim=True)
        rn = torch.where(big != 0, 1.0 / big, torch.ones_like(big))
        bn, x = bn * rn, x0[..., G.J, G.I] * rn
        r = bn - self.apply(self.A, x)
        s, eta_prev = torch.zeros_like(r), torch.ones_like(rn)
        rr = self.dot(r, r)
        K = torch.zeros_like(rn)
        for k in range(cap):
            on = rr >= tol * tol
            if k % 8 == 0 and not bool(on.any()):
                break
            z = self.apply(self.M, r)
            eta = self.dot(z, r)
            beta = eta / eta_prev
            sn = z + beta * s
            q = self.apply(self.A, sn)
            sig = self.dot(sn, q)
            alpha = eta / sig
            if keep is not None:
                keep.append((r, s, eta, eta_prev, beta, sig, alpha, on))
            x = torch.where(on, x + alpha * sn, x)
            r = torch.where(on, r - alpha * q, r)
            s = torch.where(on, sn, s)
            eta_prev = torch.where(on, eta, eta_prev)
            rr = torch.where(on, self.dot(r, r), rr)
            K = K + on
        return x, rn, K

    def padded(self, v):
        L = self.G.L
        out = torch.zeros((v.shape[0],) + tuple(L.shape2d), dtype=F64, device=DEV)
        out[..., self.G.J, self.G.I] = v
        return out

    def edges(self, u, V, sign):
        """sign (u (x) v) on the coefficient entries a tile holds, V ringed: (gW, gS, gC) on padded arrays."""
        G, L = self.G, self.G.L
        U = F.pad(u, (1, 1, 1, 1))
        v = V[:, :, 1:-1, 1:-1]
        gW, gS = (torch.zeros((u.shape[0],) + tuple(L.shape2d), dtype=F64, device=DEV) for _ in range(2))
        # face i = 0 .. ni between columns i - 1 and i, rows of the interior (and the same for j)
        gW[:, :, G.J, L.is_(1, L.sNx + 1)] = sign * (U[:, :, 1:-1, 1:] * V[:, :, 1:-1, :-1]
                                                     + U[:, :, 1:-1, :-1] * V[:, :, 1:-1, 1:])
        gS[:, :, L.js(1, L.sNy + 1), G.I] = sign * (U[:, :, 1:, 1:-1] * V[:, :, :-1, 1:-1]
                                                    + U[:, :, :-1, 1:-1] * V[:, :, 1:, 1:-1])
        return gW, gS, self.padded(sign * u * v)

    def coefficient_gradients(self, lam, x):
        return self.edges(lam / self.norm, self.G.ringed(x), -1.0)


def plain_adjoint(P, b, x0, xbar, tol, cap):
    """Reverse mode through the iterations of Plain.solve: x and the cotangents of <xbar, x>."""
    G, kept = P.G, []
    x, rn, _ = P.solve(b, x0, tol, cap, keep=kept)
    xb = xbar[..., G.J, G.I] / rn
    rb, sb, carry = torch.zeros_like(xb), torch.zeros_like(xb), torch.zeros_like(rn)
    g = [torch.zeros((xb.shape[0],) + tuple(G.L.shape2d), dtype=F64, device=DEV) for _ in range(6)]
    zero = torch.zeros((), dtype=F64, device=DEV)
    while kept:
        r, sp, eta, etap, beta, sig, alpha, on = kept.pop()
        first = not kept
        z = P.apply(P.M, r)
        s = z + beta * sp
        q = P.apply(P.A, s)
        ab = P.dot(xb, s) - P.dot(rb, q)
        sgb, etb = -ab * alpha / sig, carry + ab / sig
        qb = torch.where(on, sgb * s - alpha * rb, zero)
        s1 = sb + alpha * xb + sgb * q + P.apply(P.A, qb)
        bb = zero if first else P.dot(s1, sp)
        etb = etb + bb / etap
        carry = torch.where(on, -bb * eta / etap ** 2, carry)
        zb = torch.where(on, s1 + etb * r, zero)
        rb = torch.where(on, rb + etb * z + P.apply(P.M, zb), rb)
        sb = torch.where(on, beta * s1, sb)
        for i, (u, v) in enumerate(((qb, s), (zb, r))):
            for a, e in zip(g[3 * i:3 * i + 3], P.edges(u, G.ringed(v), 1.0)):
                a += e
    first_guess = x0[..., G.J, G.I] * rn
    for a, e in zip(g[:3], P.edges(rb, G.ringed(first_guess), -1.0)):
        a += e
    return P.padded(x / rn), dict(zip(("b",) + cg.OPS, [P.padded(rb * P.norm * rn)] + g))


def plain_pressure(s):
    """update_cg2d, cg2d_rhs, the solve and etaN of a step case."""
    m, case = s.m, s.case
    G, L, J, I = m.G, m.G.L, m.G.J, m.G.I
    one = case["count"] == 0
    hW, hS, gU, gV, em, en, eh = ((a[None] if one else a) for a in (m.hFacW, m.hFacS, m.gU, m.gV, m.EmPmR, m.etaN,
                                                                   m.etaH))
    pre = [a[None] if one else a for a in m.pre]
    g = m.g
    B = hW.shape[0]
    d = g.drF.view(-1, 1, 1)
    n4 = torch.full((B, 1, 1, 1), m.norm, dtype=F64, device=DEV)
    J1, I1 = L.js(1, L.sNy + 1), L.is_(1, L.sNx + 1)
    Ip, Jp = L.is_(2, L.sNx + 1), L.js(2, L.sNy + 1)
    aW, aS = torch.zeros_like(en), torch.zeros_like(en)
    u, v = torch.zeros_like(en), torch.zeros_like(en)
    for i in range(B):          # instance by instance: the 3-D products are large
        aW[i, :, J1, I1] = ((hW[i] * d).sum(1) * g.dyG * g.recip_dxC * m.norm)[:, J1, I1]
        aS[i, :, J1, I1] = ((hS[i] * d).sum(1) * g.dxG * g.recip_dyC * m.norm)[:, J1, I1]
        u[i] = (hW[i] * gU[i] * d).sum(1) * g.dyG / DELTA_T
        v[i] = (hS[i] * gV[i] * d).sum(1) * g.dxG / DELTA_T
    ops = finish_operator(G, aW, aS, n4, g.rA * m.recip_Bo, pre)
    b = torch.zeros_like(en)
    b[..., J, I] = (g.rA * em * g.maskInC * (m.p.mass2rUnit / DELTA_T) - g.rA / DELTA_T / DELTA_T * eh)[..., J, I] \
        + u[..., J, Ip] - u[..., J, I] + v[..., Jp, I] - v[..., J, I]
    x0 = m.Bo * en
    P = Plain(G, ops, m.norm)
    x, rn, _ = P.solve(b, x0, case["tol"], iteration_cap(case))
    full = torch.where(G.mask, P.padded(x / rn), x0)
    eta = m.recip_Bo * torch.where(G.mask, full, G.exch(full))
    cut = (lambda a: a[0]) if one else (lambda a: a)
    return {"ops": tuple(cut(a) for a in ops), "etaN": cut(eta), "b": cut(b)}


def exact(case, seed):
    s = prepare(case, seed) if case["kind"] != "graph" else None
    kind, tol = case["kind"], case["tol"]
    if kind == "step":
        return plain_pressure(s)
    if kind == "graph":
        gen = torch.Generator(device=DEV)
        gen.manual_seed(int(seed) * 7919 + 17)
        G, ops, norm, b, _ = problem(case["n"], case["ts"], case["count"], gen)
        P = Plain(G, ops, norm)
        x, rn, _ = P.solve(b, torch.zeros_like(b), tol, iteration_cap(case))
        return {"x": P.padded(x / rn)}
    if kind == "groups":
        got = []
        for gr in s.groups:
            P = Plain(s.G if gr is s.groups[0] else s.G2, gr.ops, gr.norm)
            got.append([])
            for b, x0 in zip(gr.b, gr.x0):
                x, rn, _ = P.solve(b, x0, tol, gr.max_iters[0])
                got[-1].append(P.padded(x / rn))
        return got
    one = case["count"] == 0
    ops, b, w, x0 = ([a[None] for a in s.ops], s.b[None], s.w[None], s.x0[None]) if one else (s.ops, s.b, s.w, s.x0)
    cut = (lambda a: a[0]) if one else (lambda a: a)
    P = Plain(s.G, ops, s.norm)
    cap = iteration_cap(case)
    if kind == "adjoint":
        x, grads = plain_adjoint(P, b, x0, w, tol, cap)
        # the entries of a tile's faces, one copy moved without the other, and of the preconditioner amplify the rounding of
        # the forward's sums without bound (up to 200 times their size seen): no value in 64 bits stands for them
        return {"x": x, "grads": {k: g if k in ("b", "aC2d") else None for k, g in grads.items()}}
    x, rn, _ = P.solve(b, x0, tol, cap)
    x = x / rn
    if kind == "solve":
        return {"x": cut(P.padded(x))}
    lam, ln, _ = P.solve(w, torch.zeros_like(w), s.p.adj_tolerance if kind == "grad" else tol,
                         s.p.adj_max_iters if kind == "grad" else cap)
    lam = lam / ln
    gs = () if case.get("passive") else P.coefficient_gradients(lam, x)
    if kind == "grad":
        return {"x": cut(P.padded(x)), "grads": tuple(cut(a) for a in (P.padded(lam),) + gs)}
    return {"x": P.padded(x), "lam": P.padded(lam), **dict(zip(("gW", "gS", "gC"), gs))}
