"""Solves on chip and streamed on random layouts: tiles that are not square, from 2 to 130 points wide and down to one row,
halo cells without a source, sources anywhere on the tile edges (neighbours need not be mutual), first guesses with halo
values, zero, infinite, NaN and overflowing right-hand sides, no iterations at all. The calls stream when a group with
another number of right-hand sides is added to them; both kernels make the same additions in the same order, so
solutions, halos and diagnostics are equal bit for bit."""

import random

import numpy as np
import pytest
import torch

from mit_jax_b200 import cg2d as cg
from mit_jax_b200.layout import Layout

pytestmark = pytest.mark.gpu


def _exchanger(rng, sNx, sNy, OL, T, unwritten):
    L = Layout(sNx, sNy, OL, OL, T)
    n = T * L.ny * L.nx
    src = rng.integers(0, n, n).astype(np.int32)           # corners and outer halos: anything
    comp = (rng.random(n) < 0.7).astype(np.int8)
    idx = np.arange(n).reshape(T, L.ny, L.nx)
    J, I = L.interior
    comp[idx[:, J, I].ravel()] = 0
    edge = np.zeros((sNy, sNx), bool)
    edge[[0, -1]] = edge[:, [0, -1]] = True
    pool = np.repeat(idx[:, J, I][:, edge].ravel(), 2)      # a point may feed two cells
    rng.shuffle(pool)
    ring = np.concatenate([idx[:, J, OL - 1].ravel(), idx[:, J, OL + sNx].ravel(), idx[:, OL - 1, I].ravel(),
                           idx[:, OL + sNy, I].ravel()])
    rng.shuffle(ring)
    written = ring[rng.random(len(ring)) >= unwritten][:len(pool)]
    comp[ring] = 0
    comp[written] = 1
    src[written] = pool[:len(written)]
    return cg.Exchanger(L, {"T": (src, comp, np.ones(n, np.int8))})


def _group(pick, nrhs):
    rng = np.random.default_rng(pick.getrandbits(32))
    sNx, sNy = pick.choice([2, 6, 30, 32, 34, 64, 66, 96, 98, 130]), pick.choice([1, 2, 7, 8, 9, 16, 31])
    count = pick.choice([1, 2, 7])
    ex = _exchanger(rng, sNx, sNy, pick.choice([1, 2, 4]), pick.choice([1, 2, 5, 13]), pick.choice([0.0, 0.0, 0.15]))
    shape = (count, *ex.L.shape2d)
    arr = lambda lo, hi: torch.as_tensor(rng.uniform(lo, hi, shape)).cuda()          # noqa: E731
    ops = (arr(0.1, 1), arr(0.1, 1), -arr(4.0, 4.5), arr(-0.1, 0.1), arr(-0.1, 0.1), arr(0.8, 1.2))
    b = [arr(-1, 1) * pick.choice([1.0, 1e5]) for _ in range(nrhs)]
    special = pick.choice([None] * 4 + [0.0, float("nan"), float("inf"), 1e300])
    if special == 1e300:
        b[0] *= special
    elif special is not None:
        b[0].view(-1)[rng.integers(0, b[0].numel(), 5)] = special
    return cg.GroupSpec(ex, ops, b, [arr(-1, 1) * pick.choice([0.0, 1.0]) for _ in range(nrhs)],
                        [pick.choice([0.0, 1e-5, 1e30]) for _ in range(nrhs)], [pick.choice([0, 1, 7, 24]) for _ in range(nrhs)],
                        torch.as_tensor(rng.uniform(0.5, 1.5, count)).cuda(), x_fortran=True)


def _bits(t):
    return torch.where(t.isnan(), torch.zeros_like(t), t), t.isnan()     # (which NaN it is does not matter)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("order", ["rowblock", "fortran"])
@pytest.mark.parametrize("nrhs", [1, 2])
def test_random_layouts(precision, order, nrhs):
    pick = random.Random(f"{precision} {order} {nrhs}")
    kw = dict(precision=precision, sum_order=order)
    compared = 0
    for _ in range(12):
        groups = [_group(pick, nrhs) for _ in range(pick.choice([2, 3]))]
        limit = pick.choice([0, 0, 1, 5, 40])
        other = groups + [_group(pick, 3 - nrhs)]
        assert not any(p["on_chip"] for p in cg.solve_plan(other, **kw))
        if not cg.solve_plan(groups, grid_ctas=limit, **kw)[0]["on_chip"]:
            continue
        for got, ref in zip(cg.solve_groups(groups, grid_ctas=limit, **kw), cg.solve_groups(other, **kw)):
            for (x0, f0, d0), (x1, f1, d1) in zip(ref, got):
                for a, c in ((x0, x1), (f0, f1)):
                    assert all(torch.equal(p, q) for p, q in zip(_bits(a), _bits(c)))
                for r0, r1 in zip(cg.diag_records(d0), cg.diag_records(d1)):
                    assert str(r0) == str(r1)
                compared += 1
    assert compared >= 10
