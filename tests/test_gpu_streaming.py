"""The streaming kernel (csrc/cg2d_solver.cu), which runs what does not fit on chip and groups with different numbers of
right-hand sides. Every test states that its calls stream (solve_plan). grid_ctas below the CTAs an instance needs makes any
solve stream, so the same instances solved on chip are the reference: all additions are made in the same order, and
solutions, halos and diagnostics are equal bit for bit."""

import itertools

import numpy as np
import pytest
import torch

from mit_jax_b200 import autotune
from mit_jax_b200 import cg2d as cg
from mit_jax_b200.synthetic import LLCSynthetic, make_batch

pytestmark = pytest.mark.gpu


def _group(N, count, nrhs, iters=300, tol=1e-12):
    syn, B = make_batch(N, count, with_cotangent=True, members=list(range(count)))
    ex = cg.default_exchanger(syn.L)
    t = {k: torch.as_tensor(v).cuda() for k, v in B.items()}
    w = torch.where(cg._interior_mask(syn.L, t["b"].device), t["w"], torch.zeros_like(t["w"]))
    return cg.GroupSpec(ex, tuple(t[k] for k in cg.OPS), [t["b"], w][:nrhs], [torch.zeros_like(w)] * nrhs, [tol] * nrhs,
                        [iters] * nrhs, t["cg2dNorm"], x_fortran=True)


def _same(ref, got):
    for slots0, slots1 in zip(ref, got, strict=True):
        for (x0, f0, d0), (x1, f1, d1) in zip(slots0, slots1, strict=True):
            assert torch.equal(x0, x1) and torch.equal(f0, f1) and torch.equal(d0, d1)


def _streamed(groups, **kw):
    plan = {k: v for k, v in kw.items() if k in ("precision", "sum_order", "rows_per_block", "grid_ctas", "ctas_per_sm",
                                                 "unit_deal", "stages")}
    assert not any(p["on_chip"] for p in cg.solve_plan(groups, **plan))
    return cg.solve_groups(groups, **kw)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_every_schedule_equals_the_solve_on_chip(precision):
    """Four LLC90 instances with two right-hand sides: CTAs, CTAs per SM, unit deals and pipeline depths."""
    G = _group(90, 4, 2)
    assert cg.solve_plan([G], precision=precision)[0]["on_chip"]
    ref = cg.solve_groups([G], precision=precision)
    assert all(r["status"] == "ok" for _, _, d in ref[0] for r in cg.diag_records(d))
    ran = 0
    for grid, cps, deal, stages in itertools.product((5, 12), (1, 2), (0, 1), (2, 3, 4)):
        kw = dict(precision=precision, grid_ctas=grid, ctas_per_sm=cps, unit_deal=deal, stages=stages)
        try:
            _same(ref, _streamed([G], **kw))
        except cg.capi.Cg2dError as e:           # a pipeline too deep for the shared memory is refused, not run
            assert e.status == cg.capi.CG2D_UNSUPPORTED, e
            continue
        ran += 1
    assert ran >= 8


def test_fp64_builds_for_one_and_two_ctas_per_sm():
    """One right-hand side and at least 8 work units per SM: ctas_per_sm 0 and 2 take the FP64 build for 2 CTAs per SM, 1
    the other one."""
    G = _group(90, 8, 1)
    assert cg.solve_plan([G])[0]["on_chip"]
    ref = cg.solve_groups([G])
    for cps in (0, 1, 2):
        _same(ref, _streamed([G], grid_ctas=8, ctas_per_sm=cps))


@pytest.mark.parametrize("order,widest", [("rowblock", 98), ("rowblock", 24), ("fortran", 98)])
def test_groups_with_different_numbers_of_right_hand_sides(order, widest):
    """Tiles of several widths (the builds for up to 96 and up to 288 points) and both numbers of right-hand sides in one
    launch: every group is its own solve on chip bit for bit, under every schedule of the autotuner."""
    groups = [_group(90, 2, 2, 40), _group(32, 3, 1, 40), _group(widest, 1, 1, 40)]
    kw = dict(sum_order=order)
    alone = []
    for G in groups:
        Gs = [G] if order == "rowblock" or len(G.b) == 1 else [
            cg.GroupSpec(G.ex, G.ops, [G.b[s]], [G.x0[s]], [G.tol[s]], [G.max_iters[s]], G.norm, x_fortran=True)
            for s in range(2)]   # (an LLC90 pair does not fit on chip in the FORTRAN order, one solve does)
        alone.append([slot for g in Gs for (slots,) in [cg.solve_groups([g], **kw)] for slot in slots])
    _same(alone, _streamed(groups, **kw))
    for cand in autotune.candidates(148) if order == "rowblock" else autotune.candidates(148)[:1]:
        try:
            _same(alone, _streamed(groups, **kw, **cand))
        except cg.capi.Cg2dError as e:
            assert e.status == cg.capi.CG2D_UNSUPPORTED, e


def test_mixed_precision_groups_of_several_sizes():
    """LLC270 and LLC90 in one mixed launch that streams: every candidate schedule gives the same bits, and every solve lies
    within 1e-11 of its FP64 solve."""
    groups = [_group(270, 1, 1, 1000), _group(90, 2, 2)]
    res = _streamed(groups, precision="mixed")
    for cand in autotune.candidates(148):
        try:
            _same(res, _streamed(groups, precision="mixed", **cand))
        except cg.capi.Cg2dError as e:
            assert e.status == cg.capi.CG2D_UNSUPPORTED, e
    for G, slots in zip(groups, res):
        (ref,) = cg.solve_groups([G], precision="f64")
        for (x, _, d), (x64, _, _) in zip(slots, ref):
            assert all(r["status"] == "ok" for r in cg.diag_records(d))
            for m in range(x.shape[0]):
                assert float((x[m] - x64[m]).abs().max() / x64[m].abs().max()) < 1e-11


def test_tiles_wider_than_288_points():
    """The generic row builds: a tile of 300 points, alone, in FP64 (LLC300 does not fit on chip) and in mixed precision (a
    CTA limit that streams, against the solve on chip)."""
    G = _group(300, 1, 1, 20)
    (ref,) = _streamed([G])
    for cps, deal in ((1, 1), (2, 0)):
        _same([ref], _streamed([G], ctas_per_sm=cps, unit_deal=deal))
    assert cg.solve_plan([G], precision="mixed")[0]["on_chip"]
    _same(cg.solve_groups([G], precision="mixed"), _streamed([G], precision="mixed", grid_ctas=20))


def test_time_limit_reports_status():
    """A grid-wide wait that can never complete (one arrival more than there are CTAs) runs out after the time limit; every
    solve reports barrier_timeout and the next solve is fine."""
    groups = [_group(8, 1, 1, 60), _group(16, 2, 2, 60)]
    ref = _streamed(groups)
    res = _streamed(groups, timeout_s=0.2, check_status=False, test_missing_arrivals=1)
    for slots in res:
        assert all(r["status"] == "barrier_timeout" for _, _, d in slots for r in cg.diag_records(d))
    _same(ref, _streamed(groups))


@pytest.mark.parametrize("checkpoint", [0, 5])
def test_exact_adjoint_from_a_streamed_forward(checkpoint):
    """The forward that records checkpoints and sums while it streams (LLC300 does not fit on chip): the gradients of the
    two-call path, whose recording forward repeats the iterations, bit for bit."""
    syn = LLCSynthetic(300)
    ops, norm = syn.operator()
    inner = cg._interior_mask(syn.L, torch.device("cuda"))
    t = [torch.as_tensor(np.ascontiguousarray(a)).cuda() for a in (*ops, syn.rhs(), syn.cotangent())]
    b, w = t[6], torch.where(inner, t[7], torch.zeros_like(t[7]))
    G = cg.GroupSpec(cg.default_exchanger(syn.L), tuple(a[None] for a in t[:6]), [b[None]], [torch.zeros_like(b)[None]],
                     [0.0], [12], float(norm))
    assert not cg.solve_plan([G])[0]["on_chip"]
    kw = dict(cg2dNorm=float(norm), tolerance=0.0, max_iters=12, checkpoint_every=checkpoint)
    args = (G.ex, tuple(t[:6]), b, torch.zeros_like(b), w)
    x1, d1, g1 = cg.exact_adjoint(*args, **kw)
    x2, d2, g2 = cg.exact_adjoint(*args, one_pass=False, **kw)
    assert d1["numIters"] == d2["numIters"] == 12
    assert torch.equal(x1, x2)
    for k in ("b",) + cg.OPS:
        assert torch.equal(g1[k], g2[k]), k
