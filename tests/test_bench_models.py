"""The byte models behind bench.py's roofline figures: the per-solve 12-word model (56 B per point-iteration in
mixed precision, 96 B in FP64, 96 B per replacement), and the bytes it counts twice when an instance's two solves
share one staging of the coefficients. No GPU."""

import bench


def _d(iters, rep=0):
    return {"numIters": iters, "replacements": rep}


def test_algorithmic_bytes_per_solve():
    n = bench.N_LLC90
    f, a = [_d(240, 9), _d(230, 9)], [_d(241, 9), _d(250, 10)]
    want = n * ((240 + 230 + 241 + 250) * 56 + (9 + 9 + 9 + 10) * 96)
    assert bench.algorithmic_bytes(f, a, "mixed") == want
    assert bench.algorithmic_bytes([_d(230)], [_d(225)], "f64") == n * (230 + 225) * 96


def test_shared_coefficients_counted_while_both_solves_iterate():
    n = bench.N_LLC90
    f, a = [_d(240), _d(230)], [_d(241), _d(250)]
    assert bench.shared_coefficient_bytes(f, a, "mixed") == n * 24 * (240 + 230)
    assert bench.shared_coefficient_bytes(f, a, "f64") == n * 48 * (240 + 230)
    # counted once, an instance-iteration with both solves moves 88 B in mixed precision (24 B of coefficients
    # and 32 B per solve), against the model's 2 x 56
    both = bench.algorithmic_bytes([_d(100)], [_d(100)], "mixed") - bench.shared_coefficient_bytes(
        [_d(100)], [_d(100)], "mixed")
    assert both == n * 100 * 88


def _plan(*launches, on_chip=True):
    return [{"launch": n, "on_chip": on_chip, "teams": 1, "ctas_per_team": 1} for n in launches]


def test_roofline_and_launches_follow_the_route():
    """A solve on chip is held against the shared memory (60 B a point-iteration of a right-hand side in mixed precision, 120
    B in FP64) with the streaming kernel's bytes beside it; a streamed one against HBM. The launch counts are the plan's."""
    n = bench.N_LLC90
    assert bench.on_chip_bytes([240, 230], n, "mixed") == n * 470 * 60
    assert bench.on_chip_bytes([1], 10, "f64") == 1200
    r = bench.solver_roofline(_plan(0), 4e9, 2e9, 1.0, 148, 1965.0, None)
    assert r["bound"] == "shared memory" and r["kernel"] == "cg2d_team" and r["achieved"] == 2000.0
    assert abs(r["peak"] - 148 * 128 * 1.965) < 1e-6 and r["streamed_model"]["bytes"] == 4e9
    assert bench.solver_roofline(_plan(0, 0), 4e9, 2e9, 1.0, 148, 1965.0, None)["kernel"] == "cg2d_team_groups"
    r = bench.solver_roofline(_plan(0, 0, on_chip=False), 4e9, 2e9, 1.0, 148, 1965.0, 5)
    assert r["bound"] == "hbm" and r["achieved"] == 4000.0 and r["traffic"] == 5 and r["peak"] == bench.measured_peak()[0]
    assert [bench.solver_launches(p) for p in (_plan(0), _plan(0, 0, 1), _plan(0, on_chip=False),
                                               _plan(0, 0, on_chip=False))] == [1, 2, 2, 3]
    assert bench.exact_launches(30, 30, 2) == bench.exact_launches(30, 30) + 1
