"""Sixteen right-hand sides of bodies whose coarse sums take several CTAs, with up to four coarse levels (the
ticket of the last CTA, the levels above the second), against one-at-a-time solves with
test_multi_matches_single_solves_and_oracle's bounds."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,levels", [(3, 1), (8, 3), (20, 3), (41, 4)])
def test_wide_groups_over_several_ctas(N, levels):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=120 + N, contact_pairs=8 * N)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0,
                              "precision": "fp16", "true_residual_period": 50, "check_period": 1,
                              "rhs_group": 16}})
    s.set_positions(system.positions)
    A = system.scipy()
    s.factorize(A)
    assert s.get_info()["coarse_levels"] >= levels
    B = np.stack([synthetic.rhs(system.n, seed=120 + c) for c in range(3)])
    X = s.solve_multi(B)
    counts = s.get_info()["rhs_iterations"]
    assert all(st == "Reach relative tolerance" for st in s.get_info()["rhs_status"])
    for b, x, count in zip(B, X, counts):
        assert np.linalg.norm(A @ x - b) <= 5e-8 * np.linalg.norm(b)
        x1 = np.zeros(system.n)
        s.solve(b, x1)
        assert abs(count - s.get_info()["solver_iter"]) <= 2
        assert np.linalg.norm(x - x1) <= 1e-5 * np.linalg.norm(x1)
