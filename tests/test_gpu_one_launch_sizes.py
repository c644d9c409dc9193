"""The one-launch solve of large systems of block sizes 1 and 2, bit for bit against the iteration kernels:
several items per team (more banks than teams in the grid), inverses through the ring, FP32 storage without a
natural ordering. Every one of them has to take the one launch; isolated rows (the fixed vertices) are
in all."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

pytestmark = pytest.mark.gpu

CASES = [
    # (block_dim, N, precision, banks at least)
    (1, 20, "fp32", 860),
    (1, 29, "fp64", 2500),
    (1, 36, "fp32", 4700),
    (1, 36, "fp16", 4700),
    (1, 37, "fp16", 5100),
    (2, 19, "fp32", 370),
    (2, 31, "fp64", 1500),
    (2, 34, "fp32", 2000),
    (2, 35, "fp16", 2100),
]


@pytest.mark.parametrize("block_dim,N,precision,banks", CASES)
def test_large_one_launch_solve_bit_identical(block_dim, N, precision, banks):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=110 + N)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": block_dim, "precision": precision, "relative_tolerance": 1e-8,
                              "absolute_tolerance": 0.0, "max_iter": 45, "true_residual_period": 20,
                              "check_period": 1}})
    s.factorize(system.scipy())
    assert s.get_info()["banks"] >= banks
    b = synthetic.rhs(system.n, seed=N)
    got = []
    for graphs in (False, True):
        s.set_parameters({"MAS": {"cuda_graphs": graphs}})
        x = np.zeros(system.n)
        s.solve(b, x)
        info = s.get_info()
        assert (info["kernel_launches"].get("pcg_persistent", 0) > 0) == graphs
        got.append((x, info["solver_iter"], info["solver_error"], info["solver_status"]))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
