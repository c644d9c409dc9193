"""A handle's captured iterations are kept for its solves alone and for those in batches (what stays in L2
differs between the two): alternating captures nothing anew."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import Solver, solve_batch, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_dim,N", [(3, 41), (1, 58)])
def test_alternating_solve_and_batch_keeps_the_graphs(block_dim, N):
    pairs = []
    for k in range(2):  # more banks than a one-launch solve takes
        system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=100 + k)
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": block_dim, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0,
                                  "precision": "fp16", "max_iter": 25}})
        if block_dim == 3:
            s.set_positions(system.positions)
        s.factorize(system.scipy())
        pairs.append((s, synthetic.rhs(system.n, seed=k)))
    refs = []
    for s, b in pairs:
        refs.append(np.zeros_like(b))
        s.solve(b, refs[-1])
    captures = None
    for _ in range(4):
        xs = [np.zeros_like(b) for _, b in pairs]
        solve_batch([s for s, _ in pairs], [b for _, b in pairs], xs)
        for (s, b), x, ref in zip(pairs, xs, refs):
            np.testing.assert_array_equal(x, ref)
            x[:] = 0.0
            s.solve(b, x)
            np.testing.assert_array_equal(x, ref)
        now = [s.get_info()["graph_captures"] for s, _ in pairs]
        assert min(now) >= 1 and (captures is None or now == captures)
        captures = now
