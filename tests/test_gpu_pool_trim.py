"""Memory that the handles' pool holds unused is not missing to others: an allocation of the library that
fails gives it back to the device first. The failure is injected on the host, so it is final here;
what counts is the memory that is free afterwards."""

from __future__ import annotations

import gc

import numpy as np
import pytest

from polysolve_b200 import CudaOutOfMemoryError, Solver, synthetic
from polysolve_b200.solver import debug_fail_allocation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("failing", ["factorize", "solve_multi"])
def test_failed_allocation_trims_the_pool(failing):
    torch = pytest.importorskip("torch")

    def handle(N, factorize=True):
        system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=80 + N)
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": 3, "precision": "fp16", "relative_tolerance": 1e-8,
                                  "absolute_tolerance": 0.0}})
        s.set_positions(system.positions)
        if factorize:
            s.factorize(system.scipy())
        return s, system

    kept, system = handle(10)
    # A larger handle comes and goes: the pool, which lives on with the other one, keeps some of its memory.
    large, _ = handle(30)
    del large
    third, other = handle(10, factorize=False)
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    debug_fail_allocation(0)
    try:
        with pytest.raises(CudaOutOfMemoryError):
            if failing == "factorize":  # inside the pool
                third.factorize(other.scipy())
            else:  # outside
                kept.solve_multi(synthetic.rhs(system.n, seed=80, count=4))
    finally:
        debug_fail_allocation(-1)
    assert torch.cuda.mem_get_info()[0] > before
    A, b, x = system.scipy(), synthetic.rhs(system.n, seed=81), np.zeros(system.n)
    for s in (kept, third):
        s.factorize(A)
        x[:] = 0.0
        s.solve(b, x)
        assert np.linalg.norm(A @ x - b) <= 2e-8 * np.linalg.norm(b)
