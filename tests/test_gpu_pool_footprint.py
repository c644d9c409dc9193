"""Device memory of many small handles: their factorizations share one pool, so a handle takes about its buffers
and not a pool's smallest enlargement (32 MB); everything is given back with the handles."""

from __future__ import annotations

import gc

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

pytestmark = pytest.mark.gpu

COUNT = 24


def test_small_handles_take_little_and_give_it_back():
    torch = pytest.importorskip("torch")
    system = synthetic.elasticity(8, young_sigma=1.0, jitter=0.2, seed=130)
    b = synthetic.rhs(system.n, seed=130)

    def handle():
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0}})
        s.set_positions(system.positions)
        s.factorize(system.scipy())
        x = np.zeros(system.n)
        s.solve(b, x)
        return s, x

    def free():
        gc.collect()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    # Once before, for what the driver keeps itself (modules, a stream per handle).
    handles = [handle() for _ in range(COUNT)]
    ref = handles[0][1]
    del handles
    before = free()
    handles = [handle() for _ in range(COUNT)]
    taken = before - free()
    assert all(np.array_equal(x, ref) for _, x in handles)
    # Buffers of some 6 MB each, and the temporaries of one factorization.
    assert taken <= COUNT * (12 << 20) + (64 << 20), taken >> 20
    del handles
    assert free() >= before
