"""Grid barriers of the one-launch solve that run out. ``device_wait_limit`` bounds them as it bounds every
other device-side wait (a poll of the barrier takes some 0.5 us, so a limit of one poll runs out in
any grid of several CTAs). A CTA that gave up must never be lost: the solve either reports the timeout or
its result is the right one, bit for bit, and the handle works again afterwards."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import MasError, Solver, synthetic
from polysolve_b200.solver import MAS_ERR_TIMEOUT

pytestmark = pytest.mark.gpu

DEFAULT_LIMIT = 1 << 20


@pytest.mark.parametrize("N,precision", [(9, "fp64"), (20, "fp16"), (30, "fp64")])
def test_barrier_timeout_is_reported(N, precision):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=53)
    b = synthetic.rhs(system.n, seed=53)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0,
                              "precision": precision}})
    s.set_positions(system.positions)
    s.factorize(system.scipy())
    ref = np.zeros(system.n)
    s.solve(b, ref)
    assert s.get_info()["kernel_launches"].get("pcg_persistent", 0) == 1
    for limit in (1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 64, DEFAULT_LIMIT):
        s.set_parameters({"MAS": {"device_wait_limit": limit}})
        x = np.zeros(system.n)
        timed_out = False
        try:
            s.solve(b, x)
        except MasError as e:
            assert e.code == MAS_ERR_TIMEOUT and "timed out" in str(e)
            timed_out = True
        assert timed_out or limit > 1
        if timed_out:
            assert limit < DEFAULT_LIMIT
        else:
            np.testing.assert_array_equal(x, ref)
