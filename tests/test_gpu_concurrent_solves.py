"""The one-launch solve keeps its SMs to itself, so a solve that begins beside another one and would take more
than a quarter of them uses the iteration kernels, which overlap with the other: same bits either way."""

from __future__ import annotations

import threading
import time

import numpy as np
import pytest

from polysolve_b200 import Solver, solve_batch, synthetic

pytestmark = pytest.mark.gpu


def _factorized(N, seed, **params):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=seed)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": dict({"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0}, **params)})
    s.set_positions(system.positions)
    s.factorize(system.scipy())
    return s, synthetic.rhs(system.n, seed=seed)


def _launches(s):
    return s.get_info()["kernel_launches"].get("pcg_persistent", 0)


@pytest.mark.parametrize("other", ["solve", "solve_multi", "batch"])
@pytest.mark.parametrize("N,launches", [(6, 1), (14, 0)])
def test_small_solve_beside_another(other, N, launches):
    small, b = _factorized(N, 90)
    ref = np.zeros_like(b)
    small.solve(b, ref)
    assert _launches(small) == 1
    # A long solve: no tolerance, thousands of iterations (hundreds of milliseconds).
    never = dict(relative_tolerance=0.0, max_iter=30000, precision="fp16", cuda_graphs=True)
    large, bl = _factorized(44, 91, **never)
    second, b2 = _factorized(9, 92, max_iter=1)

    def work():
        if other == "solve":
            large.solve(bl, np.zeros_like(bl))
        elif other == "solve_multi":
            large.solve_multi(np.stack([bl, bl]))
        else:
            solve_batch([large, second], [bl, b2], [np.zeros_like(bl), np.zeros_like(b2)])

    t = threading.Thread(target=work)
    t.start()
    time.sleep(0.2)
    x = np.zeros_like(b)
    small.solve(b, x)
    assert t.is_alive(), "the long solve ended before the small one"
    beside = _launches(small)
    t.join()
    np.testing.assert_array_equal(x, ref)
    assert beside == launches
    x[:] = 0.0
    small.solve(b, x)
    np.testing.assert_array_equal(x, ref)
    assert _launches(small) == 1


def test_large_solves_beside_each_other_share_the_l2():
    """A solve that keeps part of its matrix in L2 does so alone only: of two that run at the same time one
    uses its other set of captured iterations, which is then kept beside the first."""
    pairs = [_factorized(44, 93 + k, relative_tolerance=0.0, max_iter=400, precision="fp16") for k in range(2)]
    refs = []
    for s, b in pairs:
        refs.append(np.zeros_like(b))
        s.solve(b, refs[-1])
    alone = [s.get_info()["graph_captures"] for s, _ in pairs]

    def captures_after_solving_together():
        for _ in range(4):
            start = threading.Barrier(2)
            xs = [np.zeros_like(b) for _, b in pairs]

            def work(k):
                start.wait()
                pairs[k][0].solve(pairs[k][1], xs[k])

            threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            for x, ref in zip(xs, refs):
                np.testing.assert_array_equal(x, ref)
        return [s.get_info()["graph_captures"] for s, _ in pairs]

    together = captures_after_solving_together()
    assert sum(together) > sum(alone)
    for (s, b), ref in zip(pairs, refs):
        x = np.zeros_like(b)
        s.solve(b, x)
        np.testing.assert_array_equal(x, ref)
    assert all(n <= 2 * a for n, a in zip(captures_after_solving_together(), alone))
