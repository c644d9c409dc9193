"""The one-launch solve on a device it does not have to itself. A kernel of another library that keeps one
SM must delay neither the solve nor, through a launch that waits for the whole device, the work of other
streams: the iteration kernels take over, with the same bits, at the start of a solve or between the
launches of a long one."""

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
    s.set_parameters({"MAS": dict({"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0,
                                   "precision": "fp16"}, **params)})
    s.set_positions(system.positions)
    s.factorize(system.scipy())
    return s, synthetic.rhs(system.n, seed=seed)


@pytest.mark.parametrize("N", [6, 20])
def test_solve_beside_a_long_one_cta_kernel(N):
    torch = pytest.importorskip("torch")
    s, b = _factorized(N, 95)
    ref = np.zeros_like(b)
    s.solve(b, ref)
    assert s.get_info()["kernel_launches"].get("pcg_persistent", 0) == 1
    # The iteration kernels and their graphs, once (modules load with the first launch).
    second, b2 = _factorized(3, 96)
    x = np.zeros_like(b)
    solve_batch([s, second], [b, b2], [x, np.zeros_like(b2)])
    np.testing.assert_array_equal(x, ref)
    side, third = torch.cuda.Stream(), torch.cuda.Stream()
    one = torch.zeros(1, device="cuda")
    with torch.cuda.stream(third):
        one.add_(1)
    with torch.cuda.stream(side):
        torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(600_000_000)  # some 0.3 s on one SM
    ended = torch.cuda.Event()
    ended.record(side)
    time.sleep(0.005)
    held = []

    def work():
        x[:] = 0.0
        s.solve(b, x)
        held.append(ended.query())

    t = threading.Thread(target=work)
    t.start()
    with torch.cuda.stream(third):
        one.add_(1)
    third.synchronize()
    held.append(ended.query())
    t.join()
    torch.cuda.synchronize()
    assert held == [False, False], "the solve or the third stream waited for the long kernel"
    np.testing.assert_array_equal(x, ref)


@pytest.mark.parametrize("block_dim,N", [(3, 20), (2, 17), (1, 18)])
def test_long_solve_loses_its_sms_between_launches(block_dim, N):
    """More than 2,048 iterations are several launches. Matrix products of another stream fill the device
    after the first one has begun, so the second may not get its SMs."""
    torch = pytest.importorskip("torch")
    s, b = _factorized(N, 97, relative_tolerance=0.0, max_iter=2300, block_dim=block_dim, precision="fp32")
    got = []
    for graphs in (False, True):
        s.set_parameters({"MAS": {"cuda_graphs": graphs}})
        x = np.zeros_like(b)
        t = threading.Thread(target=s.solve, args=(b, x))
        m = torch.ones(4096, 4096, device="cuda")
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        t.start()
        time.sleep(0.01)
        with torch.cuda.stream(side):
            for _ in range(60):
                m @ m
        t.join()
        torch.cuda.synchronize()
        info = s.get_info()
        got.append((x, info["solver_iter"], info["solver_error"], info["solver_status"]))
        assert (info["kernel_launches"].get("pcg_persistent", 0) > 0) == graphs
        print(info["kernel_launches"])
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


def test_one_launch_off():
    """The parameter that keeps a program's other streams going beside its solves: captured iterations, the same
    bits."""
    s, b = _factorized(14, 98)
    got = []
    for on in (True, False, True):
        s.set_parameters({"MAS": {"one_launch": on}})
        x = np.zeros_like(b)
        s.solve(b, x)
        info = s.get_info()
        assert info["kernel_launches"].get("pcg_persistent", 0) == int(on)
        got.append((x, info["solver_iter"], info["solver_error"]))
    for g in got[1:]:
        np.testing.assert_array_equal(g[0], got[0][0])
        assert g[1:] == got[0][1:]
