"""The one-launch solve of small systems against the iteration kernels (``cuda_graphs`` off launches
them from the host): the same iterates, bit for bit, so solution, iteration count, residual norm
and status must be equal. Sizes from one bank to the largest that fit (several items per CTA, matrix
rows partly outside shared memory), every block size and storage, true-residual schedules,
isolated rows, starting guesses, and solves longer than one launch."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

pytestmark = pytest.mark.gpu

CASES = [
    # (block_dim, N, precision, parameters)
    (3, 2, "fp64", {}),  # one bank
    (3, 3, "fp16", {"check_period": 1, "true_residual_period": 50}),  # two banks
    (3, 9, "fp32", {"use_preconditioned_residual_norm": True}),
    (3, 9, "fp64", {"max_iter": 1}),
    (3, 9, "fp64", {"max_iter": 7, "true_residual_period": 3, "check_period": 2}),
    (3, 14, "fp16", {"apply_items_per_warp": 4, "true_residual_period": 1}),
    (3, 20, "fp64", {}),
    (3, 24, "fp32", {"true_residual_period": 5, "ordering": "graph"}),
    (3, 33, "fp16", {"check_period": 1, "true_residual_period": 50}),
    # inverses through the ring of bulk copies: two or three per batch, one per batch
    (3, 38, "fp16", {"check_period": 1, "true_residual_period": 50, "max_iter": 45}),
    (3, 36, "fp32", {"check_period": 1, "max_iter": 45}),
    (3, 30, "fp64", {"check_period": 1, "max_iter": 45}),
    (2, 6, "fp64", {}),
    (2, 19, "fp32", {"ordering": "natural"}),
    (2, 22, "fp16", {"check_period": 1}),
    (1, 6, "fp16", {}),
    (1, 17, "fp64", {"check_period": 3}),
    (1, 20, "fp32", {"ordering": "natural"}),
    (3, 6, "fp64", {"relative_tolerance": 0.0, "max_iter": 2300}),  # two launches, stalls at rounding
]


@pytest.mark.parametrize("block_dim,N,precision,extra", CASES)
def test_one_launch_solve_bit_identical_to_iteration_kernels(block_dim, N, precision, extra):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=N, contact_pairs=N)
    params = {"block_dim": block_dim, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0, "precision": precision,
              "max_iter": 400}
    params.update(extra)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": params})
    if block_dim == 3:
        s.set_positions(system.positions)
    s.factorize(system.scipy())
    b = synthetic.rhs(system.n, seed=N)
    for guess in ("zero", "input"):
        got = []
        for graphs in (False, True):
            s.set_parameters({"MAS": {"cuda_graphs": graphs, "initial_guess": guess}})
            x = np.full(system.n, 0.25)
            s.solve(b, x)
            info = s.get_info()
            used = info["kernel_launches"].get("pcg_persistent", 0)
            # (A natural ordering can leave a bank in many components, more coarse nodes than fit: then
            # the iteration kernels run in both.)
            assert (used > 0) == graphs or (graphs and extra.get("ordering") == "natural"), info["kernel_launches"]
            got.append((x, info["solver_iter"], info["solver_error"], info["solver_status"]))
        np.testing.assert_array_equal(got[0][0], got[1][0])
        assert got[0][1:] == got[1][1:]


def test_one_launch_solve_nonfinite_and_zero_right_hand_sides():
    """A NaN in b is reported as before; b = 0 gives x = 0 as the iteration kernels do."""
    from polysolve_b200 import MasError

    system = synthetic.elasticity(8, young_sigma=1.0, jitter=0.2, seed=4)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": 3}})
    s.set_positions(system.positions)
    s.factorize(system.scipy())
    b = synthetic.rhs(system.n, seed=4)
    b[5] = np.nan
    with pytest.raises(MasError):
        s.solve(b, np.zeros(system.n))
    got = []
    for graphs in (False, True):
        s.set_parameters({"MAS": {"cuda_graphs": graphs}})
        x = np.ones(system.n)
        s.solve(np.zeros(system.n), x)
        got.append((x, s.get_info()["solver_iter"], s.get_info()["solver_status"]))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


def test_one_launch_solves_from_several_threads():
    """Handles solved from several host threads at once give the bits of solves one after another."""
    import threading

    solvers, bs, refs = [], [], []
    for k, N in enumerate((5, 9, 14, 18)):
        system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=30 + k)
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": 3, "relative_tolerance": 1e-8, "absolute_tolerance": 0.0}})
        s.set_positions(system.positions)
        s.factorize(system.scipy())
        b = synthetic.rhs(system.n, seed=k)
        x = np.zeros(system.n)
        s.solve(b, x)
        solvers.append(s)
        bs.append(b)
        refs.append(x)
    bad = []

    def work(k):
        for _ in range(6):
            x = np.zeros_like(bs[k])
            solvers[k].solve(bs[k], x)
            if not np.array_equal(x, refs[k]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(solvers))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
