"""MAS apply with several matrices per team of warps: the two-stage copy pipeline runs over its ring
(3 to 16 teams per CTA, 148 CTAs), with a ragged last round, for every block size. Against the CPU
oracle's apply, with test_apply_parity's tolerance (FP64, the sums only in another order)."""

from __future__ import annotations

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

from .helpers import oracle_for, oracle_to_padded, padded_to_oracle, real_to_padded_nodes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_dim,N", [(3, 31), (2, 30), (1, 29)])
def test_fp64_apply_over_several_rounds(block_dim, N):
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=60 + block_dim)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": block_dim, "precision": "fp64"}})
    if block_dim == 3:
        s.set_positions(system.positions)
    s.factorize(system.scipy())
    orc, padded = oracle_for(system, s, block_dim)
    r2p = real_to_padded_nodes(padded, orc.perm)
    nodes = s.sizes()["nodes"]
    r_real = orc.spmv(np.random.default_rng(block_dim).standard_normal(orc.s.V * block_dim))
    z = s.debug_apply(oracle_to_padded(r_real, r2p, block_dim, nodes))
    z_ref = orc.apply(r_real, storage=0)
    got = padded_to_oracle(z, r2p, block_dim)
    assert np.linalg.norm(got - z_ref) <= 1e-10 * np.linalg.norm(z_ref)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("block_dim,N", [(3, 9), (3, 41), (1, 12), (1, 58)])
def test_apply_beside_the_coarse_sums_bit_identical(block_dim, N, precision):
    """The level-0 matrices of a chained apply go ahead while the coarse levels (two to four of them)
    are summed: same bits as with every kernel after the one before, graphs or not."""
    system = synthetic.elasticity(N, young_sigma=1.0, jitter=0.2, seed=N, contact_pairs=N)
    got = []
    for chained, graphs in ((False, False), (True, False), (True, True)):
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": block_dim, "precision": precision, "chained_launch": chained,
                                  "cuda_graphs": graphs, "true_residual_period": 7, "max_iter": 40}})
        if block_dim == 3:
            s.set_positions(system.positions)
        s.factorize(system.scipy())
        x = np.zeros(system.n)
        s.solve(synthetic.rhs(system.n, seed=N), x)
        got.append((x, s.get_info()["solver_iter"], s.get_info()["solver_error"]))
    for g in got[1:]:
        np.testing.assert_array_equal(g[0], got[0][0])
        assert g[1:] == got[0][1:]
