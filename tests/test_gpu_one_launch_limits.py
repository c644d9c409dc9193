"""Where one launch ends and the iteration kernels begin: a system of as many banks as the line allows solves in
one launch, one more bank takes the faster iteration kernels, and the bits are the same either way."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from polysolve_b200 import Solver

pytestmark = pytest.mark.gpu


def _chain(banks, block_dim):
    """A chain of 32 * banks vertices: tridiagonal blocks, positive definite."""
    V = banks * 32
    T = sp.diags([-np.ones(V - 1), np.full(V, 2.25), -np.ones(V - 1)], [-1, 0, 1])
    B = np.eye(block_dim) + 0.25 * np.ones((block_dim, block_dim))
    return sp.csc_matrix(sp.kron(T, B))


@pytest.mark.parametrize("block_dim,precision,line", [(3, "fp32", 1776), (2, "fp64", 1776), (2, "fp32", 2220),
                                                      (1, "fp32", 4930)])
def test_one_launch_up_to_the_line(block_dim, precision, line):
    for banks, launches in ((line, 1), (line + 1, 0)):
        A = _chain(banks, block_dim)
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": block_dim, "precision": precision, "ordering": "natural",
                                  "relative_tolerance": 1e-10, "absolute_tolerance": 0.0, "check_period": 1,
                                  "max_iter": 60}})
        s.factorize(A)
        assert s.get_info()["banks"] == banks
        b = np.random.default_rng(banks).standard_normal(A.shape[0])
        got = []
        for graphs in (False, True):
            s.set_parameters({"MAS": {"cuda_graphs": graphs}})
            x = np.zeros(A.shape[0])
            s.solve(b, x)
            info = s.get_info()
            assert info["kernel_launches"].get("pcg_persistent", 0) == (launches if graphs else 0)
            got.append((x, info["solver_iter"], info["solver_error"]))
        np.testing.assert_array_equal(got[0][0], got[1][0])
        assert got[0][1:] == got[1][1:]
