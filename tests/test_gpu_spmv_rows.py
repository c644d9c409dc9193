"""Scalar SpMV with several slots per trip: rows of every length around a trip (one entry to
several trips and a remainder) against one slot at a time, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

from polysolve_b200 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40, 331])
def test_scalar_rows_of_every_length(n):
    rng = np.random.default_rng(n)
    A = sp.lil_matrix((n, n))
    for i in range(n):
        for j in rng.choice(n, size=min(n, i % 19), replace=False):
            A[i, j] = A[j, i] = rng.standard_normal() * 0.1
    A = sp.csc_matrix(A)
    A.setdiag(np.abs(A).sum(axis=0).A1 + 1.0)
    A.sort_indices()
    b = rng.standard_normal(n)
    got = []
    for unroll in (1, 2, 4):
        s = Solver.create("MAS", "")
        s.set_parameters({"MAS": {"block_dim": 1, "precision": "fp64", "spmv_unroll": unroll, "cuda_graphs": False,
                                  "relative_tolerance": 1e-12, "true_residual_period": 2}})
        s.factorize(A)
        x = np.zeros(n)
        s.solve(b, x)
        got.append(x)
    assert np.linalg.norm(A @ got[0] - b) <= 1e-9 * np.linalg.norm(b)
    for x in got[1:]:
        np.testing.assert_array_equal(got[0], x)
