"""Products of mas_spmv_dot_noalloc on a stream of the caller's, or in a graph, against the release of the
matrix they read: a factorization of another pattern and the destruction of the handle must wait for
them. A delay on the caller's stream keeps the product from starting before the release is called."""

from __future__ import annotations

import gc

import numpy as np
import pytest

from polysolve_b200 import Solver, synthetic

pytestmark = pytest.mark.gpu

DELAY_CYCLES = 100_000_000  # some 50 ms


@pytest.mark.parametrize("release", ["factorize", "destroy"])
@pytest.mark.parametrize("captured", [False, True])
def test_product_in_flight_reads_its_own_matrix(release, captured):
    torch = pytest.importorskip("torch")
    system = synthetic.elasticity(9, young_sigma=1.0, jitter=0.2, seed=70)
    other = synthetic.elasticity(9, young_sigma=1.0, jitter=0.2, seed=71, contact_pairs=40)
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": {"block_dim": 3}})
    s.set_positions(system.positions)
    s.factorize(system.scipy())
    length = s.sizes()["nodes"] * 3
    x = np.random.default_rng(70).standard_normal(length)
    y_ref = s.debug_spmv(x)
    dx = torch.from_numpy(x).cuda()
    dy, dd = torch.empty_like(dx), torch.empty(1, dtype=torch.float64, device="cuda")

    def product():
        s.spmv_dot_noalloc(dx.data_ptr(), dy.data_ptr(), dd.data_ptr(), length,
                           torch.cuda.current_stream().cuda_stream)

    product()  # (the first call looks up its scratch)
    torch.cuda.synchronize()
    graph = None
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            product()
    dy.fill_(np.nan)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(DELAY_CYCLES)
        if captured:
            graph.replay()
        else:
            product()
    if release == "factorize":
        s.factorize(other.scipy())
    else:
        del s, product
        gc.collect()
    side.synchronize()
    y = dy.cpu().numpy()
    assert np.linalg.norm(y - y_ref) <= 1e-12 * np.linalg.norm(y_ref)
    del graph
