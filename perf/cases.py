"""The measured work of the MAS-PCG solver: what a program that links it calls, from the smallest
system to the headline 1.6 M DOF one, through the public Python mirror of the solver interface.

A case is a dict with a "kind":

* solve:    one system, factorized beforehand, solved for a right-hand side: host arrays
            (``Solver.solve``, what polysolve's callers pass) or device pointers
            (``Solver.solve_device``); block size 3 (elasticity), 2 (plane elasticity) or 1 (diffusion),
            inverses in any of the three storage precisions.
* newton:   steps of a Newton loop or time stepping: every step refactorizes new values on the same
            pattern and solves from the learned starting guess.
* contact:  steps whose contact pairs, and with them the pattern, change: a full factorization with
            the kept ordering, then a solve.
* multi:    several right-hand sides of one matrix (``Solver.solve_multi``).
* batch:    independent uneven systems solved together (``solve_batch``).
* gradient: the loss and the gradient of the warm-start network for one training sample.

Matrices are seeded synthetic meshes; right-hand sides are N(0, 1) or the sequence's smooth loads.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from polysolve_b200 import Solver, WarmStartTrainer, solve_batch, synthetic, warmstart
from polysolve_b200 import warmstart_train

TOL = 1e-8

# The reference's algorithm: FP64 inverses, true residual every 4 iterations, test every 10.
PLAIN = {"relative_tolerance": TOL, "absolute_tolerance": 0.0, "max_iter": 5000}
# The configuration the headline benchmark picks: test every iteration, true residual every 50.
CHOSEN = dict(PLAIN, true_residual_period=50, check_period=1)


def listed():
    return [
        # A body of 729 vertices with the library's defaults: a solve is launches and latency only.
        {"name": "solve8_fp64_host", "kind": "solve", "mesh": "solid", "edge": 8, "precision": "fp64",
         "chosen": False, "host": True},
        # The 27,783 DOF configuration through host arrays, as polysolve calls it.
        {"name": "solve20_fp16_host", "kind": "solve", "mesh": "solid", "edge": 20, "precision": "fp16",
         "chosen": True, "host": True},
        # A middling odd size, FP32 inverses, everything resident on the device.
        {"name": "solve37_fp32", "kind": "solve", "mesh": "solid", "edge": 37, "precision": "fp32",
         "chosen": True, "host": False},
        # The reference's algorithm (FP64 inverses) at 715 K DOF.
        {"name": "solve61_fp64", "kind": "solve", "mesh": "solid", "edge": 61, "precision": "fp64",
         "chosen": False, "host": False},
        # The headline benchmark: 1.6 M DOF, FP16 inverses, device arrays. The largest.
        {"name": "solve80_fp16", "kind": "solve", "mesh": "solid", "edge": 80, "precision": "fp16",
         "chosen": True, "host": False},
        # Heterogeneous diffusion, one unknown per vertex (the library's default block size).
        {"name": "scalar70_fp64", "kind": "solve", "mesh": "scalar", "edge": 70, "precision": "fp64",
         "chosen": False, "host": True},
        # Plane elasticity, two unknowns per vertex, a long thin ragged grid's worth of vertices.
        {"name": "plane201_fp16", "kind": "solve", "mesh": "plane", "edge": 201, "precision": "fp16",
         "chosen": True, "host": False},
        # Newton / time stepping: values-only refactorization plus a learned-start solve per step.
        {"name": "newton32_learned", "kind": "newton", "edge": 32, "steps": 4, "declared": False},
        # Contact: the pattern changes every step, so the whole factorization is repeated.
        {"name": "contact30_steps", "kind": "contact", "edge": 30, "pairs": 1500, "precision": "fp64"},
        # Sixteen load cases of one contact-coupled body (the several-right-hand-side workload).
        {"name": "multi40_rhs16", "kind": "multi", "edge": 40, "pairs": 2500, "rhs": 16},
        # Independent uneven systems, edges log-uniform (the batch workload's range, fewer of them).
        {"name": "batch16", "kind": "batch", "count": 16, "lo": 8, "hi": 32},
        # Training the warm-start network: one sample's reverse pass.
        {"name": "gradient24", "kind": "gradient", "edge": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    if u < 0.55:
        mesh = rng.choice(["solid", "solid", "solid", "scalar", "plane"])
        lo, hi = {"solid": (8, 64), "scalar": (12, 100), "plane": (24, 400)}[mesh]
        return {"kind": "solve", "mesh": mesh, "edge": _log_int(rng, lo, hi),
                "precision": rng.choice(["fp64", "fp32", "fp16", "fp16"]), "chosen": rng.random() < 0.6,
                "host": rng.random() < 0.5}
    if u < 0.68:
        return {"kind": "newton", "edge": _log_int(rng, 10, 40), "steps": rng.randint(3, 5),
                "declared": rng.random() < 0.3}
    if u < 0.78:
        edge = _log_int(rng, 10, 30)
        return {"kind": "contact", "edge": edge, "pairs": _log_int(rng, 2 * edge, edge * edge + 2 * edge),
                "precision": rng.choice(["fp64", "fp32", "fp16"])}
    if u < 0.88:
        edge = _log_int(rng, 10, 40)
        return {"kind": "multi", "edge": edge, "pairs": _log_int(rng, 2 * edge, edge * edge + 2 * edge),
                "rhs": rng.randint(2, 16)}
    if u < 0.95:
        return {"kind": "batch", "count": rng.randint(4, 24), "lo": 8, "hi": rng.randint(16, 32)}
    return {"kind": "gradient", "edge": _log_int(rng, 8, 32)}


# ---------------------------------------------------------------------------------------------
# Systems
# ---------------------------------------------------------------------------------------------

def _system(n, rows, cols, vals, xyz):
    """CSC (sorted columns and rows) from coordinate entries without duplicates."""
    order = np.argsort(cols.astype(np.int64) * n + rows)
    outer = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(np.bincount(cols, minlength=n), out=outer[1:])
    return synthetic.System(n=n, outer=outer, inner=rows[order].astype(np.int32), vals=vals[order], positions=xyz)


def _grid_edges(shape):
    """Vertex pairs of a box grid's axis edges, one (i, j) array pair per axis."""
    ids = np.arange(int(np.prod(shape))).reshape(shape)
    for ax in range(len(shape)):
        a = np.take(ids, range(shape[ax] - 1), axis=ax).ravel()
        b = np.take(ids, range(1, shape[ax]), axis=ax).ravel()
        yield a, b


def _scalar_system(edge, seed):
    """(K + M) u = f for -div(k grad u) + u / dt, k lognormal(0, 1) per grid edge, seven-point grid
    of (edge + 1)^3 vertices."""
    rng = np.random.default_rng([seed, edge, 1])
    shape = (edge + 1,) * 3
    n = int(np.prod(shape))
    rows, cols, vals, diag = [], [], [], np.full(n, 1e-3)
    for a, b in _grid_edges(shape):
        k = rng.lognormal(0.0, 1.0, a.size)
        rows += [a, b]
        cols += [b, a]
        vals += [-k, -k]
        diag += np.bincount(a, k, n) + np.bincount(b, k, n)
    rows.append(np.arange(n))
    cols.append(np.arange(n))
    vals.append(diag)
    xyz = np.stack(np.meshgrid(*[np.arange(s, dtype=np.float64) for s in shape], indexing="ij"), -1).reshape(-1, 3)
    return _system(n, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals), xyz / edge)


def _plane_system(edge, seed):
    """Springs of a triangulated (edge + 1) x (edge / 2 + 1) sheet plus a mass term: two unknowns per
    vertex, 2 x 2 blocks k n n^T along the axis and diagonal edges."""
    rng = np.random.default_rng([seed, edge, 2])
    nx, ny = edge + 1, edge // 2 + 1
    V = nx * ny
    ids = np.arange(V).reshape(nx, ny)
    pos = np.stack(np.meshgrid(np.arange(nx, dtype=np.float64), np.arange(ny, dtype=np.float64), indexing="ij"), -1)
    pos = pos.reshape(V, 2) + rng.uniform(-0.2, 0.2, (V, 2))
    a = np.concatenate([ids[:-1, :].ravel(), ids[:, :-1].ravel(), ids[:-1, :-1].ravel(), ids[:-1, 1:].ravel()])
    b = np.concatenate([ids[1:, :].ravel(), ids[:, 1:].ravel(), ids[1:, 1:].ravel(), ids[1:, :-1].ravel()])
    d = pos[b] - pos[a]
    d /= np.linalg.norm(d, axis=1)[:, None]
    k = rng.lognormal(0.0, 0.7, a.size)
    blk = k[:, None, None] * d[:, :, None] * d[:, None, :]
    diag = np.zeros((V, 2, 2))
    np.add.at(diag, a, blk)
    np.add.at(diag, b, blk)
    diag += 1e-2 * np.eye(2)
    bi = np.concatenate([a, b, np.arange(V)])
    bj = np.concatenate([b, a, np.arange(V)])
    bv = np.concatenate([-blk, -blk, diag])
    c = np.arange(2)
    rows = (2 * bi[:, None, None] + c[None, :, None] + np.zeros((1, 1, 2), dtype=np.int64)).ravel()
    cols = (2 * bj[:, None, None] + c[None, None, :] + np.zeros((1, 2, 1), dtype=np.int64)).ravel()
    return _system(2 * V, rows, cols, bv.ravel(), np.concatenate([pos, np.zeros((V, 1))], axis=1) / edge)


def _solid_system(edge, seed, pairs=0):
    return synthetic.elasticity(edge, young_sigma=1.0, jitter=0.2, seed=seed % (1 << 30), contact_pairs=pairs)


def _solve_system(case, seed):
    if case["mesh"] == "solid":
        return _solid_system(case["edge"], seed)
    return (_scalar_system if case["mesh"] == "scalar" else _plane_system)(case["edge"], seed)


def _block_dim(case):
    return {"solid": 3, "plane": 2, "scalar": 1}[case.get("mesh", "solid")]


def _sequence(case, seed):
    return [synthetic.workload_sequence60(10 + k, seed=seed % (1 << 30), N=case["edge"])
            for k in range(case["steps"])]


def _contact_systems(case, seed):
    """Two contact states of one body size: other pairs, so another pattern."""
    return [_solid_system(case["edge"], 2 * (seed % (1 << 29)) + k, case["pairs"]) for k in range(2)]


def _batch_systems(case, seed):
    edges = synthetic.batch_edges(case["count"], 0, case["lo"], case["hi"])
    return [synthetic.elasticity(N, young_sigma=0.5, seed=(seed % (1 << 24)) * 64 + k) for k, N in enumerate(edges)]


def _factorized(system, params):
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": params})
    s.set_positions(system.positions)
    s.analyze_pattern(system, system.n)
    s.factorize(system)
    return s


# ---------------------------------------------------------------------------------------------
# What a program holds before the call, and the call
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A = _solve_system(case, seed)
        params = dict(CHOSEN if case["chosen"] else PLAIN, block_dim=_block_dim(case), precision=case["precision"])
        s = _factorized(A, params)
        b = synthetic.rhs(A.n, seed)
        if case["host"]:
            return {"case": case, "solver": s, "b": b, "x": np.zeros(A.n)}
        s.set_stream(torch.cuda.current_stream().cuda_stream)
        return {"case": case, "solver": s, "b": torch.from_numpy(b).cuda(),
                "x": torch.zeros(A.n, dtype=torch.float64, device="cuda")}
    if kind == "newton":
        seq = _sequence(case, seed)
        s = _factorized(seq[0][0], dict(CHOSEN, block_dim=3, precision="fp16", initial_guess="learned"))
        s.set_warm_start_model()
        return {"case": case, "solver": s, "A": [A for A, _ in seq], "b": [b for _, b in seq],
                "x": [np.zeros(A.n) for A, _ in seq]}
    if kind == "contact":
        systems = _contact_systems(case, seed)
        # Created from JSON parameters, whose defaults keep the ordering while n stays the same.
        s = Solver.create({"solver": "MAS", "MAS": dict(PLAIN, block_dim=3, precision=case["precision"])})
        s.set_positions(systems[0].positions)
        s.analyze_pattern(systems[0], systems[0].n)
        s.factorize(systems[0])
        return {"case": case, "solver": s, "A": systems, "b": _contact_rhs(systems, seed),
                "x": [np.zeros(A.n) for A in systems]}
    if kind == "multi":
        A = _solid_system(case["edge"], seed, case["pairs"])
        s = _factorized(A, dict(CHOSEN, block_dim=3, precision="fp16"))
        return {"case": case, "solver": s, "b": synthetic.rhs(A.n, seed, case["rhs"])}
    if kind == "batch":
        systems = _batch_systems(case, seed)
        bs = _batch_rhs(systems, seed)
        return {"case": case, "solver": [_factorized(A, dict(CHOSEN, block_dim=3, precision="fp16")) for A in systems],
                "b": bs, "x": [np.zeros_like(b) for b in bs]}
    # gradient: a sample of a short sequence, history and exact solution from the solver itself, in the
    # training's own scaling
    scale = warmstart_train.SOLVE_SCALE
    s = Solver.create("MAS", "")
    s.set_parameters({"MAS": dict(warmstart_train.SOLVE_PARAMS)})
    xs = []
    for A, b in _sequence(dict(case, steps=4), seed):
        if not xs:
            s.set_positions(A.positions)
        A.vals *= scale
        b = b * scale
        s.factorize(A)
        xs.append(np.zeros(A.n))
        s.solve(b, xs[-1])
    trainer = WarmStartTrainer(warmstart.default_weights())
    return {"case": case, "solver": s, "trainer": trainer, "sample": trainer.add_sample(s, b, xs[-2::-1], xs[-1])}


def _contact_rhs(systems, seed):
    return [synthetic.rhs(A.n, 2 * seed + k) for k, A in enumerate(systems)]


def _batch_rhs(systems, seed):
    return [synthetic.rhs(A.n, 64 * seed + k) for k, A in enumerate(systems)]


def run(state):
    kind, s = state["case"]["kind"], state["solver"]
    if kind == "solve":
        b, x = state["b"], state["x"]
        if state["case"]["host"]:
            s.solve(b, x)
        else:
            s.solve_device(b.data_ptr(), x.data_ptr(), b.numel())
        return x
    if kind == "newton":
        s.reset_warm_start()
        for A, b, x in zip(state["A"], state["b"], state["x"]):
            if state["case"]["declared"]:
                s.factorize_values(A)
            else:
                s.factorize(A)
            s.solve(b, x)
        return state["x"]
    if kind == "contact":
        # The last state first: each factorization then meets another pattern than the one before.
        for A, b, x in list(zip(state["A"], state["b"], state["x"]))[::-1]:
            s.analyze_pattern(A, A.n)
            s.factorize(A)
            s.solve(b, x)
        return state["x"]
    if kind == "multi":
        return s.solve_multi(state["b"])
    if kind == "batch":
        return solve_batch(s, state["b"], state["x"])
    loss, grad = state["trainer"].gradient(state["sample"])
    return {"loss": loss, "gradient": grad}


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------

def _sizes(mesh, edge, pairs=0):
    """(vertices, nonzero blocks) of a system."""
    N = edge
    if mesh == "solid":
        V, E = (N + 1) ** 3, 7 * N ** 3 + 9 * N ** 2 + 3 * N + pairs
    elif mesh == "scalar":
        V, E = (N + 1) ** 3, 3 * N * (N + 1) ** 2
    else:
        m = N // 2
        V, E = (N + 1) * (m + 1), N * (m + 1) + (N + 1) * m + 2 * N * m
    return V, V + 2 * E


def _iterations(mesh, edge, pairs=0):
    """PCG iterations to 1e-8, fitted to this solver's counts (they vary by some percent with the
    seed); contact springs of lognormal stiffness raise them."""
    base = {"solid": 18 + 1.45 * edge, "scalar": 25 + 1.6 * edge, "plane": 30 + 1.2 * edge}[mesh]
    return base * (2.2 if pairs else 1.0)


def _solve_work(mesh, edge, precision, pairs=0, rhs=1, iterations=None):
    """One pass over the matrix (values and columns) and over the triangular subdomain inverses per
    iteration, serving all right-hand sides, and the four vectors (x, r, p and A p) read and written
    once per iteration; the right-hand sides in, the solutions out."""
    bd = {"solid": 3, "plane": 2, "scalar": 1}[mesh]
    V, nnzb = _sizes(mesh, edge, pairs)
    n, mats, N = V * bd, V / 32 * 33 / 32, 32 * bd
    it = _iterations(mesh, edge, pairs) if iterations is None else iterations
    width = {"fp64": 8, "fp32": 4, "fp16": 2}[precision]
    per_it = nnzb * (8 * bd * bd + 4) + mats * N * (N + 1) / 2 * width + 8 * 8 * n * rhs
    flops = rhs * (2 * nnzb * bd * bd + 2 * mats * N * N + 12 * n)
    return {"bytes": it * per_it + 16 * n * rhs, "flops": it * flops}


def _factorize_work(edge, precision, pairs=0):
    """The matrix in (values, rows and column pointers), its block form and the inverses out; a
    symmetric inversion of every subdomain."""
    V, nnzb = _sizes("solid", edge, pairs)
    mats, N = V / 32 * 33 / 32, 96
    width = {"fp64": 8, "fp32": 4, "fp16": 2}[precision]
    return {"bytes": nnzb * (9 * 12 + 76) + 12 * V + mats * N * (N + 1) / 2 * width, "flops": mats * N ** 3}


def _total(parts):
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    if kind == "solve":
        return _total([_solve_work(case["mesh"], case["edge"], case["precision"])])
    if kind == "newton":
        # The kept solutions halve the iterations of later steps.
        it = _iterations("solid", case["edge"])
        parts = [_factorize_work(case["edge"], "fp16")] * case["steps"]
        parts += [_solve_work("solid", case["edge"], "fp16", iterations=it * (1.0 if k == 0 else 0.7))
                  for k in range(case["steps"])]
        return _total(parts)
    if kind == "contact":
        one = [_factorize_work(case["edge"], case["precision"], case["pairs"]),
               _solve_work("solid", case["edge"], case["precision"], case["pairs"])]
        return _total(one * 2)
    if kind == "multi":
        return _total([_solve_work("solid", case["edge"], "fp16", case["pairs"], case["rhs"])])
    if kind == "batch":
        return _total([_solve_work("solid", N, "fp16")
                       for N in synthetic.batch_edges(case["count"], 0, case["lo"], case["hi"])])
    # Per vertex and layer: the 64-wide hidden states in 16 bits, read by the neighbours' messages and
    # written once, forward and backward; three 128 x 64 products, twice as many in the reverse pass.
    V, nnzb = _sizes("solid", case["edge"])
    return {"bytes": float(3 * 3 * V * 64 * 2 * 2 + 3 * nnzb * 4 + nnzb * 76),
            "flops": float(3 * 3 * V * 2 * 128 * 64 + 3 * 2 * nnzb * 2 * 64)}


# ---------------------------------------------------------------------------------------------
# The solutions in 64 bits
# ---------------------------------------------------------------------------------------------

def _direct(A, b):
    """A^-1 b by diagonally preconditioned conjugate gradients in torch float64, driven to rounding
    level and corrected twice with the recomputed residual. A is symmetric, so its CSC arrays are
    also its CSR arrays."""
    outer, inner = (torch.from_numpy(v.astype(np.int64)).cuda() for v in (A.outer, A.inner))
    vals = torch.from_numpy(A.vals).cuda()
    M = torch.sparse_csr_tensor(outer, inner, vals, size=(A.n, A.n))
    on_diagonal = inner == torch.repeat_interleave(torch.arange(A.n, device="cuda"), outer.diff())
    dinv = 1.0 / vals[on_diagonal]
    rhs = torch.from_numpy(np.ascontiguousarray(b)).cuda()
    x = torch.zeros_like(rhs)
    stop = float(rhs.norm()) * 1e-13
    for _ in range(3):
        r = rhs - M @ x
        if float(r.norm()) <= stop:
            break
        d = torch.zeros_like(x)
        z = dinv * r
        p = z.clone()
        rz = torch.dot(r, z)
        for k in range(4000):
            q = M @ p
            alpha = rz / torch.dot(p, q)
            d += alpha * p
            r -= alpha * q
            if k % 20 == 19 and float(r.norm()) <= stop:
                break
            z = dinv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        x += d
    return x.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A = _solve_system(case, seed)
        x = _direct(A, synthetic.rhs(A.n, seed))
        return x if case["host"] else torch.from_numpy(x)
    if kind == "newton":
        return [_direct(A, b) for A, b in _sequence(case, seed)]
    if kind == "contact":
        systems = _contact_systems(case, seed)
        return [_direct(A, b) for A, b in zip(systems, _contact_rhs(systems, seed))]
    if kind == "multi":
        A = _solid_system(case["edge"], seed, case["pairs"])
        return np.stack([_direct(A, b) for b in synthetic.rhs(A.n, seed, case["rhs"])])
    if kind == "batch":
        systems = _batch_systems(case, seed)
        return [_direct(A, b) for A, b in zip(systems, _batch_rhs(systems, seed))]
    return None
