"""The work that users of this framework have it do, as cases that can be timed.

Kinds of case (each through the package's public entry points):

  cugal     ``cugal()`` from two networkx graphs to the host P and the mapping: the drop-in call
  align     ``align()`` on device-resident graphs: the same alignment inside a GPU program
  log       ``SinkhornState.solve``, log domain, FP32 or BF16/FP16 stream: one optimal-transport solve
  standard  ``SinkhornState.solve``, scaling form (the reference's default method)
  plan      ``sinkhorn_plan`` forward and backward (implicit adjoint): a differentiable layer
  unrolled  ``sinkhorn_plan_unrolled`` forward and backward (the reference's iteration, checkpointed)
  dropin    one Frank-Wolfe step as the reference's own Python runs it on the ``cuda_kernels`` functions
  assign    exact rounding of a quasi-permutation (HungarianMethod.SCIPY)
  graph     CSR build and node features of a graph pair

Sizes, graph families, regularizations and schedules are those of the repository's workloads
(``cugal_b200/synthetic.py``: Newman-Watts-Strogatz 1000 and 4096, power-law 8192 and 65536,
Erdos-Renyi of mean degree 16) and odd sizes in between.
"""

import math

import numpy as np
import torch

from cugal_b200 import Config, HungarianMethod, SinkhornMethod, cugal
from cugal_b200 import cuda_kernels
from cugal_b200.adjacency import Adjacency
from cugal_b200.autograd import sinkhorn_plan, sinkhorn_plan_unrolled
from cugal_b200.exact_lap import exact_assign
from cugal_b200.feature_extraction import Features
from cugal_b200.pred import align
from cugal_b200.sinkhorn import SinkhornState
from cugal_b200.synthetic import Workload, noisy_permuted_copy, source_graph

DEVICE = "cuda"
STREAMS = {"fp32": None, "bf16": torch.bfloat16, "fp16": torch.float16}
L2_BYTES = 126e6


def listed():
    return [
        # a small alignment end to end: 150 Frank-Wolfe steps whose solves converge in a few sweeps,
        # so launches, host work and synchronisations are what a user waits for
        {"name": "cugal_er1000_fp32", "kind": "cugal", "n": 1000, "stream": "fp32", "steps": 10, "blocks": 15},
        # a large alignment in its fast mode (the 32768-node workload at half its size)
        {"name": "align_er16384_bf16", "kind": "align", "n": 16384, "stream": "bf16", "steps": 10, "blocks": 15},
        # the 1000-node workload's solve: runs to the 500-iteration cap, a few microseconds of work each
        {"name": "log_nws1000_fp32", "kind": "log", "n": 1000, "graph": "nws", "stream": "fp32", "reg": 1e-3,
         "share": 0.0, "iterations": 500},
        # the 8192-node workload's solve (FP32 drop-in), every solve capped
        {"name": "log_power8192_fp32", "kind": "log", "n": 8192, "graph": "power", "stream": "fp32", "reg": 1e-3,
         "share": 0.1, "iterations": 500},
        # FP16 stream at a size the L2 holds, ragged rows
        {"name": "log_nws4099_fp16", "kind": "log", "n": 4099, "graph": "nws", "stream": "fp16", "reg": 1e-2,
         "share": 0.0, "iterations": 500},
        # BF16 stream at a size only HBM holds, ragged rows
        {"name": "log_er20011_bf16", "kind": "log", "n": 20011, "graph": "er", "stream": "bf16", "reg": 1e-2,
         "share": 0.1, "iterations": 300},
        # the reference's default method at its experiments' regularization
        {"name": "standard_power6000", "kind": "standard", "n": 6000, "graph": "power", "reg": 0.3,
         "share": 0.1, "iterations": 300},
        # the 4096-node differentiation workload: plan and its gradient
        {"name": "plan_nws4096", "kind": "plan", "n": 4096, "graph": "nws", "reg": 0.1, "mu": 0.2,
         "share": 0.02, "iterations": 500},
        # gradient through the iteration itself
        {"name": "unrolled_nws1024", "kind": "unrolled", "n": 1024, "graph": "nws", "reg": 0.3, "mu": 0.2,
         "share": 0.1, "iterations": 60},
        # a cuGAL user who keeps cuGAL's Python and swaps the native module
        {"name": "dropin_power8192", "kind": "dropin", "n": 8192, "graph": "power", "reg": 0.05, "iterations": 10,
         "lam": 2},
        # exact rounding of a quasi-permutation
        {"name": "assign_4096", "kind": "assign", "n": 4096},
        # graphs of the largest workload: CSR and features, a few hundred microseconds
        {"name": "graph_power65536", "kind": "graph", "n": 65536, "graph": "power", "degree": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cugal", "align", "log", "log", "log", "standard", "plan", "unrolled", "dropin", "assign",
                       "graph"])
    graph = rng.choice(["nws", "er", "power"])
    if kind == "cugal":
        return {"kind": kind, "n": _log_int(rng, 300, 2000), "stream": rng.choice(list(STREAMS)), "steps": 10,
                "blocks": rng.choice([5, 10, 15])}
    if kind == "align":
        return {"kind": kind, "n": _log_int(rng, 3000, 14000), "stream": rng.choice(list(STREAMS)), "steps": 10,
                "blocks": rng.choice([5, 10])}
    if kind == "log":
        return {"kind": kind, "n": _log_int(rng, 200, 20000), "graph": graph, "stream": rng.choice(list(STREAMS)),
                "reg": rng.choice([1e-3, 1e-2, 0.05, 0.3]), "share": rng.choice([0.0, 0.1, 0.5]),
                "iterations": rng.choice([100, 200, 300])}
    if kind == "standard":
        return {"kind": kind, "n": _log_int(rng, 300, 12000), "graph": graph, "reg": rng.choice([0.3, 1.0]),
                "share": rng.choice([0.1, 0.5]), "iterations": rng.choice([100, 200, 300])}
    if kind == "plan":
        # the plans a gradient is taken through are diffuse: an almost integral one has almost none
        graph = rng.choice(["nws", "er"])
        return {"kind": kind, "n": _log_int(rng, 200, 4096), "graph": graph, "mu": 0.2, "iterations": 500,
                "reg": rng.choice([0.1, 0.3] if graph == "nws" else [0.3, 1.0]),
                "share": rng.choice([0.0, 0.02] if graph == "nws" else [0.0])}
    if kind == "unrolled":
        return {"kind": kind, "n": _log_int(rng, 200, 2500), "graph": graph, "reg": rng.choice([0.3, 1.0]), "mu": 0.2,
                "share": rng.choice([0.0, 0.1]), "iterations": rng.choice([20, 60])}
    if kind == "dropin":
        return {"kind": kind, "n": _log_int(rng, 500, 12000), "graph": graph, "reg": rng.choice([0.05, 0.3]),
                "iterations": rng.choice([5, 10, 20]), "lam": rng.choice([0, 1, 5])}
    if kind == "assign":
        return {"kind": kind, "n": _log_int(rng, 300, 6000)}
    return {"kind": "graph", "n": _log_int(rng, 2000, 100000), "graph": graph, "degree": rng.choice([8, 12, 16, 24])}


# ------------------------------------------------------------------ inputs


def _edges(graph, n, degree, rng):
    """n degree / 2 undirected edges (m, 2) without loops or repeats: ring with shortcuts (nws), uniform
    pairs (er), pairs with one end drawn by power-law weights (power)."""
    m = n * degree // 2
    if graph == "nws":
        k = max(1, degree // 2 - 1)
        i = np.repeat(np.arange(n), k)
        e = np.concatenate([np.stack([i, (i + np.tile(np.arange(1, k + 1), n)) % n], 1),
                            rng.integers(0, n, size=(2 * (m - n * k), 2))])
    else:
        e = rng.integers(0, n, size=(m + m // 2, 2))
        if graph == "power":
            w = np.cumsum(1.0 / np.sqrt(np.arange(1, n + 1)))
            e[:, 0] = np.searchsorted(w, rng.random(len(e)) * w[-1]).clip(0, n - 1)
    return _simple(e, m, rng)


def _simple(e, m, rng):
    """m of the distinct pairs of e."""
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    return e[np.sort(rng.permutation(len(e))[:m])]


def _pair(graph, n, degree, seed, noise=0.02):
    """(source edges, target edges, perm): the target is the source relabelled, with edges exchanged."""
    rng = np.random.default_rng(seed)
    e = _edges(graph, n, degree, rng)
    perm = rng.permutation(n)
    k = max(1, int(noise * len(e) / 2))
    t = np.concatenate([perm[e[rng.permutation(len(e))[k:]]], rng.integers(0, n, size=(k, 2))])
    return e, _simple(t, len(e) - k, rng), perm


def _directed(e):
    """Both directions of every edge, as a device int32 (2m, 2) tensor."""
    both = np.concatenate([e, e[:, ::-1]]).astype(np.int32)
    return torch.from_numpy(np.ascontiguousarray(both)).to(DEVICE)


def _sparse(e, n, dtype):
    d = torch.from_numpy(np.concatenate([e, e[:, ::-1]]).T.copy()).to(DEVICE)
    return torch.sparse_coo_tensor(d, torch.ones(d.shape[1], dtype=dtype, device=DEVICE), (n, n)).coalesce()


def _node_features(e, n, mu):
    """[degree, mean neighbour degree, mean of that, log degree] x mu (n x 4, FP32)."""
    S = _sparse(e, n, torch.float32)
    deg = torch.sparse.mm(S, torch.ones(n, 1, device=DEVICE))
    inv = 1.0 / deg.clamp(min=1.0)
    f2 = torch.sparse.mm(S, deg) * inv
    f3 = torch.sparse.mm(S, f2) * inv
    return (mu * torch.cat([deg, f2, f3, torch.log1p(deg)], 1)).contiguous()


def _cost(case, seed):
    """A Frank-Wolfe gradient on the way to the planted match: mu D - 2 A P B with
    P = (1 - share) / n + share Pi (share 0: the first step)."""
    share = case.get("share", 0.5)
    n = case["n"]
    e, t, perm = _pair(case["graph"], n, 12, seed)
    fs, ft = _node_features(e, n, 1.0), _node_features(t, n, 1.0)
    C = case.get("mu", 1.0) * torch.cdist(fs, ft, compute_mode="donot_use_mm_for_euclid_dist")
    if share:
        Bd = _sparse(t, n, torch.float32).to_dense()
        C -= torch.sparse.mm(_sparse(e, n, torch.float32), Bd[torch.from_numpy(perm).to(DEVICE)]) * (2 * share)
        del Bd
    C -= fs[:, :1] * ft[:, 0] * (2 * (1 - share) / n)
    return C.contiguous()


def _config(case, **more):
    kw = dict(device=DEVICE, dtype=torch.float32, mu=1.0, sinkhorn_method=SinkhornMethod.LOG,
              sinkhorn_regularization=case.get("reg", 1e-3), sinkhorn_iterations=case.get("iterations", 500),
              sinkhorn_threshold=1e-4, sinkhorn_eval_freq=10, use_sparse_adjacency=True,
              iter_count=case.get("blocks", 15), frank_wolfe_iter_count=case.get("steps", 10),
              hungarian_method=HungarianMethod.DOUBLE_GREEDY, stream_dtype=STREAMS[case.get("stream", "fp32")])
    kw.update(more)
    return Config(**kw)


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _host_pair(case, seed):
    w = Workload("er", "er", case["n"], seed, 0.02, case["blocks"], "DOUBLE_GREEDY", (16.0,))
    src = source_graph(w)
    k = int(0.01 * src.number_of_edges())
    return (src,) + noisy_permuted_copy(src, np.random.default_rng(seed), k, k)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "cugal":
        src, tgt, _ = _host_pair(case, seed)
        return {"kind": kind, "source": src, "target": tgt, "config": _config(case)}
    if kind == "align":
        e, t, _ = _pair("er", n, 16, seed)
        return {"kind": kind, "A": Adjacency.from_edges(_directed(e), n), "B": Adjacency.from_edges(_directed(t), n),
                "config": _config(case)}
    if kind == "log":
        return {"kind": kind, "C": _cost(case, seed), "config": _config(case)}
    if kind == "standard":
        # the reference's experiments scale the cost into the range exp(-C/reg) can hold
        C = _cost(case, seed)
        C = (C - C.min()) * (10.0 / float(C.max() - C.min()))
        return {"kind": kind, "C": C, "config": _config(case, sinkhorn_method=SinkhornMethod.STANDARD)}
    if kind in ("plan", "unrolled"):
        W = torch.randn((n, n), generator=_generator(seed), device=DEVICE)
        return {"kind": kind, "C": _cost(case, seed).requires_grad_(True), "W": W, "config": _config(case)}
    if kind == "dropin":
        e, t, perm = _pair(case["graph"], n, 12, seed)
        P = torch.full((n, n), 0.5 / n, device=DEVICE)
        P[torch.arange(n, device=DEVICE), torch.from_numpy(perm).to(DEVICE)] += 0.5
        return {"kind": kind, "A": Adjacency.from_edges(_directed(e), n), "B": Adjacency.from_edges(_directed(t), n),
                "fs": _node_features(e, n, 1.0), "ft": _node_features(t, n, 1.0), "P": P, "lam": case["lam"],
                "reg": case["reg"], "iterations": case["iterations"]}
    if kind == "assign":
        # rows split over up to three columns, as an unfinished Frank-Wolfe plan leaves them, on a faint floor
        g = _generator(seed)
        P = torch.rand((n, n), generator=g, device=DEVICE) * (1e-3 / n)
        w = torch.rand((n, 3), generator=g, device=DEVICE) ** 3
        w = w / w.sum(1, keepdim=True)
        rows = torch.arange(n, device=DEVICE)
        for k in range(3):
            P[rows, torch.randperm(n, generator=g, device=DEVICE)] += w[:, k]
        return {"kind": kind, "P": P}
    e, t, _ = _pair(case["graph"], n, case["degree"], seed)
    return {"kind": kind, "n": n, "source": _directed(e), "target": _directed(t), "config": _config(case)}


def _dropin_step(s):
    """One Frank-Wolfe step as cuGAL's Python writes it (gradient, fixed number of log-Sinkhorn
    iterations, update), on the functions of its native module."""
    A, B, P = s["A"], s["B"], s["P"]
    AP = torch.empty_like(P)
    cuda_kernels.adjacency_matmul(A.col_indices, A.row_pointers, P, AP, True)
    APt = AP.T
    G = torch.empty_like(APt)
    cuda_kernels.adjacency_matmul(B.col_indices, B.row_pointers, APt, G, False)
    G = G.T * 2
    cuda_kernels.add_distance(s["fs"], s["ft"], G)
    cuda_kernels.regularize(G, P, s["lam"])
    K = -G / s["reg"]
    Kt = K.T.contiguous()
    u = torch.zeros(K.shape[0], device=K.device)
    v = torch.zeros_like(u)
    for _ in range(s["iterations"]):
        cuda_kernels.sinkhorn_log_step(Kt, u, v, 1.0)
        cuda_kernels.sinkhorn_log_step(K, v, u, 1.0)
    error = cuda_kernels.sinkhorn_log_marginal(Kt, v, u)
    gap = cuda_kernels.update_quasi_permutation_log(P, K, u, v, 0.5, s["reg"])
    return {"P": P, "gradient": G, "u": u, "v": v, "gap": np.float32(gap), "error": np.float32(error)}


def run(s):
    kind = s["kind"]
    if kind == "cugal":
        P, mapping = cugal(s["source"], s["target"], s["config"])
        return {"P": P, "columns": np.array([c for _, c in mapping])}
    if kind == "align":
        P, columns, _ = align(s["A"], s["B"], s["config"])
        return {"P": P, "columns": columns}
    if kind in ("log", "standard"):
        C, config = s["C"], s["config"]
        K, u, v = SinkhornState(C.shape[0], config).solve(C, config)
        if kind == "standard":
            return {"K": K, "u": u, "v": v}
        # one array: log-domain duals are defined up to a constant that moves from one to the other
        return {"K": K, "duals": torch.stack([u, v])}
    if kind == "plan":
        P = sinkhorn_plan(s["C"], s["config"])
        (dC,) = torch.autograd.grad(P, s["C"], s["W"])
        return {"P": P.detach(), "dC": dC}
    if kind == "unrolled":
        P = sinkhorn_plan_unrolled(s["C"], s["config"])
        (dC,) = torch.autograd.grad(P, s["C"], s["W"])
        return {"P": P.detach(), "dC": dC}
    if kind == "dropin":
        return _dropin_step(s)
    if kind == "assign":
        columns, steps, status = exact_assign(s["P"])
        return {"columns": columns, "steps": steps, "status": status}
    A = Adjacency.from_edges(s["source"], s["n"])
    B = Adjacency.from_edges(s["target"], s["n"])
    f = Features.create(A, B, s["config"])
    return {"columns": [A.col_indices, B.col_indices], "rows": [A.row_pointers, B.row_pointers], "source": f.source,
            "target": f.target}


def work(case):
    """What one pass cannot do without: inputs read and outputs written once; a matrix larger than the
    L2 is also read once per iteration of its solve (n^2 multiply, add, exponential and add each)."""
    kind, n = case["kind"], case["n"]
    n2 = float(n) * n
    if kind in ("cugal", "align"):
        steps = case["steps"] * case["blocks"]
        b = 4 if case["stream"] == "fp32" else 2
        sweeps = 11  # iterations of a converged solve
        stream = sweeps * n2 * b if n2 * b > L2_BYTES else 0.0
        # per step: the kept A P B and P read, the cost written and read, P written
        return {"bytes": steps * (n2 * (8 + 4 + 4 + 4 + 4) + stream), "flops": steps * n2 * (4 * sweeps + 30)}
    if kind == "log":
        b = 4 if case["stream"] == "fp32" else 2
        stream = case["iterations"] * n2 * b if n2 * b > L2_BYTES else 0.0
        return {"bytes": n2 * 8 + stream, "flops": case["iterations"] * n2 * 5}
    if kind == "standard":
        stream = case["iterations"] * n2 * 4 if n2 * 4 > L2_BYTES else 0.0
        return {"bytes": n2 * 8 + stream, "flops": case["iterations"] * n2 * 4}
    if kind == "plan":
        return {"bytes": n2 * 16, "flops": case["iterations"] * n2 * 5 + 50 * n2 * 4}
    if kind == "unrolled":
        return {"bytes": n2 * 16, "flops": case["iterations"] * n2 * (5 + 10)}
    if kind == "dropin":
        stream = 2 * case["iterations"] * n2 * 4 if n2 * 4 > L2_BYTES else 0.0
        return {"bytes": n2 * 4 * 12 + stream, "flops": n2 * (4 * 12 + 2 * case["iterations"] * 5)}
    if kind == "assign":
        return {"bytes": n2 * 4, "flops": n2 * 4}
    m = float(n) * case["degree"]
    return {"bytes": 2 * (m * 8 + m * 4 + n * (4 + 16)), "flops": 2 * m * case["degree"]}


# ------------------------------------------------------------------ the same in 64 bits


def _log_solve(K, iterations, threshold, freq, u=None, v=None):
    """log-domain Sinkhorn in FP64 with the column-marginal stopping rule."""
    u = torch.zeros(K.shape[0], dtype=torch.float64, device=K.device) if u is None else u
    v = torch.zeros_like(u) if v is None else v
    for t in range(iterations):
        v = -torch.logsumexp(K + u[:, None], 0)
        X = K + v[None, :]
        u = -torch.logsumexp(X, 1)
        if threshold is not None and t % freq == 0 and t != 0:
            if float((torch.exp(X + u[:, None]).sum(0) - 1).abs().sum().detach()) < threshold:
                break
    return u, v


def _standard_solve(K, iterations, threshold, freq):
    n = K.shape[0]
    u = torch.full((n,), 1.0 / n, dtype=torch.float64, device=K.device)
    v = u.clone()
    for t in range(iterations):
        v = 1.0 / (u @ K + 1e-16)
        u = 1.0 / (K @ v + 1e-16)
        if t % freq == 0 and float(((u @ K) * v - 1).abs().sum()) < threshold:
            break
    return u, v


def _dense64(e, n):
    return _sparse(e, n, torch.float64).to_dense()


def _fugal_features(M):
    deg = M.sum(1)
    tri = ((M @ M) * M).sum(1)
    clust = torch.where(deg > 1, tri / (deg * (deg - 1)).clamp(min=1), torch.zeros_like(deg))
    inv = 1.0 / deg.clamp(min=1)
    return torch.stack([deg, clust, (M @ deg) * inv, (M @ clust) * inv], 1)


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "cugal" and n <= 1500:
        src, tgt, _ = _host_pair(case, seed)
        A, B = (_dense64(np.array(list(g.edges())), n) for g in (src, tgt))
        D = torch.cdist(_fugal_features(A), _fugal_features(B), compute_mode="donot_use_mm_for_euclid_dist")
        P = torch.full((n, n), 1.0 / n, dtype=torch.float64, device=DEVICE)
        u = v = None
        for lam in range(case["blocks"]):
            for it in range(1, case["steps"] + 1):
                K = -(-2 * A @ P @ B + D + lam * (1 - 2 * P)) / 1e-3
                u, v = _log_solve(K, 500, 1e-4, 10, u, v)
                P = P + 2.0 / (2.0 + it) * (torch.exp(K + u[:, None] + v[None, :]) - P)
        return {"P": P, "columns": None}
    if kind == "log" and n <= 12000:
        K = -_cost(case, seed).double() / case["reg"]
        return {"K": K, "duals": torch.stack(_log_solve(K, case["iterations"], 1e-4, 10))}
    if kind == "standard" and n <= 12000:
        C = prepare(case, seed)["C"].double()
        K = torch.exp(-C / case["reg"])
        u, v = _standard_solve(K, case["iterations"], 1e-4, 10)
        return {"K": K, "u": u, "v": v}
    if kind == "plan" and n <= 4096:
        s = prepare(case, seed)
        K = -s["C"].detach().double() / case["reg"]
        u, v = _log_solve(K, 500, 1e-4, 10)
        P = torch.exp(K + u[:, None] + v[None, :])
        GP = s["W"].double() * P
        a, b = GP.sum(1), GP.sum(0)
        # (I - P^T P) y = b - P^T a by conjugate gradients off the constant vector, which dC does not see
        # (and on which the system of a plan with rounded column sums is not consistent); x = a - P y
        def apart(z):
            return z - z.mean()
        y = torch.zeros_like(b)
        r = apart(b - P.T @ a)
        d, rs, small = r.clone(), r @ r, 1e-24 * (b @ b)
        for _ in range(3000):
            if rs <= small:
                break
            q = apart(d - P.T @ (P @ d))
            alpha = rs / (d @ q)
            y += alpha * d
            r -= alpha * q
            rs, old = r @ r, rs
            d = r + (rs / old) * d
        x = a - P @ y
        return {"P": P, "dC": -(P * (s["W"].double() - x[:, None] - y[None, :])) / case["reg"]}
    if kind == "unrolled" and n <= 2048 and case["iterations"] * n * n <= 8e7:
        s = prepare(case, seed)
        C = s["C"].detach().double().requires_grad_(True)
        K = -C / case["reg"]
        u, v = _log_solve(K, case["iterations"], 1e-4, 10)
        P = torch.exp(K + u[:, None] + v[None, :])
        (dC,) = torch.autograd.grad(P, C, s["W"].double())
        return {"P": P.detach(), "dC": dC}
    if kind == "dropin" and n <= 12000:
        s = prepare(case, seed)
        e, t, _ = _pair(case["graph"], n, 12, seed)
        P = s["P"].double()
        AP = torch.sparse.mm(_sparse(e, n, torch.float64), P)
        G = -2 * torch.sparse.mm(_sparse(t, n, torch.float64), AP.T.contiguous()).T
        del AP
        G += torch.cdist(s["fs"].double(), s["ft"].double(), compute_mode="donot_use_mm_for_euclid_dist")
        G += case["lam"] * (1 - 2 * P)
        K = -G / case["reg"]
        u, v = _log_solve(K, case["iterations"], None, 10)
        q = torch.exp(K + u[:, None] + v[None, :])
        error = float((q.sum(0) - 1).abs().sum())
        d = q - P
        return {"P": P + 0.5 * d, "gradient": G, "u": u, "v": v, "gap": np.float64(abs(float((d * G).sum()))),
                "error": np.float64(error)}
    return None
