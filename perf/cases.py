"""Workloads of the skeleton library, each through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a program has in hand before
the call (observations of a seeded linear-Gaussian SEM, a context, a server), ``run``
is one pass over it and returns what the pass computes. Only values that do not depend
on the order in which tests run are returned: adjacencies, the edges, potential tests
and largest degree of every level, record sizes and correlation matrices -- not which
of several separating sets was found first.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "masterthesis-heterogeneous-pc_gb300"))

import heterogpc as hg  # noqa: E402

_PRECISION = {"fp64": hg.PREC_FP64, "mixed": hg.PREC_MIXED, "tc": hg.PREC_MIXED_TC}


def listed():
    return [
        # the command line's default path on a small table: host FP64 observations in, levels
        # until exhausted, adjacency out (launch and latency bound)
        dict(name="er_p50_host", kind="skeleton", precision="mixed", source="host", dtype="f64", graph="er", degree=2.0,
             p=50, n=1000, alpha=0.01, max_level=-1, missing=0.0),
        # one problem at scale, FP32 observations resident on the device, FP64-accurate correlation
        dict(name="er_p2000_obs", kind="skeleton", precision="mixed", source="device", dtype="f32", graph="er",
             degree=4.0, p=2000, n=5000, alpha=0.01, max_level=6, missing=0.0),
        # the same shape from a correlation matrix that the caller already has
        dict(name="er_p2000_matrix", kind="matrix", precision="mixed", graph="er", degree=4.0, p=2000, n=5000,
             alpha=0.01, max_level=6),
        # gene-expression shape: hub-heavy graph, many variables, tensor-core correlation
        dict(name="pa_p9000_tc", kind="skeleton", precision="tc", source="device", dtype="f32", graph="pa", degree=2.0,
             p=9000, n=3000, alpha=0.05, max_level=3, missing=0.0),
        # the same at an ordinary, odd size, FP32 observations on the host with missing samples
        dict(name="pa_p3001_tc_host", kind="skeleton", precision="tc", source="host", dtype="f32", graph="pa",
             degree=2.0, p=3001, n=1777, alpha=0.05, max_level=3, missing=0.01),
        # all-FP64 arithmetic on a small problem
        dict(name="er_p300_fp64", kind="skeleton", precision="fp64", source="device", dtype="f64", graph="er",
             degree=3.0, p=300, n=1500, alpha=0.05, max_level=4, missing=0.0),
        # hundreds of problems of uneven sizes in one context, observations on the device
        dict(name="batch_512", kind="batch", source="device", count=512, p_lo=20, p_hi=800, n_lo=200, n_hi=8000,
             shapes=1),
        # bootstrap-sized batch end to end: observations and results in pinned host memory
        dict(name="batch_24_host", kind="batch", source="host", count=24, p_lo=20, p_hi=400, n_lo=200, n_hi=4000,
             shapes=2),
        # a burst of requests to the server, half ER and half hub-heavy
        dict(name="serve_32", kind="serve", count=32, p_lo=30, p_hi=1000, n_lo=500, n_hi=4000, alpha=0.01, max_level=4,
             shapes=3),
        # correlation matrices alone: FP64-accurate, tensor-core FP32, and allocation-free
        dict(name="corr_fp64_p1203", kind="corr", precision="mixed", dtype="f64", p=1203, n=3777, missing=0.0),
        dict(name="corr_tc_p4001", kind="corr", precision="tc", dtype="f32", p=4001, n=2999, missing=0.0),
        dict(name="corr_noalloc_p96", kind="noalloc", p=96, n=1500, missing=0.02),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "matrix", "tc", "tc", "fp64", "batch", "batch", "serve", "corr", "corr",
                       "noalloc"])
    missing = rng.choice([0.0, 0.0, 0.01])
    if kind == "mixed":
        return dict(kind="skeleton", precision="mixed", source=rng.choice(["host", "device"]),
                    dtype=rng.choice(["f32", "f64"]), graph="er", degree=round(rng.uniform(1.5, 4.0), 2),
                    p=_log_int(rng, 12, 2000), n=_log_int(rng, 300, 5000), alpha=rng.choice([0.01, 0.05]),
                    max_level=rng.choice([2, 4, 6]), missing=missing)
    if kind == "matrix":
        return dict(kind="matrix", precision=rng.choice(["mixed", "mixed", "fp64"]), graph="er",
                    degree=round(rng.uniform(1.5, 4.0), 2), p=_log_int(rng, 12, 1500), n=_log_int(rng, 300, 5000),
                    alpha=rng.choice([0.01, 0.05]), max_level=rng.choice([2, 4]))
    if kind == "tc":
        graph = rng.choice(["pa", "pa", "er"])
        return dict(kind="skeleton", precision="tc", source=rng.choice(["host", "device"]), dtype="f32", graph=graph,
                    degree=2.0 if graph == "pa" else round(rng.uniform(1.5, 4.0), 2), p=_log_int(rng, 100, 8000),
                    n=_log_int(rng, 300, 3000), alpha=rng.choice([0.01, 0.05]), max_level=rng.choice([1, 2, 3]),
                    missing=missing)
    if kind == "fp64":
        return dict(kind="skeleton", precision="fp64", source="device", dtype=rng.choice(["f32", "f64"]), graph="er",
                    degree=round(rng.uniform(1.5, 4.0), 2), p=_log_int(rng, 12, 500), n=_log_int(rng, 300, 4000),
                    alpha=rng.choice([0.01, 0.05]), max_level=rng.choice([2, 4]), missing=missing)
    if kind == "batch":
        return dict(kind="batch", source=rng.choice(["host", "device"]), count=_log_int(rng, 6, 256), p_lo=20,
                    p_hi=_log_int(rng, 100, 800), n_lo=200, n_hi=_log_int(rng, 800, 8000),
                    shapes=rng.randrange(1, 1 << 20))
    if kind == "serve":
        return dict(kind="serve", count=_log_int(rng, 4, 48), p_lo=30, p_hi=_log_int(rng, 100, 1000), n_lo=500,
                    n_hi=_log_int(rng, 1000, 4000), alpha=0.01, max_level=4, shapes=rng.randrange(1, 1 << 20))
    if kind == "corr":
        precision = rng.choice(["mixed", "tc"])
        return dict(kind="corr", precision=precision, dtype=rng.choice(["f32", "f64"]), p=_log_int(rng, 16, 4000),
                    n=_log_int(rng, 200, 5000), missing=missing)
    p = _log_int(rng, 8, 700)
    return dict(kind="noalloc", p=p, n=_log_int(rng, 100, min(20000, 4 * 1024 * 1024 // p)), missing=missing)


# ---- inputs ---------------------------------------------------------------------

def _parents_pa(rng, p, m):
    """Preferential attachment: node t takes min(m, t) distinct earlier nodes, each with
    probability proportional to its degree plus one; (parents, children)."""
    urn, src, dst = [0], [], []
    for t in range(1, p):
        chosen = set()
        while len(chosen) < min(m, t):
            chosen.add(urn[int(rng.random() * len(urn))])
        for s in chosen:
            src.append(s)
            dst.append(t)
            urn += [s, t]
        urn.append(t)
    return src, dst


def _sem(seed, graph, degree, p, n, dtype, missing=0.0):
    """Observations (p, n) of a linear-Gaussian SEM on a random DAG, on the device, each
    variable's samples contiguous; the variables in random order."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    full = torch.float64 if dtype == "f64" else torch.float32
    w_lo = 0.2 if graph == "pa" else 0.1
    W = torch.zeros((p, p), dtype=full, device="cuda")  # W[child, parent]
    if graph == "pa":
        src, dst = _parents_pa(random.Random(seed), p, 2)
        at = torch.tensor([dst, src], device="cuda")
        w = w_lo + (1.0 - w_lo) * torch.rand(at.shape[1], generator=g, device="cuda", dtype=full)
        w *= 2.0 * (torch.rand(at.shape[1], generator=g, device="cuda") < 0.5) - 1.0
        W[at[0], at[1]] = w
    else:
        u = torch.rand((p, p), generator=g, device="cuda")
        w = w_lo + (1.0 - w_lo) * torch.rand((p, p), generator=g, device="cuda", dtype=full)
        sign = 2.0 * (torch.rand((p, p), generator=g, device="cuda") < 0.5) - 1.0
        W = torch.tril((u < degree / (p - 1)) * w * sign, -1)
    E = torch.randn((p, n), generator=g, device="cuda", dtype=full)
    X = torch.linalg.solve_triangular(W.neg_(), E, upper=False, unitriangular=True)
    X = X[torch.randperm(p, generator=g, device="cuda")].contiguous()
    if missing:
        X[torch.rand((p, n), generator=g, device="cuda") < missing] = float("nan")
    return X


def _shapes(case):
    """(p, n, alpha, degree, graph) of each problem of a batch or of a served burst."""
    rng = random.Random(case["shapes"])
    out = []
    for k in range(case["count"]):
        if case["kind"] == "serve":
            out.append((_log_int(rng, case["p_lo"], case["p_hi"]), _log_int(rng, case["n_lo"], case["n_hi"]),
                        case["alpha"], 3.0, "er" if k % 2 else "pa"))
        else:
            out.append((rng.randint(case["p_lo"], case["p_hi"]), rng.randint(case["n_lo"], case["n_hi"]),
                        0.01 if k % 2 else 0.05, rng.uniform(1.0, 5.0), "er"))
    return out


def _observations(case, seed):
    return _sem(seed, case.get("graph", "er"), case.get("degree", 3.0), case["p"], case["n"], case.get("dtype", "f64"),
                case.get("missing", 0.0))


def _correlation(X):
    """FP64 correlation with missing samples skipped: the mean over the samples that are
    there, the sum of squares over n - 1, a product with a missing sample counting as 0."""
    X = X.double()
    there = ~torch.isnan(X)
    mean = torch.where(there, X, 0.0).sum(1, keepdim=True) / there.sum(1, keepdim=True)
    D = torch.where(there, X - mean, 0.0)
    Z = D / torch.sqrt((D * D).sum(1, keepdim=True) / (X.shape[1] - 1))
    return Z @ Z.T / (X.shape[1] - 1)


# ---- passes ---------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("skeleton", "corr"):
        X = _observations(case, seed)
        s["np_dtype"] = np.float64 if case["dtype"] == "f64" else np.float32
        s["X"] = X.cpu().numpy() if case.get("source") == "host" else X
        s["sk"] = hg.SkeletonCalculator(case["p"], case["n"], alpha=case.get("alpha", 0.05),
                                        max_level=case.get("max_level", 4), precision=_PRECISION[case["precision"]])
        if kind == "corr":
            s["out"] = torch.empty((case["p"], case["p"]), pin_memory=True,
                                   dtype=torch.float32 if case["precision"] == "tc" else torch.float64)
        else:
            s["out"] = torch.empty((case["p"], case["p"]), dtype=torch.uint8, pin_memory=True)
    elif kind == "matrix":
        s["C"] = _correlation(_observations(case, seed)).contiguous()
        s["sk"] = hg.SkeletonCalculator(case["p"], case["n"], alpha=case["alpha"], max_level=case["max_level"],
                                        precision=_PRECISION[case["precision"]])
        s["out"] = torch.empty((case["p"], case["p"]), dtype=torch.uint8, pin_memory=True)
    elif kind == "noalloc":
        s["X"] = _observations(case, seed)
        s["out"] = torch.empty((case["p"], case["p"]), dtype=torch.float64, device="cuda")
    elif kind == "batch":
        shapes = _shapes(case)
        b = hg.SkeletonBatch([x[0] for x in shapes], [x[1] for x in shapes], [x[2] for x in shapes], max_level=-1,
                             precision=hg.PREC_MIXED_TC)
        X = torch.empty(int(b.obs_off[-1]), dtype=torch.float32, device="cuda")
        for k, (p, n, _, degree, graph) in enumerate(shapes):
            X[int(b.obs_off[k]):int(b.obs_off[k + 1])] = _sem(seed * 1000 + k, graph, degree, p, n, "f32").view(-1)
        s["batch"] = b
        s["X"] = torch.empty(X.shape, dtype=X.dtype, pin_memory=True).copy_(X) if case["source"] == "host" else X
        s["bits"] = torch.empty(int(b.adjacency_words()[-1]), dtype=torch.int32, pin_memory=True)
        if case["source"] == "host":
            # 8 words hold a record of levels 1 and 2, where nearly all of them fall, and at least half of the
            # pairs are removed at level 0, which writes none
            s["records"] = torch.empty(4 * sum(x[0] * x[0] // 2 for x in shapes), dtype=torch.int32, pin_memory=True)
    elif kind == "serve":
        s["server"] = hg.SkeletonServer(max_level=case["max_level"])
        s["X"] = [_sem(seed * 1000 + k, graph, degree, p, n, "f32").cpu().numpy()
                  for k, (p, n, _, degree, graph) in enumerate(_shapes(case))]
        s["alpha"] = [x[2] for x in _shapes(case)]
    torch.cuda.synchronize()  # the library's streams are its own
    return s


def _levels(stats):
    out = np.zeros((hg.HPC_MAX_LEVEL + 1, 3), np.int64)  # levels not run: zeros
    for k, st in enumerate(stats):
        out[k] = st["edges_after"], st["potential_tests"], st["max_degree"]
    return out


def _check(status):
    if status != 0:
        raise hg.HpcError(status, hg.lib().hpc_last_error_string().decode())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "skeleton":
        sk, X = state["sk"], state["X"]
        if case["source"] == "host":
            sk.add_observations(X)
        else:
            sk.add_observations_device(X.data_ptr(), state["np_dtype"])
        stats = sk.run()
        sk.adjacency_into(state["out"].data_ptr())
        return {"adjacency": state["out"], "levels": _levels(stats)}
    if kind == "matrix":
        sk = state["sk"]
        sk.add_correlation_matrix_device(state["C"].data_ptr())
        stats = sk.run()
        sk.adjacency_into(state["out"].data_ptr())
        return {"adjacency": state["out"], "levels": _levels(stats)}
    if kind == "corr":
        sk, out = state["sk"], C.c_void_p(state["out"].data_ptr())
        sk.add_observations_device(state["X"].data_ptr(), state["np_dtype"])
        if case["precision"] == "tc":
            _check(hg.lib().hpc_get_correlation_f32(sk.handle, out))
        else:
            _check(hg.lib().hpc_get_correlation(sk.handle, out))
        return {"correlation": state["out"]}
    if kind == "noalloc":
        _check(hg.lib().hpc_correlation_noalloc_f64(C.c_void_p(state["X"].data_ptr()), case["n"], case["p"], 0,
                                                    C.c_void_p(state["out"].data_ptr()),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"correlation": state["out"]}
    if kind == "batch":
        b = state["batch"]
        if case["source"] == "host":
            b.add_observations_ptr(state["X"].data_ptr(), np.float32)
        else:
            b.add_observations_device(state["X"].data_ptr(), np.float32)
        stats = b.run()
        b.adjacency_bits_into(state["bits"].data_ptr(), state["bits"].numel())
        out = {"bits": state["bits"], "levels": _levels(stats)}
        if case["source"] == "host":
            out["record_words"] = b.records_packed_into(state["records"].data_ptr(), state["records"].numel())
        return out
    sv = state["server"]
    for X, alpha in zip(state["X"], state["alpha"]):
        sv.submit(X, alpha, want_adjacency=True)
    sv.drain()
    done = sorted(sv.poll(), key=lambda r: r["id"])
    return {"adjacency": [r["adjacency"] for r in done], "edges": np.array([r["edges"] for r in done], np.int64),
            "status": np.array([r["status"] for r in done], np.int64)}


def work(case):
    """Observations (or the matrix) read once, results written once; the operations of the
    correlation and one test of every pair. How many further tests a skeleton needs is
    known only from its data."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        shapes = [(p, n) for p, n, _, _, _ in _shapes(case)]
        out = sum(p * ((p + 31) // 32) * 4 if kind == "batch" else p * p for p, _ in shapes)
        return {"bytes": sum(4 * p * n for p, n in shapes) + out, "flops": sum(n * p * (p + 1) + 4 * p * p for p, n in shapes)}
    p, n = case["p"], case["n"]
    if kind == "matrix":
        return {"bytes": 9 * p * p, "flops": 4 * p * p}
    size = 4 if case.get("dtype") == "f32" else 8
    if kind == "skeleton":
        return {"bytes": size * n * p + p * p, "flops": n * p * (p + 1) + 4 * p * p}
    return {"bytes": size * n * p + (4 if case.get("precision") == "tc" else 8) * p * p, "flops": n * p * (p + 1)}


def exact(case, seed):
    if case["kind"] in ("corr", "noalloc"):
        return {"correlation": _correlation(_observations(case, seed))}
    return None  # adjacencies and counts: whole numbers
