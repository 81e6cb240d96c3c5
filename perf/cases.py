"""The measured cases: what programs that use this framework have it do.

Products of a resident H-matrix with one vector (device and host buffers), with 8 to
64 vectors (CUDA cores, tensor cores on stored operands, tensor cores on operands
split on chip), kernel-ridge solves, and construction (one set, and many small sets in
the same launches), over the point sets, kernels, tolerances and storage types of the
repository's own workloads.

A case is a dict of plain values: `kind` names the call, the other keys its sizes and
options.  Outputs are the product or solution vectors, whole; `exact` gives the FP64
direct sum over the kernel matrix (or the dense solve) in plain torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import hmglib_b200 as hmg

_PREC = {"fp64": hmg.PREC_FP64, "fp32": hmg.PREC_FP32, "mixed": hmg.PREC_MIXED}
_TC = {"bf16": hmg.PREC_BF16, "bf16x6": hmg.PREC_BF16X6, "onchip": hmg.PREC_BF16X6_ONCHIP}

# Uniform 3D points, Matern-3/2 rho 0.2, leaf 128, eps 1e-8: the batching workload.
_MATERN = dict(points="uniform", dim=3, kernel="matern32", param=0.2, leaf=128, rule="min", eps=1e-8, k=96)
# The same kernel as the serving loop compresses it: leaf 64, eps 1e-4.
_SERVE = dict(_MATERN, leaf=64, eps=1e-4)
# Gaussian mixture in 2D, Gaussian length^2 0.05, eps 1e-6: the precision workload.
_GMM = dict(points="gmm", dim=2, kernel="gaussian", param=0.05, leaf=64, rule="min", eps=1e-6, k=64)
# The reference's own arithmetic and parameters: uniform 2D, exp(-r^2/0.1), max rule,
# fixed rank 64, FP64 factors and near field.
_PLAIN = dict(points="uniform", dim=2, kernel="gaussian", param=0.1, leaf=64, rule="max", eps=0.0, k=64, prec="fp64")
# One set of the many-matrix workload: Gaussian, eps 1e-5, FP32 factors.
_SET2D = dict(points="uniform", dim=2, kernel="gaussian", param=0.05, leaf=64, rule="min", eps=1e-5, k=64, prec="fp32")


def listed():
    return [
        # the smallest sets of the many-matrix workload, one at a time: latency and launches
        dict(_SET2D, name="product small 2D", kind="product", n=1000),
        # a program written for the reference: FP64, fixed rank
        dict(_PLAIN, name="product fp64 fixed rank", kind="product", n=16384),
        # the headline product, at a size of which several matrices are resident
        dict(_MATERN, name="product mixed 3D", kind="product", n=262144, prec="mixed"),
        # a host program (C, or numpy) that hands in x and takes y back on every call
        dict(_SERVE, name="product host buffers", kind="host", n=65001, prec="fp32"),
        # the serving loop's product batches: a few requests on one matrix
        dict(_MATERN, name="multi 8 mixed 3D", kind="multi", n=131072, prec="mixed", nrhs=8),
        # 32 right-hand sides on clustered points
        dict(_GMM, name="multi 32 fp32 clustered 2D", kind="multi", n=262139, prec="fp32", nrhs=32),
        # a full batch at FP32 accuracy, no operand copy
        dict(_MATERN, name="multi 64 on chip 3D", kind="tc", n=65536, prec="mixed", nrhs=64, tc="onchip"),
        # batched products where BF16 accuracy is enough
        dict(_MATERN, name="multi 32 bf16 3D", kind="tc", n=100003, prec="fp32", nrhs=32, tc="bf16"),
        # 8 kernel-ridge solves sharing their products, as the serving loop runs them
        dict(_SERVE, name="solve 8 mixed 3D", kind="solve", n=32768, prec="mixed", nrhs=8, tol=1e-4),
        # compress and multiply once, as a program written for the reference does
        dict(_PLAIN, name="build fp64 fixed rank", kind="build", n=16384),
        # a new point set of the headline kind: cluster, compress, multiply once
        dict(_MATERN, name="build mixed 3D", kind="build", n=131071, prec="mixed"),
        # many independent small sets, clustered, compressed and multiplied once each
        dict(name="build 48 small sets", kind="group", count=48, lo=10.0, hi=14.0, eps=1e-5, k=64, prec="fp32"),
    ]


def _size(rng, lo, hi):
    """Log-uniform, odd half of the time."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng: random.Random):
    pick = rng.choice(["product", "product", "host", "multi", "multi", "tc", "solve", "build", "build", "group"])
    if pick == "group":
        return dict(kind="group", count=rng.randint(4, 48), lo=10.0, hi=rng.uniform(11.0, 14.0), eps=1e-5, k=64, prec="fp32")
    if pick == "solve":
        return dict(_SERVE, kind="solve", n=_size(rng, 4096, 32768), prec=rng.choice(["mixed", "fp32"]), nrhs=rng.randint(2, 12),
                    tol=1e-4)
    if pick == "tc":
        tc = rng.choice(["bf16", "bf16x6", "onchip"])
        return dict(_MATERN, kind="tc", n=_size(rng, 8192, 65536), prec=rng.choice(["mixed", "fp32"]) if tc == "onchip" else "fp32",
                    nrhs=rng.randint(17, 64), tc=tc)
    base = rng.choice([_MATERN, _SERVE, _GMM, _SET2D, _PLAIN])
    if base is _PLAIN:
        c = dict(base, n=_size(rng, 1024, 16384), k=rng.choice([16, 32, 64]))
    elif base is _SET2D:
        c = dict(base, n=_size(rng, 1024, 65536))
    else:
        c = dict(base, n=_size(rng, 4096, 131072), prec=rng.choice(["mixed", "mixed", "fp32", "fp64"]))
    c["kind"] = pick
    if pick == "multi":
        c["nrhs"] = rng.randint(2, 40)
        c["n"] = min(c["n"], 65536) if c["prec"] == "fp64" else c["n"]
    return c


# ---- inputs -----------------------------------------------------------------------


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _points(case, seed, n=None, dim=None):
    """(dim, n) FP64 coordinates: uniform in the unit box, or 16 Gaussian clusters."""
    dev = _device()
    n, dim = n or case["n"], dim or case["dim"]
    g = _generator(2 * seed + 1, dev)
    if case.get("points", "uniform") == "uniform":
        return torch.rand(dim, n, dtype=torch.float64, device=dev, generator=g)
    mean = torch.rand(16, dim, dtype=torch.float64, device=dev, generator=g)
    std = 0.02 + 0.08 * torch.rand(16, dtype=torch.float64, device=dev, generator=g)
    comp = torch.randint(16, (n,), device=dev, generator=g)
    z = torch.randn(n, dim, dtype=torch.float64, device=dev, generator=g)
    return (mean[comp] + std[comp, None] * z).T.contiguous()


def _vectors(seed, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=_device(), generator=_generator(2 * seed, _device())) * 2.0 - 1.0


def _sets(case, seed):
    """The point sets of a group: sizes 2^U[lo, hi] (the case's own), alternating 2D and 3D, length^2 U[0.01, 0.2]."""
    sizes, r = random.Random(case["count"]), random.Random(int(seed))
    out = []
    for i in range(case["count"]):
        n = int(round(2.0 ** sizes.uniform(case["lo"], case["hi"])))
        l2 = r.uniform(0.01, 0.2)
        out.append((_points({}, seed * 1000 + i, n, 2 if i % 2 == 0 else 3), l2))
    return out


def _kind(case):
    return hmg.KERNEL_GAUSSIAN if case["kernel"] == "gaussian" else hmg.KERNEL_MATERN32


def _build(case, p):
    n = p.shape[1]
    H = hmg.HMatrix(n, n, case["dim"])
    H.set_points(0, p)
    H.set_points(1, p)
    H.setup(1.5, case["leaf"], rule=hmg.ADMISSIBLE_MIN if case["rule"] == "min" else hmg.ADMISSIBLE_MAX)
    H.set_kernel(_kind(case), case["param"], 0.0)
    H.precompute_aca(case["k"], case["eps"], _PREC[case["prec"]])
    H.precompute_dense(_PREC[case["prec"]])
    return H


def _build_group(case, sets):
    hs = []
    for p, l2 in sets:
        H = hmg.HMatrix(p.shape[1], p.shape[1], p.shape[0])
        H.set_points(0, p)
        H.set_points(1, p)
        H.set_kernel(hmg.KERNEL_GAUSSIAN, l2, 0.0)
        hs.append(H)
    G = hmg.group_setup(hs, 1.5, [64 if p.shape[0] == 2 else 128 for p, _ in sets], rule=hmg.ADMISSIBLE_MIN)
    for H in hs:
        H.close()
    G.precompute_aca(case["k"], case["eps"], _PREC[case["prec"]])
    G.precompute_dense(_PREC[case["prec"]])
    return G


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "group":
        s["sets"] = _sets(case, seed)
        n = sum(p.shape[1] for p, _ in s["sets"])
        s["x"], s["y"] = _vectors(seed, n), torch.zeros(n, dtype=torch.float64, device="cuda")
        return s
    n = case["n"]
    p = _points(case, seed)
    if kind == "build":
        s["p"], s["x"], s["y"] = p, _vectors(seed, n), torch.zeros(n, dtype=torch.float64, device="cuda")
        return s
    s["H"] = _build(case, p)
    if kind == "tc":
        s["H"].build_bf16_factors(near=_TC[case["tc"]])
    if kind == "product":
        s["x"], s["y"] = _vectors(seed, n), torch.zeros(n, dtype=torch.float64, device="cuda")
    elif kind == "host":
        s["x"] = _vectors(seed, n).cpu().numpy()
    else:
        s["X"] = _vectors(seed, case["nrhs"], n)
        s["Y"] = torch.zeros_like(s["X"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "product":
        return s["H"].matvec(s["x"], s["y"])
    if kind == "host":
        return s["H"].matvec(s["x"])
    if kind in ("multi", "tc"):
        return s["H"].matvec_multi(s["X"], s["Y"])
    if kind == "solve":
        s["Y"].zero_()  # the initial guess
        s["H"].cg_solve_multi(s["X"], s["Y"], 1e-3 * case["n"], tol=case["tol"], maxit=300, refine=True)
        return s["Y"]
    with (_build(case, s["p"]) if kind == "build" else _build_group(case, s["sets"])) as H:
        return H.matvec(s["x"], s["y"])


# ---- what a pass cannot do without ------------------------------------------------


def work(case):
    """Bytes and operations of one pass.

    Products: the stored H-matrix (or tensor-core operands) and the vectors once; two
    operations per stored entry and vector.  Solves: that for 10 iterations.
    Construction: points in, factors and near field out; of operations, the kernel
    entries of the factors' rows and columns and of the near field (20 each) and the
    factors' residuals, 2 (m1 + m2) r^2 / 2 per block at the mean rank.
    """
    s = prepare(case if case["kind"] != "tc" else dict(case, kind="multi"), 1)
    kind, nrhs = case["kind"], case.get("nrhs", 1)
    H = s.get("H") or (_build(case, s["p"]) if kind == "build" else _build_group(case, s["sets"]))
    i = H.info()
    H.close()
    n, entries = i["n1"], i["near_entries"] + i["far_entries"]
    stored = i["matvec_bytes"] - 16 * n
    if kind in ("build", "group"):
        rank = i["far_entries"] / max(1, i["far_rows"])
        return {"bytes": float(stored + 32 * n), "flops": float(20 * entries + i["far_entries"] * rank)}
    if kind == "tc" and case["tc"] != "onchip":
        stored = entries * 2 * (3 if case["tc"] == "bf16x6" else 1)
    passes = 10 if kind == "solve" else 1
    return {"bytes": float(passes * (stored + 16 * n * nrhs)), "flops": float(passes * 2 * entries * nrhs)}


# ---- the same in 64 bits ----------------------------------------------------------


def _kernel_rows(p, kernel, param, a, b):
    d2 = torch.zeros(b - a, p.shape[1], dtype=torch.float64, device=p.device)
    for c in p:
        t = c[a:b, None] - c[None, :]
        d2.addcmul_(t, t)
    if kernel == "gaussian":
        return d2.mul_(-1.0 / param).exp_()
    r = d2.sqrt_().mul_(math.sqrt(3.0) / param)
    return (-r).exp_().mul_(r.add_(1.0))


def _direct(p, kernel, param, X):
    """K X for X of shape (nrhs, n)."""
    n = p.shape[1]
    out = torch.empty_like(X)
    step = max(1, (1 << 28) // n)
    for a in range(0, n, step):
        b = min(n, a + step)
        out[:, a:b] = X @ _kernel_rows(p, kernel, param, a, b).T
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "group":
        sets = _sets(case, seed)
        x = _vectors(seed, sum(p.shape[1] for p, _ in sets))
        parts, at = [], 0
        for p, l2 in sets:
            n = p.shape[1]
            parts.append(_direct(p, "gaussian", l2, x[None, at:at + n])[0])
            at += n
        return torch.cat(parts)
    p = _points(case, seed)
    n = case["n"]
    if kind in ("product", "host", "build"):
        y = _direct(p, case["kernel"], case["param"], _vectors(seed, 1, n))[0]
        return y.cpu().numpy() if kind == "host" else y
    X = _vectors(seed, case["nrhs"], n)
    if kind != "solve":
        return _direct(p, case["kernel"], case["param"], X)
    K = _kernel_rows(p, case["kernel"], case["param"], 0, n)
    K.diagonal().add_(1e-3 * n)
    L = torch.linalg.cholesky(K)
    del K
    return torch.cholesky_solve(X.T.contiguous(), L).T.contiguous()
