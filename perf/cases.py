"""Performance cases: the calls a user of this framework makes, at the sizes,
types and options they are made with.

One case is one call of a public entry point (or, for the serving loop, one
burst of requests through the server's handle).  Inputs are the framework's own
seeded workloads (superman_b200/workloads.py): U[0,1) real matrices, blocks of
Haar-random unitaries, Bernoulli(0.5) 0/1 matrices with the identity OR-ed in,
and sparse permutation-plus-k patterns.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import superman_b200 as spb
from superman_b200 import _lib, serving
from superman_b200 import workloads as W


def listed():
    return [
        # A single small permanent: a latency-bound library call.
        {"name": "dense_n13_fp64", "kind": "dense", "n": 13, "precision": "fp64"},
        # The plain dense configuration, checked against exact values: n=24.
        {"name": "dense_n24_dd", "kind": "dense", "n": 24, "precision": "dd"},
        # An odd mid-range size in the default precision.
        {"name": "dense_n29_fp64", "kind": "dense", "n": 29, "precision": "fp64"},
        # The headline configuration: n=32 at <= 1e-12 relative error.
        {"name": "dense_n32_dd", "kind": "dense", "n": 32, "precision": "dd"},
        # Boson-sampling amplitudes: blocks of a Haar-random unitary, small ...
        {"name": "complex_n19_fp64", "kind": "complex", "n": 19, "precision": "fp64"},
        # ... at the configured size, refined ...
        {"name": "complex_n28_dd", "kind": "complex", "n": 28, "precision": "dd"},
        # ... and where FP32 products are accurate enough for the caller.
        {"name": "complex_n27_fp32", "kind": "complex", "n": 27, "precision": "fp32"},
        # Exact count of perfect matchings of a dense bipartite graph.
        {"name": "binary_n36", "kind": "binary", "n": 36},
        # A sparse matrix through the whole pipeline (pruning, components,
        # decomposition, drivers).
        {"name": "sparse_n40_pipeline_dd", "kind": "pipeline", "n": 40, "extra": 3, "precision": "dd"},
        # Many small permanents at once from device memory.
        {"name": "batch_n20_real", "kind": "batch", "n": 20, "count": 4096, "complex": False},
        # A sampling estimate beyond the exact paths' n <= 63.
        {"name": "approx_n100", "kind": "approx", "n": 100, "extra": 3, "samples": 1 << 20},
        # A burst of mixed requests to the serving loop, half real, half complex.
        {"name": "serve_n8_24", "kind": "serve", "n_lo": 8, "n_hi": 24, "count": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "complex", "complex", "binary", "sparse", "pipeline", "batch", "batch",
                       "approx", "serve"])
    if kind == "dense":
        return {"kind": kind, "n": rng.randint(4, 32), "precision": rng.choice(["fp64", "dd"])}
    if kind == "complex":
        p = rng.choice(["fp64", "dd", "dd", "fp32"])
        return {"kind": kind, "n": rng.randint(12 if p == "fp32" else 4, 30), "precision": p}
    if kind == "binary":
        return {"kind": kind, "n": rng.randint(6, 35)}
    if kind == "sparse":
        return {"kind": kind, "n": rng.randint(20, 34), "extra": rng.randint(2, 4),
                "precision": rng.choice(["fp64", "dd"])}
    if kind == "pipeline":
        return {"kind": kind, "n": rng.randint(20, 40), "extra": rng.randint(2, 3),
                "precision": rng.choice(["fp64", "dd"])}
    if kind == "batch":
        n = rng.randint(4, 22)
        cplx = rng.random() < 0.5
        most = max(1, min(16384, (4 if cplx else 12) << max(0, 30 - n)))
        return {"kind": kind, "n": n, "count": _log_int(rng, 16, max(17, min(most, 8192 >> max(0, n - 18)))),
                "complex": cplx}
    if kind == "approx":
        return {"kind": kind, "n": _log_int(rng, 40, 200), "extra": rng.randint(2, 4),
                "samples": _log_int(rng, 1 << 14, 1 << 20)}
    lo = rng.randint(6, 16)
    return {"kind": "serve", "n_lo": lo, "n_hi": rng.randint(lo + 2, 24), "count": _log_int(rng, 64, 1024)}


# --------------------------------------------------------------- inputs ----

_SERVER = []  # one serving loop per program, as a user's service keeps it


def _server():
    if not _SERVER:
        _SERVER.append(serving.Server())
    return _SERVER[0]


def _haar(n, seed):
    """n x n block of a Haar unitary of at least twice the size."""
    return W.haar_block(n, seed, N=64)


def _matrix(case, seed):
    n = case["n"]
    if case["kind"] == "dense":
        return W.dense_uniform(n, seed)
    if case["kind"] == "complex":
        return _haar(n, seed)
    if case["kind"] == "binary":
        return W.binary_bernoulli(n, seed)
    return W.sparse_perm_plus(n, seed, case["extra"])


def _batch(case, seed):
    n, count = case["n"], case["count"]
    if not case["complex"]:
        return W.uniform(seed, count * n * n).reshape(count, n, n)
    u = [W.haar_unitary(64, seed * 31 + k) for k in range(2)]
    rng = np.random.default_rng(seed)
    at = rng.integers(0, 64 - n + 1, size=(count, 2))
    return np.stack([u[k % 2][r:r + n, c:c + n] for k, (r, c) in enumerate(at)])


def _requests(case, seed):
    u = [W.haar_unitary(64, seed * 17 + k) for k in range(2)]
    rng = np.random.default_rng(seed)
    mats = []
    for k in range(case["count"]):
        n = int(rng.integers(case["n_lo"], case["n_hi"] + 1))
        if rng.random() < 0.5:
            mats.append(rng.random((n, n)))
        else:
            r, c = rng.integers(0, 64 - n + 1, size=2)
            mats.append(np.ascontiguousarray(u[k % 2][r:r + n, c:c + n]))
    return mats


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        m = _batch(case, seed)
        flat = np.ascontiguousarray(m).view(np.float64) if case["complex"] else m
        comps = 2 if case["complex"] else 1
        return {"case": case, "mats": torch.from_numpy(np.ascontiguousarray(flat)).cuda(),
                "out": torch.empty((case["count"], comps, 2), dtype=torch.float64, device="cuda")}
    if kind == "serve":
        mats = _requests(case, seed)
        return {"case": case, "server": _server(),
                "flat": np.concatenate([np.ascontiguousarray(a).view(np.float64).ravel() for a in mats]),
                "ns": np.array([a.shape[0] for a in mats], dtype=np.int32),
                "cx": np.array([int(np.iscomplexobj(a)) for a in mats], dtype=np.int32)}
    state = {"case": case, "a": _matrix(case, seed), "seed": seed}
    if kind == "sparse":  # the compressed-column arrays such a program holds
        a = state["a"]
        c_idx, r_idx = np.nonzero(a.T)
        cptrs = np.concatenate([[0], np.cumsum(np.bincount(c_idx, minlength=a.shape[0]))])
        state["csc"] = (cptrs.astype(np.int32), r_idx.astype(np.int32), np.ascontiguousarray(a.T[c_idx, r_idx]))
    return state


# ---------------------------------------------------------------- calls ----

def _words(v, bits=320):
    v &= (1 << bits) - 1
    return np.array([(v >> (32 * i)) & 0xFFFFFFFF for i in range(bits // 32)], dtype=np.int64)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dense":
        return np.array([spb.perm_dense(state["a"], precision=case["precision"]).permanent])
    if kind == "complex":
        kw = {"rel_tol": 1e-2} if case["precision"] == "fp32" else {}
        return np.array([spb.perm_complex(state["a"], precision=case["precision"], **kw).permanent])
    if kind == "binary":
        return _words(spb.perm_binary(state["a"]).permanent)
    if kind == "sparse":
        return np.array([spb.perm_sparse(state["csc"], precision=case["precision"]).permanent])
    if kind == "pipeline":
        a = state["a"]
        args = [b"calculation_precision=dd"] if case["precision"] == "dd" else []
        arr = (ctypes.c_char_p * max(1, len(args)))(*args)
        out = _lib.spb_pipeline_result()
        _lib.check(_lib.lib().spb_perm_pipeline(a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), a.shape[0], arr,
                                                len(args), ctypes.byref(out)))
        return np.array([out.permanent])
    if kind == "batch":
        _lib.check(_lib.lib().spb_perm_batch_dev(
            ctypes.c_void_p(state["mats"].data_ptr()), case["n"], int(case["complex"]), case["count"],
            ctypes.c_void_p(state["out"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["out"]
    if kind == "approx":
        return np.array([spb.perm_approx(state["a"], samples=case["samples"], seed=state["seed"]).permanent])
    srv = state["server"]
    tickets = srv.submit_flat(state["flat"], state["ns"], state["cx"])
    return np.array([complex(srv.wait(t)["permanent"]) for t in tickets])


# ----------------------------------------------- what a pass cannot avoid ----

def _ryser_flops(n, cplx):
    """Row adds and products of Ryser's formula over 2^(n-1) subsets."""
    return (8.0 if cplx else 2.0) * n * 2.0 ** (n - 1)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        ns = range(case["n_lo"], case["n_hi"] + 1)
        per = case["count"] / len(ns)
        return {"bytes": sum(per * 12.0 * n * n for n in ns),
                "flops": sum(per * 0.5 * (_ryser_flops(n, False) + _ryser_flops(n, True)) for n in ns)}
    n = case["n"]
    if kind == "batch":
        c = 2 if case["complex"] else 1
        return {"bytes": case["count"] * 8.0 * c * (n * n + 2), "flops": case["count"] * _ryser_flops(n, c == 2)}
    if kind == "approx":
        nnz = n * (case["extra"] + 1)
        # per sample and row: ten scaling passes over the row's columns
        return {"bytes": 8.0 * nnz, "flops": case["samples"] * 10.0 * nnz * (case["extra"] + 2)}
    if kind in ("sparse", "pipeline"):
        nnz = n * (case["extra"] + 1)
        # what a sparse permanent costs depends on its pattern; the entries
        # are read once and each takes part in a product and a sum at the least
        return {"bytes": 16.0 * nnz, "flops": 2.0 * nnz}
    cplx = kind == "complex"
    return {"bytes": (16.0 if cplx else 1.0 if kind == "binary" else 8.0) * n * n, "flops": _ryser_flops(n, cplx)}


def tolerance(case):
    kind = case["kind"]
    if kind == "binary":
        return "exact"
    if kind == "dense" and case["precision"] == "fp64":
        # FP64 products in Ryser's alternating sum: ~kappa sqrt(n/6) 2^-52
        return {"rel": 1e-12 if case["n"] <= 24 else 2e-11}
    if kind == "complex" and case["precision"] == "fp32":
        # ~kappa n 2^-24 on Haar blocks
        return {"rel": 4e-5}
    # the accuracy bar of the real, complex and sparse paths; the sampling
    # estimate's samples are fixed by the seed, only their sum's order is free
    return {"rel": 1e-12}


# ------------------------------------------------ plain 64-bit evaluation ----

def _ryser(a, device):
    """Nijenhuis-Wilf Ryser in float64 / complex128, subsets in a low and a
    high half, products over rows as plain tensor operations."""
    a = torch.as_tensor(np.ascontiguousarray(a), device=device)
    n = a.shape[-1]
    if n == 1:
        return a[0, 0].cpu().item()
    x0 = a[:, n - 1] - a.sum(dim=1) / 2

    def sums(cols):  # [rows, 2^cols] subset sums, [2^cols] signs
        s = torch.zeros((n, 1), dtype=a.dtype, device=device)
        g = torch.ones(1, dtype=torch.float64, device=device)
        for j in cols:
            s = torch.cat([s, s + a[:, j:j + 1]], dim=1)
            g = torch.cat([g, -g])
        return s, g

    w = min(n - 1, 11)
    low, gl = sums(range(w))
    low = low + x0[:, None]
    high, gh = sums(range(w, n - 1))
    step, parts = 1 << 12, []
    for h in range(0, high.shape[1], step):
        p = torch.ones((1, 1), dtype=a.dtype, device=device)
        for r in range(n):
            p = p * (high[r, h:h + step, None] + low[r, None, :])
        parts.append((p * gl).sum(dim=1).mul(gh[h:h + step]).sum())
    v = torch.stack(parts).sum() * (4 * (n % 2) - 2)
    return v.cpu().item()


def _ryser_batch(mats, device):
    out = [_ryser(m, device) for m in mats]
    return np.array(out)


def _binary_words(a):
    """Exact 0/1 permanent: Ryser modulo primes below 2^31, joined by the
    Chinese remainder theorem."""
    n = a.shape[0]
    dev = "cuda"
    m = torch.as_tensor(a.astype(np.int64), device=dev)
    bound = 1
    for r in range(n):
        bound *= max(1, int(a[r].sum()))
    value, mod, p = 0, 1, (1 << 31) - 1
    while mod <= bound:
        while any(p % q == 0 for q in range(3, int(p ** 0.5) + 1, 2)):
            p -= 2
        w = min(n, 11)

        def sums(cols):
            s = torch.zeros((n, 1), dtype=torch.int64, device=dev)
            g = torch.ones(1, dtype=torch.int64, device=dev)
            for j in cols:
                s = torch.cat([s, s + m[:, j:j + 1]], dim=1)
                g = torch.cat([g, -g])
            return s, g

        low, gl = sums(range(w))
        high, gh = sums(range(w, n))
        total = 0
        for h in range(0, high.shape[1], 1 << 12):
            t = torch.ones((1, 1), dtype=torch.int64, device=dev)
            for r in range(n):
                t = t * (high[r, h:h + (1 << 12), None] + low[r, None, :]) % p
            total += int(((t * gl).sum(dim=1) * gh[h:h + (1 << 12)]).sum())
        total = total * (-1) ** n % p
        k = (total - value) * pow(mod, -1, p) % p
        value += mod * k
        mod *= p
        p -= 2
    return _words(value)


def _sparse_expansion(a):
    """Row-by-row expansion over the sets of used columns (sums of products
    only, no cancellation on positive entries); None when the sets grow past
    what a few seconds allow."""
    n = a.shape[0]
    rows = [np.flatnonzero(a[r]) for r in range(n)]
    left, order, used = list(range(n)), [], set()
    while left:  # next: the row that opens fewest new columns
        r = min(left, key=lambda i: (sum(c not in used for c in rows[i]), i))
        left.remove(r)
        order.append(r)
        used.update(rows[r])
    last = {}
    for k, r in enumerate(order):
        for c in rows[r]:
            last[int(c)] = k
    masks, vals = np.zeros(1, dtype=np.uint64), np.ones(1)
    for k, r in enumerate(order):
        nm, nv = [], []
        for c in rows[r]:
            bit = np.uint64(1 << int(c))
            free = (masks & bit) == 0
            nm.append(masks[free] | bit)
            nv.append(vals[free] * a[r, c])
        m, v = np.concatenate(nm), np.concatenate(nv)
        must = np.uint64(sum(1 << c for c, l in last.items() if l == k))
        keep = (m & must) == must
        masks, inv = np.unique(m[keep], return_inverse=True)
        vals = np.bincount(inv, weights=v[keep], minlength=masks.size)
        if masks.size > 4_000_000:
            return None
        if masks.size == 0:
            return 0.0
    return float(vals.sum())


def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        return np.array([_ryser(_matrix(case, seed), "cuda")])
    if kind == "complex":
        return np.array([_ryser(_matrix(case, seed), "cuda")])
    if kind == "binary":
        return _binary_words(_matrix(case, seed)) if case["n"] <= 28 else None
    if kind in ("sparse", "pipeline"):
        v = _sparse_expansion(_matrix(case, seed))
        return None if v is None else np.array([v])
    if kind == "batch":
        if case["count"] * 2.0 ** case["n"] * case["n"] > 2e11 or case["count"] > 1024:
            return None
        m = _ryser_batch(_batch(case, seed), "cuda")
        out = np.zeros((case["count"], 2 if case["complex"] else 1, 2))
        out[:, 0, 0] = m.real
        if case["complex"]:
            out[:, 1, 0] = m.imag
        return torch.from_numpy(out)
    if kind == "serve":
        if case["count"] > 512:
            return None
        return np.array([complex(_ryser(m, "cuda")) for m in _requests(case, seed)])
    return None  # a sampling estimate: no plain 64-bit value of its own
