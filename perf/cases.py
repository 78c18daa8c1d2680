"""Workloads of the permanent engine that its speed is judged on.

Every case goes through the public Python entry points (the ctypes mirror of
include/perman_b200.h) the way a user's program calls them: host numpy
matrices in, permanents or estimates out; the batch keeps its plan between
runs, everything else is a single call.  Matrices are synthetic with the
shapes and value distributions of the repository's own configurations,
benchmark and tests.

Kinds:
  policy     Engine.exact_dense: one exact permanent with the default accuracy
             policy (error at most 1e-10, estimate included)
  reference  gpu_perman64_xshared_coalescing_mshared: one evaluation through
             the reference's own signature, no policy
  sparse     Engine.exact_sparse on CRS/CCS arrays after skipOrder
  batch      Batch.run: a resident batch of mixed matrices
  rasmussen, scaling   Monte-Carlo estimates of a 0/1 matrix
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[1]


def _package():
    """The engine's Python mirror (its directory name is not an identifier)."""
    if "perman_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "perman_b200", ROOT / "matrix-permanent-calculator_b200" / "__init__.py")
        mod = importlib.util.module_from_spec(spec)
        sys.modules["perman_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["perman_b200"]


_engine = None


def _get_engine():
    global _engine
    if _engine is None:
        _engine = _package().Engine(0)
    return _engine


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # smallest calls, where host work, copies and launches count
        {"name": "policy_real_n12", "kind": "policy", "n": 12, "density": 0.5, "values": "real"},
        # an ordinary small request of the request loop, odd order, FP32 input
        {"name": "policy_float_n23", "kind": "policy", "n": 23, "density": 0.5, "values": "float"},
        # the plain exact configuration: binary matrix of order 30
        {"name": "policy_binary_n30", "kind": "policy", "n": 30, "density": 0.5, "values": "binary"},
        # a large request of the request loop: real matrix, certified walk
        {"name": "policy_real_n32", "kind": "policy", "n": 32, "density": 0.5, "values": "real"},
        # an integer matrix at the order between the parity instance and the headline, certified
        {"name": "policy_int_n36", "kind": "policy", "n": 36, "density": 0.5, "values": "int"},
        # one plain FP64 evaluation of a real matrix through the reference's signature
        {"name": "reference_real_n33", "kind": "reference", "n": 33, "density": 0.5, "values": "real"},
        # the headline: order 40, values 1..4, one evaluation through the reference's signature
        {"name": "reference_int_n40", "kind": "reference", "n": 40, "density": 0.5, "values": "int"},
        # the sparse exact configuration: order 36, density 0.2, values (0,1]
        {"name": "sparse_real_n36", "kind": "sparse", "n": 36, "density": 0.2, "values": "real"},
        # very sparse binary matrix (about three nonzeros a row): most Gray terms vanish
        {"name": "sparse_binary_n36", "kind": "sparse", "n": 36, "density": 0.0834, "values": "binary"},
        # the batch configuration (orders 12..28, density 0.2..0.9, half binary), an eighth of its count
        {"name": "batch_1024", "kind": "batch", "count": 1024, "n_lo": 12, "n_hi": 28, "d_lo": 0.2, "d_hi": 0.9},
        # the approximate requests of the request loop
        {"name": "rasmussen_n64", "kind": "rasmussen", "n": 64, "density": 0.5, "trials": 200000},
        {"name": "scaling_n57", "kind": "scaling", "n": 57, "density": 0.5, "trials": 200000,
         "scale_intervals": 4, "scale_times": 5},
    ]


def draw(rng):
    kind = rng.choice(["policy", "policy", "policy", "reference", "reference", "sparse", "batch", "rasmussen",
                       "scaling"])
    if kind == "policy":
        values = rng.choice(["real", "real", "float", "int", "binary"])
        n = rng.randint(10, 37 if values in ("int", "binary") else 33)
        return {"kind": kind, "n": n, "density": round(rng.uniform(0.3, 0.9), 3), "values": values}
    if kind == "reference":
        values = rng.choice(["real", "float", "int", "binary"])
        # a single FP64 evaluation of a larger or denser real matrix cancels too much to be of use
        n = rng.randint(14, 37 if values in ("int", "binary") else 32)
        d_hi = 0.9 if values in ("int", "binary") else 0.7
        return {"kind": kind, "n": n, "density": round(rng.uniform(0.3, d_hi), 3), "values": values}
    if kind == "sparse":
        if rng.random() < 0.5:
            return {"kind": kind, "n": rng.randint(24, 36), "density": round(rng.uniform(0.15, 0.3), 3),
                    "values": "real"}
        n = rng.randint(24, 36)
        return {"kind": kind, "n": n, "density": round(rng.uniform(2.7, 3.3) / n, 4), "values": "binary"}
    if kind == "batch":
        lo = rng.randint(8, 20)
        return {"kind": kind, "count": int(round(2 ** rng.uniform(4, 10.5))), "n_lo": lo,
                "n_hi": rng.randint(lo + 3, 28), "d_lo": 0.2, "d_hi": 0.9}
    trials = int(round(10 ** rng.uniform(3.5, 5.4)))
    case = {"kind": kind, "n": rng.randint(30, 64), "density": round(rng.uniform(0.35, 0.7), 3), "trials": trials}
    if kind == "scaling":
        case["scale_intervals"] = rng.choice([2, 4, 4, 8])
        case["scale_times"] = rng.choice([3, 5, 5])
    return case


# ---- inputs -------------------------------------------------------------------

def _matrix(r, n, density, values):
    """n x n matrix, entries nonzero with probability `density`; every row and
    column has a nonzero and the pattern a perfect matching (a hidden
    permutation), so that the permanent is positive."""
    mask = r.random((n, n)) < density
    mask[np.arange(n), r.permutation(n)] = True
    if values == "binary":
        return mask.astype(np.int32)
    if values == "int":
        return np.where(mask, r.integers(1, 5, (n, n)), 0).astype(np.int32)
    a = np.where(mask, 1.0 - r.random((n, n)), 0.0)
    return a.astype(np.float32) if values == "float" else a


def _batch_matrices(case, seed):
    r = np.random.default_rng([seed, 7])
    mats = []
    for i in range(case["count"]):
        n = int(r.integers(case["n_lo"], case["n_hi"] + 1))
        density = float(r.uniform(case["d_lo"], case["d_hi"]))
        mats.append(_matrix(r, n, density, "binary" if i % 2 else "real").astype(np.float64))
    return mats


class _ResidentBatch:
    """A batch plan and its lifetime."""

    def __init__(self, mats):
        self.batch = _get_engine().batch(mats)

    def __del__(self):
        try:
            self.batch.free()
        except Exception:
            pass


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"case": case, "plan": _ResidentBatch(_batch_matrices(case, seed))}
    _get_engine()
    r = np.random.default_rng([seed, case["n"]])
    a = _matrix(r, case["n"], case["density"], case.get("values", "binary"))
    state = {"case": case, "a": a, "seed": seed % (1 << 31) + 1}
    if kind == "sparse":
        state["c"] = _package().compress(2, a)
    return state


def _number(x):
    """A result in its own 64 bits."""
    return np.array([x], dtype=np.float64)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "policy":
        return {"value": _number(_get_engine().exact_dense(state["a"]).value)}
    if kind == "reference":
        return {"value": _number(_package().gpu_perman64_xshared_coalescing_mshared(state["a"]))}
    if kind == "sparse":
        c = state["c"]
        r = _get_engine().exact_sparse(c["n"], c["rptrs"], c["cols"], c["rvals"], c["cptrs"], c["rows"], c["cvals"])
        return {"value": _number(r.value)}
    if kind == "batch":
        return {"values": state["plan"].batch.run()[0]}
    if kind == "rasmussen":
        e = _get_engine().rasmussen(state["a"], case["trials"], seed=state["seed"])
    else:
        e = _get_engine().scaling(state["a"], case["trials"], case["scale_intervals"], case["scale_times"],
                                  seed=state["seed"])
    return {"mean": _number(e.mean), "std_error": _number(e.std_error), "zero_trials": int(e.zero_trials)}


# ---- work and exact values ----------------------------------------------------

def work(case):
    """Bytes: the matrix in, the results out.  Operations: exact kinds 2n FP64
    operations (n row-sum updates, n multiplies) for each of the 2^(n-1) terms
    of the plain Gray walk; estimators one comparison per available entry."""
    kind = case["kind"]
    if kind == "batch":
        span = range(case["n_lo"], case["n_hi"] + 1)
        each = case["count"] / len(span)
        return {"bytes": sum(each * (8.0 * n * n + 16) for n in span),
                "flops": sum(each * 2.0 * n * 2.0 ** (n - 1) for n in span)}
    n = case["n"]
    if kind in ("rasmussen", "scaling"):
        per_trial = n * n * case["density"] / 2
        if kind == "scaling":
            per_trial += 4.0 * case["scale_times"] / case["scale_intervals"] * case["density"] * n ** 3 / 3
        return {"bytes": n * n / 8 + 32.0, "flops": per_trial * case["trials"]}
    size = 4.0 if case["values"] != "real" else 8.0
    nonzeros = n * n * case["density"] if kind == "sparse" else n * n
    return {"bytes": size * nonzeros + 16, "flops": 2.0 * n * 2.0 ** (n - 1)}


def _permanent(a):
    """Permanent by the subset recurrence: f_i(S) = sum over c in S of
    a[i][c] f_{i-1}(S without c), S the columns used by the first i rows.  For
    nonnegative matrices nothing cancels, so 64-bit sums are good to n units
    in the last place."""
    import torch

    n = a.shape[0]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = torch.zeros(1 << n, dtype=torch.float64, device=dev)
    f[0] = 1.0
    g = torch.empty_like(f)
    for i in range(n):
        g.zero_()
        for c in range(n):
            v = float(a[i, c])
            if v != 0.0:
                shape = (1 << (n - 1 - c), 2, 1 << c)
                g.view(shape)[:, 1].add_(f.view(shape)[:, 0], alpha=v)
        f, g = g, f
    return float(f[-1])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rasmussen", "scaling"):
        return None  # a random estimate: defined by its streams alone
    if kind == "batch":
        if case["count"] * 2.0 ** case["n_hi"] * case["n_hi"] ** 2 > 1e13:
            return None
        return {"values": np.array([_permanent(m) for m in _batch_matrices(case, seed)])}
    n = case["n"]
    if n > 32:
        return None
    r = np.random.default_rng([seed, n])
    a = _matrix(r, n, case["density"], case["values"]).astype(np.float64)
    v = _permanent(a)
    return {"value": _number(v)} if math.isfinite(v) else None
