"""The work that programs have this solver do, as cases that can be timed and compared.

Each case is a dict of plain values with a "kind":

  factor      LUSolver.factor_solve: FP64 P A = L U in place and x = A^-1 b
  solve       LUSolver.solve: right-hand sides against factors kept from before
  mixed       LUSolver.refine_solve: low-precision factors, FP64 refinement
  grad        autograd.lu_solve, forward and backward, FP64
  grad_mixed  autograd.lu_solve_mixed, forward and backward
  batched     BatchedSystems.factor_solve: many systems of uneven order

Matrices and right-hand sides are i.i.d. uniform [-0.5, 0.5), the inputs of the
repository's benchmark.  The in-place entry points overwrite their inputs, so a pass
copies them first, as a program that keeps its matrix does.  The mixed solves refine
until the scaled residual is below 1e-3, the default of lu_solve_mixed, which is where
their solution has the accuracy of an FP64 solve.
"""
import math

import torch

from charmlu_b200 import LU_PREC_FP16X3, LU_PREC_FP32, LU_PREC_FP64, LUConfig, LUSolver
from charmlu_b200.autograd import lu_solve, lu_solve_mixed
from charmlu_b200.batched import BatchedSystems, log_uniform_orders

IR_TARGET = 1e-3


def listed():
    return [
        # one small system in a larger program's loop: launches and latency
        {"name": "factor_256", "kind": "factor", "n": 256, "b": 64, "lookahead": False, "graph": False},
        # the plain FP64 configuration that the reference runs as it is
        {"name": "factor_2048", "kind": "factor", "n": 2048, "b": 128, "lookahead": False, "graph": False},
        # an odd order (padded row pitch, ragged tiles and last panel) under look-ahead
        {"name": "factor_4999_lookahead", "kind": "factor", "n": 4999, "b": 192, "lookahead": True, "graph": False},
        # the large FP64 configuration
        {"name": "factor_32768_lookahead", "kind": "factor", "n": 32768, "b": 256, "lookahead": True, "graph": False},
        # new right-hand sides for a system factored earlier
        {"name": "solve_8192x16", "kind": "solve", "n": 8192, "nrhs": 16, "trans": False},
        # a mixed-precision solve of ordinary size with direct launches, ragged
        {"name": "mixed_10000", "kind": "mixed", "n": 10000, "b": 256, "lookahead": False, "graph": False},
        # the headline configuration: look-ahead schedule replayed from a graph
        {"name": "mixed_65536_lookahead", "kind": "mixed", "n": 65536, "b": 512, "lookahead": True, "graph": True},
        # a training step through the solve: forward, and both gradients
        {"name": "grad_4096x16", "kind": "grad", "n": 4096, "nrhs": 16, "b": 128},
        # the same through low-precision factors, refined in both directions
        {"name": "grad_mixed_16384x16", "kind": "grad_mixed", "n": 16384, "nrhs": 16, "b": 256},
        # thousands of independent systems of uneven order, FP64
        {"name": "batched_fp64_4096", "kind": "batched", "count": 4096, "lo": 32, "hi": 1024, "fp32": False},
        # the same with FP32 factors and FP64 refinement
        {"name": "batched_fp32_4096", "kind": "batched", "count": 4096, "lo": 32, "hi": 1024, "fp32": True},
        # many small systems, fewer than fill the GPU for long
        {"name": "batched_fp64_small", "kind": "batched", "count": 1000, "lo": 5, "hi": 120, "fp32": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["factor", "factor", "solve", "mixed", "grad", "grad_mixed", "batched", "batched"])
    if kind == "factor":
        return {"kind": kind, "n": _log_int(rng, 64, 20000), "b": rng.choice([64, 128, 192, 256]),
                "lookahead": rng.random() < 0.5, "graph": rng.random() < 0.25}
    if kind == "solve":
        return {"kind": kind, "n": _log_int(rng, 128, 16384), "nrhs": rng.randint(1, 16), "trans": rng.random() < 0.5}
    if kind == "mixed":
        return {"kind": kind, "n": _log_int(rng, 512, 40000), "b": rng.choice([128, 256, 512]),
                "lookahead": rng.random() < 0.5, "graph": rng.random() < 0.5}
    if kind == "grad":
        return {"kind": kind, "n": _log_int(rng, 128, 8192), "nrhs": rng.randint(1, 16), "b": rng.choice([64, 128, 256])}
    if kind == "grad_mixed":
        return {"kind": kind, "n": _log_int(rng, 512, 16384), "nrhs": rng.randint(1, 16), "b": rng.choice([128, 256])}
    lo = _log_int(rng, 1, 128)
    hi = max(lo, _log_int(rng, 32, 1024))
    return {"kind": kind, "count": _log_int(rng, 50, 4096), "lo": lo, "hi": hi, "fp32": rng.random() < 0.5}


def _uniform(gen, *shape):
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=gen).sub_(0.5)


def _pitched(n):
    """n x n with rows on 16-byte boundaries, as the factorisation takes them."""
    return torch.empty(n, n + (n & 1), dtype=torch.float64, device="cuda")[:, :n]


def _inputs(case, seed):
    """The arrays that make up the problem, from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "batched":
        n = log_uniform_orders(case["count"], case["lo"], case["hi"])  # the orders belong to the case, the values to the seed
        n64 = n.astype("int64")
        return {"orders": n, "A": _uniform(gen, int((n64 * n64).sum())), "B": _uniform(gen, int(n64.sum()))}
    n = case["n"]
    A = _pitched(n)
    if n & 1:
        A.copy_(_uniform(gen, n, n))
    else:
        torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen, out=A)
        A.sub_(0.5)
    k = case.get("nrhs", 0)
    d = {"A": A, "B": _uniform(gen, n, k) if k else _uniform(gen, n)}
    if case["kind"].startswith("grad"):
        d["W"] = _uniform(gen, n, k).mul_(2.0)  # upstream gradient, uniform [-1, 1)
    return d


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    s.update(_inputs(case, seed))
    if kind == "batched":
        s["plan"] = BatchedSystems(s.pop("orders"))
        s["precision"] = LU_PREC_FP32 if case["fp32"] else LU_PREC_FP64
        s["plan"].work(s["precision"])
        s["x"] = torch.empty_like(s["B"])
        if not case["fp32"]:  # overwritten by the factors
            s["LU"] = torch.empty_like(s["A"])
        return s
    n = case["n"]
    if kind in ("grad", "grad_mixed"):
        s["A"].requires_grad_()
        s["B"].requires_grad_()
        return s
    if kind == "mixed":
        s["solver"] = LUSolver(LUConfig(n, case["b"], precision=LU_PREC_FP16X3, lookahead=case["lookahead"],
                                        use_graph=case["graph"], ir_target=IR_TARGET))
        s["x"] = torch.empty_like(s["B"])
        return s
    if kind == "factor":
        s["solver"] = LUSolver(LUConfig(n, case["b"], lookahead=case["lookahead"], use_graph=case["graph"]))
        s["LU"] = _pitched(n)
        s["x"] = torch.empty_like(s["B"])
        s["ipiv"] = torch.empty(n, dtype=torch.int32, device="cuda")
        return s
    s["solver"] = LUSolver(LUConfig(n, 128))
    s["LU"] = s.pop("A")
    s["ipiv"] = s["solver"].factor(s["LU"])
    s["x"] = torch.empty_like(s["B"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "factor":
        s["LU"].copy_(s["A"])
        s["x"].copy_(s["B"])
        s["solver"].factor_solve(s["LU"], s["x"], s["ipiv"])
        return {"LU": s["LU"], "x": s["x"], "ipiv": s["ipiv"]}
    if kind == "solve":
        s["x"].copy_(s["B"])
        return {"x": s["solver"].solve(s["LU"], s["ipiv"], s["x"], trans=case["trans"])}
    if kind == "mixed":
        return {"x": s["solver"].refine_solve(s["A"], s["B"], s["x"])[0]}
    if kind in ("grad", "grad_mixed"):
        solve = lu_solve if kind == "grad" else lu_solve_mixed
        X = solve(s["A"], s["B"], case["b"])
        gA, gB = torch.autograd.grad(X, (s["A"], s["B"]), s["W"])
        return {"X": X.detach(), "gA": gA, "gB": gB}
    s["x"].copy_(s["B"])
    if case["fp32"]:
        info = s["plan"].factor_solve(s["A"], s["x"], s["precision"])
        return {"x": s["x"], "info": info}
    s["LU"].copy_(s["A"])
    info = s["plan"].factor_solve(s["LU"], s["x"], s["precision"])
    return {"LU": s["LU"], "x": s["x"], "info": info}


def work(case):
    """Factor 2/3 n^3 flops and solve 2 n^2 per right-hand side; inputs read once, outputs written once."""
    kind = case["kind"]
    if kind == "batched":
        # mean of n^p over the log-uniform law of the orders
        lo, hi = case["lo"], case["hi"] + 1
        span = math.log(hi / lo)
        m1, m2, m3 = ((hi ** p - lo ** p) / (p * span) for p in (1, 2, 3))
        return {"bytes": case["count"] * (8 * m2 * (1 if case["fp32"] else 2) + 16 * m1),
                "flops": case["count"] * (2 / 3 * m3 + 2 * m2)}
    n, k = case["n"], case.get("nrhs", 1)
    if kind == "solve":
        return {"bytes": 8 * n * n + 16 * n * k, "flops": 2 * n * n * k}
    if kind == "factor":
        return {"bytes": 16 * n * n + 20 * n, "flops": 2 / 3 * n ** 3 + 2 * n * n}
    if kind == "mixed":
        return {"bytes": 8 * n * n + 16 * n, "flops": 2 / 3 * n ** 3 + 2 * n * n}
    # solve, transposed solve and the rank-k gradient of A
    return {"bytes": 16 * n * n + 40 * n * k, "flops": 2 / 3 * n ** 3 + 6 * n * n * k}


def exact(case, seed):
    kind = case["kind"]
    if case.get("n", 0) > 40000:  # the matrix and its factors do not fit beside each other
        return None
    d = _inputs(case, seed)
    if kind == "batched":
        x, LU, a, b = torch.empty_like(d["B"]), None if case["fp32"] else torch.empty_like(d["A"]), 0, 0
        for n in d["orders"].tolist():
            f, p = torch.linalg.lu_factor(d["A"][a:a + n * n].view(n, n))
            x[b:b + n] = torch.linalg.lu_solve(f, p, d["B"][b:b + n].view(n, 1)).view(n)
            if LU is not None:
                LU[a:a + n * n] = f.reshape(-1)
            a, b = a + n * n, b + n
        return {"x": x, "info": None} if LU is None else {"LU": LU, "x": x, "info": None}
    A, B = d["A"], d["B"]
    B2 = B if B.dim() == 2 else B.view(-1, 1)
    f, p = torch.linalg.lu_factor(A)
    if kind == "solve" and case["trans"]:
        return {"x": torch.linalg.lu_solve(f, p, B2, adjoint=True)}
    X = torch.linalg.lu_solve(f, p, B2).view(B.shape)
    if kind in ("solve", "mixed"):
        return {"x": X}
    if kind == "factor":
        return {"LU": f, "x": X, "ipiv": None}
    lam = torch.linalg.lu_solve(f, p, d["W"], adjoint=True)
    return {"X": X, "gA": -lam @ X.T, "gB": lam}
