"""The work that programs give this package, as cases that can be timed and compared.

listed() holds fixed sizes over the range in use, draw() more of the same
ranges, prepare() what a program has in hand before the call, run() one pass
through the public entry points, work() the bytes and operations that the pass
cannot do without, tolerance() how far another correct implementation at the
same precision may be off, and exact() the same results from torch in FP64
without this package.  Matrices are column-major throughout, so a tensor here
is the transpose of the matrix: T[j, i] = M[i, j].
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rochpl_b200.autograd import hpl_solve
from rochpl_b200.batch import BatchPlan, batch_flops, workload_sizes
from rochpl_b200.hpl import Algo, HPL_pdgesv, HPL_pdmatgen, default_ld, hpl_flops
from rochpl_b200.lib import HPLB_BATCH_RECURSIVE, PREC_BF16X3, PREC_FP16X3, library

F64 = torch.float64
PRECISIONS = {"bf16x3": PREC_BF16X3, "fp16x3": PREC_FP16X3}
# Panel widths by size class as the tuner picks them; without it the plan has its own table.
TUNED = [32, 32] + [HPLB_BATCH_RECURSIVE] * 4


def _dev() -> torch.device:
    return torch.device("cuda", torch.cuda.current_device())


def listed() -> list:
    return [
        # One small system: the smallest problem an HPL.dat sweep runs, where
        # launches and latency are all there is.
        {"name": "solve_n100", "kind": "solve", "n": 100, "nb": 32, "nbmin": 8, "rfact": 2},
        # A ragged size: neither N nor NB is a multiple of a tile.
        {"name": "solve_n1031", "kind": "solve", "n": 1031, "nb": 96, "nbmin": 32, "rfact": 2},
        # The small HPL configuration of the benchmark.
        {"name": "solve_n4096", "kind": "solve", "n": 4096, "nb": 256, "nbmin": 32, "rfact": 2},
        # The benchmark's parity solve.
        {"name": "solve_n16384", "kind": "solve", "n": 16384, "nb": 512, "nbmin": 32, "rfact": 2},
        # The largest FP64 solve that takes under a second or so: the trailing
        # update carries most of it, as at the headline size.
        {"name": "solve_n32768", "kind": "solve", "n": 32768, "nb": 512, "nbmin": 32, "rfact": 2},
        # The other half of an HPL test: regenerate [A|b], then the scaled
        # residual of a solution.
        {"name": "check_n16384", "kind": "check", "n": 16384, "stored": True},
        # Low-precision LU and GMRES refinement to FP64 accuracy, the matrix
        # never stored in FP64 (the benchmark's smaller mixed size).
        {"name": "mixed_n32768", "kind": "mixed", "n": 32768, "nb": 512, "precision": "fp16x3",
         "stored": False},
        # The batched workload: thousands of systems of uneven size at once.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 32, "hi": 1024, "nrhs": 16,
         "tuned": True},
        # A batch of a few small systems with one right-hand side: latency.
        {"name": "batch_48_small", "kind": "batch", "count": 48, "lo": 16, "hi": 96, "nrhs": 1,
         "tuned": False},
        # A solve inside a differentiated program, forward and backward, at
        # the benchmark's size and at a small one.
        {"name": "grad_n16384", "kind": "grad", "n": 16384, "nrhs": 32, "nb": 512},
        {"name": "grad_n1000", "kind": "grad", "n": 1000, "nrhs": 3, "nb": 256},
        # New right-hand sides for a matrix factored earlier.
        {"name": "getrs_n8192", "kind": "getrs", "n": 8192, "nb": 512, "nrhs": 32, "trans": 0},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _nb(rng, n: int) -> int:
    """The panel widths in use at a size: narrow for small systems, wide for large."""
    if n < 512:
        return rng.choice([16, 32, 64])
    return rng.choice([64, 96, 128, 256] if n < 4096 else [256, 384, 512])


def draw(rng) -> dict:
    kind = rng.choice(["solve", "solve", "check", "mixed", "batch", "grad", "getrs"])
    if kind == "solve":
        n = _log(rng, 64, 30000)
        return {"kind": kind, "n": n, "nb": _nb(rng, n), "nbmin": rng.choice([16, 32]),
                "rfact": rng.choice([0, 1, 2, 2])}
    if kind == "check":
        return {"kind": kind, "n": _log(rng, 1000, 24000), "stored": rng.random() < 0.5}
    if kind == "mixed":
        n = _log(rng, 1000, 30000)
        return {"kind": kind, "n": n, "nb": _nb(rng, n),
                "precision": rng.choice(["fp16x3", "bf16x3"]), "stored": rng.random() < 0.5}
    if kind == "batch":
        lo, hi = rng.choice([(32, 1024), (16, 96), (64, 512), (200, 700)])
        return {"kind": kind, "count": _log(rng, 16, 2048), "lo": lo, "hi": hi,
                "nrhs": rng.choice([1, 2, 4, 16, 64]), "tuned": rng.random() < 0.5}
    n = _log(rng, 64, 12000)
    if kind == "grad":
        return {"kind": kind, "n": n, "nrhs": _log(rng, 1, 64), "nb": rng.choice([256, 512])}
    return {"kind": kind, "n": n, "nb": _nb(rng, n), "nrhs": _log(rng, 1, 64),
            "trans": rng.choice([0, 1])}


def _uniform(seed: int, *shape) -> torch.Tensor:
    """Entries uniform in [-0.5, 0.5), as HPL's."""
    g = torch.Generator(device=_dev()).manual_seed(seed)
    return torch.rand(*shape, generator=g, dtype=F64, device=_dev()) - 0.5


def _sizes(case) -> np.ndarray:
    return workload_sizes(case["count"], case["lo"], case["hi"])


def _dense(case, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """A (n x n) and B (n x nrhs) of the stored-factor and differentiated solves."""
    return _uniform(seed, case["n"], case["n"]), _uniform(seed + 1, case["n"], case["nrhs"])


def prepare(case, seed: int) -> dict:
    lib = library(_dev().index)
    kind, n = case["kind"], case.get("n", 0)
    s = {"case": case, "seed": seed, "lib": lib}
    if kind == "solve":
        s["algo"] = Algo(case["nb"], min(case["nbmin"], case["nb"]), 2, 2, case["rfact"], 1, 0)
        s["mat"] = HPL_pdmatgen(n, case["nb"], seed, _dev().index, lib)
    elif kind == "check":
        s["mat"] = HPL_pdmatgen(n, 512, seed, _dev().index, lib)
        # A vector of a solution's length.  With the solution itself the
        # residual is the rounding error of the sums and no two correct
        # implementations agree on it.
        s["mat"].X.copy_(_uniform(seed, n))
    elif kind == "mixed":
        s["algo"] = Algo(case["nb"], 32, 2, 2, 2, 1, 0)
        s["x"] = torch.zeros(n, dtype=F64, device=_dev())
        if case["stored"]:
            s["mat"] = HPL_pdmatgen(n, case["nb"], seed, _dev().index, lib)
    elif kind == "batch":
        p = s["plan"] = BatchPlan(lib, _sizes(case), case["nrhs"],
                                  TUNED if case["tuned"] else None)
        s["A0"], s["B0"] = _uniform(seed, p.a_elems), _uniform(seed + 1, p.b_elems)
        s["A"], s["B"] = torch.empty_like(s["A0"]), torch.empty_like(s["B0"])
        s["ipiv"] = torch.zeros(p.p_elems, dtype=torch.int32, device=_dev())
        s["info"] = torch.zeros(p.count, dtype=torch.int32, device=_dev())
    elif kind == "grad":
        A, B = _dense(case, seed)
        s["A"], s["B"] = A.requires_grad_(), B.requires_grad_()
        s["Xbar"] = _uniform(seed + 2, n, case["nrhs"])
    else:
        A, B = _dense(case, seed)
        ld = int(default_ld(n))
        s["ld"] = ld
        s["LU"] = torch.zeros(n, ld, dtype=F64, device=_dev())
        s["LU"][:, :n].copy_(A.t())
        s["ipiv"] = torch.zeros(n, dtype=torch.int32, device=_dev())
        nb = min(case["nb"], n)
        lib.getrf(Algo(nb, min(32, nb), 2, 2, 2, 1, 0).c(), n, s["LU"].data_ptr(), ld,
                  s["ipiv"].data_ptr())
        s["B0"] = B.t().contiguous()
        s["B"] = torch.empty_like(s["B0"])
    return s


def run(s: dict):
    case, lib = s["case"], s["lib"]
    kind = case["kind"]
    if kind == "solve":
        # One repetition of an HPL test: generate (the solve overwrites
        # [A|b]), factor and solve.
        m = s["mat"]
        lib.matgen(m.n, m.n + 1, s["seed"], m.A.data_ptr(), m.ld, m.nb)
        info = HPL_pdgesv(s["algo"], m, lib)
        return {"LUy": m.A.view(m.n + 1, m.ld)[:, : m.n], "x": m.X, "ipiv": m.ipiv, "info": info}
    if kind == "check":
        m = s["mat"]
        if case["stored"]:
            lib.matgen(m.n, m.n + 1, s["seed"], m.A.data_ptr(), m.ld, m.nb)
            r = lib.residual(m.n, m.A.data_ptr(), m.ld, m.X.data_ptr())
            return {"A": m.A.view(m.n + 1, m.ld)[:, : m.n], **r}
        return lib.residual_lcg(m.n, s["seed"], m.X.data_ptr())
    if kind == "mixed":
        m = s.get("mat")
        r = lib.pdgesv_mixed(s["algo"].c(), case["n"], s["x"].data_ptr(), seed=s["seed"],
                             A=m.A.data_ptr() if m else None, ld=m.ld if m else 0,
                             precision=PRECISIONS[case["precision"]])
        # The rest of the report is times, counts and a residual at rounding
        # level; the low-precision pivots are not the caller's result.
        return {"x": s["x"], "converged": r["converged"]}
    if kind == "batch":
        s["A"].copy_(s["A0"])
        s["B"].copy_(s["B0"])
        s["plan"].gesv(s["A"].data_ptr(), s["B"].data_ptr(), s["ipiv"].data_ptr(),
                       s["info"].data_ptr())
        return {"LU": s["A"], "X": s["B"], "ipiv": s["ipiv"], "info": s["info"]}
    if kind == "grad":
        X = hpl_solve(s["A"], s["B"], nb=case["nb"])
        gA, gB = torch.autograd.grad(X, (s["A"], s["B"]), s["Xbar"])
        return {"X": X, "gA": gA, "gB": gB}
    s["B"].copy_(s["B0"])
    lib.getrs(case["trans"], case["n"], min(case["nb"], case["n"]), case["nrhs"],
              s["LU"].data_ptr(), s["ld"], s["ipiv"].data_ptr(), s["B"].data_ptr(), case["n"])
    return s["B"]


def work(case) -> dict:
    kind, n, nrhs = case["kind"], case.get("n", 0), case.get("nrhs", 0)
    if kind == "solve":
        return {"bytes": 8 * n * (n + 2) + 4 * n, "flops": hpl_flops(n)}
    if kind == "check":
        return {"bytes": (8 * n * (n + 1) if case["stored"] else 0) + 8 * n, "flops": 4 * n * n}
    if kind == "mixed":
        return {"bytes": (8 * n * (n + 1) if case["stored"] else 0) + 8 * n,
                "flops": hpl_flops(n)}
    if kind == "batch":
        sizes = _sizes(case).astype(np.float64)
        return {"bytes": float(np.sum(16 * sizes * (sizes + nrhs) + 4 * sizes)),
                "flops": batch_flops(sizes, nrhs)}
    if kind == "grad":
        # A, B and the cotangent read; X, dA and dB written.  LU, both
        # triangular solves forward and backward, and the outer product.
        return {"bytes": 16 * n * n + 32 * n * nrhs,
                "flops": 2 / 3 * n ** 3 + 6 * n * n * nrhs}
    return {"bytes": 8 * n * n + 16 * n * nrhs + 4 * n, "flops": 2 * n * n * nrhs}


def tolerance(case) -> dict:
    """Four times the error against exact(), for a condition number that few
    seeds exceed.  The error of a solution is eps kappa, and kappa of a random
    matrix is over t times its median for about one seed in t, so a single
    seed's error (seen: 6e-11 for a solve, 8e-10 for the worst of 4096 systems
    of a batch, 1e-9 after refinement) says little about the next one's."""
    if case["kind"] == "check":
        return {"rel": 1e-12}
    if case["kind"] == "mixed":
        # Refinement stops below the HPL threshold, at a residual that the
        # factors' precision decides: near 1 with bf16x3, near 0.02 with fp16x3.
        return {"rel": 1e-5 if case["precision"] == "bf16x3" else 1e-6}
    return {"rel": 1e-7 if case["kind"] == "batch" else 1e-8}


# ---------------------------------------------------------------------------
# The same results in FP64 from torch alone
# ---------------------------------------------------------------------------

_MASK = (1 << 64) - 1
_MULT, _ADD = 6364136223846793005, 1


def _signed(values) -> torch.Tensor:
    return torch.from_numpy(np.array(values, dtype=np.uint64).view(np.int64)).to(_dev())


def _lcg_matrix(n: int, seed: int) -> torch.Tensor:
    """HPL's n x (n + 1) [A|b] as T[j, i]: entry (i, j) from the state
    X(1 + i + j n) of X(k + 1) = mult X(k) + add mod 2^64, X(0) = seed."""
    mult, add, a, c = [], [], 1, 0
    for _ in range(n):  # jump by i
        mult.append(a)
        add.append(c)
        a, c = a * _MULT & _MASK, (c * _MULT + _ADD) & _MASK
    start, x = [], (_MULT * seed + _ADD) & _MASK
    for _ in range(n + 1):
        start.append(x)
        x = (a * x + c) & _MASK
    mult, add, start = _signed(mult), _signed(add), _signed(start)
    T = torch.empty(n + 1, n, dtype=F64, device=_dev())
    for j in range(0, n + 1, 2048):
        r = start[j:j + 2048, None] * mult + add
        low, high = (r & 0xFFFFFFFF).to(F64), ((r >> 32) & 0xFFFFFFFF).to(F64)
        T[j:j + 2048] = 0.5 - (low * 2.0 ** -32 + high) * 2.0 ** -32
    return T


def _swaps(piv, lo: int, hi: int, n: int) -> np.ndarray:
    """The rows after interchanges lo .. hi - 1: row r holds old row out[r]."""
    out = np.arange(n)
    for k in range(lo, hi):
        p = piv[k]
        out[k], out[p] = out[p], out[k]
    return out


def _exact_solve(case, seed: int) -> dict:
    n, nb = case["n"], case["nb"]
    T = _lcg_matrix(n, seed)
    LU, piv = torch.linalg.lu_factor(T.t())  # n x (n + 1): the last column is y
    del T
    piv = piv.long().cpu().numpy() - 1
    x = torch.linalg.solve_triangular(LU[:, :n], LU[:, n:], upper=True)[:, 0]
    # Later panels' interchanges move LAPACK's multipliers and not HPL's.
    later = np.arange(n)
    for j in reversed(range(0, n, nb)):
        at = torch.from_numpy(later).to(LU.device)
        cols = LU[:, j:j + nb].clone()
        LU[at, j:j + nb] = cols
        later = _swaps(piv, j, min(j + nb, n), n)[later]
    return {"LUy": LU.t(), "x": x, "ipiv": torch.from_numpy(piv.astype(np.int32)), "info": 0}


def _exact_check(case, seed: int) -> dict:
    n = case["n"]
    T, x, eps = _lcg_matrix(n, seed), _uniform(seed, n), 2.0 ** -53
    A, b = T[:n], T[n]
    anorm_inf = float(A.abs().sum(0).max())
    out = {"rnorm_inf": float((b - x @ A).abs().max()), "anorm_1": float(A.abs().sum(1).max()),
           "anorm_inf": anorm_inf, "xnorm_1": float(x.abs().sum()),
           "xnorm_inf": float(x.abs().max()), "bnorm_inf": float(b.abs().max()), "eps": eps}
    out["resid"] = out["rnorm_inf"] / (
        eps * (anorm_inf * out["xnorm_inf"] + out["bnorm_inf"]) * n)
    return {"A": T, **out} if case["stored"] else out


def _exact_batch(case, seed: int) -> dict:
    """LAPACK, one system after another."""
    sizes, nrhs = _sizes(case), case["nrhs"]
    A = _uniform(seed, int(np.sum(sizes.astype(np.int64) ** 2))).cpu()
    B = _uniform(seed + 1, int(np.sum(sizes.astype(np.int64)) * nrhs)).cpu()
    ipiv, a, b = [], 0, 0
    for n in map(int, sizes):
        At, Bt = A[a:a + n * n].view(n, n), B[b:b + n * nrhs].view(nrhs, n)
        LU, piv = torch.linalg.lu_factor(At.t())
        Bt.copy_(torch.linalg.lu_solve(LU, piv, Bt.t()).t())
        At.copy_(LU.t())
        ipiv.append(piv - 1)
        a, b = a + n * n, b + n * nrhs
    return {"LU": A, "X": B, "ipiv": torch.cat(ipiv).to(torch.int32),
            "info": torch.zeros(len(sizes), dtype=torch.int32)}


def exact(case, seed: int):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "check":
        return _exact_check(case, seed)
    if kind == "mixed":
        T = _lcg_matrix(n, seed)
        return {"x": torch.linalg.solve(T[:n].t(), T[n]), "converged": 1}
    if kind == "batch":
        return _exact_batch(case, seed)
    A, B = _dense(case, seed)
    LU, piv = torch.linalg.lu_factor(A)
    if kind == "grad":
        Xbar = _uniform(seed + 2, n, case["nrhs"])
        X = torch.linalg.lu_solve(LU, piv, B)
        gB = torch.linalg.lu_solve(LU, piv, Xbar, adjoint=True)
        return {"X": X, "gA": -gB @ X.t(), "gB": gB}
    return torch.linalg.lu_solve(LU, piv, B, adjoint=bool(case["trans"])).t()
