"""The work whose speed counts: what a program asks of this eigensolver through
glagpu's public entry points, from one small matrix to one of order 4096 and
batches of thousands.

Every case is a dict of plain values; its "kind" names the entry point:

  one        glagpu.eigen / glagpu.eigvals of one dense symmetric matrix
  hermitian  glagpu.eigen of one complex Hermitian matrix
  tridiag    glagpu.eigen / eigvals of a SymTridiagonal
  factor     glagpu.symtri and a product with its EigenQ
  batch      Plan.execute over many matrices of uneven orders
  grad       eigh_autograd and its backward pass, a training step's use
  mixed      Plan.execute and Plan.adjoint over orders on both sides of 128

An eigenvector is determined up to its sign (a complex one up to a unit
factor), and a program that stores or compares eigenvectors fixes it; so does
each run() here, and losses use the squared components. The spectra keep their
gaps wide enough (Gaussian ensembles, or prescribed with a gap) that the
eigenvectors are determined by the data to far better than 1e-9.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genericlinearalgebra.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import glagpu  # noqa: E402

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the smallest call: one matrix of a physics or statistics code, default
        # precision; latency is all there is
        {"name": "one_64_f64", "kind": "one", "n": 64, "precision": "f64", "jobz": "V", "uplo": "L"},
        # an ordinary single matrix of an order that fits no tile
        {"name": "one_777_f64", "kind": "one", "n": 777, "precision": "f64", "jobz": "V", "uplo": "U"},
        # the largest plain FP64 solve (the order the benchmark reports)
        {"name": "one_4096_f64", "kind": "one", "n": 4096, "precision": "f64", "jobz": "V", "uplo": "L"},
        # a large matrix through the FP32 solve and FP64 refinement
        {"name": "one_2048_refined", "kind": "one", "n": 2048, "precision": "f32_refined", "jobz": "V", "uplo": "L"},
        # a complex Hermitian matrix, as quantum codes have them
        {"name": "hermitian_333", "kind": "hermitian", "n": 333, "uplo": "L"},
        # eigenpairs of a tridiagonal that a Lanczos code or symtri left
        {"name": "tridiag_1500", "kind": "tridiag", "n": 1500, "jobz": "V"},
        # the Householder factorisation alone, and Q applied to a block
        {"name": "factor_400", "kind": "factor", "n": 400, "cols": 200, "uplo": "L"},
        # the benchmark's batch: thousands of small matrices, plain FP64
        {"name": "batch_4096_f64", "kind": "batch", "count": 4096, "lo": 8, "hi": 128, "precision": "f64",
         "jobz": "V", "alg": "QL", "uplo": "L", "orders": 2},
        # the same batch through the refined route, the headline
        {"name": "batch_4096_refined", "kind": "batch", "count": 4096, "lo": 8, "hi": 128,
         "precision": "f32_refined", "jobz": "V", "alg": "QL", "uplo": "L", "orders": 2},
        # eigenvalues only in single precision (spectral statistics, screening)
        {"name": "values_1000_f32", "kind": "batch", "count": 1000, "lo": 8, "hi": 128, "precision": "f32",
         "jobz": "N", "alg": "QL", "uplo": "L", "orders": 3},
        # a training step through the decomposition, forward and backward
        {"name": "grad_1024_refined", "kind": "grad", "count": 1024, "lo": 32, "hi": 96,
         "precision": "f32_refined", "orders": 4},
        # orders from 16 to 1024 in one plan, forward and adjoint
        {"name": "mixed_48_refined", "kind": "mixed", "count": 48, "top": 1024, "precision": "f32_refined",
         "orders": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "one", "hermitian", "tridiag", "factor", "batch", "batch", "batch", "grad",
                       "mixed"])
    orders = rng.randrange(1 << 20)
    uplo = rng.choice("LU")
    if kind == "one":
        precision = rng.choice(["f64", "f32_refined"])
        return {"kind": kind, "n": _log_int(rng, 4, 3600), "precision": precision,
                "jobz": "N" if rng.random() < 0.2 else "V", "uplo": uplo}
    if kind == "hermitian":
        return {"kind": kind, "n": _log_int(rng, 8, 600), "uplo": uplo}
    if kind == "tridiag":
        return {"kind": kind, "n": _log_int(rng, 16, 3000), "jobz": "N" if rng.random() < 0.2 else "V"}
    if kind == "factor":
        return {"kind": kind, "n": _log_int(rng, 16, 450), "cols": _log_int(rng, 1, 450), "uplo": uplo}
    if kind == "batch":
        precision, jobz = rng.choice([("f64", "V"), ("f32_refined", "V"), ("f64", "N"), ("f32", "N")])
        hi = _log_int(rng, 8, 128)
        return {"kind": kind, "count": _log_int(rng, 16, 4096), "lo": rng.randint(1, hi), "hi": hi,
                "precision": precision, "jobz": jobz, "alg": rng.choice(["QL", "QL", "QR"]), "uplo": uplo,
                "orders": orders}
    if kind == "grad":
        hi = rng.randint(16, 96)
        return {"kind": kind, "count": _log_int(rng, 16, 2048), "lo": rng.randint(4, hi), "hi": hi,
                "precision": rng.choice(["f64", "f32_refined"]), "orders": orders}
    return {"kind": kind, "count": _log_int(rng, 4, 48), "top": _log_int(rng, 150, 1024),
            "precision": rng.choice(["f64", "f32_refined"]), "orders": orders}


def _orders(case):
    """The orders of a batch's matrices: part of the case, not of the inputs."""
    rng = np.random.Generator(np.random.PCG64(case["orders"]))
    if case["kind"] == "mixed":
        return np.round(np.exp(rng.uniform(math.log(16), math.log(case["top"]), case["count"]))).astype(np.int64)
    return rng.integers(case["lo"], case["hi"] + 1, case["count"]).astype(np.int64)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _goe(n, g, dtype=F64):
    B = torch.randn(n, n, dtype=dtype, device=DEV, generator=g)
    return (B + B.mT) / 2


def _goe_arena(ns, g, dtype):
    """GOE matrices, packed one after another."""
    A = torch.randn(int((ns * ns).sum()), dtype=dtype, device=DEV, generator=g)
    off = 0
    for n in ns.tolist():
        M = A[off:off + n * n].view(n, n)
        M.copy_((M + M.T) / 2)
        off += n * n
    return A


def _spectrum(n, k, rng):
    """An even spectrum on [-1, 1], jittered (k even), or values of both signs
    over two decades (k odd); either keeps its neighbours apart."""
    t = (np.arange(n) + 0.5 + 0.3 * rng.uniform(-1, 1, n)) / n
    if k % 2 == 0:
        return 2 * t - 1
    return 10.0 ** (-2 * t) * rng.choice([-1.0, 1.0], n)


def _prescribed_arena(ns, seed):
    """Q diag(lam) Q' with Haar Q, packed one after another."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    parts = []
    for k, n in enumerate(ns.tolist()):
        lam = _spectrum(n, k, rng)
        if n <= 128:
            Q, R = np.linalg.qr(rng.standard_normal((n, n)))
            Q = Q * np.sign(np.diag(R))
            A = (Q * lam) @ Q.T
            parts.append(torch.from_numpy(((A + A.T) / 2).ravel()))
        else:
            B = torch.randn(n, n, dtype=F64, device=DEV, generator=_gen(rng.integers(1 << 31)))
            Q, R = torch.linalg.qr(B)
            Q = Q * torch.sign(torch.diagonal(R))
            A = (Q * torch.from_numpy(lam).to(DEV)) @ Q.T
            parts.append(((A + A.T) / 2).reshape(-1))
    out, small = [], []
    for p in parts:  # the small ones go up in few copies
        if p.is_cuda:
            if small:
                out.append(torch.cat(small).to(DEV))
                small = []
            out.append(p)
        else:
            small.append(p)
    if small:
        out.append(torch.cat(small).to(DEV))
    return torch.cat(out)


def _beta_hermite(n, seed):
    """The tridiagonal of a GOE matrix (Dumitriu and Edelman, 2002)."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    d = rng.standard_normal(n)
    e = np.sqrt(rng.chisquare(np.arange(n - 1, 0, -1)) / 2)
    return torch.from_numpy(d).to(DEV), torch.from_numpy(e).to(DEV)


class _Signs:
    """Signs of packed eigenvectors: the last component of each is made positive."""

    def __init__(self, ns):
        lens = torch.from_numpy(np.repeat(ns, ns)).to(DEV)
        self.last = torch.cumsum(lens, 0) - 1
        self.col = torch.repeat_interleave(torch.arange(lens.numel(), device=DEV), lens)

    def fix(self, V):
        one = torch.ones((), dtype=V.dtype, device=V.device)
        return V * torch.copysign(one, V[self.last])[self.col]


def _fix_columns(V):
    """The largest component of every column made positive."""
    big = V.gather(0, V.abs().argmax(0, keepdim=True))
    return V * (big.conj() / big.abs())


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": dict(case)}
    if kind == "one":
        st["A"] = _goe(case["n"], _gen(seed))
    elif kind == "hermitian":
        n, g = case["n"], _gen(seed)
        B = torch.complex(torch.randn(n, n, dtype=F64, device=DEV, generator=g),
                          torch.randn(n, n, dtype=F64, device=DEV, generator=g))
        st["A"] = (B + B.mH) / 2
    elif kind == "tridiag":
        st["T"] = glagpu.SymTridiagonal(*_beta_hermite(case["n"], seed))
    elif kind == "factor":
        g = _gen(seed)
        st["A"] = _goe(case["n"], g)
        st["B"] = torch.randn(case["n"], case["cols"], dtype=F64, device=DEV, generator=g)
    else:
        ns = _orders(case)
        jobz = case.get("jobz", "V")
        plan = glagpu.Plan(ns, precision=case["precision"], jobz=jobz, uplo=case.get("uplo", "L"),
                           alg=case.get("alg", "QL"))
        dt = torch.float32 if case["precision"] == "f32" else F64
        st["plan"] = plan
        st["A"] = _goe_arena(ns, _gen(seed), dt) if kind == "batch" else _prescribed_arena(ns, seed)
        if jobz == "V":
            st["signs"] = _Signs(ns)
        if kind in ("batch", "mixed"):
            st["w"] = torch.empty(plan.w_elems, dtype=dt, device=DEV)
            st["V"] = torch.empty(plan.a_elems, dtype=dt, device=DEV) if jobz == "V" else None
            st["info"] = torch.zeros(len(ns), dtype=torch.int32, device=DEV)
        if kind in ("grad", "mixed"):
            g = _gen(seed + 1)
            st["cw"] = torch.randn(plan.w_elems, dtype=F64, device=DEV, generator=g)
            st["cv"] = torch.randn(plan.a_elems, dtype=F64, device=DEV, generator=g)
        if kind == "mixed":
            st["Abar"] = torch.empty(plan.a_elems, dtype=F64, device=DEV)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "one":
        if case["jobz"] == "N":
            return {"w": glagpu.eigvals(st["A"], uplo=case["uplo"], precision=case["precision"])}
        r = glagpu.eigen(st["A"], uplo=case["uplo"], precision=case["precision"])
        return {"w": r.values, "V": _fix_columns(r.vectors)}
    if kind == "hermitian":
        r = glagpu.eigen(st["A"], uplo=case["uplo"])
        return {"w": r.values, "V": _fix_columns(r.vectors)}
    if kind == "tridiag":
        if case["jobz"] == "N":
            return {"w": glagpu.eigvals(st["T"])}
        r = glagpu.eigen(st["T"])
        return {"w": r.values, "V": _fix_columns(r.vectors)}
    if kind == "factor":
        F = glagpu.symtri(st["A"], uplo=case["uplo"])
        return {"d": F.diagonals.dv, "e": F.diagonals.ev, "QB": F.reflectors.lmul(st["B"])}
    plan = st["plan"]
    if kind == "batch":
        plan.execute(st["A"], st["w"], st["V"], st["info"])
        if case["jobz"] == "N":
            return {"w": st["w"], "info": st["info"]}
        return {"w": st["w"], "V": st["signs"].fix(st["V"]), "info": st["info"]}
    if kind == "grad":
        A = st["A"].detach().requires_grad_()
        w, V = glagpu.eigh_autograd(A, plan)
        loss = (st["cw"] * w).sum() + (st["cv"] * V * V).sum()
        loss.backward()
        return {"w": w.detach(), "V": st["signs"].fix(V.detach()), "grad": A.grad}
    plan.execute(st["A"], st["w"], st["V"], st["info"])
    Vbar = 2 * st["cv"] * st["V"]
    plan.adjoint(st["w"], st["V"], st["cw"], Vbar, st["Abar"])
    return {"w": st["w"], "V": st["signs"].fix(st["V"]), "info": st["info"], "grad": st["Abar"]}


def work(case):
    """Bytes of the matrices in and the results out; operations: 4/3 n^3 of the
    reduction, and for vectors 4/3 n^3 of the tridiagonal's and 2 n^3 of the
    back-transformation; 5 n^3 of the adjoint's products."""
    kind = case["kind"]
    if kind == "one":
        n, v = case["n"], case["jobz"] == "V"
        return {"bytes": 8 * (n * n * (2 if v else 1) + n), "flops": n ** 3 * (14 / 3 if v else 4 / 3)}
    if kind == "hermitian":
        n = case["n"]
        return {"bytes": 8 * (4 * n * n + n), "flops": 4 * n ** 3 * 14 / 3}
    if kind == "tridiag":
        n, v = case["n"], case["jobz"] == "V"
        return {"bytes": 8 * (3 * n + (n * n if v else 0)), "flops": n ** 3 * 4 / 3 if v else 30.0 * n * n}
    if kind == "factor":
        n, m = case["n"], case["cols"]
        return {"bytes": 8 * (2 * n * n + 2 * n * m), "flops": n ** 3 * 4 / 3 + 2.0 * n * n * m}
    ns = _orders(case).astype(float)
    n2, n3 = float((ns ** 2).sum()), float((ns ** 3).sum())
    size = 4 if case["precision"] == "f32" else 8
    if kind == "batch":
        v = case["jobz"] == "V"
        return {"bytes": size * (n2 * (2 if v else 1) + float(ns.sum())), "flops": n3 * (14 / 3 if v else 4 / 3)}
    return {"bytes": size * (4 * n2 + 2 * float(ns.sum())), "flops": n3 * (14 / 3 + 5)}


def _eigh(M):
    """Ascending eigenpairs in 64 bits."""
    return torch.linalg.eigh(M) if M.shape[0] > 160 else \
        tuple(torch.from_numpy(x).to(DEV) for x in np.linalg.eigh(M.cpu().numpy()))


def _tridiagonalise(A, uplo):
    """Householder's reduction with the reflectors' usual signs (beta against the
    column's head): d, e and Q."""
    A = A.copy() if uplo == "L" else A[::-1, ::-1].copy()
    n = A.shape[0]
    Q = np.eye(n)
    for j in range(n - 2):
        x = A[j + 1:, j].copy()
        s = np.linalg.norm(x[1:])
        if s == 0:
            continue
        beta = -math.copysign(math.hypot(x[0], s), x[0])
        v = x.copy()
        v[0] -= beta
        v /= np.linalg.norm(v)
        S = A[j + 1:, j + 1:]
        p = S @ v
        q = p - (p @ v) * v
        S -= 2 * (np.outer(v, q) + np.outer(q, v))
        A[j + 1:, j] = A[j, j + 1:] = 0
        A[j + 1, j] = A[j, j + 1] = beta
        Q[:, j + 1:] -= 2 * np.outer(Q[:, j + 1:] @ v, v)
    d, e = np.diag(A).copy(), np.diag(A, -1).copy()
    return (d, e, Q) if uplo == "L" else (d[::-1].copy(), e[::-1].copy(), Q[::-1, ::-1].copy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "factor":
        st = prepare(case, seed)
        d, e, Q = _tridiagonalise(st["A"].cpu().numpy(), case["uplo"])
        return {"d": d, "e": e, "QB": torch.from_numpy(np.ascontiguousarray(Q)).to(DEV) @ st["B"]}
    if kind in ("one", "hermitian"):
        w, V = torch.linalg.eigh(prepare(case, seed)["A"])
        return {"w": w} if case.get("jobz") == "N" else {"w": w, "V": _fix_columns(V)}
    if kind == "tridiag":
        d, e = _beta_hermite(case["n"], seed)
        w, V = torch.linalg.eigh(torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1))
        return {"w": w} if case["jobz"] == "N" else {"w": w, "V": _fix_columns(V)}
    st = prepare(case, seed)
    ns = _orders(case)
    ws, Vs, grads, ao, wo = [], [], [], 0, 0
    for n in ns.tolist():
        w, V = _eigh(st["A"][ao:ao + n * n].view(n, n).to(F64))
        ws.append(w)
        if case.get("jobz", "V") == "V":
            Vs.append(V.T.reshape(-1))
        if kind in ("grad", "mixed"):
            wbar = st["cw"][wo:wo + n]
            Vbar = 2 * st["cv"][ao:ao + n * n].view(n, n).T * V
            gap = w[None, :] - w[:, None]
            gap.fill_diagonal_(math.inf)
            M = (V.T @ Vbar) / gap
            grads.append((V @ (torch.diag(wbar) + (M + M.T) / 2) @ V.T).reshape(-1))
        ao += n * n
        wo += n
    out = {"w": torch.cat(ws)}
    if Vs:
        out["V"] = st["signs"].fix(torch.cat(Vs))
    if grads:
        out["grad"] = torch.cat(grads)
    return out
