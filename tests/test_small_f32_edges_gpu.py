"""The FP32 reduction and the application of Q with the matrix in registers, at
the edges of their 16 x 16 thread grid and of their four register shapes, for
each caller: FP32 by chase (QL), FP32 values, and the refined route (with the
tridiagonal solver, and with what that leaves to the chase).

Bounds: backward errors of Householder reductions are a modest multiple of
n eps ||A||_F (n eps for the orthogonality of their products); 10 of them are
allowed, eps = 2^-24 for FP32. The refined route works on 48-bit products and
stops at 1e-14 ||A||: 1e-12 ||A||_F."""
import numpy as np
import pytest
import torch

import glagpu

SIZES = [1, 2, 3, 4, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 80, 95, 96, 97, 112, 113, 127, 128]


def _matrix(n, kind, rng):
    if kind == "dense":
        A = rng.standard_normal((n, n))
        A = A + A.T
    elif kind == "split":  # columns that are zero below the subdiagonal, and whole zero rows
        A = rng.standard_normal((n, n))
        A = A + A.T
        h = n // 2
        A[:h, h:] = 0
        A[h:, :h] = 0
        A[n // 3, :] = 0
        A[:, n // 3] = 0
    elif kind == "tiny":  # columns whose squares leave the range of FP32
        s = np.where(np.arange(n) % 3 == 0, 1.0, 2.0 ** -70)
        A = rng.standard_normal((n, n))
        A = (A + A.T) * np.sqrt(np.outer(s, s)) + np.diag(np.arange(1.0, n + 1))
    else:  # diagonal, with a repeated value
        A = np.diag(np.where(np.arange(n) < n // 4, 1.0, np.arange(1.0, n + 1)))
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "split", "tiny", "diagonal"])
@pytest.mark.parametrize("precision,jobz,uplo", [("f32", "V", "L"), ("f32", "V", "U"), ("f32", "N", "L"),
                                                 ("f32_refined", "V", "L"), ("f32_refined", "V", "U")])
def test_small_f32_edges(kind, precision, jobz, uplo):
    rng = np.random.default_rng(11)
    mats = [_matrix(n, kind, rng) for n in SIZES]
    dt = np.float32 if precision == "f32" else np.float64
    arena, off = [], [0]
    for A in mats:
        B = A.astype(dt)
        n = len(B)
        # the other triangle is not to be read
        B = np.tril(B) + np.triu(np.full((n, n), 7.0, dt), 1) if uplo == "L" else np.triu(B) + np.tril(np.full((n, n), 7.0, dt), -1)
        arena.append(B.T.reshape(-1))  # column-major
    woff = np.cumsum([0] + SIZES)
    aoff = np.cumsum([0] + [n * n for n in SIZES])
    plan = glagpu.Plan(SIZES, precision=precision, jobz=jobz, uplo=uplo)
    Ad = torch.from_numpy(np.concatenate(arena)).cuda()
    w = torch.full((int(woff[-1]),), float("nan"), dtype=Ad.dtype, device="cuda")
    V = torch.full((int(aoff[-1]),), float("nan"), dtype=Ad.dtype, device="cuda") if jobz == "V" else None
    info = torch.full((len(SIZES),), -7, dtype=torch.int32, device="cuda")
    plan.execute(Ad, w, V, info)
    torch.cuda.synchronize()
    assert not info.any()
    for b, n in enumerate(SIZES):
        A = mats[b].astype(dt).astype(np.float64)
        nrm = np.linalg.norm(A)
        rel = 10 * n * 2.0 ** -24 if precision == "f32" else 1e-12
        wb = w[woff[b]:woff[b + 1]].cpu().numpy().astype(np.float64)
        assert np.abs(wb - np.linalg.eigvalsh(A)).max() <= rel * nrm, (n, "values")
        if jobz == "V":
            Vb = V[aoff[b]:aoff[b + 1]].cpu().numpy().astype(np.float64).reshape(n, n).T
            assert np.linalg.norm(Vb.T @ Vb - np.eye(n)) <= rel * max(1.0, np.sqrt(n)), (n, "orthogonality")
            assert np.linalg.norm(A @ Vb - Vb * wb) <= rel * nrm, (n, "residual")
