"""Small matrices (orders up to 128) of low rank, whose reduction leaves columns
of rounding errors of rounding errors down to zero, and matrices with columns
far below the others."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu
ORDERS = (2, 3, 8, 16, 24, 33, 57, 64, 87, 100, 128)


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def low_rank(n, r):
    X = np.random.default_rng(n + r).integers(-3, 4, (n, r)).astype(float)
    return X @ X.T


def graded(n, decades):
    s = 10.0 ** (-decades * np.arange(n) / max(n - 1, 1))
    return goe(n, 1) * np.outer(s, s)


def far_column(n, c):
    A = goe(n, 2)
    A[0, 1:] *= c
    A[1:, 0] *= c
    return A


CASES = {
    "ones": lambda n: np.ones((n, n)),
    "rank 1": lambda n: low_rank(n, 1),
    "rank 3": lambda n: low_rank(n, 3),
    "graded 10": lambda n: graded(n, 10),
    "graded 20": lambda n: graded(n, 20),
    "far column 1e-20": lambda n: far_column(n, 1e-20),
}
FAR = {"graded 150": lambda n: graded(n, 150), "far column 1e-160": lambda n: far_column(n, 1e-160),
       "far column 1e-300": lambda n: far_column(n, 1e-300)}


def check(A, r, eps, n):
    w, V = r.values.astype(np.float64), r.vectors.astype(np.float64)
    nA = np.linalg.norm(A, 2)
    bound = max(1e-13, 8 * n * eps)
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= bound * nA
    assert np.linalg.norm(A @ V - V * w, 2) <= bound * nA
    assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= bound


@pytest.mark.parametrize("alg", ["QL", "QR"])
@pytest.mark.parametrize("precision", ["f64", "f32", "f32_refined"])
def test_eigenpairs(G, precision, alg):
    cases = dict(CASES, **FAR) if precision == "f64" else CASES
    for name, make in cases.items():
        mats = [make(n) for n in ORDERS]
        if precision == "f32":
            mats = [A.astype(np.float32).astype(np.float64) for A in mats]
        res = G.eigen_batched([A.astype(np.float32) if precision == "f32" else A for A in mats], precision=precision,
                              alg=alg)
        for A, r, n in zip(mats, res, ORDERS):
            check(A, r, 2.0 ** -23 if precision == "f32" else 2.0 ** -52, n)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_values_and_two_rows(G, precision):
    eps = 2.0 ** -23 if precision == "f32" else 2.0 ** -52
    for name, make in CASES.items():
        for n in ORDERS:
            A = make(n).astype(np.float32).astype(np.float64)
            nA, want = np.linalg.norm(A, 2), np.linalg.eigvalsh(A)
            X = A.astype(np.float32) if precision == "f32" else A
            if precision == "f32" or name in ("ones", "rank 1", "rank 3"):
                assert np.abs(G.eigvals(X, precision=precision) - want).max() <= 8 * n * eps * nA, (name, n)
            r = G.eigen2(X, precision=precision)
            assert np.abs(r.values - want).max() <= 8 * n * eps * nA, (name, n)
