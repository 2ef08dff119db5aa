"""Large matrices whose tridiagonal has blocks far below its largest entry:
matrices of low rank (each step of the reduction leaves rounding errors of the
step before) and graded ones."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu
EPS = {"f64": 2.0 ** -52, "f32_refined": 2.0 ** -52, "f32": 2.0 ** -23}


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def graded(n, decades):
    s = 10.0 ** (-decades * np.arange(n) / (n - 1))
    return goe(n, 1) * np.outer(s, s)


def low_rank(n, r):
    X = np.random.default_rng(n + r).integers(-3, 4, (n, r)).astype(float)
    return X @ X.T


def check(G, A, precision):
    import torch
    n = A.shape[0]
    A = A.astype(np.float32).astype(np.float64) if precision == "f32" else A
    r = G.eigen(torch.tensor(A, device="cuda", dtype=torch.float32 if precision == "f32" else torch.float64),
                precision=precision)
    w, V = r.values.cpu().numpy().astype(np.float64), r.vectors.cpu().numpy().astype(np.float64)
    nA = np.linalg.norm(A, 2)
    bound = max(1e-13, 8 * n * EPS[precision])
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= bound * nA
    assert np.linalg.norm(A @ V - V * w, 2) <= bound * nA
    assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= bound


@pytest.mark.parametrize("precision", ["f64", "f32", "f32_refined"])
@pytest.mark.parametrize("n", [150, 257, 371, 513, 1100])
def test_low_rank(G, n, precision):
    check(G, np.ones((n, n)), precision)
    check(G, low_rank(n, 1), precision)
    check(G, low_rank(n, 5), precision)


@pytest.mark.parametrize("precision", ["f64", "f32", "f32_refined"])
@pytest.mark.parametrize("n", [200, 371, 513])
def test_graded(G, n, precision):
    for decades in (5, 10, 15, 20, 40):
        check(G, graded(n, decades), precision)
