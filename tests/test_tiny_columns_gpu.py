"""Reflector columns that are tiny beside the rest of the matrix, in the large
FP64 reduction: one row and column coupled to an O(1) block, as a kernel matrix
with one far point has it. Orders whose trailing matrix is reduced in fixed
point and orders that never are."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu
EPS64 = 2.0 ** -52


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def coupled(n, c):
    """[0.3, c v'; c v, B]: to 1e-100 the eigenvalues of B and 0.3."""
    B = goe(n - 1, n)
    A = np.zeros((n, n))
    A[1:, 1:] = B
    A[0, 0] = 0.3
    A[1:, 0] = A[0, 1:] = c * np.random.default_rng(n).standard_normal(n - 1)
    return A, np.sort(np.append(np.linalg.eigvalsh(B), 0.3))


@pytest.mark.parametrize("n", [300, 1056, 1089])
def test_tiny_first_column(G, n):
    import torch
    for c in (1e-125, 1e-140, 1e-150):
        A, want = coupled(n, c)
        w = G.eigvals(torch.tensor(A, device="cuda")).cpu().numpy()
        assert np.abs(w - want).max() <= 8 * n * EPS64 * np.abs(want).max(), c
    r = G.eigen(torch.tensor(A, device="cuda"))
    V = r.vectors.cpu().numpy()
    assert np.linalg.norm(A @ V - V * r.values.cpu().numpy(), 2) <= 1e-13 * np.abs(want).max()
    assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= 1e-13


@pytest.mark.parametrize("precision,c", [("f64", 1e-154), ("f64", 1e-157), ("f64", 1e-165), ("f32", 1e-19),
                                         ("f32", 1e-20), ("f32", 1e-22), ("f32_refined", 1e-20)])
@pytest.mark.parametrize("n", [150, 300, 1056])
def test_first_column_whose_square_underflows(G, n, precision, c):
    # the squared norm of the column is subnormal or zero in the working precision
    import torch
    A, want = coupled(n, c)
    dt = torch.float32 if precision == "f32" else torch.float64
    eps = 2.0 ** -23 if precision == "f32" else EPS64
    r = G.eigen(torch.tensor(A, device="cuda", dtype=dt), precision=precision)
    w, V = r.values.cpu().numpy().astype(np.float64), r.vectors.cpu().numpy().astype(np.float64)
    nA = np.abs(want).max()
    assert np.abs(w - want).max() <= 8 * n * eps * nA
    if precision != "f32":
        assert np.linalg.norm(A @ V - V * w, 2) <= 1e-13 * nA
        assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= 1e-13
