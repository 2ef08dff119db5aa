"""Divide and conquer on tridiagonals whose merges deflate by pairs (copies of
one block glued by small entries, equal diagonals), by size (tiny couplings)
or hardly at all, below and above the length that the pair deflation stages
at a time."""
import numpy as np
import pytest

from helpers import residual, orth

pytestmark = pytest.mark.gpu
EPS64 = 2.0 ** -52


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def tridiagonal(kind, n):
    rng = np.random.default_rng(n)
    if kind == "glued":  # Wilkinson blocks W21+ glued by 1e-9
        d = np.abs(np.arange(n) % 21 - 10.0)
        e = np.ones(n - 1)
        e[20::21] = 1e-9
        return d, e
    if kind == "equal":
        return np.full(n, 0.5), 1e-17 * rng.standard_normal(n - 1)
    if kind == "toeplitz":
        return np.full(n, 2.0), np.full(n - 1, -1.0)
    d = rng.standard_normal(n)  # signs and magnitudes over twelve decades
    return d, rng.standard_normal(n - 1) * 10.0 ** rng.uniform(-12, 0, n - 1)


@pytest.mark.parametrize("kind", ["glued", "equal", "toeplitz", "mixed"])
@pytest.mark.parametrize("n", [129, 143, 272, 1030, 2205])
def test_tridiagonal_deflation(G, kind, n):
    d, e = tridiagonal(kind, n)
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    r = G.eigen(G.SymTridiagonal(d, e))
    nT = np.abs(r.values).max()
    assert np.all(np.diff(r.values) >= 0)
    assert np.abs(r.values - np.linalg.eigvalsh(T)).max() <= 8 * n * EPS64 * nT
    assert residual(T, r.vectors, r.values) <= 1e-13 and orth(r.vectors) <= 1e-13
