"""The FP64 reduction with its products in fixed point (trailing orders above
1000): orders at the edges of its 64 x 32 units and where only the first panels
take it, both triangles, and entries of very different size.

Bound: the normwise backward error of a Householder reduction with FP64 sums is
a small multiple of sqrt(n) u ||A|| in each column, n u ||A||_F over all of
them in the worst case; fixed point must stay within the same 8 n u ||A||_F."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def _matrix(n, kind):
    A = goe(n, 3 * n)
    if kind == "graded":  # units whose entries span 2^-52 .. 1, in rows and columns
        s = np.logspace(0, -8, n)
        A = A * s[:, None] * s[None, :]
    elif kind == "spikes":  # one large entry among tiny ones in most units
        B = A * 2.0 ** -60
        i = np.arange(0, n - 40, 37)
        B[i, i + 33] = B[i + 33, i] = A[i, i + 33]
        A = B
    elif kind == "split":  # whole units of zeros
        A[: n // 2, n // 2:] = 0
        A[n // 2:, : n // 2] = 0
    return A


@pytest.mark.parametrize("n,kind,uplo", [
    (1001, "dense", "L"), (1002, "dense", "U"), (1033, "dense", "L"), (1056, "graded", "L"), (1057, "spikes", "U"),
    (1088, "split", "L"), (1089, "graded", "U"), (1151, "dense", "U"), (1216, "spikes", "L")])
def test_fixed_point_panels(G, n, kind, uplo):
    A = _matrix(n, kind)
    B = np.tril(A) if uplo == "L" else np.triu(A)
    B = B + (np.triu(np.full((n, n), 3.0), 1) if uplo == "L" else np.tril(np.full((n, n), 3.0), -1))
    w, V = G.eigen(B, uplo=uplo)
    w, V = np.asarray(w), np.asarray(V)
    nrm = np.linalg.norm(A)
    assert np.linalg.norm(A @ V - V * w) <= 8 * n * U * nrm
    assert np.linalg.norm(V.T @ V - np.eye(n)) <= 8 * n * U * np.sqrt(n)
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 8 * n * U * np.linalg.norm(A, 2) + 8 * n * U * nrm / np.sqrt(n)
