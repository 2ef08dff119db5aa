"""symtri of matrices near the ends of the FP64 range, and symtri and its
products where blocks of very different size do not touch one another."""
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


@pytest.mark.parametrize("n", [1, 2, 90, 300, 1056])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_matrices_of_any_size(G, n, uplo):
    A = goe(n, 5)
    F = G.symtri(A, uplo=uplo)
    U = np.tril(F.reflectors.factors.cpu().numpy(), -2) if uplo == "L" else \
        np.triu(F.reflectors.factors.cpu().numpy(), 2)
    for k in (-900, -465, -201, -199, 199, 201, 465, 900):
        S = G.symtri(np.ldexp(A, k), uplo=uplo)
        assert np.array_equal(S.diagonals.dv.cpu().numpy(), np.ldexp(F.diagonals.dv.cpu().numpy(), k)), k
        assert np.array_equal(S.diagonals.ev.cpu().numpy(), np.ldexp(F.diagonals.ev.cpu().numpy(), k)), k
        if n > 1:
            assert np.array_equal(S.reflectors.tau.cpu().numpy(), F.reflectors.tau.cpu().numpy()), k
        factors = S.reflectors.factors.cpu().numpy()
        assert np.array_equal(np.tril(factors, -2) if uplo == "L" else np.triu(factors, 2), U), k
        assert np.array_equal(np.diag(factors), S.diagonals.dv.cpu().numpy()), k


@pytest.mark.parametrize("n,h", [(150, 40), (200, 60), (300, 100), (300, 170)])
def test_products_of_blocks_that_do_not_touch(G, n, h):
    # Q = diag(Q1, Q2): the second block's rows of a product owe nothing to the
    # first block's, however large these are
    A = np.zeros((n, n))
    A[:h, :h], A[h:, h:] = goe(h, 1), goe(n - h, 2)
    F = G.symtri(A)
    B = np.random.default_rng(3).standard_normal((n, 70))
    for trans in (False, True):
        want = F.reflectors.lmul(B, trans=trans)
        for s in (1e-20, 1e10, 1e20):
            Bs = B.copy()
            Bs[:h] *= s
            X = F.reflectors.lmul(Bs, trans=trans)
            bound = 8 * n * EPS64 * np.linalg.norm(B, axis=0)
            assert (np.linalg.norm(X[h:] - want[h:], axis=0) <= bound).all(), s
            assert (np.linalg.norm(X[:h] - s * want[:h], axis=0) <= s * bound).all(), s
            Y = F.reflectors.rmul(Bs.T.copy(), trans=not trans)
            assert (np.linalg.norm(Y.T[h:] - want[h:], axis=0) <= bound).all(), s


@pytest.mark.parametrize("n,h", [(300, 100), (1100, 50), (1200, 300)])
def test_blocks_of_two_sizes(G, n, h):
    # the second block's part of the tridiagonal to its own accuracy
    A1, A2 = goe(h, 1), goe(n - h, 2)
    w2 = np.linalg.eigvalsh(A2)
    for s in (1e10, 1e20):
        A = np.zeros((n, n))
        A[:h, :h], A[h:, h:] = s * A1, A2
        T = G.symtri(A).diagonals
        d, e = T.dv.cpu().numpy(), T.ev.cpu().numpy()
        assert e[h - 1] == 0
        w = np.linalg.eigvalsh(np.diag(d[h:]) + np.diag(e[h:], 1) + np.diag(e[h:], -1))
        assert np.abs(w - w2).max() <= 8 * n * EPS64 * np.abs(w2).max(), s
