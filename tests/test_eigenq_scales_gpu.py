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
