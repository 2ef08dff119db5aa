"""The FP64 chase with four lanes per matrix, the shear replay and the FP64
reduction at the orders where they can go wrong (one and two entries, the
edges of a warp and of a 32-bit word, the largest), on graded and split
spectra, and on matrices scaled so far that the fast rotation and the fast
reflector scalars do not apply."""
import numpy as np
import pytest

from helpers import goe, residual, orth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS64 = 2.0 ** -52
ORDERS = (1, 2, 3, 4, 5, 16, 31, 32, 33, 63, 65, 96, 97, 127, 128)


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def matrix(kind, n):
    A = goe(n, 4100 + n)
    if kind == "graded":  # rows and columns falling over 24 decades
        s = 10.0 ** np.linspace(0, -12, n)
        A = A * s[:, None] * s[None, :]
    elif kind == "split":  # exact zeros leave blocks of their own
        h = n // 2
        A[:h, h:] = 0
        A[h:, :h] = 0
    return A


@pytest.mark.parametrize("alg", ["QL", "QR"])
@pytest.mark.parametrize("kind,scale", [("goe", 0), ("goe", 500), ("goe", -500), ("graded", 0), ("split", 0)])
def test_chase_orders_and_ranges(G, alg, kind, scale):
    mats = [matrix(kind, n) for n in ORDERS]
    res = G.eigen_batched([m * 2.0 ** scale for m in mats], alg=alg)
    for A, r in zip(mats, res):
        n = A.shape[0]
        w, V = r.values * 2.0 ** -scale, r.vectors  # exact
        nA = max(np.linalg.norm(A, 2), 1e-300)
        wo, _, _ = O.syev(A)
        assert np.all(np.diff(w) >= 0)
        assert np.abs(w - wo).max() <= 8 * n * EPS64 * nA
        assert residual(A, V, w) <= 1e-13 and orth(V) <= 1e-13
