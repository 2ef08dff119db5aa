"""Tridiagonal matrices of orders up to 128 whose entries, or couplings, lie
where the square of an FP64 number leaves the normal range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def graded(n, decades, seed):
    """d and e with the sizes s_i s_i and s_i s_i+1, s from 1 to 10^-decades."""
    rng = np.random.default_rng(seed)
    s = 10.0 ** (-decades * np.arange(n) / (n - 1))
    return rng.standard_normal(n) * s * s, rng.standard_normal(n - 1) * s[:-1] * s[1:]


def far_block(n, c, seed):
    """The lower half in units of c."""
    rng = np.random.default_rng(seed)
    s = np.where(np.arange(n) < n // 2, 1.0, c)
    return rng.standard_normal(n) * s, rng.standard_normal(n - 1) * np.minimum(s[:-1], s[1:])


@pytest.mark.parametrize("alg", ["QL", "QR"])
@pytest.mark.parametrize("flip", [False, True])
def test_tridiagonal(G, alg, flip):
    for n in (3, 4, 17, 64, 128):
        cases = [graded(n, p, n) for p in (20, 75, 150)] + [far_block(n, c, n) for c in (1e-140, 1e-160, 1e-200, 1e-290)]
        for d, e in cases:
            if flip:
                d, e = d[::-1].copy(), e[::-1].copy()
            w, V = G.eigen(G.SymTridiagonal(d, e), alg=alg)
            T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
            nT = np.linalg.norm(T, 2)
            assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 8 * n * EPS * nT
            assert np.linalg.norm(T @ V - V * w, 2) <= 1e-13 * nT
            assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= 1e-13
