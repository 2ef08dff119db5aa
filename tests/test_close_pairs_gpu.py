"""Complex and quaternion matrices with eigenvalues 1e-6 to 1e-13 ||A|| apart:
far enough for one real eigenvector each, too near for one orthonormalisation
step."""
import numpy as np
import pytest

from helpers import haar, qeye, qH, qmul, qnorm

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def wilkinson(n):
    return np.diag(np.abs(np.arange(n) - (n - 1) / 2)) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)


def gaps(n):
    rng = np.random.default_rng(n)
    lam = np.repeat(np.linspace(-1, 1, (n + 2) // 3), 3)[:n]
    lam[1::3] += 10.0 ** -rng.uniform(6, 13, len(lam[1::3]))
    lam[2::3] -= 10.0 ** -rng.uniform(6, 13, len(lam[2::3]))
    Q = haar(n, rng)
    A = (Q * lam) @ Q.T
    return (A + A.T) / 2


def gauss(n):
    x = np.random.default_rng(n).standard_normal((n, 2))
    return np.exp(-((x[:, None] - x[None]) ** 2).sum(-1))


KINDS = {"wilkinson": wilkinson, "gaps": gaps, "gauss": gauss}


@pytest.mark.parametrize("kind", KINDS)
def test_complex(G, kind):
    for n in (17, 32, 71, 128, 200):
        A = KINDS[kind](n)
        p = np.exp(2j * np.pi * np.random.default_rng(n).random(n))
        H = A * np.outer(p, p.conj())
        H = (H + H.conj().T) / 2
        nA = np.linalg.norm(A, 2)
        w, V = G.eigen(H)
        assert np.abs(w - np.linalg.eigvalsh(H)).max() <= 16 * n * EPS * nA
        assert np.linalg.norm(H @ V - V * w, 2) <= 1e-13 * nA
        assert np.linalg.norm(V.conj().T @ V - np.eye(n), 2) <= 1e-13


@pytest.mark.parametrize("kind", KINDS)
def test_quaternion(G, kind):
    for n in (17, 32, 71, 128):
        A = KINDS[kind](n)
        q = np.random.default_rng(n).standard_normal((n, 4))
        q /= np.linalg.norm(q, axis=1, keepdims=True)
        D, Aq = np.zeros((n, n, 4)), np.zeros((n, n, 4))
        D[np.arange(n), np.arange(n)], Aq[..., 0] = q, A
        H = qmul(qmul(D, Aq), qH(D))
        H = (H + qH(H)) / 2
        nA = np.linalg.norm(A, 2)
        w, V = G.eigen(G.QuaternionMatrix(H))
        assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 32 * n * EPS * nA
        assert qnorm(qmul(H, V) - V * w[None, :, None]) <= 1e-13 * nA
        assert qnorm(qmul(qH(V), V) - qeye(n)) <= 1e-13
