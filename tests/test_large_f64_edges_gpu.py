"""The FP64 path above order 128, whose trailing updates, eigenvector updates
and back-transformation run on the tensor cores: orders at the edges of its
128-row blocks, 32-wide slabs and merge sizes, operands of odd widths, and
non-finite columns."""
import numpy as np
import pytest

from helpers import goe, prescribed, residual, orth

pytestmark = pytest.mark.gpu
EPS64 = 2.0 ** -52


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


@pytest.mark.parametrize("n", [129, 130, 159, 160, 161, 255, 256, 257, 258, 289, 384, 385, 512, 513, 641])
def test_eigen_block_edges(G, n):
    rng = np.random.default_rng(n)
    lam = np.logspace(-6, 0, n) * rng.choice([-1.0, 1.0], n)
    for A in (goe(n, n), prescribed(lam, n)):
        r = G.eigen(A)
        nA = np.linalg.norm(A, 2)
        assert np.abs(r.values - np.linalg.eigvalsh(A)).max() <= 8 * n * EPS64 * nA
        assert residual(A, r.vectors, r.values) <= 1e-13 and orth(r.vectors) <= 1e-13


def explicit_q(F):
    """Q of symtri's lower factors, one reflector after another."""
    f, tau = F.reflectors.factors.cpu().numpy(), F.reflectors.tau.cpu().numpy()
    n = f.shape[0]
    Q = np.eye(n)
    for k in range(n - 2, -1, -1):
        v = np.concatenate([[1.0], f[k + 2:, k]])
        Q[k + 1:] -= tau[k] * np.outer(v, v @ Q[k + 1:])
    return Q


@pytest.mark.parametrize("n,cols", [(129, 1), (200, 63), (256, 64), (257, 65), (300, 700), (385, 130)])
def test_eigenq_products(G, n, cols):
    import torch
    rng = np.random.default_rng(n + cols)
    F = G.symtri(torch.tensor(goe(n, 3 * n), device="cuda"))
    Q = explicit_q(F)
    B = rng.standard_normal((n, cols)) * 10.0 ** rng.integers(-6, 7, cols)
    nB = np.linalg.norm(B, axis=0)
    for trans in (False, True):
        X = F.reflectors.lmul(B, trans=trans)
        err = np.linalg.norm(X - (Q.T if trans else Q) @ B, axis=0)
        assert (err <= 8 * n * EPS64 * nB).all()
    # a column with a NaN or an infinity loses itself and no other
    Bad = B.copy()
    Bad[n // 2, 0] = np.nan
    if cols > 2:
        Bad[n - 1, 2] = np.inf
    Y, X = F.reflectors.lmul(Bad), F.reflectors.lmul(B)
    lost = [0, 2] if cols > 2 else [0]
    kept = [j for j in range(cols) if j not in lost]
    assert not np.isfinite(Y[1:, lost]).any()
    assert np.array_equal(Y[:, kept], X[:, kept])


@pytest.mark.parametrize("n", [127, 128, 129, 200])
def test_complex_and_quaternion_orthonormalisation(G, n):
    # the Newton-Schulz step's products change from the FP64 pipe to the
    # tensor cores at order 128
    from helpers import qherm_random, qmul, qH, qeye, qnorm
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A = (B + B.conj().T) / 2
    r = G.eigen(A)
    nA = np.linalg.norm(A, 2)
    assert np.abs(r.values - np.linalg.eigvalsh(A)).max() <= 16 * n * EPS64 * nA
    assert np.linalg.norm(A @ r.vectors - r.vectors * r.values, 2) <= 1e-13 * nA
    assert np.linalg.norm(r.vectors.conj().T @ r.vectors - np.eye(n), 2) <= 1e-13
    m = n // 2 if n < 200 else n
    A = qherm_random(m, rng)
    r = G.eigen(G.QuaternionMatrix(A))
    V, nA = r.vectors, qnorm(A)
    assert qnorm(qmul(A, V) - V * r.values[None, :, None]) <= 1e-13 * nA
    assert qnorm(qmul(qH(V), V) - qeye(m)) <= 1e-13
