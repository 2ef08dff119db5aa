"""Tridiagonal input above order 128: a call with a NaN or an infinity leaves
nothing behind for the next one of its order, and entries near the ends of the
FP64 range; dense input whose largest entry is subnormal."""
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


def half_kept(n):
    """Two halves, coupled at the rounding level: the upper one's vectors are
    spread out and drop out of the last merge, of the lower one's, unit vectors,
    a single one stays (an entry z of a half's end row stays when
    100 u |z| sqrt(2) > 8 u |T|, |T| = 4)."""
    h = n // 2
    d = np.concatenate([np.full(h, 2.0), np.linspace(0.1, 3.9, n - h)])
    e = np.concatenate([np.full(h - 1, -1.0), [100 * 2.0 ** -53], np.zeros(n - h - 1)])
    return d, e


@pytest.mark.parametrize("n", [129, 256, 512, 1001])
def test_after_a_non_finite_call(G, n):
    rng = np.random.default_rng(n)
    cases = [half_kept(n), (rng.standard_normal(n), rng.standard_normal(n - 1))]
    fresh = []
    for d, e in cases:
        G.release_workspaces()
        fresh.append(G.eigen(G.SymTridiagonal(d, e)))
    for bad in (np.nan, np.inf):
        for where in (0, 1):
            d, e = cases[1][0].copy(), cases[1][1].copy()
            (d, e)[where][n // 3] = bad
            with pytest.raises(G.NonFiniteError):
                G.eigen(G.SymTridiagonal(d, e))
            with pytest.raises(G.NonFiniteError):
                G.eigvals(G.SymTridiagonal(d, e))
        for (d, e), want in zip(cases, fresh):
            r = G.eigen(G.SymTridiagonal(d, e))
            assert np.array_equal(r.values, want.values) and np.array_equal(r.vectors, want.vectors)
    T = np.diag(cases[0][0]) + np.diag(cases[0][1], 1) + np.diag(cases[0][1], -1)
    w, V = fresh[0]
    assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 8 * n * EPS64 * 4
    assert np.linalg.norm(T @ V - V * w, 2) <= 1e-13 * 4 and np.linalg.norm(V.T @ V - np.eye(n), 2) <= 1e-13


@pytest.mark.parametrize("k", [-1000, -600, 600, 1000])
def test_tridiagonal_of_any_size(G, k):
    n = 300
    rng = np.random.default_rng(7)
    d, e = rng.uniform(0.5, 2, n), rng.uniform(0.5, 2, n - 1)
    r = G.eigen(G.SymTridiagonal(d, e))
    s = G.eigen(G.SymTridiagonal(np.ldexp(d, k), np.ldexp(e, k)))
    assert np.array_equal(s.values, np.ldexp(r.values, k)) and np.array_equal(s.vectors, r.vectors)


def test_subnormal_dense_matrix(G):
    n = 200
    A = np.ldexp(goe(n, 4), -1060)  # entries of up to 16 bits
    r = G.eigen(A)
    up = np.ldexp(A, 1060)
    nA = np.linalg.norm(up, 2)
    w = np.ldexp(r.values, 1060)
    assert np.abs(w - np.linalg.eigvalsh(up)).max() <= 8 * n * EPS64 * nA + 2.0 ** -14
    assert np.linalg.norm(r.vectors.T @ r.vectors - np.eye(n), 2) <= 1e-13
