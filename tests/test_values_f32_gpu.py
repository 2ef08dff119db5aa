"""FP32 eigenvalues by bisection (jobz 'N', default tolerance): orders at the
edges of a warp, diagonal matrices (exact), graded and split ones, matrices
near the ends of the FP32 range, and non-finite input."""
import numpy as np
import pytest

from helpers import goe
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS32 = 2.0 ** -23
ORDERS = (1, 2, 3, 31, 32, 33, 64, 65, 96, 127, 128)


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


@pytest.mark.parametrize("scale", [0, 100, -100])
def test_goe_values(G, scale):
    mats = [np.float32(goe(n, 60 + n)) for n in ORDERS]
    ws = G.eigvals_batched([m * np.float32(2.0 ** scale) for m in mats], precision="f32")
    for A, w in zip(mats, ws):
        n = A.shape[0]
        wo = O.syev(A.astype(np.float64), "N")[0]
        w = w.astype(np.float64) * 2.0 ** -scale
        assert np.all(np.diff(w) >= 0)
        assert np.abs(w - wo).max() <= 8 * n * EPS32 * max(np.linalg.norm(A.astype(np.float64), 2), 1e-30)


def test_values_with_a_known_spectrum(G):
    rng = np.random.default_rng(3)
    diag = np.float32(rng.standard_normal(100) * 10.0 ** rng.uniform(-20, 3, 100))
    zero = np.zeros((40, 40), np.float32)
    two = np.zeros((65, 65), np.float32)  # 2 x 2 blocks [[1, h], [h, 1]], h = 2^-k: eigenvalues 1 +- h exactly
    for k in range(20):
        two[2 * k, 2 * k] = two[2 * k + 1, 2 * k + 1] = 1
        two[2 * k, 2 * k + 1] = two[2 * k + 1, 2 * k] = 2.0 ** -k
    ws = G.eigvals_batched([np.diag(diag), zero, two], precision="f32")
    assert np.array_equal(ws[0], np.sort(diag))
    assert np.array_equal(ws[1], np.zeros(40, np.float32))
    want = np.sort(np.concatenate([1 + 2.0 ** -np.arange(20), 1 - 2.0 ** -np.arange(20), np.zeros(25)]))
    assert np.abs(ws[2] - want).max() <= 2 * EPS32


def test_non_finite_and_other_tolerance(G):
    A, B = np.float32(goe(50, 1)), np.float32(goe(50, 2))
    A[3, 2] = A[2, 3] = np.nan
    plan = G.Plan([50, 50], precision="f32", jobz="N")
    w, info = np.zeros(100, np.float32), np.zeros(2, np.int32)
    plan.execute_host(plan.pack([A, B]), w, None, info)
    assert list(info) == [-1, 0] and np.isnan(w[:50]).all()
    wt = G.eigvals(B, precision="f32", tol=1e-6)  # the chase
    assert np.abs(w[50:] - wt).max() <= 50 * 8 * EPS32 * np.linalg.norm(B, 2)
