"""FP32 eigenvalues by bisection at the ends of the range: a reduction that
overflowed is reported, and small eigenvalues of entries that stand alone come
back as they are."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def values(G, mats):
    plan = G.Plan([m.shape[0] for m in mats], precision="f32", jobz="N")
    w, info = np.zeros(plan.w_elems, np.float32), np.zeros(len(mats), np.int32)
    plan.execute_host(plan.pack(mats), w, None, info)
    return plan.unpack(w)[0], info


def test_overflow_is_reported(G):
    mats = [np.full((100, 100), 1e37, np.float32), np.float32(goe(60, 1)), np.full((33, 33), 3e37, np.float32)]
    w, info = values(G, mats)
    assert info[0] > 0 and info[1] == 0 and info[2] > 0
    assert np.isnan(w[0]).all() and np.isnan(w[2]).all()
    assert np.abs(w[1] - np.linalg.eigvalsh(mats[1].astype(np.float64))).max() <= 8 * 60 * 2.0 ** -23 * 20
    with pytest.raises(G.NonConvergenceError):
        G.eigvals(mats[0], precision="f32")


def test_small_values_that_stand_alone(G):
    rng = np.random.default_rng(2)
    lists = [[1e8, 1e-29], [1e38, 1e-38, -3e-38, 0, 1e-38], [1, 1e-40, 2e-20, -1e-44], [-2e38, 1e-45, 0, 0, -1e-45, 3],
             [1e-45], [0, 0], list(rng.standard_normal(128) * 10.0 ** rng.uniform(-44, 37, 128))]
    ds = [np.float32(x) for x in lists]
    w, info = values(G, [np.diag(d) for d in ds])
    assert not info.any()
    for d, x in zip(ds, w):
        assert np.array_equal(x, np.sort(d)), d
    # beside a block of size 1e30: its eigenvalues to FP32 accuracy, the others as they are
    B = np.float32(goe(20, 3) * 1e30)
    d = np.float32([1e-38, -1e-40, 0, 7e-20, -5e-30])
    A = np.zeros((25, 25), np.float32)
    A[:20, :20] = B
    A[20:, 20:] = np.diag(d)
    x = values(G, [A])[0][0]
    small = np.abs(x) < 1e20
    assert np.array_equal(x[small], np.sort(d))
    want = np.linalg.eigvalsh(B.astype(np.float64))
    assert np.abs(x[~small] - want).max() <= 8 * 20 * 2.0 ** -23 * np.abs(want).max()


def test_graded_and_rank_deficient(G):
    rng = np.random.default_rng(5)
    X = np.float32(rng.integers(-3, 4, (40, 10)))
    A = X @ X.T  # rank 10, whole numbers
    T = np.diag(np.float32(2.0 ** -np.arange(0, 100, 5.0)))
    w, info = values(G, [A, T])
    assert not info.any()
    nA = np.linalg.norm(A, 2)
    assert np.abs(w[0] - np.linalg.eigvalsh(A.astype(np.float64))).max() <= 8 * 40 * 2.0 ** -23 * nA
    assert np.array_equal(w[1], np.sort(np.diag(T)))
