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
