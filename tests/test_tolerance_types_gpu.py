"""The tolerance of a one-shot call as any one-valued number: the plan that is
kept for it is the same one."""
import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu


def test_tolerance_of_any_type():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu as G
    A = goe(40, 1)
    G.release_workspaces()
    want = G.eigen(A, tol=1e-13)
    for tol in (np.float64(1e-13), np.array(1e-13), torch.tensor(1e-13, dtype=torch.float64)):
        r = G.eigen(A, tol=tol)
        assert np.array_equal(r.values, want.values) and np.array_equal(r.vectors, want.vectors)
        assert np.array_equal(G.eigen2(A, tol=tol).values, G.eigen2(A, tol=1e-13).values)
    assert len(G._plan_pool._plans) == 1
