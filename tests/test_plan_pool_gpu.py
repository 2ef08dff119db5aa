"""The plans that the one-shot calls keep: repeated calls with new inputs,
several threads on their own streams, the bound, and giving everything back."""
import threading

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


def check(A, r):
    w, V = r.values.cpu().numpy(), r.vectors.cpu().numpy()
    n = A.shape[0]
    assert np.linalg.norm(A @ V - V * w, 2) <= 1e-13 * np.linalg.norm(A, 2)
    assert np.linalg.norm(V.T @ V - np.eye(n), 2) <= 1e-13


@pytest.mark.parametrize("precision", ["f64", "f32_refined"])
def test_repeated_calls_and_threads(G, precision):
    import torch
    mats = {n: [goe(n, 10 * n + k) for k in range(3)] for n in (40, 200)}
    first = {n: G.eigen(torch.tensor(m[0], device="cuda"), precision=precision) for n, m in mats.items()}
    errors = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for n, m in mats.items():
                    for A in m[k:] + m[:k]:
                        check(A, G.eigen(torch.tensor(A, device="cuda"), precision=precision))
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for n, m in mats.items():  # a kept plan gives a new one's bits
        again = G.eigen(torch.tensor(m[0], device="cuda"), precision=precision)
        assert torch.equal(first[n].values, again.values) and torch.equal(first[n].vectors, again.vectors)


def test_bounded_and_given_back(G):
    import torch
    pool = G._plan_pool
    for n in range(20, 20 + pool.entries + 5):
        G.eigvals(torch.tensor(goe(n, n), device="cuda"))
    assert len(pool._plans) <= pool.entries and 0 < pool._bytes <= pool.limit
    G.release_workspaces()
    assert len(pool._plans) == 0 and pool._bytes == 0
    with pytest.raises(G.NonFiniteError):
        G.eigen(np.full((30, 30), np.nan))
    check(goe(30, 1), G.eigen(torch.tensor(goe(30, 1), device="cuda")))
