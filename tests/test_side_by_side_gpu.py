"""Several large matrices of one plan, solved side by side on streams and host
threads of their own: accuracy, repeated orders, the same bits from call to
call, other threads and streams at the same time, non-finite input."""
import threading

import numpy as np
import pytest

from helpers import goe, prescribed, residual, orth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    return glagpu


def matrices(ns, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k, n in enumerate(ns):
        if k % 2:
            out.append(prescribed(np.logspace(-8, 0, n) * rng.choice([-1.0, 1.0], n), seed + k))
        else:
            out.append(goe(n, seed + k))
    return out


def run(G, plan, mats, stream=None):
    import torch
    A = plan.pack(mats, device="cuda")
    w = torch.empty(plan.w_elems, dtype=torch.float64, device="cuda")
    V = torch.empty(plan.a_elems, dtype=torch.float64, device="cuda")
    info = torch.full((len(mats),), 7, dtype=torch.int32, device="cuda")
    plan.execute(A, w, V, info)
    return plan.unpack(w.cpu().numpy(), V.cpu().numpy()), info.cpu().numpy()


@pytest.mark.parametrize("precision", ["f64", "f32_refined"])
@pytest.mark.parametrize("ns", [[129, 130], [200] * 11 + [40, 3], [1024, 513, 300, 300, 1025, 128, 257, 700, 150, 151]])
def test_side_by_side(G, precision, ns):
    mats = matrices(ns, 5)
    plan = G.Plan(ns, precision=precision)
    (ws, Vs), info = run(G, plan, mats)
    assert (info == 0).all()
    for A, w, V in zip(mats, ws, Vs):
        nA = np.linalg.norm(A, 2)
        assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-13 * nA
        assert residual(A, V, w) <= 1e-13 and orth(V) <= 1e-13
    (w2, V2), _ = run(G, plan, mats)
    for a, b in zip(ws + Vs, w2 + V2):
        assert np.array_equal(a, b)


def test_non_finite_and_two_plans_at_once(G):
    import torch
    ns = [300, 200, 301, 200]
    mats = matrices(ns, 50)
    mats[1][5, 3] = mats[1][3, 5] = np.inf
    plans = [G.Plan(ns, precision=p) for p in ("f64", "f32_refined")]
    alone = [run(G, p, mats) for p in plans]
    for _, info in alone:
        assert list(info) == [0, -1, 0, 0]
    got = [None, None]

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[k] = run(G, plans[k], mats)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for ((w, V), info), ((w2, V2), info2) in zip(alone, got):
        assert np.array_equal(info, info2)
        for a, b in zip(w + V, w2 + V2):
            assert np.array_equal(a, b, equal_nan=True)
