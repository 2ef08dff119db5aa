"""Adjoints of several orders above 128 in one plan, which run side by side on
streams of their own: the same bits as each matrix's own plan gives (the same
kernels on the same inputs), next to small orders, from a stream of the
caller's and in a captured graph. And the FP32 back-transformation with columns
off the 16-byte boundaries (odd orders of the refined route)."""
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


def _adjoint(G, ns, mats, seeds):
    import torch
    plan = G.Plan(ns, precision="f32_refined")
    A = plan.pack(mats, device="cuda")
    w = torch.empty(plan.w_elems, dtype=torch.float64, device="cuda")
    V = torch.empty(plan.a_elems, dtype=torch.float64, device="cuda")
    info = torch.zeros(len(ns), dtype=torch.int32, device="cuda")
    plan.execute(A, w, V, info)
    assert not info.any()
    wbar = torch.cat([torch.from_numpy(np.random.default_rng(s).standard_normal(n)) for n, s in zip(ns, seeds)]).cuda()
    Vbar = torch.cat([torch.from_numpy(np.random.default_rng(s + 1).standard_normal(n * n)) for n, s in zip(ns, seeds)]).cuda()
    return plan, w, V, wbar, Vbar


@pytest.mark.parametrize("ns", [[129, 200], [301, 64, 257, 130, 511, 128, 300, 222, 190, 333, 401]])
def test_side_by_side_adjoints(G, ns):
    import torch
    mats = [goe(n, 40 + n) for n in ns]
    seeds = [100 + 2 * i for i in range(len(ns))]
    plan, w, V, wbar, Vbar = _adjoint(G, ns, mats, seeds)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    out = torch.full_like(V, float("nan"))
    plan.adjoint(w, V, wbar, Vbar, out, stream=s)
    s.synchronize()
    assert torch.isfinite(out).all()
    ao = np.cumsum([0] + [n * n for n in ns])
    wo = np.cumsum([0] + ns)
    for b, n in enumerate(ns):
        one = G.Plan([n], precision="f32_refined")
        sl, sw = slice(int(ao[b]), int(ao[b + 1])), slice(int(wo[b]), int(wo[b + 1]))
        ref = torch.empty_like(V[sl])
        one.adjoint(w[sw].clone(), V[sl].clone(), wbar[sw].clone(), Vbar[sl].clone(), ref)
        torch.cuda.synchronize()
        assert torch.equal(ref, out[sl]), n
    # captured: the streams fork from the capturing one and join it again
    g = torch.cuda.CUDAGraph()
    out2 = torch.zeros_like(out)
    with torch.cuda.graph(g):
        plan.adjoint(w, V, wbar, Vbar, out2, stream=torch.cuda.current_stream())
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, out2)


@pytest.mark.parametrize("n", [129, 130, 131, 197, 322, 641])
def test_refined_orders_off_the_boundary(G, n):
    # the refined route's own bound: 1e-14 ||A|| (its products) times sqrt(n), and a factor of 10
    A = goe(n, 7 * n)
    w, V = G.eigen(A, precision="f32_refined")
    w, V = np.asarray(w), np.asarray(V)
    nrm = np.linalg.norm(A, 2)
    tol = 1e-13 * np.sqrt(n)
    assert np.linalg.norm(A @ V - V * w) <= tol * nrm
    assert np.linalg.norm(V.T @ V - np.eye(n)) <= tol
