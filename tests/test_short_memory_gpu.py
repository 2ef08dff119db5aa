"""Calls with little device memory left: most of it is held by the test while
they run, and given back afterwards."""
import contextlib

import numpy as np
import pytest

from helpers import goe

pytestmark = pytest.mark.gpu
OUT_OF_MEMORY = -1002  # cudaErrorMemoryAllocation


@pytest.fixture(scope="module")
def G():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    glagpu.eigvals(goe(300, 1))  # kernels loaded
    return glagpu


@contextlib.contextmanager
def only(leave):
    """At most `leave` bytes of device memory free inside."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    for unit in (1 << 30, 16 << 20, 2 << 20):
        n = (torch.cuda.mem_get_info()[0] - leave) // unit
        if n > 0:
            held.append(torch.empty(n * unit, dtype=torch.uint8, device="cuda"))
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_a_failed_allocation_is_told_once(G):
    G.release_workspaces()
    A = goe(200, 2)
    want = G.symtri(A).diagonals.dv.cpu().numpy()
    with only(40 << 20):
        with pytest.raises(G.GLAError) as e:
            G.Plan([2000])
        assert e.value.status == OUT_OF_MEMORY
    assert np.array_equal(G.symtri(A).diagonals.dv.cpu().numpy(), want)


@pytest.mark.parametrize("precision", ["f64", "f32_refined"])
@pytest.mark.parametrize("ns", [[1000] * 8, [700, 700, 700, 300, 300, 500]])
def test_repeated_orders_share_a_context(G, precision, ns):
    # memory for one context an order, but not for one a matrix
    import torch
    G.release_workspaces()
    plan = G.Plan(ns, precision=precision)
    A = plan.pack([torch.tensor(goe(n, k + n), device="cuda") for k, n in enumerate(ns)], device="cuda")
    outs = []
    for short in (False, True):
        w, V = torch.empty(plan.w_elems, dtype=A.dtype, device="cuda"), torch.empty_like(A)
        wbar, Vbar, Abar = torch.ones_like(w), torch.ones_like(V), torch.empty_like(V)
        info = torch.zeros(len(ns), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        need = plan.workspace_bytes() * 4 // 5 if not short else need
        if short:
            plan.close()
        with only(need) if short else contextlib.nullcontext():
            if short:
                plan = G.Plan(ns, precision=precision)
            plan.execute(A, w, V, info)
            torch.cuda.synchronize()
            if short:
                assert plan.workspace_bytes() < need
        assert (info.cpu().numpy() == 0).all()
        # the adjoint's workspaces: 84 n^2 bytes each
        with only((128 << 20) + 120 * max(ns) ** 2) if short else contextlib.nullcontext():
            for _ in range(2):
                plan.adjoint(w, V, wbar, Vbar, Abar)
            torch.cuda.synchronize()
        outs.append([x.cpu().numpy() for x in (w, V, Abar)])
    plan.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b)


def test_other_calls_take_the_kept_plans_memory(G):
    # the kept plans hold 0.9 GB; what is left beside them is too little for a context of order 1000
    import torch
    rng = np.random.default_rng(1)
    mats = [torch.tensor(goe(1000, k), device="cuda") for k in range(8)]
    C = rng.standard_normal((500, 500)) + 1j * rng.standard_normal((500, 500))
    Q = rng.standard_normal((250, 250, 4))
    Q = np.concatenate([(Q + Q.swapaxes(0, 1))[..., :1], (Q - Q.swapaxes(0, 1))[..., 1:]], axis=-1) / 2
    calls = [lambda: G.symtri(mats[0]).diagonals.dv, lambda: G.eigvals(torch.tensor(C + C.conj().T, device="cuda")),
             lambda: G.eigvals(G.QuaternionMatrix(torch.tensor(Q, device="cuda"))),
             lambda: G.eigvals(G.SymTridiagonal(mats[0][0], mats[0][1, 1:])),
             lambda: torch.tensor(G.Plan([1000, 999]).workspace_bytes())]
    for f in calls:
        G.release_workspaces()
        want = f()
        G.release_workspaces()
        G.eigen_batched(mats)
        assert len(G._plan_pool._plans) == 1
        with only(64 << 20):
            got = f()
        assert len(G._plan_pool._plans) == 0 and torch.equal(got, want)
    G.release_workspaces()


def test_refined_batch_with_fewer_ctas(G):
    # every CTA of the persistent kernel has 0.9 MB of slices (twice that where the host pipeline runs)
    rng = np.random.default_rng(3)
    ns = rng.integers(8, 17, 2000)
    G.release_workspaces()
    outs = []
    for leave in (None, 400 << 20, 160 << 20):
        with only(leave) if leave else contextlib.nullcontext():
            plan = G.Plan(ns, precision="f32_refined")
            A = plan.pack([goe(int(n), 10 * k + int(n)) for k, n in enumerate(ns)])
            w, V, info = np.zeros(plan.w_elems), np.zeros(plan.a_elems), np.zeros(len(ns), np.int32)
            plan.execute_host(A, w, V, info)
            if leave:
                assert plan.workspace_bytes() < leave
            plan.close()
        assert not info.any()
        outs.append((w, V))
    for w, V in outs[1:]:
        assert np.array_equal(w, outs[0][0]) and np.array_equal(V, outs[0][1])
