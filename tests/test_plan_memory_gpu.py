"""Device memory of plans: the figure a plan gives for itself, and the bound of
the plans kept for the one-shot calls."""
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


def free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", ["f64", "f32", "f32_refined"])
@pytest.mark.parametrize("ns", [[1000] * 8, [700, 700, 300, 300, 90, 20], [1500], [100] * 200])
def test_the_figure_is_what_is_held(G, precision, ns):
    G.release_workspaces()
    for _ in range(2):  # (the first plan of the process also loads kernels)
        f0 = free()
        plan = G.Plan(ns, precision=precision)
        A = plan.pack([goe(n, n) for n in ns])
        w, V = np.zeros(plan.w_elems, plan.dtype), np.zeros(plan.a_elems, plan.dtype)
        plan.execute_host(A, w, V, np.zeros(len(ns), np.int32))
        if precision != "f32":
            plan.adjoint_host(w, V, w, V, np.zeros_like(V))
        held, said = f0 - free(), plan.workspace_bytes()
        plan.close()
    # the driver hands memory out in blocks of 2 MiB, so small buffers hold more than they say
    assert said <= held and held <= 1.3 * said + (64 << 20)


def test_the_kept_plans_stay_within_the_bound(G):
    import torch
    G.release_workspaces()
    pool = G._plan_pool
    mats = [torch.tensor(goe(1000, k), device="cuda") for k in range(8)]
    G.eigvals(mats[0])  # kernels loaded
    G.release_workspaces()
    f0 = free()
    for uplo in "LU":
        for precision in ("f64", "f32_refined"):
            G.eigen_batched(mats, uplo=uplo, precision=precision)
            G.eigvals_batched(mats, uplo=uplo, precision=precision)
            held = f0 - free()
            assert held <= pool.limit + (256 << 20), (uplo, precision)
            assert sum(n for _, n in pool._plans.values()) == pool._bytes <= pool.limit
    G.release_workspaces()
    assert len(pool._plans) == 0
