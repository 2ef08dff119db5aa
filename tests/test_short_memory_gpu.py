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
