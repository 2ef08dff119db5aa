"""A tensor-core product of a complex or quaternion call whose bounded wait ran
out: that call reports it, and the next one is clean. The mark such a wait
leaves is set by the test; no kernel waits in vain here."""
import numpy as np
import pytest

from device_harness import compile_cuda
from helpers import qherm_random

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "gla_large.h"
extern "C" int mark(int quaternion) {
  gla::Oz64Gemm* w = quaternion ? gla::quaternion_gemm() : gla::complex_gemm();
  return w ? (int)gla::oz64_gemm_mark(w) : -1;
}
"""


def test_a_wait_that_ran_out_is_reported_once(tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu as G
    lib = compile_cuda(SOURCE, tmp_path, link=[G._lib.LIB_PATH])
    rng = np.random.default_rng(1)
    n = 130
    B = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    for quaternion, A in ((0, B + B.conj().T), (1, G.QuaternionMatrix(qherm_random(n, rng)))):
        first = G.eigen(A)
        assert lib.mark(quaternion) == 0
        with pytest.raises(G.GLAError) as e:
            G.eigen(A)
        assert e.value.status == -1702  # cudaErrorLaunchTimeout
        again = G.eigen(A)
        assert np.array_equal(first.values, again.values) and np.array_equal(first.vectors, again.vectors)
