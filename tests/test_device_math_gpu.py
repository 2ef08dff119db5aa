"""Device functions that stand in for an FP64 instruction or two, against the
host's arithmetic."""
import ctypes

import numpy as np
import pytest

from device_harness import compile_cuda

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "df64.cuh"
#include "gla_common.cuh"
using namespace gla;
__global__ void k(int what, int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  double r, s;
  if (what == 0) out[i] = f3_diff(f3_from(x), f3_from(y));
  if (what == 1) out[i] = rcp64(x);
  if (what == 2) out[i] = sqrt64(x);
  if (what >= 3) sqrt_rsqrt64(x, r, s);
  if (what == 3) out[i] = r;
  if (what == 4) out[i] = s;
}
extern "C" int run(int what, int n, const double* a, const double* b, double* out) {
  double* d;
  if (cudaMalloc((void**)&d, sizeof(double) * 3 * n)) return 1;
  cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(what, n, d, d + n, d + 2 * n);
  int rc = cudaGetLastError() != cudaSuccess;
  rc |= cudaMemcpy(out, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = compile_cuda(SOURCE, tmp_path_factory.mktemp("math"))

    def call(what, a, b=None):
        a = np.ascontiguousarray(a, np.float64)
        b = np.zeros_like(a) if b is None else np.ascontiguousarray(b, np.float64)
        out = np.empty_like(a)
        assert lib.run(what, a.size, *(ctypes.c_void_p(x.ctypes.data) for x in (a, b, out))) == 0
        return out

    return call


def test_differences_of_three_floats(device):
    # pairs at every distance, from size 1 down to one unit in the last place:
    # within four float roundings of the exact difference (two_sum's parts, their
    # sum, and the last sum)
    rng = np.random.default_rng(1)
    a = rng.uniform(-2, 2, 400000)
    b = a * (1 + 2.0 ** -rng.uniform(0, 53, a.size) * rng.choice([-1, 1], a.size))
    b[:1000] = a[:1000]
    b[1000:2000] = np.nextafter(a[1000:2000], 9)
    b[2000:3000] = -a[2000:3000]
    exact = a.astype(np.longdouble) - b.astype(np.longdouble)
    got = device(0, a, b).astype(np.longdouble)
    assert (np.abs(got - exact) <= 4 * 2.0 ** -24 * np.abs(exact)).all()


def test_seeded_reciprocals_and_roots(device):
    # relative errors: the last rounding (2^-53) for 1/x; for the roots half of
    # that of x y as well; 1% for what the third-order step leaves out
    u = np.longdouble(2.0) ** -53
    rng = np.random.default_rng(2)
    x = rng.uniform(1, 2, 500000) * 2.0 ** rng.integers(-1000, 1001, 500000)
    x[:5] = 1, 2, 4, 2.0 ** 1000, 2.0 ** -1000
    X = x.astype(np.longdouble)
    for sign in (1, -1):
        got = device(1, sign * x).astype(np.longdouble)
        assert (np.abs(sign * got * X - 1) <= 1.01 * u).all()
    for what in (2, 3):
        root = np.sqrt(X)
        assert (np.abs(device(what, x).astype(np.longdouble) - root) <= 1.01 * 1.5 * u * root).all()
    assert (np.abs(device(4, x).astype(np.longdouble) * np.sqrt(X) - 1) <= 1.01 * 1.5 * u).all()
