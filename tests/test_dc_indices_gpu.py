"""Divide and conquer's merged order on values that are not numbers: every index
it leaves stays inside the merge, whatever its memory held before."""
import ctypes

import numpy as np
import pytest

from device_harness import compile_cuda

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "large_dc.cu"
using namespace gla;
// k_dc_prep of one merge of m1 + m2 values; out: ssrc, ksrc, fsrc (m each), then k, nf
extern "C" int prep(int m1, int m2, const double* dd, double beta, int* out) {
  const int m = m1 + m2;
  double *f, *Z;
  int* w;
  if (cudaMalloc((void**)&f, sizeof(double) * 9 * m) || cudaMalloc((void**)&Z, sizeof(double) * m * m) ||
      cudaMalloc((void**)&w, sizeof(int) * (7 * m + 64)))
    return 1;
  cudaMemset(f, 0, sizeof(double) * 9 * m);
  cudaMemset(w, 0x3f, sizeof(int) * (7 * m + 64));  // what malloc might leave: far outside
  double* z = new double[m * m];
  for (int i = 0; i < m * m; i++) z[i] = 1.0 / (1 + i % 7);
  cudaMemcpy(Z, z, sizeof(double) * m * m, cudaMemcpyHostToDevice);
  delete[] z;
  DcArrays<double> a{};
  a.dd = f;
  a.e = f + m;
  a.sD = f + 2 * m;
  a.sZ = f + 3 * m;
  a.kd = f + 4 * m;
  a.kz = f + 5 * m;
  a.fd = f + 6 * m;
  a.rc = f + 7 * m;
  a.rs = f + 8 * m;
  a.ssrc = w;
  a.ksrc = w + m;
  a.fsrc = w + 2 * m;
  a.zdef = w + 3 * m;
  a.ctype = w + 4 * m;
  a.rp = w + 5 * m;
  a.rt = w + 6 * m;
  a.info = (MergeInfo*)(w + 7 * m);
  a.Zin = Z;
  a.ld = m;
  MergeInfo mi{};
  mi.m1 = m1;
  mi.m2 = m2;
  cudaMemcpy(a.info, &mi, sizeof(mi), cudaMemcpyHostToDevice);
  cudaMemcpy(a.dd, dd, sizeof(double) * m, cudaMemcpyHostToDevice);
  cudaMemcpy(f + m + m1 - 1, &beta, sizeof(double), cudaMemcpyHostToDevice);
  k_dc_prep<double><<<1, kPrepThreads>>>(a);
  int rc = cudaGetLastError() != cudaSuccess;
  rc |= cudaMemcpy(out, w, sizeof(int) * 3 * m, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaMemcpy(&mi, a.info, sizeof(mi), cudaMemcpyDeviceToHost);
  out[3 * m] = mi.k;
  out[3 * m + 1] = mi.nf;
  cudaFree(f);
  cudaFree(Z);
  cudaFree(w);
  return rc;
}
"""


def test_indices_stay_inside(tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import glagpu
    lib = compile_cuda(SOURCE, tmp_path, link=[glagpu._lib.LIB_PATH])
    lib.prep.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p]
    rng = np.random.default_rng(1)
    for m1, m2 in ((8, 8), (40, 41), (700, 600)):
        m = m1 + m2
        base = np.concatenate([np.sort(rng.standard_normal(m1)), np.sort(rng.standard_normal(m2))])
        for share in (0.0, 0.3, 1.0):
            dd = np.where(rng.random(m) < share, np.nan, base)
            out = np.zeros(3 * m + 2, np.int32)
            assert lib.prep(m1, m2, dd.ctypes.data, 0.5, out.ctypes.data) == 0
            ssrc, ksrc, fsrc, k, nf = out[:m], out[m:2 * m], out[2 * m:3 * m], out[-2], out[-1]
            assert 0 <= k and 0 <= nf and k + nf == m
            for idx in (ssrc, ksrc[:k], fsrc[:nf]):
                assert ((0 <= idx) & (idx < m)).all()
            if share == 0.0:
                assert (np.sort(ssrc) == np.arange(m)).all() and (np.diff(dd[ssrc]) >= 0).all()
