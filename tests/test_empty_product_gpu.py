"""A product with no terms in the grouped tensor-core GEMM (a merge of divide
and conquer whose kept vectors all come from one half): zeros, whatever an
earlier product left in the words of its exponents."""
import ctypes

import numpy as np
import pytest

from device_harness import compile_cuda

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "ozaki64.cuh"
using namespace gla;
using namespace gla::oz64;
// C (m x n, leading dimension m) = the product of k = 0 terms, its exponents' words holding `word`
extern "C" int empty_product(int m, int n, int word, double* host) {
  const int rows = (m + kBM - 1) / kBM * kBM, cols = (n + kBM - 1) / kBM * kBM;
  double* C;
  int* w;
  GemmDesc* d;
  if (cudaMalloc((void**)&C, sizeof(double) * m * n) || cudaMalloc((void**)&w, sizeof(int) * (rows + cols + 1)) ||
      cudaMalloc((void**)&d, sizeof(GemmDesc)))
    return 1;
  GemmDesc h{};
  h.m = m;
  h.n = n;
  h.k = 0;
  h.C = C;
  h.ldc = m;
  int* words = new int[rows + cols + 1];
  for (int i = 0; i < rows + cols; i++) words[i] = word;
  words[rows + cols] = 0;  // the error word
  cudaMemcpy(w, words, sizeof(int) * (rows + cols + 1), cudaMemcpyHostToDevice);
  cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
  cudaMemset(C, 0xff, sizeof(double) * m * n);
  Group g{};
  g.d = d;
  g.ea = w;
  g.eb = w + rows;
  g.a_rows = rows;
  g.b_rows = cols;
  g.err = w + rows + cols;
  cudaFuncSetAttribute((const void*)k_group_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  const int tiles = rows / kBM * ((n + kBN - 1) / kBN);
  k_group_gemm<<<dim3(tiles, 1), kThreads, kSmem>>>(g);
  int rc = cudaGetLastError() != cudaSuccess;
  rc |= cudaMemcpy(host, C, sizeof(double) * m * n, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(C);
  cudaFree(w);
  cudaFree(d);
  delete[] words;
  return rc;
}
"""


def test_product_without_terms(tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = compile_cuda(SOURCE, tmp_path)
    for m, n in ((128, 1), (130, 65), (129, 192)):
        for word in (0, 5, 1 << 20):  # 2^20 marks a row with a non-finite entry
            C = np.empty((n, m))
            assert lib.empty_product(m, n, word, ctypes.c_void_p(C.ctypes.data)) == 0
            assert (C == 0).all(), (m, n, word)
