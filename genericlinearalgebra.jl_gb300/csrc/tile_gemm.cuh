// Batched small-matrix GEMM building blocks (one CTA of kTileThreads per
// matrix, 64 x 64 output tiles, 4 x 4 outputs per thread, operands read
// through accessor functors so that transposes, triangles and on-the-fly
// conversions cost nothing extra). Used by the eigenpair refinement and the
// adjoint kernel.
#pragma once
#include "df64.cuh"

namespace gla {

constexpr int kRT = 256;  // threads per CTA of the tile GEMMs

// C(i, j) = init(i, j) + sum_k la(i, k) * lb(k, j) over 64 x 64 output tiles;
// 256 threads, 4 x 4 outputs per thread, double-float accumulation.
// `upper` skips tiles strictly below the diagonal and stores i <= j only.
// Operand slices (16 x 64) are staged in shared memory with a padded row
// (kTP = 65 elements: conflict-free stores of the k-fastest global reads) and
// the next slice is prefetched into registers while the current one is used.
constexpr int kTP = 65;
template <class TB, class LA, class LB, class IN, class ST>
GLA_DEV void tile_gemm_df(int n, const LA& la, const LB& lb, const IN& init, const ST& store, df64* As, TB* Bs,
                          bool upper) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kk_ld = tid & 15, ii_ld = tid >> 4;  // this thread loads (kk_ld, ii_ld + 16 q), q < 4
  for (int i0 = 0; i0 < n; i0 += 64) {
    for (int j0 = 0; j0 < n; j0 += 64) {
      if (upper && j0 + 63 < i0) continue;
      df64 acc[4][4];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const int i = i0 + tx + 16 * u, j = j0 + ty + 16 * v;
          acc[u][v] = (i < n && j < n) ? init(i, j) : df_make(0.f, 0.f);
        }
      df64 ra[4];
      TB rb[4];
      auto fetch = [&](int k0) {
        const int k = k0 + kk_ld;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int i = i0 + ii_ld + 16 * q, j = j0 + ii_ld + 16 * q;
          ra[q] = (i < n && k < n) ? la(i, k) : df_make(0.f, 0.f);
          rb[q] = (j < n && k < n) ? lb(k, j) : TB();
        }
      };
      fetch(0);
      for (int k0 = 0; k0 < n; k0 += 16) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
          As[kk_ld * kTP + ii_ld + 16 * q] = ra[q];
          Bs[kk_ld * kTP + ii_ld + 16 * q] = rb[q];
        }
        __syncthreads();
        if (k0 + 16 < n) fetch(k0 + 16);
#pragma unroll 2
        for (int kk = 0; kk < 16; kk++) {
          df64 a[4];
          TB b[4];
#pragma unroll
          for (int u = 0; u < 4; u++) a[u] = As[kk * kTP + tx + 16 * u];
#pragma unroll
          for (int v = 0; v < 4; v++) b[v] = Bs[kk * kTP + ty + 16 * v];
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int v = 0; v < 4; v++) acc[u][v] = df_mac(acc[u][v], a[u], b[v]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const int i = i0 + tx + 16 * u, j = j0 + ty + 16 * v;
          if (i < n && j < n && (!upper || i <= j)) store(i, j, acc[u][v]);
        }
    }
  }
  __syncthreads();
}

// C(i, j) = sum_k la(i, k) lb(k, j) in FP32 for n <= 128 (the X E update):
// one tile of 16 TM x 16 TM outputs, TM x TM per thread in quads of rows and
// columns 64 apart, so that the operands come as float4 (TM = 8: 64 FMAs per
// four shared-memory loads; with 4 x 4 outputs read word by word the product
// of order 128 took 49 us with two CTAs on the SM). As, Bs: 16 x kTPF each.
constexpr int kTPF = 132;
template <int TM, class LA, class LB, class ST>
GLA_DEV void tile_gemm_f32_tm(int n, const LA& la, const LB& lb, const ST& store, float* As, float* Bs) {
  constexpr int NG = TM / 4;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kk_ld = tid & 15, ii_ld = tid >> 4;  // this thread loads (kk_ld, ii_ld + 16 q), q < TM
  float acc[TM][TM];
#pragma unroll
  for (int u = 0; u < TM; u++)
#pragma unroll
    for (int v = 0; v < TM; v++) acc[u][v] = 0.f;
  float ra[TM], rb[TM];
  auto fetch = [&](int k0) {
    const int k = k0 + kk_ld;
#pragma unroll
    for (int q = 0; q < TM; q++) {
      const int i = ii_ld + 16 * q;
      const bool in = i < n && k < n;
      ra[q] = in ? la(i, k) : 0.f;
      rb[q] = in ? lb(k, i) : 0.f;
    }
  };
  fetch(0);
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += 16) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TM; q++) {
      As[kk_ld * kTPF + ii_ld + 16 * q] = ra[q];
      Bs[kk_ld * kTPF + ii_ld + 16 * q] = rb[q];
    }
    __syncthreads();
    if (k0 + 16 < n) fetch(k0 + 16);
#pragma unroll 2
    for (int kk = 0; kk < 16; kk++) {
      float a[TM], b[TM];
#pragma unroll
      for (int g = 0; g < NG; g++) {
        const float4 x = *reinterpret_cast<const float4*>(As + kk * kTPF + 64 * g + 4 * tx);
        const float4 y = *reinterpret_cast<const float4*>(Bs + kk * kTPF + 64 * g + 4 * ty);
        a[4 * g] = x.x, a[4 * g + 1] = x.y, a[4 * g + 2] = x.z, a[4 * g + 3] = x.w;
        b[4 * g] = y.x, b[4 * g + 1] = y.y, b[4 * g + 2] = y.z, b[4 * g + 3] = y.w;
      }
#pragma unroll
      for (int u = 0; u < TM; u++)
#pragma unroll
        for (int v = 0; v < TM; v++) acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
    }
  }
#pragma unroll
  for (int u = 0; u < TM; u++)
#pragma unroll
    for (int v = 0; v < TM; v++) {
      const int i = 64 * (u >> 2) + 4 * tx + (u & 3), j = 64 * (v >> 2) + 4 * ty + (v & 3);
      if (i < n && j < n) store(i, j, acc[u][v]);
    }
  __syncthreads();
}
template <class LA, class LB, class ST>
GLA_DEV void tile_gemm_f32(int n, const LA& la, const LB& lb, const ST& store, float* As, float* Bs) {
  if (n <= 64) tile_gemm_f32_tm<4>(n, la, lb, store, As, Bs);
  else tile_gemm_f32_tm<8>(n, la, lb, store, As, Bs);
}

}  // namespace gla
