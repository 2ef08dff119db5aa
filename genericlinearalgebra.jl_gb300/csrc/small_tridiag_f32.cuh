// FP32 Householder reduction and application of Q with the matrix in the
// registers of one CTA (256 threads, n <= 128), used by tridiag_body
// (small_tridiag.cuh) for float.
//
// What bounds it: a column is a chain of dependent steps (norm, reflector,
// product, correction, update), and with the matrix in shared memory every
// step was a loop of dependent shared-memory accesses: about 5000 cycles a
// column at n = 128 with the FP32 pipe 5% busy. Here thread (tx, ty) of a
// 16 x 16 grid keeps the entries (ty + 16 u, tx + 16 v) of the full symmetric
// matrix, so that a step is at most NB^2 independent FMAs per thread, and the
// cyclic distribution lets whole register rows and columns drop out as the
// trailing matrix shrinks (the loops over u and v start at the block KB of
// the current column, for which the code is unrolled; one loop with a switch
// around the FMAs took 196 us where this takes 128). Two barriers a column: 1900 to 2100
// cycles with two CTAs on the SM (order 128: 385 -> 128 us a matrix).
//
// The reflectors are applied to X = Q Y by warps that own whole columns of X
// (no barrier at all), which takes the place of forming Q and the product
// Q Y (order 128: 282 -> 60 us); Q itself, where it is asked for, is Y = I.
#pragma once
#include "gla_small.cuh"

namespace gla {

constexpr int kRegNT = 256;     // threads the register path takes
constexpr int kXsStride = 12;   // 8 values of a thread row or column, padded: 16 lanes' float4 reads fall on all banks
constexpr int kXsWords = 16 * kXsStride;

// Words of the staged reflectors: n - 2 rows of 16 NB values.
__host__ __device__ inline size_t reg_v_words(int n) {
  const size_t row = n <= 32 ? 32 : n <= 64 ? 64 : n <= 96 ? 96 : 128;
  return (size_t)(n > 2 ? n - 2 : 0) * row;
}

// Place of entry i of a reflector in its row of RU * 8 words: lane i % 8 of a
// column group reads its entries i / 8 four at a time, eight lanes on
// different banks (RU = 16 and 8 need the exclusive or, 12 and 4 do not).
template <int RU>
GLA_DEV int v_place(int i) {
  constexpr int NG = RU / 4;
  const int lr = i & 7, u = i >> 3;
  const int x = NG == 4 ? (lr >> 1) & 3 : NG == 2 ? (lr >> 2) & 1 : 0;
  return ((lr * NG + ((u >> 2) ^ x)) << 2) + (u & 3);
}

// The values v >= KB & ~3 of a thread row or column (p: 16-byte aligned).
template <int NB, int KB>
GLA_DEV void load_vals(const float* p, float (&o)[8]) {
#pragma unroll
  for (int g = KB / 4; g < (NB + 3) / 4; g++) {
    const float4 q = *reinterpret_cast<const float4*>(p + 4 * g);
    o[4 * g] = q.x;
    o[4 * g + 1] = q.y;
    o[4 * g + 2] = q.z;
    o[4 * g + 3] = q.w;
  }
}

// Sum over the 16 lanes of a half warp of p[0 .. L), value index r of the
// padded power of two left in the lanes whose upper bits spell r (the value
// is returned by all of them).
template <int L>
GLA_DEV float half_warp_rowsum(float (&p)[8], int& r) {
  constexpr int P = L > 4 ? 8 : L > 2 ? 4 : L > 1 ? 2 : 1;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = L; q < P; q++) p[q] = 0.f;
  int s = 8;
  r = 0;
#pragma unroll
  for (int w = P / 2; w >= 1; w /= 2, s /= 2) {
    const bool up = lane & s;
#pragma unroll
    for (int q = 0; q < w; q++) {
      const float keep = up ? p[q + w] : p[q], send = up ? p[q] : p[q + w];
      p[q] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
    r += up ? w : 0;
  }
#pragma unroll
  for (; s >= 1; s /= 2) p[0] += __shfl_xor_sync(0xffffffffu, p[0], s);
  return p[0];
}

// symtriLower! (GenericLinearAlgebra.jl src/eigenSelfAdjoint.jl:450-504) with
// reflector! as tridiag_body restates it. S: the lower triangle staged with
// leading dimension ld. Leaves the diagonals in dd and ee (ee[n-1] = 0), the
// scalars in taus, and hands entry i of reflector k (all n of them, zeros
// above k + 1 and from n to 16 NB) to storev(k, i, v). xs: 3 kXsWords words of shared scratch.
template <int NB, int KB, class SV>
GLA_DEV void tridiag_regs_block(float (&a)[NB][NB], int n, float* dd, float* ee, float* taus, float* xs,
                                const SV& storev);
template <int NB, class SV>
GLA_DEV void tridiag_regs(int n, const float* S, int ld, float* dd, float* ee, float* taus, float* xs,
                          const SV& storev) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  float a[NB][NB];
#pragma unroll
  for (int u = 0; u < NB; u++)
#pragma unroll
    for (int v = 0; v < NB; v++) {
      const int i = ty + 16 * u, j = tx + 16 * v;
      const int lo = min(i, j), hi = max(i, j);
      a[u][v] = hi < n ? S[lo * ld + hi] : 0.f;
    }
  __syncthreads();  // S is free (storev may write there)
  tridiag_regs_block<NB, 0>(a, n, dd, ee, taus, xs, storev);
  __syncthreads();
}

// Columns 16 KB .. of tridiag_regs.
template <int NB, int KB, class SV>
GLA_DEV void tridiag_regs_block(float (&a)[NB][NB], int n, float* dd, float* ee, float* taus, float* xs,
                                const SV& storev) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, wid = tid >> 5;
  const unsigned half = 0xffffu << (tid & 16);
  float* ps = xs + 2 * kXsWords;
#pragma unroll 1
  for (int kk = 0; kk < 16; kk++) {
    const int k = 16 * KB + kk;
    if (k >= n) return;
    float* xk = xs + (k & 1) * kXsWords;
    if (wid == (kk >> 1)) {  // the warp that holds row k makes its reflector
      float x[NB], s2 = 0.f;
      unsigned mb = 0;
#pragma unroll
      for (int v = KB; v < NB; v++) {
        x[v] = tx + 16 * v > k ? a[KB][v] : 0.f;
        s2 = fmaf(x[v], x[v], s2);
        mb = max(mb, __float_as_uint(x[v]) & 0x7fffffffu);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
      }
      const float x0 = __shfl_sync(0xffffffffu, kk < 15 ? a[KB][KB] : a[KB][KB + 1 < NB ? KB + 1 : KB], (kk + 1) & 15, 16);
      const bool mine = ty == kk;
      if (mine && tx == kk) dd[k] = a[KB][KB];
      if (k + 2 >= n) {
        if (mine && tx == 0) ee[k] = k + 1 < n ? x0 : 0.f;
      } else {
        float tau = 0.f, scl = 0.f, nu = 0.f;
        if (mb != 0) {  // (alike in the 16 lanes of a row)
          const float maxabs = __uint_as_float(mb), mm = maxabs * maxabs;
          float y0 = x0, up = 1.f;
          if (!(isfinite((float)(n - k - 1) * mm) && mm >= 0x1p-100f)) {
            // squares (nearly) out of range: the column by an exact power of
            // two, so that 1/x1 and, where it is subnormal, nu keep their digits
            const int ex = min(max((int)(mb >> 23) - 127, -126), 126);
            const float dn = __int_as_float((127 - ex) << 23);
            up = __int_as_float((127 + ex) << 23);
            y0 *= dn;
            s2 = 0.f;
#pragma unroll
            for (int v = KB; v < NB; v++) {
              x[v] *= dn;
              s2 = fmaf(x[v], x[v], s2);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s2 += __shfl_xor_sync(half, s2, o);
          }
          nu = copysignf(prec<float>::sqrt_ieee(s2), y0);
          const float xi1 = y0 + nu;
          tau = prec<float>::div_ieee(xi1, nu);
          scl = prec<float>::tame(xi1) ? prec<float>::rcp(xi1) : prec<float>::div_ieee(1.f, xi1);
          nu *= up;
        }
        if (mine) {
#pragma unroll
          for (int v = 0; v < NB; v++) {
            const int j = tx + 16 * v;
            const float vj = (v < KB || j <= k || j >= n) ? 0.f : (j == k + 1 && mb != 0) ? 1.f : x[v < KB ? KB : v] * scl;
            if (v >= KB) xk[tx * kXsStride + v] = vj;
            storev(k, j, vj);
          }
          if (tx == 0) {
            taus[k] = tau;
            ee[k] = -nu;
          }
        }
      }
    }
    __syncthreads();
    if (k + 2 >= n) continue;
    float cv[8], p[8];
    load_vals<NB, KB>(xk + tx * kXsStride, cv);
#pragma unroll
    for (int u = KB; u < NB; u++) {
      float s = 0.f;
#pragma unroll
      for (int v = KB; v < NB; v++) s = fmaf(a[u][v], cv[v], s);
      p[u - KB] = s;
    }
    int r;
    const float sum = half_warp_rowsum<NB - KB>(p, r);
    if (r < NB - KB) ps[ty * kXsStride + KB + r] = sum;  // (lanes of one r write the same)
    __syncthreads();
    // u = tau A v, w = tau (v'u) v - u: A += v w' - u v'. Rows and columns up
    // to k are dead: what they hold stays finite and meets zeros in v.
    const float tau = taus[k];
    float w[8], dot = 0.f;
    load_vals<NB, KB>(ps + tx * kXsStride, w);
#pragma unroll
    for (int v = KB; v < NB; v++) dot = fmaf(cv[v], w[v], dot);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float xiv = tau * (tau * dot);
#pragma unroll
    for (int v = KB; v < NB; v++) w[v] = fmaf(xiv, cv[v], -tau * w[v]);
    float vr[8], pr[8];
    load_vals<NB, KB>(xk + ty * kXsStride, vr);
    load_vals<NB, KB>(ps + ty * kXsStride, pr);
#pragma unroll
    for (int u = KB; u < NB; u++) {
      const float ui = tau * pr[u];
#pragma unroll
      for (int v = KB; v < NB; v++) a[u][v] = fmaf(-ui, cv[v], fmaf(vr[u], w[v], a[u][v]));
    }
  }
  if constexpr (KB + 1 < NB) tridiag_regs_block<NB, KB + 1>(a, n, dd, ee, taus, xs, storev);
}

// The reflectors 32 QB + 31 .. 0 of apply_q_regs, in that order.
template <int NB, int QB>
GLA_DEV void apply_q_block(float (&x)[2 * NB][NB / 2], int n, const float* Vs, const float* taus) {
  constexpr int RU = 2 * NB, CV = NB / 2, U0 = 4 * QB;  // rows below 8 U0 are zero in v
  const int lr = threadIdx.x & 7;
#pragma unroll 1
  for (int k = min(32 * QB + 31, n - 3); k >= 32 * QB; k--) {
    const float* vk = Vs + (size_t)k * (8 * RU);
    float v[RU], d[CV];
#pragma unroll
    for (int u = U0; u < RU; u += 4) {
      const float4 q = *reinterpret_cast<const float4*>(vk + v_place<RU>(lr + 8 * u));
      v[u] = q.x;
      v[u + 1] = q.y;
      v[u + 2] = q.z;
      v[u + 3] = q.w;
    }
#pragma unroll
    for (int c = 0; c < CV; c++) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int u = U0; u < RU; u += 2) {
        s0 = fmaf(v[u], x[u][c], s0);
        s1 = fmaf(v[u + 1], x[u + 1][c], s1);
      }
      d[c] = s0 + s1;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < CV; c++) d[c] += __shfl_xor_sync(0xffffffffu, d[c], o);
    const float tau = taus[k];
#pragma unroll
    for (int c = 0; c < CV; c++) {
      const float t = -tau * d[c];
#pragma unroll
      for (int u = U0; u < RU; u++) x[u][c] = fmaf(v[u], t, x[u][c]);
    }
  }
  if constexpr (QB > 0) apply_q_block<NB, QB - 1>(x, n, Vs, taus);
}

// X = H_0 H_1 ... H_{n-3} Y for Y read through y(i, c), X stored through
// x(i, c, value). Vs: the reflectors in shared memory, row k at Vs + k RU 8
// with its entries at v_place, zeros from n on. Warp w holds the columns
// w 2 NB .. (w + 1) 2 NB - 1, lane (lr, lc) the rows lr + 8 u of the columns
// lc + 4 c, so that a reflector is 2 RU CV FMAs and two reductions over 8
// lanes. y is read by all threads before `ready` (which must end with a
// barrier) puts the reflectors in place.
template <int NB, class Y, class RD, class ST>
GLA_DEV void apply_q_regs(int n, const float* Vs, const float* taus, const Y& y, const RD& ready, const ST& store) {
  constexpr int RU = 2 * NB, CV = NB / 2;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, lr = lane & 7;
  const int c0 = wid * 2 * NB + (lane >> 3);
  float x[RU][CV];
#pragma unroll
  for (int u = 0; u < RU; u++)
#pragma unroll
    for (int c = 0; c < CV; c++) {
      const int i = lr + 8 * u, cc = c0 + 4 * c;
      x[u][c] = (i < n && cc < n) ? y(i, cc) : 0.f;
    }
  ready();
  if (wid * 2 * NB < n) apply_q_block<NB, NB / 2 - 1>(x, n, Vs, taus);
#pragma unroll
  for (int u = 0; u < RU; u++)
#pragma unroll
    for (int c = 0; c < CV; c++) {
      const int i = lr + 8 * u, cc = c0 + 4 * c;
      if (i < n && cc < n) store(i, cc, x[u][c]);
    }
}

}  // namespace gla
