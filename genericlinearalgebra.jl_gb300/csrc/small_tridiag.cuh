// Device body of the batched Householder tridiagonalisation (one CTA per
// matrix, n <= 128), shared by its kernel (small_tridiag.cu) and by the
// persistent FP32 + refinement kernel (refine.cu). See small_tridiag.cu.
#pragma once
#include <type_traits>

#include "df64.cuh"
#include "gla_small.cuh"
#include "small_stein.cuh"
#include "small_tridiag_f32.cuh"

namespace gla {

template <class T> struct AbsBits;
template <> struct AbsBits<double> {
  static GLA_DEV unsigned long long get(double x) { return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull; }
  static GLA_DEV double from(unsigned long long b) { return __longlong_as_double((long long)b); }
};
template <> struct AbsBits<float> {
  static GLA_DEV unsigned long long get(float x) { return (unsigned long long)(__float_as_uint(x) & 0x7fffffffu); }
  static GLA_DEV float from(unsigned long long b) { return __uint_as_float((unsigned)b); }
};

// Sum and max (of non-negative bit patterns) over the block.
GLA_DEV void block_sum_max(double v, unsigned long long m, double* red, unsigned long long* redm, double& sum,
                           unsigned long long& mx) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(0xffffffffu, v, o);
    unsigned long long w = __shfl_xor_sync(0xffffffffu, m, o);
    m = w > m ? w : m;
  }
  __syncthreads();
  if (lane == 0) {
    red[wid] = v;
    redm[wid] = m;
  }
  __syncthreads();
  // the warps' sums by three shuffles (nw <= 8): every warp would queue
  // nw - 1 additions on the FP64 pipe
  double s = (lane & 7) < nw ? red[lane & 7] : 0.0;
  unsigned long long x = (lane & 7) < nw ? redm[lane & 7] : 0ull;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    unsigned long long w = __shfl_xor_sync(0xffffffffu, x, o);
    x = w > x ? w : x;
  }
  sum = s;
  mx = x;
}

// The same for a sum alone.
GLA_DEV double block_sum8(double v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double s = (lane & 7) < nw ? red[lane & 7] : 0.0;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The reflector's scalars from x1 and the column's squared norm (FP64, both
// well inside the normal range): nu = copysign(norm, x1), tau = (x1 + nu)/nu
// and 1/(x1 + nu), each from one hardware seed (12 FP64 instructions; the IEEE
// square root and two divisions have a latency of about 30; with block_sum8
// and two threads per row, the reduction and Q of one matrix of order 64 went
// from 0.62 to 0.42 ms, of 512 of order 128 from 7.7 to 5.8).
GLA_DEV void reflector_scalars(double x0, double sumsq, double& nu, double& tau, double& scl) {
  double norm, rnorm;
  sqrt_rsqrt64(sumsq, norm, rnorm);
  nu = copysign(norm, x0);
  tau = fma(fabs(x0), rnorm, 1.0);
  scl = rcp64(x0 + nu);
}

// Leading dimension of the staged matrix: odd, so that transposed accesses
// (stride ld across the lanes of a warp) spread over all shared-memory banks.
__host__ __device__ inline int stage_ld(int n) { return (n + 1) | 1; }
// Words of the staged matrix (FP32: of the staged reflectors if these take
// more, and a multiple of 16 bytes).
__host__ __device__ inline size_t stage_words(int n, int elem) {
  const size_t s = (size_t)n * stage_ld(n);
  if (elem == 8) return s;
  const size_t v = reg_v_words(n);
  return ((s > v ? s : v) + 3) & ~(size_t)3;
}

// The part of tridiag_body after the staging, float with the matrix in
// registers (small_tridiag_f32.cuh). vv: the words after the staged matrix.
template <int NB, bool WANTQ, bool STEIN>
GLA_DEV void tridiag_body_regs(int mid, const SmallDesc& dsc, float* S, int ld, float* vv, float* __restrict__ dout,
                               float* __restrict__ eout, float* __restrict__ Qout, ChaseState* __restrict__ cst,
                               float* __restrict__ wout, float* __restrict__ qtmp, int sexp,
                               float* __restrict__ rows2) {
  constexpr int RU = 2 * NB;
  const int n = dsc.n, tid = threadIdx.x;
  float *dd = vv + n, *ee = vv + 2 * n, *taus = vv + 3 * n, *part = vv + 4 * n;
  float* Qt = STEIN ? qtmp + dsc.a_off : nullptr;
  // STEIN: S holds the vectors of the tridiagonal while the reflectors wait in
  // Qt; else they stay in S
  tridiag_regs<NB>(n, S, ld, dd, ee, taus, part, [&](int k, int i, float v) {
    if (!WANTQ && !rows2) return;
    if (!STEIN)
      S[(size_t)k * (8 * RU) + v_place<RU>(i)] = v;
    else if (i < n)
      Qt[(size_t)k * n + i] = v;
  });
  for (int i = tid; i < n; i += kRegNT) {
    dout[dsc.w_off + i] = dd[i];
    eout[dsc.w_off + i] = ee[i];
  }
  if constexpr (!WANTQ) {
    if (!rows2) return;
    // eigen2!'s rows 1 and n of Q (see tridiag_body_shared), row n in the
    // registers of warp 0
    __syncthreads();
    const int lane = tid & 31;
    float* R2 = rows2 + 2 * dsc.w_off;
    if (tid >= 32) return;
    float r[4];
#pragma unroll
    for (int q = 0; q < 4; q++) r[q] = lane + 32 * q == n - 1 ? 1.f : 0.f;
    for (int k = 0; k + 2 < n; k++) {
      float v[4], dot = 0.f;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        v[q] = lane + 32 * q < n ? S[(size_t)k * (8 * RU) + v_place<RU>(lane + 32 * q)] : 0.f;
        dot = fmaf(r[q], v[q], dot);
      }
      const float f = taus[k] * warp_sum(dot);
#pragma unroll
      for (int q = 0; q < 4; q++) r[q] = fmaf(-f, v[q], r[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = lane + 32 * q;
      if (i < n) {
        R2[2 * i] = i == 0 ? 1.f : 0.f;
        R2[2 * i + 1] = r[q];
      }
    }
  } else {
    float* Qg = Qout + dsc.a_off;
    auto identity = [&](int i, int c) { return i == c ? 1.f : 0.f; };
    auto store = [&](int i, int c, float v) { Qg[(size_t)c * n + i] = v; };
    if constexpr (STEIN) {
      auto fetch = [&]() {
        __syncthreads();
        batched<8>(
            max(n - 2, 0) * (8 * RU),
            [&](int idx) {
              const int k = idx / (8 * RU), i = idx % (8 * RU);
              return i < n ? Qt[(size_t)k * n + i] : 0.f;
            },
            [&](int idx, float v) {
              const int k = idx / (8 * RU), i = idx % (8 * RU);
              S[(size_t)k * (8 * RU) + v_place<RU>(i)] = v;
            });
        __syncthreads();
      };
      // Y in S (leading dimension ld), e^2, eigenvalues and flags in part
      // (8 x 256 >= 3 n + 104 + 3 x 256 words)
      float* e2s = part;
      float* lams = e2s + n;
      int* misc = reinterpret_cast<int*>(lams + n);  // [0] give up, [1] clusters, [2 + 2c], [3 + 2c] bounds
      const bool solved = stein_solve(n, dd, ee, e2s, lams, S, ld, misc, reinterpret_cast<float*>(misc + n + 8),
                                      misc + n + 104);
      if (solved) {
        for (int k = tid; k < n; k += kRegNT) wout[dsc.w_off + k] = sexp ? ldexpf(lams[k], sexp) : lams[k];
        if (tid == 0) {
          ChaseState st;
          st.bs = n;
          st.nsweeps = 0;
          st.nrot = 0;
          st.nhdr = 0;
          st.status = kChaseDone;
          st.applied = 1;
          cst[mid] = st;
        }
      }
      // X = Q Y, or Q for the QL chase (whose state stays "running")
      apply_q_regs<NB>(
          n, S, taus, [&](int i, int c) { return solved ? S[(size_t)i * ld + c] : identity(i, c); }, fetch, store);
    } else {
      apply_q_regs<NB>(n, S, taus, identity, []() {}, store);
    }
  }
}

// The part of tridiag_body after the staging, FP64: the matrix in shared memory.
template <bool WANTQ>
GLA_DEV void tridiag_body_shared(const SmallDesc& dsc, double* S, int ld, double* vv, double* red,
                                 unsigned long long* redm, double* __restrict__ dout, double* __restrict__ eout,
                                 double* __restrict__ Qout, double* __restrict__ rows2) {
  using T = double;
  const int n = dsc.n, tid = threadIdx.x, NT = blockDim.x;
  T* uu = vv + n;
  T* ww = uu + n;
  T* taus = ww + n;
  T* part = taus + n;
  // ---- symtriLower!: k = 0 .. n-3
  for (int k = 0; k + 2 < n; k++) {
    const int m = n - k - 1;
    T* xc = S + (size_t)k * ld + (k + 1);
    T xi = (tid < m) ? xc[tid] : T(0);
    const T x0 = xc[0];  // read before the reduction's barriers; thread 0 rewrites xc[0] below
    T sumsq;
    unsigned long long mb;
    block_sum_max(xi * xi, (tid < m) ? AbsBits<T>::get(xi) : 0ull, red, redm, sumsq, mb);
    T tau = 0;
    if (mb != 0) {
      // LinearAlgebra.reflector!: nu = copysign(norm, x1), x1 += nu,
      // x[2:] /= x1, tau = x1/nu, x[1] = -nu. A column far from 1 is brought
      // there first by an exact power of two: its squares, 1/x1 and, where it
      // is subnormal, nu keep their digits, and I - tau v v' stays orthogonal.
      T nu, scl;
      const int mbe = (int)(mb >> 52);  // (FP64) biased exponent of the largest entry
      if (mbe > 1023 - 400 && mbe < 1023 + 400) {
        reflector_scalars(x0, sumsq, nu, tau, scl);
      } else {
        const int ex = min(max(mbe - 1023, -1022), 1022);
        const T dn = __hiloint2double((1023 - ex) << 20, 0), up = __hiloint2double((1023 + ex) << 20, 0);
        xi *= dn;
        T s2;
        unsigned long long dummy;
        block_sum_max(xi * xi, 0ull, red, redm, s2, dummy);
        const T y0 = x0 * dn, nus = copysign(prec<T>::sqrt_ieee(s2), y0), y1 = y0 + nus;
        tau = prec<T>::div_ieee(y1, nus);
        scl = prec<T>::rcp(y1);
        nu = nus * up;
      }
      if (tid < m) {
        const T v = (tid == 0) ? T(1) : xi * scl;
        vv[tid] = v;
        xc[tid] = (tid == 0) ? -nu : v;
      }
    }
    if (tid == 0) taus[k] = tau;
    __syncthreads();
    if (mb == 0) continue;  // zero column: H = I, nothing to update

    // ---- u = tau * A~ * v (lower-triangle SYMV); rows x P column parts
    T* At = S + (size_t)(k + 1) * ld + (k + 1);
    {
      const int R = (m + 31) & ~31;
      int P = NT / R;
      P = P > 8 ? 8 : P;
      const int p = tid / R, i = tid - p * R;
      if (p < P && i < m) {
        const int j0 = (p * m) / P, j1 = ((p + 1) * m) / P;
        T acc0 = 0, acc1 = 0;
        int j = j0;
        for (; j + 1 < j1; j += 2) {
          const int a0 = (j <= i) ? (j * ld + i) : (i * ld + j);
          const int a1 = (j + 1 <= i) ? ((j + 1) * ld + i) : (i * ld + j + 1);
          acc0 = fma(At[a0], vv[j], acc0);
          acc1 = fma(At[a1], vv[j + 1], acc1);
        }
        if (j < j1) acc0 = fma(At[(j <= i) ? (j * ld + i) : (i * ld + j)], vv[j], acc0);
        part[p * R + i] = acc0 + acc1;
      }
      __syncthreads();
      T ui = 0;
      if (tid < m) {
        T s = part[tid];
        for (int q = 1; q < P; q++) s += part[q * R + tid];
        ui = tau * s;
        uu[tid] = ui;
      }
      // xi = tau * (v' u)
      const T vi = (tid < m) ? vv[tid] : T(0);
      const T xsum = block_sum8(vi * ui, red);
      const T xiv = tau * xsum;
      if (tid < m) ww[tid] = xiv * vi - ui;
      __syncthreads();
    }
    // ---- A~ += v w' - u v'   (== x(xi x)' - x u' - u x' of :484-491), lower triangle:
    // a warp per column (columns dealt in snake order, w, 2 nw - 1 - w, 2 nw + w,
    // ..., which evens out their lengths), lanes over its rows
    {
      const int lane = tid & 31, wid = tid >> 5, nw = NT >> 5;
      for (int r = 0;; r++) {
        const int j = r * nw + ((r & 1) ? (nw - 1 - wid) : wid);
        if (j >= m) break;
        const T wj = ww[j], vj = vv[j];
        T* col = At + (size_t)j * ld;
        for (int i = j + lane; i < m; i += 32) {
          T a = col[i];
          a = fma(vv[i], wj, a);
          a = fma(-uu[i], vj, a);
          col[i] = a;
        }
      }
    }
    __syncthreads();
  }

  // ---- diagonals
  T* dg = dout + dsc.w_off;
  T* eg = eout + dsc.w_off;
  for (int i = tid; i < n; i += NT) {
    const T di = S[(size_t)i * ld + i], ei = (i + 1 < n) ? S[(size_t)i * ld + i + 1] : T(0);
    dg[i] = di;
    eg[i] = ei;
  }
  if (!WANTQ && rows2) {
    // eigen2! (src/eigenSelfAdjoint.jl:633-644): only rows 1 and n of Q,
    // [e_1'; e_n'] Q = rmul!(V, Q) (:62-80), in place of Array(Q): row 1 is
    // e_1' (Q = diag(1, Qt)); row n is e_n' H_0 H_1 ... H_{n-3}, one
    // reflector at a time (H_k on indices k+1.., v = [1; column k below its
    // subdiagonal], tau_k). Stored 2 x n column-major at 2 w_off.
    __syncthreads();
    T* r = vv;  // the row being formed (n entries); uu holds the dot-product partials
    for (int i = tid; i < n; i += NT) r[i] = (i == n - 1) ? T(1) : T(0);
    __syncthreads();
    for (int k = 0; k + 2 < n; k++) {
      const T tau = taus[k];
      if (tau == T(0)) continue;  // uniform: taus is shared
      T part = T(0);
      for (int i = k + 1 + tid; i < n; i += NT) part = fma(r[i], (i == k + 1) ? T(1) : S[(size_t)k * ld + i], part);
      const T dot = block_sum8(part, red);
      const T f = tau * dot;
      for (int i = k + 1 + tid; i < n; i += NT) r[i] = fma(-f, (i == k + 1) ? T(1) : S[(size_t)k * ld + i], r[i]);
      __syncthreads();
    }
    T* R2 = rows2 + 2 * dsc.w_off;
    for (int i = tid; i < n; i += NT) {
      R2[2 * i] = (i == 0) ? T(1) : T(0);
      R2[2 * i + 1] = r[i];
    }
    return;
  }
  if (!WANTQ) return;
  __syncthreads();

  // ---- Q = H_0 H_1 ... H_{n-3} (Array(EigenQ) of the reference), in place.
  // Q = diag(1, Qt); reflector kk lives in column kk (rows kk+2..), Qt's
  // column kk is global column kk+1, formed after H_kk is applied to the
  // trailing columns kk+2.. (rows kk+1..).
  for (int r = tid; r < n; r += NT) S[(size_t)(n - 1) * ld + r] = (r == n - 1) ? T(1) : T(0);
  __syncthreads();
  for (int kk = n - 3; kk >= 0; kk--) {
    const T tau = taus[kk];
    const int M = n - kk - 1;
    if (tid < M) vv[tid] = (tid == 0) ? T(1) : S[(size_t)kk * ld + kk + 1 + tid];
    __syncthreads();
    const int C = n - kk - 2;
    if (tau != T(0)) {
      // two lanes per column (row halves), partial dots combined by shuffle
      const int half = (M + 1) >> 1;
      for (int t2 = tid; t2 < 2 * ((C + 15) / 16) * 16; t2 += NT) {
        const int t = t2 >> 1, h = t2 & 1;
        const bool live = t < C;
        T* col = S + (size_t)(kk + 2 + (live ? t : 0)) * ld + (kk + 1);
        const int r0 = h * half, r1 = h ? M : half;
        T d0 = 0, d1 = 0;
        if (live) {
          int r = r0;
          for (; r + 1 < r1; r += 2) {
            d0 = fma(vv[r], col[r], d0);
            d1 = fma(vv[r + 1], col[r + 1], d1);
          }
          if (r < r1) d0 = fma(vv[r], col[r], d0);
        }
        T dot = d0 + d1;
        dot += __shfl_xor_sync(0xffffffffu, dot, 1);
        const T tmp = tau * dot;
        if (live)
          for (int r = r0; r < r1; r++) col[r] = fma(-vv[r], tmp, col[r]);
      }
    }
    __syncthreads();
    {
      T* col = S + (size_t)(kk + 1) * ld;
      for (int r = tid; r < n; r += NT)
        col[r] = (r <= kk) ? T(0) : ((r == kk + 1) ? T(1) - tau : -tau * vv[r - kk - 1]);
    }
    __syncthreads();
  }
  for (int r = tid; r < n; r += NT) S[r] = (r == 0) ? T(1) : T(0);
  __syncthreads();
  T* Qg = Qout + dsc.a_off;
  for (int j = 0; j < n; j++)
    for (int i = tid; i < n; i += NT) Qg[(size_t)j * n + i] = S[(size_t)j * ld + i];
}

// Float runs with the matrix in registers (256 threads). STEIN (float only): after the reduction, solve the
// tridiagonal in the same CTA (small_stein.cuh) and write X = Q Y and the
// ascending eigenvalues (times 2^scale) to wout, marking the matrix done for
// the chase; a matrix the solver leaves to the QL chase gets Q as usual. The
// reflectors wait in qtmp (an n x n float scratch per matrix, arena layout)
// meanwhile, so that the solver's arrays reuse the shared memory of the
// reduction.
template <class T, class Tin, bool WANTQ, bool STEIN>
GLA_DEV void tridiag_body(int mid, unsigned char* smem_raw, const SmallDesc* __restrict__ descs,
                          const Tin* __restrict__ A, int lower, T* __restrict__ dout, T* __restrict__ eout,
                          T* __restrict__ Qout, int* __restrict__ info, ChaseState* __restrict__ cst,
                          int* __restrict__ scale_exp, T* __restrict__ wout, T* __restrict__ qtmp,
                          T* __restrict__ rows2 = nullptr) {
  const SmallDesc dsc = descs[mid];
  const int n = dsc.n;
  const int ld = stage_ld(n);
  const int tid = threadIdx.x, NT = blockDim.x;
  unsigned long long* redm = reinterpret_cast<unsigned long long*>(smem_raw);
  T* red = reinterpret_cast<T*>(smem_raw + 256);
  T* S = reinterpret_cast<T*>(smem_raw + 512);
  T* vv = S + stage_words(n, (int)sizeof(T));

  const Tin* Ag = A + dsc.a_off;
  // ---- load the referenced triangle (mirroring 'U' into 'L'), check finiteness
  // (flat over the n^2 entries; column j = idx / n by a float reciprocal,
  // exact for idx < 2^14: the quotient's fraction stays >= 1/(2n) from 1;
  // entries outside the triangle are not read and count as zero)
  int bad = 0;
  unsigned long long amax = 0;
  const float inv_n = 1.f / (float)n;
  auto in_triangle = [&](int idx, int& i, int& j) {
    j = (int)(((float)idx + 0.5f) * inv_n);
    i = idx - j * n;
    return lower ? (i >= j) : (i <= j);
  };
  auto entry = [&](int idx) {
    int i, j;
    return in_triangle(idx, i, j) ? Ag[idx] : Tin(0);
  };
  batched<sizeof(T) == 8 ? 4 : 8>(n * n, entry, [&](int, Tin v) {
    bad |= !isfinite(v);
    const unsigned long long b = AbsBits<Tin>::get(v);
    amax = b > amax ? b : amax;
  });
  bad = __syncthreads_or(bad);
  if (tid == 0) {
    ChaseState st;
    st.bs = 0;
    st.nsweeps = 0;
    st.nrot = 0;
    st.nhdr = 0;
    st.status = bad ? kChaseDone : kChaseRunning;
    st.applied = 0;
    cst[mid] = st;
    info[mid] = bad ? -1 : 0;
  }
  if (bad) return;
  // Reduced-precision runs scale the matrix by an exact power of two so that
  // its largest entry is near 1 (no overflow/underflow in the narrow type).
  int sexp = 0;
  if (sizeof(Tin) != sizeof(T)) {
    unsigned long long mx = amax;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = w > mx ? w : mx;
    }
    if ((tid & 31) == 0) redm[tid >> 5] = mx;
    __syncthreads();
    mx = redm[0];
    for (int w = 1; w < (NT >> 5); w++) mx = redm[w] > mx ? redm[w] : mx;
    __syncthreads();
    if (mx != 0) {
      int e2;
      frexp(AbsBits<Tin>::from(mx), &e2);
      sexp = e2;  // max |A| * 2^-sexp in [0.5, 1)
    }
    if (tid == 0) scale_exp[mid] = sexp;
  }
  batched<sizeof(T) == 8 ? 4 : 8>(n * n, entry, [&](int idx, Tin v) {
    int i, j;
    if (!in_triangle(idx, i, j)) return;
    const T t = (sizeof(Tin) != sizeof(T)) ? (T)df_scaled((double)v, sexp).hi : (T)v;
    if (lower) S[j * ld + i] = t;
    else S[i * ld + j] = t;
  });
  __syncthreads();

  if constexpr (sizeof(T) == 8) {
    tridiag_body_shared<WANTQ>(dsc, S, ld, vv, red, redm, dout, eout, Qout, rows2);
  } else {
    auto body = [&](auto nb) {
      tridiag_body_regs<decltype(nb)::value, WANTQ, STEIN>(mid, dsc, S, ld, vv, dout, eout, Qout, cst, wout, qtmp, sexp,
                                                           rows2);
    };
    if (n <= 32) body(std::integral_constant<int, 2>());
    else if (n <= 64) body(std::integral_constant<int, 4>());
    else if (n <= 96) body(std::integral_constant<int, 6>());
    else body(std::integral_constant<int, 8>());
  }
}

}  // namespace gla
