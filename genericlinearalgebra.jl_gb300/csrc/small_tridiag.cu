// Batched Householder tridiagonalisation and explicit Q, one CTA per matrix,
// the whole matrix staged in shared memory (n <= 128).
//
// Replaces, per matrix:
//   symtriLower! (GenericLinearAlgebra.jl src/eigenSelfAdjoint.jl:450-504)
//   with LinearAlgebra.reflector! (called at :466) and BLAS symv (:477),
//   and Array(Q::EigenQ) = lmul!(Q, I) (:101, :23-41).
// uplo 'U' input is mirrored into the lower triangle on load, so both
// triangles run the 'L' reduction (the 'U' variant :507-564 reduces the
// mirrored matrix in reverse order and yields the same eigenpairs).
//
// FP32: the matrix in registers, see small_tridiag_f32.cuh.
// FP64 work split (FP64 on GB300 costs ~68 cycles per warp instruction no matter
// how many lanes are active, so every FP64 loop is spread over all lanes):
//   norm / dot products: one element per thread + block reduction,
//   SYMV: rows x (1, 2 or 4 column parts),
//   rank-2 update: flat index over the trailing lower triangle,
//   Q formation: dorg2l-style backward accumulation in place of the
//   reflectors (H_k applied only to the already-formed trailing block).
#include <algorithm>

#include "gla_launch.h"
#include "gla_small.cuh"
#include "small_stein.cuh"
#include "small_tridiag.cuh"

namespace gla {

size_t tridiag_smem_bytes(int n, int nt, int elem, bool) {
  // redm[32] u64 | red[32] (8-byte slots) | S[n*ld] | vv,uu,ww,taus [n] | part: FP64 [nt], FP32 [8*256]
  // (the FP32 tridiagonal solver reuses S and part once the reflectors are in global memory)
  return 512 + (size_t)elem * (stage_words(n, elem) + 4 * (size_t)n + (elem == 8 ? (size_t)nt : 8 * (size_t)kRegNT));
}

template <class T, class Tin, bool WANTQ, bool STEIN>
__global__ void __launch_bounds__(256) k_tridiag(const SmallDesc* __restrict__ descs, const int* __restrict__ perm,
                                                 const Tin* __restrict__ A, int lower, T* __restrict__ dout,
                                                 T* __restrict__ eout, T* __restrict__ Qout, int* __restrict__ info,
                                                 ChaseState* __restrict__ cst, int* __restrict__ scale_exp,
                                                 T* __restrict__ wout, T* __restrict__ qtmp,
                                                 T* __restrict__ rows2) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  tridiag_body<T, Tin, WANTQ, STEIN>(perm[blockIdx.x], smem_raw, descs, A, lower, dout, eout, Qout, info, cst,
                                     scale_exp, wout, qtmp, rows2);
}

size_t stein_tri_smem_bytes(int n) { return 512 + 4 * (2 * (size_t)n + stein_extra_words(n) + 3 * 128); }

// Tridiagonal input on the FP32 stage (the leaves of the divide and conquer
// of the FP32 + refinement path): the per-eigenvalue solver of
// small_stein.cuh on (d, e) as the chase would take them, one CTA per
// matrix (blockDim >= n). A solved matrix gets its ascending eigenvalues in
// wout and its eigenvectors in Q, and is marked done for the chase and the
// rotation replay; the others keep Q = I and their "running" chase state.
__global__ void __launch_bounds__(128) k_stein_tri(const SmallDesc* __restrict__ descs, const int* __restrict__ perm,
                                                   const float* __restrict__ dg_all, const float* __restrict__ eg_all,
                                                   float* __restrict__ Qout, float* __restrict__ wout,
                                                   ChaseState* __restrict__ cst, const int* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int mid = perm[blockIdx.x];
  const SmallDesc dsc = descs[mid];
  const int n = dsc.n, tid = threadIdx.x;
  if (n < 1 || info[mid] != 0 || cst[mid].status != kChaseRunning) return;
  float* fscr = reinterpret_cast<float*>(smem_raw);  // 128 floats
  float* dd = reinterpret_cast<float*>(smem_raw + 512);
  float* ee = dd + n;
  const int ldy = stein_ldy(n);
  float* Ys = ee + n;
  float* e2s = Ys + (size_t)n * ldy;
  float* lams = e2s + n;
  int* misc = reinterpret_cast<int*>(lams + n);
  for (int i = tid; i < n; i += blockDim.x) {
    dd[i] = dg_all[dsc.w_off + i];
    ee[i] = (i + 1 < n) ? eg_all[dsc.w_off + i] : 0.f;
  }
  __syncthreads();
  if (!stein_solve(n, dd, ee, e2s, lams, Ys, ldy, misc, fscr, misc + n + 8)) return;
  float* Qg = Qout + dsc.a_off;
  for (int j = 0; j < n; j++)
    for (int i = tid; i < n; i += blockDim.x) Qg[(size_t)j * n + i] = Ys[(size_t)i * ldy + j];
  for (int k = tid; k < n; k += blockDim.x) wout[dsc.w_off + k] = lams[k];
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

cudaError_t launch_stein_tri(int nblocks, int nmax, cudaStream_t st, const SmallDesc* descs, const int* perm,
                             const void* d, const void* e, void* Q, void* w, ChaseState* cst, const int* info) {
  if (nblocks <= 0) return cudaSuccess;
  const int nt = std::max(32, (nmax + 31) / 32 * 32);
  k_stein_tri<<<nblocks, nt, stein_tri_smem_bytes(nmax), st>>>(descs, perm, (const float*)d, (const float*)e,
                                                               (float*)Q, (float*)w, cst, info);
  return cudaGetLastError();
}

// Eigenvalues of FP32 matrices (jobz 'N'): one CTA per matrix, one thread per
// eigenvalue, bisection on Sturm counts of (d, e) scaled by an exact power of
// two (the largest to about 2^62: its square is in range and the squares of
// entries 2^-136 as large are too), to the last bit, in place of the root-free chase and the sort. That
// chase is one serial recurrence of about n^2 steps per matrix (550 cycles
// each: 5.1 ms for 1000 matrices of orders 8 .. 128 with everything beside
// it), bisection 15 to 20 passes of n steps for all eigenvalues at once.
__global__ void __launch_bounds__(128) k_bisect_values(const SmallDesc* __restrict__ descs,
                                                       const int* __restrict__ perm, const float* __restrict__ dg_all,
                                                       const float* __restrict__ eg_all, float* __restrict__ wout,
                                                       int* __restrict__ info) {
  __shared__ float dd[kSmallMaxN], e2[kSmallMaxN], xs[kSmallMaxN], red[3][4];
  __shared__ int cnt[3 * kSmallMaxN];
  const int mid = perm[blockIdx.x];
  const SmallDesc dsc = descs[mid];
  const int n = dsc.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  if (info[mid] == -1) {
    if (tid < n) wout[dsc.w_off + tid] = NAN;
    return;
  }
  const float d = tid < n ? dg_all[dsc.w_off + tid] : 0.f;
  const float e = tid + 1 < n ? eg_all[dsc.w_off + tid] : 0.f;
  // a reduction that left the range (entries near the largest float): no
  // eigenvalue is found, as the chase would report it
  if (__syncthreads_or(!isfinite(d) || !isfinite(e))) {
    if (tid < n) wout[dsc.w_off + tid] = NAN;
    if (tid == 0) info[mid] = max(n - 1, 1);
    return;
  }
  float m = fmaxf(fabsf(d), fabsf(e));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[0][wid] = m;
  __syncthreads();
  for (int w = 0; w < nw; w++) m = fmaxf(m, red[0][w]);
  const int ex = m > 0.f ? ilogbf(m) - 62 : 0;
  const float ds = ldexpf(d, -ex), es = ldexpf(e, -ex);
  if (tid < n) {
    dd[tid] = ds;
    e2[tid] = es * es;
  }
  // Gershgorin interval: |e| of the entry before through the warp and, at its edge, shared memory
  __syncthreads();
  const float ep = tid > 0 && tid < n ? sqrtf(e2[tid - 1]) : 0.f;
  const float ai = (fabsf(es) + ep) * 1.0001f;
  float lo = tid < n ? ds - ai : 3.0e38f, hi = tid < n ? ds + ai : -3.0e38f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    red[1][wid] = lo;
    red[2][wid] = hi;
  }
  __syncthreads();
  for (int w = 0; w < nw; w++) {
    lo = fminf(lo, red[1][w]);
    hi = fmaxf(hi, red[2][w]);
  }
  const float pivmin = 0x1p-120f;
  const float widen = 2.f * (float)n * prec<float>::eps * fmaxf(fabsf(lo), fabsf(hi)) + 2.f * pivmin;
  lo -= widen;
  hi += widen;
  grid_bracket<true>(n, dd, e2, lo, hi, pivmin, cnt);
  const float zero = 4.f * pivmin;
  const float x = tid < n ? eig_bisect_full(n, dd, e2, tid, lo, hi, pivmin, zero) : 0.f;
  if (tid < n) xs[tid] = x;
  __syncthreads();
  if (tid >= n) return;
  float out = ldexpf(x, ex);
  if (fabsf(x) <= zero) {
    // Zero to within the guarded pivots (2^-180 of the matrix): zero, but for
    // the entries that stand alone, which are eigenvalues as they are. Those
    // below zero come first here, those above it last.
    const float* dg = dg_all + dsc.w_off;
    auto alone = [&](int i) {
      return (i == 0 || e2[i - 1] == 0.f) && e2[i] == 0.f && fabsf(dd[i]) <= zero;  // (e2[n - 1] is zero)
    };
    int before = 0, here = 0, neg = 0, pos = 0;
    for (int i = 0; i < n; i++) {
      before += xs[i] < -zero;
      here += fabsf(xs[i]) <= zero;
      neg += alone(i) && dg[i] < 0.f;
      pos += alone(i) && dg[i] > 0.f;
    }
    const int r = tid - before;
    out = 0.f;
    if (r < neg || r >= here - pos) {
      const int want = r < neg ? r : r - (here - pos);
      const bool up = r >= neg;
      for (int i = 0; i < n; i++) {
        if (!alone(i) || (up ? dg[i] <= 0.f : dg[i] >= 0.f)) continue;
        int rank = 0;
        for (int j = 0; j < n; j++)
          rank += alone(j) && (up ? dg[j] > 0.f : dg[j] < 0.f) && (dg[j] < dg[i] || (dg[j] == dg[i] && j < i));
        if (rank == want) out = dg[i];
      }
    }
  }
  wout[dsc.w_off + tid] = out;
}

cudaError_t launch_bisect_values(int nblocks, int nmax, cudaStream_t st, const SmallDesc* descs, const int* perm,
                                 const void* d, const void* e, void* w, int* info) {
  if (nblocks <= 0) return cudaSuccess;
  const int nt = std::max(32, (nmax + 31) / 32 * 32);
  k_bisect_values<<<nblocks, nt, 0, st>>>(descs, perm, (const float*)d, (const float*)e, (float*)w, info);
  return cudaGetLastError();
}

template <class T, class Tin, bool Q, bool ST = false> static void set_tri_attr() {
  cudaFuncSetAttribute(k_tridiag<T, Tin, Q, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)tridiag_smem_bytes(kSmallMaxN, 256, sizeof(T), ST));
}

cudaError_t tridiag_kernels_init() {
  set_tri_attr<double, double, true>();
  set_tri_attr<double, double, false>();
  set_tri_attr<float, float, true>();
  set_tri_attr<float, float, false>();
  set_tri_attr<float, double, true>();
  set_tri_attr<float, double, false>();
  set_tri_attr<float, double, true, true>();
  set_tri_attr<float, float, true, true>();
  cudaFuncSetAttribute(k_stein_tri, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)stein_tri_smem_bytes(kSmallMaxN));
  return cudaGetLastError();
}

cudaError_t launch_tridiag(int tcode, bool wantq, int nblocks, int nt, size_t smem, cudaStream_t st,
                           const SmallDesc* descs, const int* perm, const void* A, int lower, void* d, void* e,
                           void* Q, int* info, ChaseState* cst, int* scale_exp, bool stein, void* w,
                           void* qtmp, void* rows2) {
  if (nblocks <= 0) return cudaSuccess;
  if (tcode != kF64) nt = kRegNT;  // (small_tridiag_f32.cuh)
#define GLA_TRI(T, Tin, WQ, ST)                                                                                 \
  k_tridiag<T, Tin, WQ, ST><<<nblocks, nt, smem, st>>>(descs, perm, (const Tin*)A, lower, (T*)d, (T*)e, (T*)Q, \
                                                       info, cst, scale_exp, (T*)w, (T*)qtmp, (T*)rows2)
  if (tcode == kF64) {
    if (wantq) GLA_TRI(double, double, true, false);
    else GLA_TRI(double, double, false, false);
  } else if (tcode == kF32) {
    if (wantq && stein) GLA_TRI(float, float, true, true);
    else if (wantq) GLA_TRI(float, float, true, false);
    else GLA_TRI(float, float, false, false);
  } else {
    if (wantq && stein) GLA_TRI(float, double, true, true);
    else if (wantq) GLA_TRI(float, double, true, false);
    else GLA_TRI(float, double, false, false);
  }
#undef GLA_TRI
  return cudaGetLastError();
}

}  // namespace gla
