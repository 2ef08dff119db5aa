// Householder tridiagonalisation of one large symmetric matrix (lower
// triangle), blocked in panels of kSytrdNB columns: the LAPACK dsytrd/dlatrd
// organisation of the reference's symtriLower! (src/eigenSelfAdjoint.jl:450-504).
//
// Column j of a panel (c = j - k0 columns into it), s = j + 1:
//   x  = A[s:, j] after the panel's earlier rank-2 terms
//   reflector H_j = I - tau v v' from x (reflector! convention: beta = -sign(x1)|x|,
//   v[s] = 1, v stored in A[s+1:, j] like the reference)
//   y  = A_t v - V (W' v) - W (V' v)     A_t = A[s:, s:] without this panel
//   w  = tau y - (tau^2 / 2)(y' v) v     (so A_t - v w' - w v' = H A_t H)
// and after the panel one rank-2k update A_t -= V W' + W V' (a GEMM over
// the lower tiles). Every panel is one cooperative launch over all SMs with
// two grid barriers per column:
//   phase A (all CTAs): the SYMV of A_t with the raw column a (a_i = x_i
//     below row s, so it needs no reflector scalars and starts at once), in
//     warp units of 32 columns x 64 rows of the lower triangle (each unit
//     adds A_IJ a_J to its rows and A_IJ' a_I to its columns, into
//     deterministic partial buffers), the dot products V'a, W'a,
//     a'A[:, s] and the quadratic form a'A_t a;
//   phase B (rows split over CTAs): the reflector scalars from the norm
//     partials, v = scale a + e_s applied to the phase A results by
//     linearity, y, w, the reflector stored, and the next column updated
//     with this column's terms plus its norm partial.
// Each phase issues all of its global loads before its first reduction:
// on GB300 an L2 round trip costs about a microsecond and is the unit of
// cost at the small trailing orders. Phase B's rows are split over the CTAs
// once per panel (rows k0 + 1 .. n - 1; a row above the current column's s
// is idle), so each CTA computes V and W for the same rows in every column
// of the panel and keeps them in shared memory for the rank-2 corrections
// of the later columns, instead of reading them back from L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gla_common.cuh"
#include "gla_large.h"
#include "tc_gemm.cuh"

namespace gla {

// Shapes of a SYMV unit (one warp): CW columns, NQ rows per lane. A unit is
// a serial chain of FP64 instructions of 64 cycles each (2 CW NQ products,
// and CW or so additions to reduce its column sums), so small trailing
// orders, where every warp has at most one unit, want small units, and large
// ones, which fill the FP64 units anyway, those with the fewest additions
// per product. FP64 panels take the first shape whose max_m holds their
// trailing order (other limits by a factor of 0.7 or 1.4 cost 1 to 4%); FP32
// panels, bound by latency, the last.
struct UnitShape {
  int cw, nq, max_m;
};
constexpr int kMaxOrder = 16384;
constexpr UnitShape kShapes[] = {{8, 1, 560}, {16, 1, 1000}, {16, 2, 1500}, {32, 2, kMaxOrder}};
constexpr int kNumShapes = 4;
constexpr int kMaxTC = kMaxOrder / 32;  // tile columns a launch may cover (560/8 and 1500/16 are fewer)
// Trailing orders up to these run a panel on one cluster of 16 CTAs: the
// cluster's barrier saves what the other SMs would have shortened the column
// by (FP32 order 500: 4.7 us a column on the cluster, 5.7 on 152 SMs; order
// 1000 with its last 700 columns, its last 400 or none on the cluster: 5.6,
// 5.5 and 5.9. FP64 order 200: 7.3 and 8.5; order 400: 10.2 and 9.3).
// A plan that solves several matrices side by side runs all of their panels
// so (SytrdPlan::cluster_only), each on SMs of its own.
constexpr int kClusterG = 16, kClusterMaxF64 = 200, kClusterMaxF32 = 700;
static_assert(kClusterMaxF64 <= kSideBySideMaxN && kClusterMaxF32 <= kSideBySideMaxN,
              "the cluster kernels' shared memory is set for kSideBySideMaxN");
// Rows per dot-product unit. An FP32 unit waits for L2 (eight rows a lane, in
// two batches of loads, 6.6 us a column at order 2048; 32 rows 7.6); in FP64
// the warps are occupied as it is, and shorter units add their reductions
// (order 1500: 10.9 us with 1024 rows, 11.4 with 256).
template <class T>
constexpr int kDotRows = sizeof(T) == 8 ? 1024 : 256;
constexpr int kPT = 256;       // threads per CTA
constexpr long long kSpinLimit = 1ll << 26;

template <class T>
struct SytrdArgs {
  T* A;
  long long ld;
  int n, k0, nbp;
  T* V;              // column c of the panel's V (n rows, leading dimension ldv)
  T* W;
  long long ldv;
  T* d;
  T* e;
  T* tau;
  T* P;              // row partials    [tile column - Jbase][n]
  T* Qp;             // column partials [chunk of rows][n]
  T* normp;          // [G]
  T* qfp;            // [G]
  T* dots;           // [3][kSytrdNB][nDCH]
  int nDCH;
  const int2* F;     // fixed-point panels: the trailing matrix (leading dimension n), see fix_of
  const int* fe;     // its exponents, [tile column][fch]
  int fch;
  const int* ustart; // of this shape: first SYMV unit of each tile column; ustart[nTC] = total
  int nTC;
  unsigned* bar;     // arrival counter (monotonic over the launches of one tridiagonalisation)
  unsigned bar_base; // counter value when this launch starts
  int* err;
};

// Sum over the lanes of the warp that differ in the lane bits of [lo, 32).
template <class T>
GLA_DEV T lane_sum(T v, int lo) {
  for (int o = 16; o >= lo; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Four sums over the warp at once, six additions in all: lane 8 k ends with
// the sum of v[k].
template <class T>
GLA_DEV T warp_sum4(const T (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const bool u = lane & 16, w = lane & 8;
  const T a = (u ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, u ? v[0] : v[2], 16);
  const T b = (u ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, u ? v[1] : v[3], 16);
  T x = (w ? b : a) + __shfl_xor_sync(0xffffffffu, w ? a : b, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x + __shfl_xor_sync(0xffffffffu, x, 1);
}

// Grid barrier on a monotonic arrival counter: barrier number k of a launch
// completes when the counter reaches (k + 1) * gridDim.x. Thread 0 of each
// CTA arrives with a release add and polls with acquire loads; the wait is
// bounded (kSpinLimit polls) and a timeout sets the error word, which every
// waiting CTA also watches now and then. The verdict is broadcast through shared memory
// so that all threads of a CTA return the same value. Before it arrives, the
// CTA's part of a sum goes out: the warps' parts in part[0 .. 8), added by
// warp 0 into *out.
//
// CL: the grid is one thread-block cluster, and the barrier is the cluster's
// (0.4 us instead of 1.7; release and acquire at cluster scope cover the
// CTAs' global writes). The hardware schedules a cluster as a whole, so there
// is nothing to spin on.
template <class T, bool CL>
GLA_DEV bool grid_sync(unsigned* bar, int* err, unsigned& target, const T* part, T* out) {
  __shared__ int s_ok;
  target += gridDim.x;
  __syncthreads();
  if (CL) {
    if (threadIdx.x < 32) {
      T v = part[threadIdx.x & 7];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (threadIdx.x == 0) *out = v;
      __syncwarp();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  if (threadIdx.x < 32) {
    T v = part[threadIdx.x & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) {
      *out = v;
      // (cumulative: it also releases what the CTA's other threads wrote
      // before the __syncthreads above)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      volatile int* verr = err;
      bool ok = false;
      for (long long it = 1; it <= kSpinLimit; it++) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
        ok = (int)(c - target) >= 0;
        if (ok || ((it & 255) == 0 && *verr)) break;
      }
      if (!ok) atomicExch(err, 1);
      s_ok = ok;
    }
  }
  __syncthreads();
  return s_ok != 0;
}

// a_i = A[i, j] below row s (the raw reflector column), 0 elsewhere. The
// SYMV runs on a (no reflector scalars needed yet); phase B restores
// v = scale a + e_s by linearity.
template <class T>
GLA_DEV T a_at(const T* __restrict__ A, long long ld, int j, int s, int i) {
  return i > s ? A[i + (long long)j * ld] : T(0);
}

// One warp: SYMV unit (tile column J, chunk ch) of the trailing lower
// triangle on the raw column a, row by row (lane l holds row r0 + l + 32 q);
// all loads of the unit are issued before its FMAs. Adds the row sums to
// P[J - Jbase][r] and the column sums to Qp[ch][c]; returns the unit's part
// of a'A_t a.
template <class T, int CW, int NQ>
__device__ T symv_unit(const SytrdArgs<T>& a, int j, int s, int J, int ch, T* svcol) {
  constexpr int RC = 32 * NQ;
  const int lane = threadIdx.x & 31, n = a.n;
  const long long ld = a.ld;
  const T* __restrict__ A = a.A;
  const int c0 = J * CW, r0 = c0 + ch * RC;
  constexpr int kRep = 32 / CW;  // lanes that end with the same column sum
  const int cc = c0 + lane / kRep;
  const T vc = cc < n ? a_at(A, ld, j, s, cc) : T(0);
  const T* __restrict__ base = A + (long long)c0 * ld + r0 + lane;
  const int ncol = min(CW, n - c0);
  T x[NQ][CW], vr[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int r = r0 + lane + 32 * q;
    const bool rin = r < n;
    const T* rowp = base + 32 * q;
#pragma unroll
    for (int ci = 0; ci < CW; ci++) x[q][ci] = (rin && ci < ncol) ? rowp[(long long)ci * ld] : T(0);
    vr[q] = rin ? a_at(A, ld, j, s, r) : T(0);
  }
  if (lane % kRep == 0) svcol[lane / kRep] = vc;
  __syncwarp();
  T colacc[CW];
#pragma unroll
  for (int ci = 0; ci < CW; ci++) colacc[ci] = T(0);
  T qf = T(0);
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    if (r0 + 32 * q >= n) break;  // warp-uniform
    const bool diag = ch == 0 && q == 0;  // diagonal tile: lower part only (row >= column)
    T rowacc = T(0);
#pragma unroll
    for (int ci = 0; ci < CW; ci++) {
      const T xr = (diag && lane < ci) ? T(0) : x[q][ci];
      const T xc = (diag && lane <= ci) ? T(0) : x[q][ci];
      rowacc = fma(xr, svcol[ci], rowacc);
      colacc[ci] = fma(xc, vr[q], colacc[ci]);
    }
    const int r = r0 + lane + 32 * q;
    if (r < n) a.P[(long long)(J - a.k0 / CW) * n + r] = rowacc;
    qf = fma(rowacc, vr[q], qf);
  }
  // reduce-scatter the column sums across the warp: lane l keeps column l / kRep
#pragma unroll
  for (int half = CW / 2; half >= 1; half >>= 1) {
    const int bit = half * kRep;
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const T send = up ? colacc[i] : colacc[i + half];
      const T keep = up ? colacc[i + half] : colacc[i];
      colacc[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
#pragma unroll
  for (int o = kRep / 2; o >= 1; o >>= 1) colacc[0] += __shfl_xor_sync(0xffffffffu, colacc[0], o);
  if (lane % kRep == 0) {
    if (cc < n) a.Qp[(long long)ch * n + cc] = colacc[0];
    qf = fma(colacc[0], vc, qf);
  }
  __syncwarp();
  return qf;
}

// ---- The FP64 SYMV in fixed point, for trailing orders above kFixedMin.
//
// Every entry of the trailing matrix meets the vector twice (row and column
// sums), and an FP64 product costs a sub-partition 64 cycles: at order 4096
// the SYMV took 16 of the 27 us of a column, at 70% of the FP64 rate. The
// trailing matrix is the same for the 32 columns of a panel, so it is turned
// once per panel into integers of 57 bits, scaled by the largest entry of
// their 64 x 32 unit, as two digits of 28 bits; the vector is split alike
// unit by unit. A product is then three 32 x 32 -> 64-bit multiply-adds of 4
// cycles (the product of the low digits, 2^-58 of the unit's largest, is left
// out), the sums are exact in 64 bits, and the reductions over lanes are
// integer additions. (The matrix given to gla_dsytrd keeps the FP64 units: see
// large_keep_entries.) What is rounded is the entries, at 2^-57 of their unit's
// largest, and the unit's sums, at 2^-56: below the 2^-53 of each FP64 sum
// (residual and orthogonality of orders 1100 .. 4096, also of graded
// matrices, as with FP64 products to 3%).
//
// Reduction of order 4096: 26.9 -> 18.5 us a column, 1500: 10.9 -> 10.3. Below
// about 1000 a warp has less than a unit of this size, and smaller FP64 units
// are faster (a limit of 600: order 777 9.8 us a column instead of 9.1).
constexpr int kFixedMin = 1000;
constexpr int kFixW = 32, kFixR = 64;  // columns and rows of a unit (the last of kShapes)

// e with |x| < 2^e for the top word of the largest |x|; subnormal numbers share
// the least exponent. A reflector's column may be as small as it likes beside
// the rest of the matrix (one coupled by 1e-140 to a block of size 1): it is
// scaled up to size 1 after the product, so its digits keep their own exponent.
GLA_DEV int fix_exp(unsigned top) { return max((int)(top >> 20), 1) - 1022; }
GLA_DEV unsigned fix_top(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// x 2^(56 - e), |x| < 2^e, rounded: digits (hi, lo) with hi 2^28 + lo, |lo| <= 2^27.
GLA_DEV int2 fix_of(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(b >> 52) & 0x7ff, s = max(ex, 1) - 1019 - e;  // the mantissa's shift, at most 3
  const unsigned long long m = (b & 0xfffffffffffffull) | (ex ? 1ull << 52 : 0ull);
  const unsigned long long f = s >= 0 ? m << s : s > -64 ? ((m >> (-s - 1)) + 1) >> 1 : 0ull;
  const long long v = (long long)b < 0 ? -(long long)f : (long long)f;
  const int hi = (int)((v + (1ll << 27)) >> 28);
  return make_int2(hi, (int)(v - ((long long)hi << 28)));
}
// The sum s1 2^56 + s2 2^28 of products of digits, in units of 2^56.
GLA_DEV long long fix_sum(long long s1, long long s2) { return s1 + ((s2 + (1ll << 27)) >> 28); }
// v 2^(e - 56), zero where that is below 2^-960 (a unit of the matrix and a
// column that are both tiny: times the column's scale, at most 2^511, that is
// below 2^-440 of the matrix). e <= 1078, as the eigensolvers scale their matrix.
GLA_DEV double fix_value(long long v, int e) {
  return (double)v * __hiloint2double(max(1023 - 56 + e, 0) << 20, 0);
}

// The units of the tile columns J0 .. of the lower triangle (grid: chunk of
// rows, tile column).
__global__ void __launch_bounds__(256) k_sytrd_fix(const double* __restrict__ A, long long ld, int n, int J0,
                                                   int2* __restrict__ F, int* __restrict__ fe, int fch) {
  __shared__ unsigned red[8];
  const int J = J0 + blockIdx.y, c0 = J * kFixW, r0 = c0 + (int)blockIdx.x * kFixR, tid = threadIdx.x;
  if (r0 >= n) return;
  const int r = r0 + (tid & (kFixR - 1)), cb = c0 + (tid >> 6);
  double x[8];
  unsigned m = 0;
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int c = cb + 4 * u;
    x[u] = (r < n && c <= r) ? A[r + c * ld] : 0.0;
    m = max(m, fix_top(x[u]));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; w++) m = max(m, red[w]);
  const int e = fix_exp(m);
  if (tid == 0) fe[J * fch + blockIdx.x] = e;
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int c = cb + 4 * u;
    if (r < n && c < n) F[r + (long long)c * n] = fix_of(x[u], e);
  }
}

// symv_unit<double, 32, 2> on F, eight columns at a time.
GLA_DEV double symv_unit_fixed(const SytrdArgs<double>& a, int j, int s, int J, int ch, int2* sv) {
  const int lane = threadIdx.x & 31, n = a.n;
  const int c0 = J * kFixW, r0 = c0 + ch * kFixR, cc = c0 + lane;
  int2 nx[2][8];  // the next eight columns, on their way while these are multiplied
  auto fetch = [&](int h) {
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int r = r0 + lane + 32 * q;
      const int2* base = a.F + r + (long long)(c0 + h) * n;
#pragma unroll
      for (int i = 0; i < 8; i++) nx[q][i] = (r < n && c0 + h + i < n) ? base[(long long)i * n] : make_int2(0, 0);
    }
  };
  fetch(0);
  const double vc = cc < n ? a_at(a.A, a.ld, j, s, cc) : 0.0;
  double vr[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int r = r0 + lane + 32 * q;
    vr[q] = r < n ? a_at(a.A, a.ld, j, s, r) : 0.0;
  }
  const int ea = a.fe[J * a.fch + ch];
  const int ec = fix_exp(__reduce_max_sync(0xffffffffu, fix_top(vc)));
  const int er = fix_exp(__reduce_max_sync(0xffffffffu, max(fix_top(vr[0]), fix_top(vr[1]))));
  sv[lane] = fix_of(vc, ec);
  const int2 w[2] = {fix_of(vr[0], er), fix_of(vr[1], er)};
  __syncwarp();
  long long r1[2] = {0, 0}, r2[2] = {0, 0};
  double qf = 0.0;
#pragma unroll 1
  for (int h = 0; h < kFixW; h += 8) {
    int2 x[2][8];
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
      for (int i = 0; i < 8; i++) x[q][i] = nx[q][i];
    if (h + 8 < kFixW) fetch(h + 8);
    long long v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int2 xc = sv[h + i];
      const bool diag = ch == 0 && lane == h + i;  // F is zero above the diagonal; on it only the row sum counts
      long long c1 = 0, c2 = 0;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int2 f = x[q][i];
        r1[q] += (long long)f.x * xc.x;
        r2[q] += (long long)f.x * xc.y;
        r2[q] += (long long)f.y * xc.x;
        const int wx = q == 0 && diag ? 0 : w[q].x, wy = q == 0 && diag ? 0 : w[q].y;
        c1 += (long long)f.x * wx;
        c2 += (long long)f.x * wy;
        c2 += (long long)f.y * wx;
      }
      v[i] = fix_sum(c1, c2);
    }
    // column sums across the warp: lane l keeps column h + l / 4
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
      const bool up = (lane & (4 * half)) != 0;
#pragma unroll
      for (int i = 0; i < half; i++) {
        const long long send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * half);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    const int ci = h + (lane >> 2);
    const double xv = __shfl_sync(0xffffffffu, vc, ci);
    if ((lane & 3) == 0 && c0 + ci < n) {
      const double y = fix_value(v[0], ea + er);
      a.Qp[(long long)ch * n + c0 + ci] = y;
      qf = fma(y, xv, qf);
    }
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int r = r0 + lane + 32 * q;
    if (r < n) {
      const double y = fix_value(fix_sum(r1[q], r2[q]), ea + ec);
      a.P[(long long)(J - a.k0 / kFixW) * n + r] = y;
      qf = fma(y, vr[q], qf);
    }
  }
  __syncwarp();
  return qf;
}

// Rows of the trailing range [s, n) owned by CTA g.
GLA_DEV void own_rows(int s, int n, int& lo, int& hi) {
  const int m = n - s, G = gridDim.x;
  const int R = (m + G - 1) / G;
  lo = min(n, s + (int)blockIdx.x * R);
  hi = min(n, lo + R);
}

// Rows per CTA of phase B in the panel starting at column k0 (the split of
// rows k0 + 1 .. n - 1, fixed for the panel).
GLA_DEV __host__ int panel_rows(int k0, int n, int G) { return (n - k0 - 1 + G - 1) / G; }

// beta = -copysign(norm, alpha), tau = (beta - alpha) / beta and 1 / (alpha -
// beta) from alpha and sigma, the squared norm below it; beta = alpha and
// zeros when sigma is zero, or when the whole column is so small (2^-500 beside
// a matrix of size 1; FP32 2^-60) that its square leaves the normal range and
// the seeds below: leaving it out moves the matrix by no more than its norm.
// FP64: the steps of sqrt_rsqrt64 and rcp64, 10 instructions in a row; the norm
// in even lanes and its reciprocal in odd ones.
GLA_DEV void panel_scalars(double alpha, double sigma, double& beta, double& tau, double& scale) {
  const double nrm2 = fma(alpha, alpha, sigma);
  if ((__double_as_longlong(sigma) << 1) == 0 || prec<double>::biased_exp(nrm2) < 1023 - 1000) {
    beta = alpha;
    tau = scale = 0.0;
    return;
  }
  const bool odd = threadIdx.x & 1;
  const double y = rsqrt_seed64(nrm2), h = nrm2 * y;
  const double e = fma(-h, y, 1.0);
  const double q = e * fma(e, 0.375, 0.5);
  const double hy = odd ? y : h;
  const double r = fma(hy, q, hy);
  const double nrm = __shfl_sync(0xffffffffu, r, 0), rn = __shfl_sync(0xffffffffu, r, 1);
  beta = copysign(nrm, -alpha);
  // even: alpha - beta = sign(alpha) (|alpha| + norm); odd: tau = 1 + |alpha| / norm
  const double d = fma(odd ? fabs(alpha) : 1.0, odd ? rn : nrm, odd ? 1.0 : fabs(alpha));
  tau = __shfl_sync(0xffffffffu, d, 1);
  scale = rcp64(copysign(__shfl_sync(0xffffffffu, d, 0), alpha));
}
GLA_DEV void panel_scalars(float alpha, float sigma, float& beta, float& tau, float& scale) {
  const float nrm2 = fmaf(alpha, alpha, sigma);
  if (sigma == 0.f || nrm2 < 0x1p-120f) {
    beta = alpha;
    tau = scale = 0.f;
    return;
  }
  const float nrm = nrm2 * prec<float>::rsqrt(nrm2);
  beta = -copysignf(nrm, alpha);
  tau = (beta - alpha) * prec<float>::rcp(beta);
  scale = prec<float>::rcp(alpha - beta);
}

// Dot-product unit kinds, in work-list order after the SYMV units.
constexpr int kDotA = 0;  // 2 sum_r a_r A[r, s]      (cross term of v'A_t v)
constexpr int kDotV = 1;  // sum_r a_r V[r, q], q < c
constexpr int kDotW = 2;  // sum_r a_r W[r, q]

// Microseconds per column (reduction of order 777 / 4096 in FP64, of order
// 2048 in FP32): 9.1 / 18.5 and 6.0, of which the two grid barriers are about
// 3.5; before units by shape, this split and the short serial chains below
// 19.4 / 32.9 and 7.9.
//
// Work split of phase B. FP64: warps 0 .. 3 read and add up the column's
// scalars, warp 0 derives the reflector's from them (warp 1 the sums over the
// panel's earlier columns), warps 4 .. 7 hold the CTA's rows: an FP64
// addition costs 64 cycles per warp whatever its lanes hold, and the two
// warps of a sub-partition queue for it, so sums go through as few additions
// as there are (four sums in six), and by one warp. FP32, bound by the round
// trips to L2: all warps do both, with as many loads in flight as there are
// threads.
template <class T, int CW, int NQ, bool CL, bool FX = false>
__global__ void __launch_bounds__(kPT, 1) k_sytrd_panel(const SytrdArgs<T> a) {
  constexpr int RC = 32 * NQ;
  constexpr bool kSplit = sizeof(T) == 8;
  constexpr int kRowT = kSplit ? kPT / 2 : kPT, kRedT = kRowT, kRedW = kRedT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = a.n, G = gridDim.x, g = blockIdx.x;
  const long long ld = a.ld, ldv = a.ldv;
  T* __restrict__ A = a.A;
  __shared__ T spart[8];       // the warps' parts of the sum that the next barrier carries
  __shared__ T sred[kRedW][4];  // the scalars' sums by warp
  __shared__ T svcol[kPT / 32][32];
  __shared__ T sdotV[kSytrdNB], sdotW[kSytrdNB], sVs[kSytrdNB], sWs[kSytrdNB];
  __shared__ T spv[kSytrdNB], sqv[kSytrdNB], sS[4];
  __shared__ int sust[kMaxTC + 1];
  __shared__ T sscal[4];
  // this CTA's V and W rows of the panel (rows lo0 .. lo0 + R0 - 1, columns
  // 0 .. nbp - 1), dynamic shared memory
  extern __shared__ __align__(16) unsigned char vw_raw[];
  T* sVr = reinterpret_cast<T*>(vw_raw);
  const int R0 = panel_rows(a.k0, n, G);
  T* sWr = sVr + (size_t)R0 * kSytrdNB;
  const int lo0 = min(n, a.k0 + 1 + g * R0), hi0 = min(n, lo0 + R0);
  for (int i = tid; i < 2 * R0 * kSytrdNB; i += kPT) sVr[i] = T(0);
  unsigned bar_target = a.bar_base;
  const int Jb = a.k0 / CW, nJ = a.nTC - Jb;  // tile columns of the panel's trailing matrix
  for (int i = tid; i <= nJ; i += kPT) sust[i] = a.ustart[Jb + i];
  // rows: tpr threads per row
  int tpr = 1;
  while (tpr < 32 && tpr * 2 * R0 <= kRowT) tpr *= 2;
  const int rpp = kRowT / tpr;  // rows per pass (more rows than threads take several)

  // panel start: norm partial of column k0 below the subdiagonal
  {
    const int j = a.k0, s = j + 1;
    int lo, hi;
    own_rows(s, n, lo, hi);
    T part = T(0);
    for (int i = lo + tid; i < hi; i += kPT)
      if (i > s) {
        const T x = A[i + (long long)j * ld];
        part = fma(x, x, part);
      }
    part = lane_sum(part, 1);
    if (lane == 0) spart[wid] = part;
  }
  if (!grid_sync<T, CL>(a.bar, a.err, bar_target, spart, a.normp + g)) return;

  for (int c = 0; c < a.nbp; c++) {
    const int j = a.k0 + c, s = j + 1, m = n - s;
    const int J0 = s / CW;
    const int ndch = (m + kDotRows<T> - 1) / kDotRows<T>;
    // ---------------- phase A: SYMV and dot products on the raw column a
    {
      const int usym0 = sust[J0 - Jb], nsym = sust[nJ] - usym0;
      const int ndot = (2 * c + 1) * ndch;
      T qf = T(0);
      // unit u goes to CTA u % G, so every CTA gets an even share
      for (int k = wid;; k += kPT / 32) {
        const int u = g + G * k;
        if (u >= nsym + ndot) break;
        if (u < nsym) {
          const int ug = usym0 + u;
          int lo = J0 - Jb, hi = nJ - 1;  // tile column: last J with sust[J] <= ug
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sust[mid] <= ug) lo = mid; else hi = mid - 1;
          }
          if constexpr (FX)
            qf += symv_unit_fixed(a, j, s, Jb + lo, ug - sust[lo], reinterpret_cast<int2*>(svcol[wid]));
          else
            qf += symv_unit<T, CW, NQ>(a, j, s, Jb + lo, ug - sust[lo], svcol[wid]);
        } else {
          const int du = u - nsym;
          const int kind = du < ndch ? kDotA : (du - ndch) / (c * ndch) + 1;
          const int rem = du < ndch ? du : (du - ndch) % (c * ndch);
          const int q = rem / ndch, chn = rem % ndch;
          const T* __restrict__ X = kind == kDotA ? A + (long long)s * ld
                                                  : (kind == kDotV ? a.V : a.W) + (long long)q * ldv;
          const int r0 = s + 1 + chn * kDotRows<T>, r1 = min(n, r0 + kDotRows<T>);
          T acc = T(0);
#pragma unroll 4
          for (int r = r0 + lane; r < r1; r += 32) acc = fma(X[r], A[r + (long long)j * ld], acc);
          acc = lane_sum(acc, 1);
          if (kind == kDotA) acc += acc;  // the quadratic form has it twice
          if (lane == 0) a.dots[((long long)kind * kSytrdNB + q) * a.nDCH + chn] = acc;
        }
      }
      qf = lane_sum(qf, 1);
      if (lane == 0) spart[wid] = qf;
    }
    if (!grid_sync<T, CL>(a.bar, a.err, bar_target, spart, a.qfp + g)) return;

    // ---------------- phase B: reflector scalars, y, w, reflector store, next column
    const int Js = s / CW;
    const bool rows = !kSplit || wid >= 4;
    const int rt = kSplit ? tid & (kRowT - 1) : tid, sub = rt % tpr, rl0 = rt / tpr;
    // (1) every load of the phase is issued before the first sum needs one
    // (loops that load and add would each wait for L2 in turn); what does not
    // fit the registers follows in a loop. Rows: kU parts of a row's y in P
    // and in Qp per thread; cP, cQ: those the CTA's rows have at most. More
    // than four parts cost FP32 more in predicated instructions than the
    // loop does (16 parts: 6.6 us a column at order 2048, 8: 6.1, 4: 5.9).
    constexpr int kU = 4;
    const int Jhi = (max(hi0, lo0 + 1) - 1) / CW, Jlo = max(lo0, s) / CW;
    const int cP = (min(Jhi, a.nTC - 1) - J0 + tpr) / tpr;
    const int cQ = ((n - min(Jlo, a.nTC - 1) * CW + RC - 1) / RC + tpr - 1) / tpr;
    T tp[kU], tq[kU], ai = T(0), Ais = T(0);
    auto load_parts = [&](int ii) {
      const int Ji = ii / CW, nch = (n - Ji * CW + RC - 1) / RC;
      const T* pp = a.P + (long long)(J0 - Jb) * n + ii;
      const T* pq = a.Qp + ii;
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const int k = sub + u * tpr;
        if (u < cP) tp[u] = k <= Ji - J0 ? pp[(long long)k * n] : T(0);
        if (u < cQ) tq[u] = k < nch ? pq[(long long)k * n] : T(0);
      }
    };
    auto add_parts = [&](T& y) {
#pragma unroll
      for (int u = 0; u < kU; u++) {
        if (u < cP) y += tp[u];
        if (u < cQ) y += tq[u];
      }
    };
    auto row_of = [&](int rl) {  // idle threads read row s (always in range)
      const int i = lo0 + rl;
      return (rl < R0 && i < hi0 && i >= s) ? i : s;
    };
    const T alpha = A[s + (long long)j * ld];
    const T Ass = A[s + (long long)s * ld];
    if (rows) {
      const int ii = row_of(rl0);
      ai = a_at(A, ld, j, s, ii);
      Ais = A[ii + (long long)s * ld];
      load_parts(ii);
    }
    T yraw = T(0);
    if (!kSplit || !rows) {
      const int nchs = (n - Js * CW + RC - 1) / RC;
      constexpr int kN = kSplit ? 2 : 1, kD = kSplit ? 4 : 8;
      T pn[kN], pf[kN], pc[kN], da = T(0), px = T(0), vs = T(0), ws = T(0), dv[kD], dw[kD];
#pragma unroll
      for (int u = 0; u < kN; u++) {
        const int t = tid + u * kRedT;
        pn[u] = t < G ? a.normp[t] : T(0);
        pf[u] = t < G ? a.qfp[t] : T(0);
        pc[u] = t < nchs ? a.Qp[(long long)t * n + s] : T(0);
      }
      if (tid < ndch) da = a.dots[((long long)kDotA * kSytrdNB) * a.nDCH + tid];
      if (tid == 0) px = a.P[(long long)(Js - Jb) * n + s];
      const T* pv = a.dots + ((long long)kDotV * kSytrdNB + lane) * a.nDCH;
      const T* pw = a.dots + ((long long)kDotW * kSytrdNB + lane) * a.nDCH;
      if (wid == 1) {
        if (lane < c) {
          vs = a.V[s + (long long)lane * ldv];
          ws = a.W[s + (long long)lane * ldv];
        }
#pragma unroll
        for (int u = 0; u < kD; u++) {
          dv[u] = lane < c && u < ndch ? pv[u] : T(0);
          dw[u] = lane < c && u < ndch ? pw[u] : T(0);
        }
      }
      T red[4] = {pn[0], pf[0], da, pc[0]};  // sigma, a'A_t a, 2 sum a_r A[r,s], y_s raw
      if (kN > 1 && G > kRedT) {
        red[0] += pn[kN - 1];
        red[1] += pf[kN - 1];
      }
      if (kN > 1 && nchs > kRedT) red[3] += pc[kN - 1];
      if (wid == 0) red[3] += px;
      for (int t = tid + kN * kRedT; t < G; t += kRedT) {
        red[0] += a.normp[t];
        red[1] += a.qfp[t];
      }
      for (int k = tid + kN * kRedT; k < nchs; k += kRedT) red[3] += a.Qp[(long long)k * n + s];
      for (int k = tid + kRedT; k < ndch; k += kRedT) red[2] += a.dots[((long long)kDotA * kSytrdNB) * a.nDCH + k];
      const T x = warp_sum4(red);
      if ((lane & 7) == 0) sred[wid][lane >> 3] = x;
      if (wid == 1) {
        T dV = dv[0], dW = dw[0];
#pragma unroll
        for (int u = 1; u < kD; u++)
          if (u < ndch) {
            dV += dv[u];
            dW += dw[u];
          }
        for (int k = kD; k < ndch; k++)
          if (lane < c) {
            dV += pv[k];
            dW += pw[k];
          }
        sdotV[lane] = dV;
        sdotW[lane] = dW;
        sVs[lane] = vs;
        sWs[lane] = ws;
      }
    }
    if (rows) add_parts(yraw);
    __syncthreads();
    // (2) The reflector's scalars in warp 0; meanwhile the sums over the
    // panel's earlier columns in warp 1, and with them the coefficients of
    // what depends on scale. With v = scale a + e_s, p = V'v, q = W'v:
    //   v'A_t v - 2 p'q = (k2 scale + k1) scale + k0,  y_s = k3 scale + k0,
    //   k2 = a'A_t a - 2 sum dV dW, k1 = 2 a'A[:, s] - 2 sum (dV Ws + Vs dW),
    //   k0 = A[s, s] - 2 sum Vs Ws, k3 = y_s raw - sum (dV Ws + Vs dW).
    // Every step is one instruction of a serial chain (64 cycles in FP64), so
    // lanes 0 and 1 do two different products at once where the chain forks.
    if (wid < 2) {
      T x = sred[(lane >> 2) & (kRedW - 1)][lane & 3];
#pragma unroll
      for (int o = 4; o < 4 * kRedW; o *= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (wid == 1) {
        const T dV = sdotV[lane], dW = sdotW[lane], vs = sVs[lane], ws = sWs[lane];
        const T v[4] = {dV * dW, fma(dV, ws, vs * dW), vs * ws, T(0)};
        const T S = warp_sum4(v);
        // lane 0: k2, 1: k1, 2: k0, 3: k3
        const T Sk = __shfl_sync(0xffffffffu, S, lane == 0 ? 0 : lane == 2 ? 16 : 8);
        const T b = __shfl_sync(0xffffffffu, x, lane == 0 ? 1 : lane == 1 ? 2 : 3);
        const T k = fma(lane == 3 ? T(-1) : T(-2), Sk, lane == 2 ? Ass : b);
        if (lane < 4) sS[lane] = k;
        asm volatile("bar.sync 1, 64;" ::: "memory");
      } else {
        const T sigma = __shfl_sync(0xffffffffu, x, 0);
        T beta, tau, scale;
        panel_scalars(alpha, sigma, beta, tau, scale);
        spv[lane] = fma(scale, sdotV[lane], sVs[lane]);
        sqv[lane] = fma(scale, sdotW[lane], sWs[lane]);
        const T h2 = T(0.5) * tau * tau;
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const T k0 = sS[2];
        // lane 0: k2 scale + k1, lane 1: y_s
        const T u = fma(scale, lane == 0 ? sS[0] : sS[3], lane == 0 ? sS[1] : k0);
        const T hw = h2 * fma(u, scale, k0);  // (lane 0) w = tau y - hw v
        const T y_s = __shfl_sync(0xffffffffu, u, 1);
        if (lane == 0) {
          sscal[0] = tau;
          sscal[1] = scale;
          sscal[2] = hw;
          sscal[3] = fma(tau, y_s, -hw);  // w_s
          if (g == 0) {
            if (c == 0) a.d[j] = A[j + (long long)j * ld];  // later columns: written by the previous step
            a.e[j] = beta;
            a.tau[j] = tau;
          }
        }
      }
    }
    __syncthreads();
    const bool last_in_panel = c + 1 == a.nbp;
    const bool update_next = !last_in_panel || s == n - 1;
    // (3) own rows
    T npart = T(0);
    if (rows) {
      const T tau = sscal[0], scale = sscal[1], hw = sscal[2], w_s = sscal[3];
      for (int rl = rl0; rl < rpp * ((R0 + rpp - 1) / rpp); rl += rpp) {
        const int i = lo0 + rl, ii = row_of(rl);
        const bool act = rl < R0 && i < hi0 && i >= s;
        int k0p = sub + kU * tpr;  // the parts beyond the first batch
        if (rl != rl0) {
          ai = a_at(A, ld, j, s, ii);
          Ais = A[ii + (long long)s * ld];
          yraw = T(0);
          k0p = sub;
        }
        if (rl != rl0 || max(cP, cQ) > kU) {
          const int Ji = ii / CW, nch = (n - Ji * CW + RC - 1) / RC;
          const T* pp = a.P + (long long)(J0 - Jb) * n + ii;
          const T* pq = a.Qp + ii;
#pragma unroll 4
          for (int k = k0p; k <= Ji - J0; k += tpr) yraw += pp[(long long)k * n];
#pragma unroll 4
          for (int k = k0p; k < nch; k += tpr) yraw += pq[(long long)k * n];
        }
        const int rc = rl < R0 ? rl : R0 - 1;  // (idle threads: any cached row)
        T y = T(0), xn = T(0);
        for (int q = sub; q < c; q += tpr) {
          const T vq = sVr[(size_t)rc * kSytrdNB + q], wq = sWr[(size_t)rc * kSytrdNB + q];
          y = fma(vq, sqv[q], fma(wq, spv[q], y));
          xn = fma(vq, sWs[q], fma(wq, sVs[q], xn));
        }
        y = fma(scale, yraw, -y);
        // y and xn over the row's tpr lanes: the halves swap one of the two first
        if (tpr > 1) {
          const int h = tpr / 2;
          const bool up = sub >= h;
          T z = (up ? xn : y) + __shfl_xor_sync(0xffffffffu, up ? y : xn, h);
          for (int o = h / 2; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
          const T other = __shfl_xor_sync(0xffffffffu, z, h);
          y = up ? other : z;
          xn = up ? z : other;
        }
        y += Ais;
        const T vi = ii == s ? T(1) : scale * ai;
        const T wi = fma(tau, y, -hw * vi);
        xn += fma(vi, w_s, wi);  // the q = c term: v_s = 1, w_s
        if (act && sub == 0) {
          a.V[ii + (long long)c * ldv] = vi;
          a.W[ii + (long long)c * ldv] = wi;
          sVr[(size_t)rl * kSytrdNB + c] = vi;
          sWr[(size_t)rl * kSytrdNB + c] = wi;
          if (ii > s) A[ii + (long long)j * ld] = vi;
          if (update_next) {
            // A[s, s] is read by every CTA in this phase: its new value goes to d[s]
            const T x = Ais - xn;
            if (ii == s)
              a.d[s] = x;
            else
              A[ii + (long long)s * ld] = x;
            if (ii > s + 1) npart = fma(x, x, npart);
          }
        }
      }
      npart = lane_sum(npart, tpr);  // (lanes with sub > 0 hold zero)
    }
    if (lane == 0) spart[wid] = npart;
    if (c + 1 < a.nbp)
      if (!grid_sync<T, CL>(a.bar, a.err, bar_target, spart, a.normp + g)) return;
  }
}

// ---------------------------------------------------------------- host side

struct SytrdPlan {
  int n = 0, G = 0;
  int nDCH = 0;
  int* ustart = nullptr;  // the shapes' tables, one after another
  int uoff[kNumShapes] = {};
  void* P = nullptr;
  void* Qp = nullptr;
  void* normp = nullptr;
  void* qfp = nullptr;
  void* dots = nullptr;
  void* VW = nullptr;     // [V | W] panel buffer, n x 2 kSytrdNB
  float* VWt = nullptr;   // FP32: [V | W] transposed (2 kSytrdNB x n), the tensor-core update's K-major operand
  int* bkidx = nullptr;   // SYR2K k remaps: [2 nb] for nbp = kSytrdNB, then for the last panel
  unsigned* bar = nullptr;
  int* err = nullptr;
  bool f64 = true;
  size_t bytes = 0;       // device memory held
  bool cluster = false;   // the device can hold a cluster: small trailing orders run on it
  bool cluster_only = false;  // and all others too
  int2* F = nullptr;      // FP64, orders above kFixedMin: the trailing matrix in fixed point, n x n
  int* fe = nullptr;      // exponents of its units, [tile column][fch]
  int fch = 0;
  Oz64* oz = nullptr;     // FP64: trailing updates on the tensor cores (set by sytrd_set_oz64)
};

// [V | W] of a panel with nbp reflectors (V at VW, W at VW + nbp n, rows
// t.. of interest) into VWt: row kk < 32 = V column kk, row 32 + kk = W
// column kk (zero for kk >= nbp), column i = row i.
__global__ void k_vw_transpose(const float* __restrict__ VW, int n, int nbp, int t, float* __restrict__ VWt) {
  __shared__ float tile[32][65];
  const int i0 = t + blockIdx.x * 32;
  for (int idx = threadIdx.x; idx < 32 * 64; idx += blockDim.x) {
    const int ii = idx % 32, kk = idx / 32;
    const int i = i0 + ii;
    const int c = kk < 32 ? kk : kk - 32;
    float v = 0.f;
    if (i < n && c < nbp) v = VW[i + (long long)(kk < 32 ? c : nbp + c) * n];
    tile[ii][kk] = v;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 32 * 64; idx += blockDim.x) {
    const int kk = idx % 64, ii = idx / 64;
    const int i = i0 + ii;
    if (i < n) VWt[kk + (long long)i * 64] = tile[ii][kk];
  }
}

}  // namespace gla

namespace {
using namespace gla;

// The trailing update A[t:, t:] -= V W' + W V' (lower tiles) as two K
// segments of the 3xTF32 tensor-core GEMM: A operand rows = V / W rows
// (K-major through VWt), B operand columns = W / V rows. False when the
// shapes do not allow the tensor maps (the SIMT GEMM then runs).
bool sytrd_update_tc(SytrdPlan& sp, float* A, long long lda, int n, int t, int nbp, cudaStream_t st,
                     cudaError_t* err) {
  *err = cudaSuccess;
  if (sp.VWt == nullptr || kSytrdNB != 32) return false;
  CUtensorMap m;
  if (!tc::tc_make_map(&m, sp.VWt, 64, n, 64, tc::kBM)) return false;
  k_vw_transpose<<<(n - t + 31) / 32, 256, 0, st>>>((const float*)sp.VW, n, nbp, t, sp.VWt);
  if ((*err = cudaGetLastError()) != cudaSuccess) return true;
  tc::TcArgs g{};
  g.M = g.N = n - t;
  g.nseg = 2;
  g.K[0] = g.K[1] = 32;
  g.a_x[0] = 0;   // V
  g.b_x[0] = 32;  // W
  g.a_x[1] = 32;  // W
  g.b_x[1] = 0;   // V
  g.a_y = g.b_y = t;
  g.D = A + t + (long long)t * lda;
  g.ldd = lda;
  g.alpha = -1.f;
  g.beta = 1.f;
  g.lower = 1;
  g.err = sp.err;
  *err = tc::tc_gemm_launch(m, m, g, 1, st);
  return true;
}

int panel_shape(int m, bool f64) {
  int sh = 0;
  while (sh + 1 < kNumShapes && (!f64 || m > kShapes[sh].max_m)) sh++;
  return sh;
}
template <class T>
const void* panel_kernel(int sh, bool cluster, bool fixed = false) {
  static_assert(kNumShapes == 4, "one kernel per shape");
  if constexpr (sizeof(T) == 8) {
    if (fixed) return (const void*)k_sytrd_panel<T, kFixW, kFixR / 32, false, true>;
    if (cluster && sh == 0) return (const void*)k_sytrd_panel<T, kShapes[0].cw, kShapes[0].nq, true>;
    if (cluster && sh == 1) return (const void*)k_sytrd_panel<T, kShapes[1].cw, kShapes[1].nq, true>;
    if (cluster && sh == 2) return (const void*)k_sytrd_panel<T, kShapes[2].cw, kShapes[2].nq, true>;
    if (sh == 0) return (const void*)k_sytrd_panel<T, kShapes[0].cw, kShapes[0].nq, false>;
    if (sh == 1) return (const void*)k_sytrd_panel<T, kShapes[1].cw, kShapes[1].nq, false>;
    if (sh == 2) return (const void*)k_sytrd_panel<T, kShapes[2].cw, kShapes[2].nq, false>;
  }
  if (cluster) return (const void*)k_sytrd_panel<T, kShapes[3].cw, kShapes[3].nq, true>;
  return (const void*)k_sytrd_panel<T, kShapes[3].cw, kShapes[3].nq, false>;
}
// One panel: over the whole GPU as a cooperative launch, or as one cluster.
template <class T>
cudaError_t launch_panel(const SytrdPlan& sp, const SytrdArgs<T>& a, int sh, bool cluster, bool fixed,
                         cudaStream_t st) {
  const int G = cluster ? kClusterG : sp.G;
  cudaLaunchAttribute at[1];
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClusterG;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(kPT);
  cfg.dynamicSmemBytes = 2 * (size_t)panel_rows(a.k0, a.n, G) * kSytrdNB * sizeof(T);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {(void*)&a};
  return cudaLaunchKernelExC(&cfg, panel_kernel<T>(sh, cluster, fixed), args);
}

template <class T>
cudaError_t sytrd_run(SytrdPlan& sp, T* A, long long lda, T* d, T* e, T* tau, cudaStream_t st) {
  const int n = sp.n;
  cudaError_t err;
  if ((err = cudaMemsetAsync(sp.bar, 0, 2 * sizeof(unsigned), st)) != cudaSuccess) return err;
  if ((err = cudaMemsetAsync(sp.err, 0, sizeof(int), st)) != cudaSuccess) return err;
  SytrdArgs<T> a;
  a.A = A;
  a.ld = lda;
  a.n = n;
  a.ldv = n;
  a.d = d;
  a.e = e;
  a.tau = tau;
  a.P = (T*)sp.P;
  a.Qp = (T*)sp.Qp;
  a.normp = (T*)sp.normp;
  a.qfp = (T*)sp.qfp;
  a.dots = (T*)sp.dots;
  a.nDCH = sp.nDCH;
  a.F = sp.F;
  a.fe = sp.fe;
  a.fch = sp.fch;
  a.bar = sp.bar;
  a.err = sp.err;
  T* VW = (T*)sp.VW;
  unsigned bar_base = 0;
  const int nsteps = n - 1;  // reflectors 0 .. n-2
  for (int k0 = 0; k0 < nsteps; k0 += kSytrdNB) {
    const int nbp = std::min(kSytrdNB, nsteps - k0);
    a.k0 = k0;
    a.nbp = nbp;
    a.V = VW;
    a.W = VW + (long long)nbp * n;
    const int m = n - k0 - 1;
    const bool cluster = sp.cluster && (sp.cluster_only || m <= (sizeof(T) == 8 ? kClusterMaxF64 : kClusterMaxF32));
    a.bar_base = bar_base;
    if (!cluster) bar_base += 2u * (unsigned)nbp * (unsigned)sp.G;  // barriers per launch: 1 + nbp + (nbp - 1)
    // (a cluster has a tenth of the warps: the shape of a trailing order
    // with that many units per warp)
    const bool fixed = sp.F && m > kFixedMin && !cluster;
    const int sh = fixed ? kNumShapes - 1 : panel_shape(cluster ? std::min(3 * m, kMaxOrder) : m, sizeof(T) == 8);
    if constexpr (sizeof(T) == 8) {
      if (fixed) {
        const int J0 = k0 / kFixW;
        k_sytrd_fix<<<dim3((n - k0 + kFixR - 1) / kFixR, (n + kFixW - 1) / kFixW - J0), 256, 0, st>>>(
            A, lda, n, J0, sp.F, sp.fe, sp.fch);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
      }
    }
    a.nTC = (n + kShapes[sh].cw - 1) / kShapes[sh].cw;
    a.ustart = sp.ustart + sp.uoff[sh];
    if ((err = launch_panel(sp, a, sh, cluster, fixed, st)) != cudaSuccess) return err;
    const int t = k0 + nbp;
    if (t < n - 1) {  // trailing update A[t:, t:] -= V W' + W V' (lower tiles)
      if (sizeof(T) == 4 && sytrd_update_tc(sp, (float*)A, lda, n, t, nbp, st, &err)) {
        if (err != cudaSuccess) return err;
        continue;
      }
      // (down to the last columns: an order of 96 takes 25 us there, 70 on the
      // few CTAs of the FP64 loops)
      if (sizeof(T) == 8 && sp.oz) {
        err = oz64_rank2k(sp.oz, (const double*)VW, nbp, t, (double*)A, lda, st);
        if (err != cudaSuccess) return err;
        continue;
      }
      GemmDesc g{};
      g.m = n - t;
      g.n = n - t;
      g.k = 2 * nbp;
      g.A = VW + t;
      g.lda = n;
      g.B = VW + t;
      g.ldb = n;
      g.C = A + t + (long long)t * lda;
      g.ldc = lda;
      g.b_kidx = sp.bkidx + (nbp == kSytrdNB ? 0 : 2 * kSytrdNB);
      g.alpha = -1.0;
      g.beta = 1.0;
      err = gemm_launch(sizeof(T) == 8, false, true, true, g, 1, st);
      if (err != cudaSuccess) return err;
    }
  }
  return cudaSuccess;
}

}  // namespace

namespace gla {

cudaError_t sytrd_plan_create(SytrdPlan** out, int n, bool f64, bool tc) {
  *out = nullptr;
  SytrdPlan* sp = new SytrdPlan();
  sp->n = n;
  sp->f64 = f64;
  int dev = 0, nsm = 0, per = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // phase B's V / W row cache: 2 rows-per-CTA x kSytrdNB values. The limit
  // is a property of the kernel, shared by every plan: always the largest
  // order's, so that a plan made later never lowers it below an earlier
  // plan's launches.
  const int vwbytes = 2 * panel_rows(0, kMaxOrder, std::max(nsm, 1)) * kSytrdNB * (f64 ? 8 : 4);
  const bool fx = f64 && n > kFixedMin;
  for (int sh = f64 ? 0 : kNumShapes - 1; sh < kNumShapes + fx; sh++) {  // (with fx the fixed-point kernel, last)
    const void* kfn = f64 ? panel_kernel<double>(sh, false, sh == kNumShapes) : panel_kernel<float>(sh, false);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, vwbytes);
    if (err == cudaSuccess) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kfn, kPT, vwbytes);
    if (err == cudaSuccess && per < 1) err = cudaErrorCooperativeLaunchTooLarge;
  }
  if (err == cudaSuccess) {  // a cluster of kClusterG CTAs, where the device can hold one
    const int csmem = 2 * ((kSideBySideMaxN + kClusterG) / kClusterG) * kSytrdNB * (f64 ? 8 : 4);
    const void* kfn = nullptr;
    for (int sh = f64 ? 0 : kNumShapes - 1; sh < kNumShapes; sh++) {
      kfn = f64 ? panel_kernel<double>(sh, true) : panel_kernel<float>(sh, true);
      if (err == cudaSuccess) err = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, csmem);
      if (err == cudaSuccess) err = cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    if (err == cudaSuccess) {
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kClusterG;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(kClusterG);
      cfg.blockDim = dim3(kPT);
      cfg.dynamicSmemBytes = csmem;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nc = 0;
      sp->cluster = cudaOccupancyMaxActiveClusters(&nc, kfn, &cfg) == cudaSuccess && nc >= 1;
      if (!sp->cluster) cudaGetLastError();
    }
  }
  if (err != cudaSuccess) {
    delete sp;
    return err;
  }
  sp->G = nsm;  // one CTA per SM (co-residency of a cooperative launch)
  const int dot_rows = f64 ? kDotRows<double> : kDotRows<float>;
  sp->nDCH = (n + dot_rows - 1) / dot_rows;
  // unit tables of the shapes, and the partial buffers that hold any of them
  std::vector<int> ustart;
  size_t np = 0, nq = 0;
  for (int sh = 0; sh < kNumShapes; sh++) {
    const UnitShape& u = kShapes[sh];
    const int ntc = (n + u.cw - 1) / u.cw, rc = 32 * u.nq, m = std::min(n, f64 || sh == kNumShapes - 1 ? u.max_m + 1 : 0);
    sp->uoff[sh] = (int)ustart.size();
    int total = 0;
    for (int J = 0; J < ntc; J++) {
      ustart.push_back(total);
      total += (n - J * u.cw + rc - 1) / rc;  // chunks of tile column J
    }
    ustart.push_back(total);
    np = std::max(np, (size_t)(m + u.cw - 1) / u.cw + 1);
    nq = std::max(nq, (size_t)(m + u.cw + rc - 1) / rc + 1);
  }
  std::vector<int> bk(4 * kSytrdNB);
  const int last = (n - 1) % kSytrdNB == 0 ? kSytrdNB : (n - 1) % kSytrdNB;
  for (int kk = 0; kk < 2 * kSytrdNB; kk++) bk[kk] = kk < kSytrdNB ? kSytrdNB + kk : kk - kSytrdNB;
  for (int kk = 0; kk < 2 * last; kk++) bk[2 * kSytrdNB + kk] = kk < last ? last + kk : kk - last;
  const size_t el = f64 ? 8 : 4;
  auto alloc = [&](void** p, size_t bytes) {
    if (err == cudaSuccess) err = counted_malloc(p, bytes, &sp->bytes);
  };
  alloc((void**)&sp->ustart, sizeof(int) * ustart.size());
  alloc(&sp->P, el * np * n);
  alloc(&sp->Qp, el * nq * n);
  alloc(&sp->normp, el * sp->G);
  alloc(&sp->qfp, el * sp->G);
  alloc(&sp->dots, el * 3 * kSytrdNB * sp->nDCH);
  alloc(&sp->VW, el * (size_t)n * 2 * kSytrdNB);
  alloc((void**)&sp->bkidx, sizeof(int) * bk.size());
  if (fx) {
    sp->fch = (n + kFixR - 1) / kFixR;
    alloc((void**)&sp->F, sizeof(int2) * (size_t)n * n);
    alloc((void**)&sp->fe, sizeof(int) * (size_t)((n + kFixW - 1) / kFixW) * sp->fch);
  }
  alloc((void**)&sp->bar, 2 * sizeof(unsigned));
  alloc((void**)&sp->err, sizeof(int));
  if (err == cudaSuccess)
    err = cudaMemcpy(sp->ustart, ustart.data(), sizeof(int) * ustart.size(), cudaMemcpyHostToDevice);
  if (err == cudaSuccess) err = cudaMemcpy(sp->bkidx, bk.data(), sizeof(int) * bk.size(), cudaMemcpyHostToDevice);
  if (err == cudaSuccess) err = cudaMemset(sp->VW, 0, el * (size_t)n * 2 * kSytrdNB);
  if (err == cudaSuccess && !f64 && tc && tc::tc_available()) alloc((void**)&sp->VWt, sizeof(float) * 64 * (size_t)n);
  if (err != cudaSuccess) {
    sytrd_plan_destroy(sp);
    return err;
  }
  *out = sp;
  return cudaSuccess;
}

void sytrd_plan_destroy(SytrdPlan* sp) {
  if (!sp) return;
  cudaFree(sp->ustart);
  cudaFree(sp->P);
  cudaFree(sp->Qp);
  cudaFree(sp->normp);
  cudaFree(sp->qfp);
  cudaFree(sp->dots);
  cudaFree(sp->VW);
  cudaFree(sp->VWt);
  cudaFree(sp->bkidx);
  cudaFree(sp->F);
  cudaFree(sp->fe);
  cudaFree(sp->bar);
  cudaFree(sp->err);
  delete sp;
}

cudaError_t sytrd_enqueue(SytrdPlan* sp, void* A, long long lda, void* d, void* e, void* tau, cudaStream_t st) {
  if (sp->f64) return sytrd_run<double>(*sp, (double*)A, lda, (double*)d, (double*)e, (double*)tau, st);
  return sytrd_run<float>(*sp, (float*)A, lda, (float*)d, (float*)e, (float*)tau, st);
}

int* sytrd_error_word(SytrdPlan* sp) { return sp->err; }
size_t sytrd_plan_bytes(const SytrdPlan* sp) { return sp->bytes; }
void sytrd_set_oz64(SytrdPlan* sp, Oz64* oz) { sp->oz = oz; }
void sytrd_keep_entries(SytrdPlan* sp) {
  cudaFree(sp->F);
  cudaFree(sp->fe);
  sp->F = nullptr;
  sp->fe = nullptr;
}
bool sytrd_set_cluster_only(SytrdPlan* sp) {
  sp->cluster_only = sp->cluster && sp->n <= kSideBySideMaxN;
  return sp->cluster_only;
}

}  // namespace gla
