// FP64-accurate GEMM on the tcgen05 tensor cores (Ozaki scheme), the
// products of the FP64 large-matrix path: C = alpha A B + beta C with FP64
// operands and results, alpha = +-1, beta = 0 or 1.
//
// GB300's FP64 pipe gives 1.19 TFLOP/s, the bf16 tensor pipe 1900; the 34
// slice products below run at about 30 TFLOP/s of FP64-equivalent work. The
// scheme is the one of ozaki.cuh with wider digits and all of its sums in
// integers: every row of A and column of B is scaled by 2^-e, 2^e above its
// largest entry, rounded to 56 bits and written as seven balanced 8-bit
// digits (|d_1| <= 256, |d_s| <= 128 after), exact in bf16. Pairs with
// s + t <= 9 accumulate exactly in eight TMEM level accumulators of 64
// columns (all 512) over at most 96 k (the largest level, L = 8, adds
// 2 x 256 x 128 + 5 x 128^2 = 147,456 per k, and 96 x 147,456 < 2^24); the
// drained levels are summed in 64-bit integers and rounded to FP64 once.
//
// Error: 2^-57 of 2^e per entry of A and of B, while the pairs left out
// (s + t >= 10) stay below 2^-61; the sum itself is exact, where an FP64 loop
// rounds K times. Eight 7-bit digits with the same eight levels (36 pairs)
// have the same operands but leave out pairs of 2^-53: a reflector's unit
// element is 30 times its other entries, and |V'V - I| / sqrt(n) of order-4096
// eigenvectors came out at 1.4e-14 (Frobenius norm). It is 4.0e-15 with these
// digits, 5.6e-15 with the FP64 loops; residuals 1.9e-15 and 2.5e-15 |A|.
//
// A row or column with an infinity or NaN gives NaN.
//
// Kernel: CTA tile 128 x 64, 18 warps. Warp 0 streams 32-k slabs (84 KB, two
// stages) with bulk copies, warp 1 issues the MMAs, sixteen warps drain
// (quarter of the TMEM lanes = warp mod 4, 16 columns each). Operands of
// either side are stored in row blocks of 128, so one sliced matrix serves
// as both; a tile's 64 right-hand rows are one half of each slice. Every
// wait is bounded as in ozaki.cuh.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm_simt.cuh"
#include "oz_prims.cuh"

namespace gla {
namespace oz64 {

using oz::kKS;
constexpr int kS = 7;                 // slices (digits of 8 bits)
constexpr int kBM = 128, kBN = 64;    // C tile
constexpr int kMaxLevel = 9;          // levels 2 .. 9
constexpr int kGroupK = 96;           // k per TMEM drain (exactness)
constexpr int kStages = 2;
constexpr int kDrainWarps = 16;
constexpr int kThreads = 64 + 32 * kDrainWarps;
constexpr int kBadExp = 1 << 20;      // exponent of a row with a non-finite entry
__host__ __device__ constexpr int block_bytes(int rows) { return rows * kKS * 2; }
constexpr uint32_t kAAll = kS * block_bytes(kBM), kBAll = kS * block_bytes(kBN);
constexpr size_t kStageBytes = (size_t)kAAll + kBAll;
constexpr size_t kSmem = kStages * kStageBytes;
__host__ __device__ constexpr uint32_t idesc(int nn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}
static_assert((kMaxLevel - 1) * kBN <= 512 && kSmem + 1024 <= 232448, "TMEM columns, shared memory");

// A matrix as a sliced operand: row block b (128 rows), slab q, slice s at
// base + ((b nks + q) kS + s) block_bytes(128); exps: one exponent per row.
struct Operand {
  unsigned char* base;
  int* exps;
  unsigned* mx;  // slicing scratch: high word of the largest |entry| of each row
};

// Where an operand comes from: row c, index k is src[c ld + k'] (rows =
// false) or src[c + k' ld] (rows = true), k' = kidx ? kidx[k] : k.
struct Source {
  const double* src;
  long long ld;
  int count, len;
  const int* kidx;
};

// ---------------------------------------------------------------- slicing

// Exponent e of a row from the high word of its largest |entry|: all entries
// are below 2^e.
GLA_DEV int row_exp(unsigned mx) {
  const int be = (int)(mx >> 20);
  if (be >= 0x7ff) return kBadExp;
  return (be > 0 ? be : 1) - 1022;
}

// x 2^(56 - e) rounded to an integer (|x| < 2^e; round half away).
GLA_DEV long long fixed56(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int be = (int)((b >> 52) & 0x7ff);
  unsigned long long m = b & 0xfffffffffffffull;
  if (be > 0) m |= 1ull << 52;
  const int r = (be > 0 ? be : 1) - 1019 - e;  // <= 3
  if (r >= 0)
    m <<= r;
  else if (r > -55)
    m = ((m >> (-r - 1)) + 1) >> 1;
  else
    m = 0;
  return (b >> 63) ? -(long long)m : (long long)m;
}

// bf16 bits of two small integers (|d| <= 256: exact).
GLA_DEV unsigned bf16_pair(int d0, int d1) {
  const float f0 = __int_as_float(0x4b400000 + d0) - 12582912.f;
  const float f1 = __int_as_float(0x4b400000 + d1) - 12582912.f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// The seven digits of X (|X| <= 2^56): d[0] the leading one.
GLA_DEV void digits(long long X, int (&d)[kS]) {
  // low 24 bits as a balanced number (three digits), the rest above (four)
  int l = (int)((unsigned)X << 8) >> 8;
  const long long up = (X - l) >> 24;          // |up| <= 2^32
  const int l2 = (int)((unsigned)up << 8) >> 8;  // its low 24 bits: three digits
  const int top = (int)((up - l2) >> 24);      // |top| <= 256
  d[6] = (int)(signed char)l;
  l = (l - d[6]) >> 8;
  d[5] = (int)(signed char)l;
  d[4] = (l - d[5]) >> 8;  // |.| <= 128
  int h = l2;
  d[3] = (int)(signed char)h;
  h = (h - d[3]) >> 8;
  d[2] = (int)(signed char)h;
  d[1] = (h - d[2]) >> 8;
  d[0] = top;
}

// Largest |entry| of every operand row (bits of its high word).
// rows = false: one warp per operand row.
GLA_DEV void max_cols_body(const Source& s, int rows_pad, unsigned* __restrict__ mx) {
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= rows_pad) return;
  unsigned m = 0;
  if (c < s.count)
    for (int k = lane; k < s.len; k += 32) {
      const int kk = s.kidx ? s.kidx[k] : k;
      m = max(m, (unsigned)__double2hiint(s.src[(long long)c * s.ld + kk]) & 0x7fffffffu);
    }
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) mx[c] = m;
}
__global__ void __launch_bounds__(256) k_max_cols(Source s, int rows_pad, unsigned* __restrict__ mx) {
  max_cols_body(s, rows_pad, mx);
}
// rows = true: one thread per operand row and chunk of 64 k; mx zero on entry.
GLA_DEV void max_rows_body(const Source& s, unsigned* __restrict__ mx) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= s.count) return;
  const int k0 = blockIdx.y * 64, k1 = min(s.len, k0 + 64);
  unsigned m = 0;
  for (int k = k0; k < k1; k++) {
    const int kk = s.kidx ? s.kidx[k] : k;
    m = max(m, (unsigned)__double2hiint(s.src[c + (long long)kk * s.ld]) & 0x7fffffffu);
  }
  if (m) atomicMax(&mx[c], m);
}
__global__ void __launch_bounds__(256) k_max_rows(Source s, unsigned* __restrict__ mx) { max_rows_body(s, mx); }

constexpr int kBB = block_bytes(kBM);

// The digits of two neighbouring k of row r into the slab image at dst0.
GLA_DEV void put_pair(unsigned char* slab, int r, int k, double x0, double x1, int e) {
  int d0[kS], d1[kS];
  const bool bad = e == kBadExp;
  digits(bad ? 0 : fixed56(x0, e), d0);
  digits(bad ? 0 : fixed56(x1, e), d1);
  unsigned char* dst = slab + oz::tile_off(r, k);
#pragma unroll
  for (int j = 0; j < kS; j++) *reinterpret_cast<unsigned*>(dst + j * kBB) = bf16_pair(d0[j], d1[j]);
}
GLA_DEV void copy_slab(unsigned char* dst, const unsigned char* slab) {
  uint4* g = reinterpret_cast<uint4*>(dst);
  const uint4* sv = reinterpret_cast<const uint4*>(slab);
  for (int v = threadIdx.x; v < kS * kBB / 16; v += 256) g[v] = sv[v];
}

// One row block's slab q: the seven slices laid out in shared memory and
// written with 16-byte stores; each thread takes pairs of neighbouring k.
// Bound by the integer pipe (about 30 instructions per entry and slice set)
// and by writing 14 bytes per entry.
template <bool ROWS>
GLA_DEV void tile_body(const Source& s, const Operand& out, int b, int q, int nks, unsigned char* tsm) {
  const int tid = threadIdx.x;
#pragma unroll 1
  for (int t = tid; t < kBM * kKS / 2; t += 256) {
    const int r = ROWS ? t % kBM : t / (kKS / 2), kp = ROWS ? t / kBM : t % (kKS / 2);
    const int c = b * kBM + r, k = q * kKS + 2 * kp;
    double x0 = 0, x1 = 0;
    int e = 0;
    if (c < s.count) {
      e = row_exp(out.mx[c]);
      const int i0 = k < s.len ? (s.kidx ? s.kidx[k] : k) : -1;
      const int i1 = k + 1 < s.len ? (s.kidx ? s.kidx[k + 1] : k + 1) : -1;
      if (i0 >= 0) x0 = ROWS ? s.src[c + (long long)i0 * s.ld] : s.src[(long long)c * s.ld + i0];
      if (i1 >= 0) x1 = ROWS ? s.src[c + (long long)i1 * s.ld] : s.src[(long long)c * s.ld + i1];
    }
    put_pair(tsm, r, 2 * kp, x0, x1, e);
  }
  if (q == 0)
    for (int r = tid; r < kBM; r += 256) {
      const int c = b * kBM + r;
      out.exps[c] = c < s.count ? row_exp(out.mx[c]) : 0;
    }
  __syncthreads();
  copy_slab(out.base + ((size_t)b * nks + q) * kS * (size_t)kBB, tsm);
}
template <bool ROWS>
__global__ void __launch_bounds__(256) k_tile(Source s, Operand out) {
  extern __shared__ __align__(16) unsigned char tsm[];
  tile_body<ROWS>(s, out, blockIdx.x, blockIdx.y, gridDim.y, tsm);
}

// The panel factors of a trailing update, X = V or W (grid.y): rows t .. t +
// m - 1 and nbp <= 32 columns of X as an operand of one slab. V at VW, W nbp
// columns further.
struct VwArgs {
  const double* VW;
  long long ld;
  int t, m, nbp;
  Operand op[2];
};
__global__ void __launch_bounds__(256) k_slice_vw(const VwArgs a) {
  extern __shared__ __align__(16) unsigned char tsm[];
  __shared__ unsigned smx[2][kBM];
  const int b = blockIdx.x, w = blockIdx.y, tid = threadIdx.x;
  const int r = tid % kBM, h = tid / kBM;  // row of the block, half of the columns
  const int row = b * kBM + r;
  const double* X = a.VW + (long long)w * a.nbp * a.ld + a.t + row;
  double x[kKS / 2];
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < kKS / 2; k++) {
    const int kk = h * (kKS / 2) + k;
    x[k] = row < a.m && kk < a.nbp ? X[(long long)kk * a.ld] : 0.0;
    m = max(m, (unsigned)__double2hiint(x[k]) & 0x7fffffffu);
  }
  smx[h][r] = m;
  __syncthreads();
  // one bit more than the largest entry needs: |d_1| <= 128 (see NSEG = 2)
  const int e0 = row_exp(max(smx[0][r], smx[1][r])), e = e0 == kBadExp ? e0 : e0 + 1;
#pragma unroll
  for (int k = 0; k < kKS / 2; k += 2) put_pair(tsm, r, h * (kKS / 2) + k, x[k], x[k + 1], e);
  if (h == 0) a.op[w].exps[row] = e;
  __syncthreads();
  copy_slab(a.op[w].base + (size_t)b * kS * kBB, tsm);
}

// Rows of a block column of 128 (grid: row block, block column): rows 128 b
// .., columns 128 y .. of X (n x n) as the row-form operand of that block
// column, four slabs, exponents of row r at exps[y rows_pad + r]. Row blocks
// above the diagonal block are left out (X is zero there).
__global__ void __launch_bounds__(256) k_slice_blockcol(const double* __restrict__ X, long long ld, int n, int rows_pad,
                                                        unsigned char* __restrict__ base, int* __restrict__ exps) {
  extern __shared__ __align__(16) unsigned char tsm[];
  __shared__ unsigned smx[2][kBM];
  const int b = blockIdx.x, y = blockIdx.y, tid = threadIdx.x;
  if (b < y) return;
  const int r = tid % kBM, h = tid / kBM, row = b * kBM + r;
  const double* src = X + row + (long long)y * kBM * ld;
  const int ncol = min(kBM, n - y * kBM);
  unsigned m = 0;
  if (row < n)
    for (int k = h; k < ncol; k += 2) m = max(m, (unsigned)__double2hiint(src[(long long)k * ld]) & 0x7fffffffu);
  smx[h][r] = m;
  __syncthreads();
  const int e = row_exp(max(smx[0][r], smx[1][r]));
  if (h == 0) exps[(size_t)y * rows_pad + row] = e;
  const size_t nb = rows_pad / kBM;
  for (int q = 0; q < 4; q++) {
#pragma unroll 1
    for (int k = 0; k < kKS / 2; k += 2) {
      const int kk = h * (kKS / 2) + k, col = q * kKS + kk;
      const double x0 = row < n && col < ncol ? src[(long long)col * ld] : 0.0;
      const double x1 = row < n && col + 1 < ncol ? src[(long long)(col + 1) * ld] : 0.0;
      put_pair(tsm, r, kk, x0, x1, e);
    }
    __syncthreads();
    copy_slab(base + (((size_t)y * nb + b) * 4 + q) * kS * kBB, tsm);
    __syncthreads();
  }
}

// Columns of W = sum of its split-K partials (128 x ncol, leading dimension
// 128) as an operand of four slabs (grid: column block, slab).
__global__ void __launch_bounds__(256) k_slice_w(const double* __restrict__ Wp, int splits, long long pstride, int ncol,
                                                 Operand out) {
  extern __shared__ __align__(16) unsigned char tsm[];
  const int b = blockIdx.x, q = blockIdx.y, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int cc = wid; cc < kBM; cc += 8) {  // one column per warp, lane l: k = 4 l .. 4 l + 3
    const int c = b * kBM + cc;
    double x[4] = {0, 0, 0, 0};
    if (c < ncol)
      for (int s = 0; s < splits; s++) {
        const double2* p = reinterpret_cast<const double2*>(Wp + s * pstride + (long long)c * kBM) + 2 * lane;
        const double2 u = p[0], v = p[1];
        x[0] += u.x;
        x[1] += u.y;
        x[2] += v.x;
        x[3] += v.y;
      }
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) m = max(m, (unsigned)__double2hiint(x[i]) & 0x7fffffffu);
    m = __reduce_max_sync(0xffffffffu, m);
    const int e = row_exp(m);
    if (q == 0 && lane == 0) out.exps[c] = e;
    if (lane / 8 == q) {
      put_pair(tsm, cc, 4 * (lane % 8), x[0], x[1], e);
      put_pair(tsm, cc, 4 * (lane % 8) + 2, x[2], x[3], e);
    }
  }
  __syncthreads();
  copy_slab(out.base + ((size_t)b * 4 + q) * kS * kBB, tsm);
}

// ---------------------------------------------------------------- GEMM

struct Seg {
  const unsigned char* A;  // first row block of the left operand, first slab
  const unsigned char* B;
  const int* ea;           // exponents of C's rows, of C's columns
  const int* eb;
  int nks;                 // slabs to multiply
  int a_nks, b_nks;        // slabs per row block in the operands' buffers
};
struct Args {
  Seg seg[2];
  int M, N;
  double* C;
  long long ldc;
  const int* c_nidx;  // output column of column j (null: j)
  int neg, add;       // alpha = -1; beta = 1
  int lower;          // only i >= j (and only the tiles that hold such entries)
  int ksplit;         // slabs per split (0: none); split y writes to C + y split_stride
  long long split_stride;
  int* err;
};

// (H 2^32 + L) 2^(ex - 72) rounded to FP64.
GLA_DEV double to_double(long long H, long long L, int ex) {
  __int128 v = ((__int128)H << 32) + L;
  const bool neg = v < 0;
  const unsigned __int128 u = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
  const unsigned long long uh = (unsigned long long)(u >> 64), ul = (unsigned long long)u;
  if ((uh | ul) == 0) return 0.0;
  const int lz = uh ? __clzll((long long)uh) : 64 + __clzll((long long)ul);
  const unsigned __int128 w = u << lz;
  unsigned long long m = (unsigned long long)(w >> 75);
  const unsigned long long rest = (unsigned long long)(w >> 11);  // the 64 bits below the mantissa
  const bool sticky = ((unsigned)w & 0x7ffu) != 0;
  m += (rest >> 63) && ((rest << 1) != 0 || sticky || (m & 1));
  const int be = 127 - lz - 72 + ex + 1022;  // exponent field before the implicit bit is added
  double x;
  if (be >= 0 && be < 2045)
    x = __longlong_as_double((long long)(((unsigned long long)be << 52) + m));
  else
    x = ldexp((double)m, be - 1022 - 52);
  return neg ? -x : x;
}

// X 2^ex rounded to FP64 (|X| < 2^63; ties away from zero).
GLA_DEV double to_double(long long X, int ex) {
  const unsigned long long u = (unsigned long long)(X < 0 ? -X : X);
  if (u == 0) return 0.0;
  const int lz = __clzll((long long)u);
  const unsigned long long m = (((u << lz) >> 10) + 1) >> 1;
  const int be = 63 - lz + ex + 1022;  // exponent field before the implicit bit is added
  double x;
  if (be >= 0 && be < 2045)
    x = __longlong_as_double((long long)(((unsigned long long)be << 52) + m));
  else
    x = ldexp((double)m, be - 1022 - 52);
  return X < 0 ? -x : x;
}
// X >> k with rounding, any k >= 0.
GLA_DEV long long shift_down(long long X, int k) {
  return k == 0 ? X : k > 62 ? 0 : ((X >> (k - 1)) + 1) >> 1;
}

// NSEG = 1: one product over any k. NSEG = 2: the sum of two products of one
// slab each, every one with its own exponents: with |d_1| <= 128 a level's
// sum stays below 32 x 114,688 < 2^22, so it converts by a float addition, a
// product is kept as one integer in units of 2^(e - 55) and the two are added
// as integers (one FP64 addition per entry of C is left, to C itself).
template <int NSEG>
GLA_DEV void gemm_body(const Args& g, int tile, int split) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], drain_full, drain_empty, fin_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_abort_raw;
  volatile int* s_abort = &s_abort_raw;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int ntn = (g.N + kBN - 1) / kBN;
  const int tm = tile / ntn, tn = tile % ntn;
  const int row0 = tm * kBM, col0 = tn * kBN;
  // (uniform, no TMEM touched yet) nothing to store
  if (row0 >= g.M || col0 >= g.N || (g.lower && row0 + kBM <= col0)) return;
  int kbeg = 0, kend = g.seg[0].nks;
  double* C = g.C;
  if (g.ksplit > 0) {
    kbeg = split * g.ksplit;
    kend = min(kend, kbeg + g.ksplit);
    C += (long long)split * g.split_stride;
  }
  const int n0 = kend - kbeg;                          // slabs of segment 0
  const int total = n0 + (NSEG == 2 ? g.seg[1].nks : 0);
  constexpr int spg = kGroupK / kKS;                   // slabs per drain group
  const int ngroups = NSEG == 2 ? 2 : (n0 + spg - 1) / spg;
  volatile int* err = g.err;
  if (tid == 0) {
    for (int i = 0; i < kStages; i++) {
      oz::mbar_init(&full_bar[i], 1);
      oz::mbar_init(&empty_bar[i], 1);
    }
    oz::mbar_init(&drain_full, 1);
    oz::mbar_init(&drain_empty, 32 * kDrainWarps);
    oz::mbar_init(&fin_bar, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz::smem_u32(&tmem_base)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;

  if (wid == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int q = 0; q < total && !*s_abort; q++) {
        const int st = q % kStages;
        if (q >= kStages && !oz::mbar_wait(&empty_bar[st], ((q / kStages) - 1) & 1, (volatile int*)err)) {
          *s_abort = 1;
          break;
        }
        issued = q + 1;
        const Seg& sg = g.seg[NSEG == 2 && q >= n0 ? 1 : 0];
        const int qs = q >= n0 ? q - n0 : kbeg + q;
        unsigned char* dst = sm + st * kStageBytes;
        oz::mbar_expect_tx(&full_bar[st], (uint32_t)kStageBytes);
        oz::bulk_g2s(dst, sg.A + ((size_t)tm * sg.a_nks + qs) * kAAll, kAAll, &full_bar[st]);
        const unsigned char* bs = sg.B + ((size_t)(tn >> 1) * sg.b_nks + qs) * kAAll + (tn & 1) * (kBB / 2);
#pragma unroll
        for (int j = 0; j < kS; j++)
          oz::bulk_g2s(dst + kAAll + j * (kBB / 2), bs + (size_t)j * kBB, kBB / 2, &full_bar[st]);
      }
      for (int q = (issued > kStages ? issued - kStages : 0); q < issued; q++)
        for (long long it = 0; it < oz::kWaitLimit && !oz::mbar_try(&full_bar[q % kStages], (q / kStages) & 1); it++) {
        }
    }
  } else if (wid == 1) {
    if (lane == 0) {
      int q = 0;
      for (int gi = 0; gi < ngroups && !*s_abort; gi++) {
        if (gi > 0 && !oz::mbar_wait(&drain_empty, (gi - 1) & 1, err)) {
          *s_abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const int qend = NSEG == 2 ? (gi == 0 ? n0 : total) : min(total, (gi + 1) * spg);
        bool first = true;
        for (; q < qend; q++) {
          const int st = q % kStages;
          if (!oz::mbar_wait(&full_bar[st], (q / kStages) & 1, err)) {
            *s_abort = 1;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint64_t a0 = oz::make_desc(oz::smem_u32(sm + st * kStageBytes));
          const uint64_t b0 = a0 + (uint64_t)(kAAll >> 4);
          // left slice s times right slices t0 .. t0 + cnt - 1 at once: their
          // row blocks and their levels' accumulators are adjacent
#pragma unroll
          for (int ks = 0; ks < kKS / 16; ks++)
#pragma unroll
            for (int s = 1; s <= kS; s++) {
              constexpr int kMaxT = 256 / kBN;
              const int tmax = kMaxLevel - s < kS ? kMaxLevel - s : kS;
#pragma unroll
              for (int t0 = 1; t0 <= kS; t0 += kMaxT) {
                const int nt = tmax - t0 + 1;
                if (nt <= 0) continue;
                // s = 1 starts levels 2 .. 8 from zero; level 9 starts with
                // the pair (2, 7), issued by itself
                const bool split = s == 2 && t0 + kMaxT > kS;
                const int cnt = (nt < kMaxT ? nt : kMaxT) - (split ? 1 : 0);
                const uint32_t accumulate = (first && ks == 0 && s == 1) ? 0u : 1u;
                if (split)
                  oz::mma_f16(tmem + (uint32_t)((s + kS - 2) * kBN),
                              a0 + (uint64_t)(((s - 1) * block_bytes(kBM) + ks * 256) >> 4),
                              b0 + (uint64_t)(((kS - 1) * block_bytes(kBN) + ks * 256) >> 4), idesc(kBN),
                              (first && ks == 0) ? 0u : 1u);
                oz::mma_f16(tmem + (uint32_t)((s + t0 - 2) * kBN),
                            a0 + (uint64_t)(((s - 1) * block_bytes(kBM) + ks * 256) >> 4),
                            b0 + (uint64_t)(((t0 - 1) * block_bytes(kBN) + ks * 256) >> 4), idesc(cnt * kBN),
                            accumulate);
              }
            }
          first = false;
          oz::mma_commit(&empty_bar[st]);
        }
        oz::mma_commit(&drain_full);
      }
    }
  } else {
    // drain warps: TMEM lanes 32 (wid % 4) .., columns cbase .. cbase + 15
    const int quarter = wid & 3;
    const int cbase = ((wid - 2) / 4) * 16;
    const int r = row0 + quarter * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)cbase;
    long long H[NSEG == 1 ? 16 : 1], L[NSEG == 1 ? 16 : 1];
    long long X[2][NSEG == 2 ? 16 : 1];
    if (NSEG == 1)
#pragma unroll
      for (int c = 0; c < 16; c++) H[c] = L[c] = 0;
    bool ok = true;
#pragma unroll (NSEG == 2 ? 2 : 1)
    for (int gi = 0; gi < (NSEG == 2 ? 2 : ngroups); gi++) {
      if (!ok) break;
      if (!oz::mbar_wait(&drain_full, gi & 1, err)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      if (NSEG == 1) {
#pragma unroll
        for (int lv = 2; lv <= kMaxLevel; lv++) {
          uint32_t v[16];
          oz::tmem_ld16(taddr + (uint32_t)((lv - 2) * kBN), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;");
          const int sh = lv <= 5 ? 8 * (5 - lv) : 8 * (9 - lv);
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const long long x = (long long)__float2int_rn(__uint_as_float(v[c])) * (1 << sh);
            if (lv <= 5) H[c] += x; else L[c] += x;
          }
        }
      } else {
#pragma unroll
        for (int c0 = 0; c0 < 16; c0 += 8) {
          long long h[8], l[8];
#pragma unroll
          for (int c = 0; c < 8; c++) h[c] = l[c] = 0;
#pragma unroll
          for (int lv = 2; lv <= kMaxLevel; lv++) {
            uint32_t v[8];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                           "=r"(v[7])
                         : "r"(taddr + (uint32_t)((lv - 2) * kBN + c0)));
            asm volatile("tcgen05.wait::ld.sync.aligned;");
            const int sh = lv <= 5 ? 8 * (5 - lv) : 8 * (9 - lv);
#pragma unroll
            for (int c = 0; c < 8; c++) {
              const int iv = __float_as_int(__uint_as_float(v[c]) + 12582912.f) - 0x4b400000;
              const long long x = (long long)iv * (1 << sh);
              if (lv <= 5) h[c] += x; else l[c] += x;
            }
          }
#pragma unroll
          for (int c = 0; c < 8; c++) {
            X[gi & 1][c0 + c] = (h[c] << 15) + ((l[c] + 65536) >> 17);  // units of 2^(e - 55), below 2^62
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      oz::mbar_arrive(&drain_empty);
    }
    // (the TMEM loads above are warp-wide: nothing diverges before this point;
    // after a wait that ran out the results are NaN)
    const bool lost = !ok || *err;
    if (r < g.M) {
      const int a0 = g.seg[0].ea[r], a1 = NSEG == 2 ? g.seg[1].ea[r] : 0;
#pragma unroll
      for (int c = 0; c < 16; c++) {
        const int col = col0 + cbase + c;
        if (col >= g.N || (g.lower && r < col)) continue;
        const int b0 = g.seg[0].eb[col];
        double x;
        bool bad;
        if (NSEG == 1) {
          // (a product without terms has no slices either: its exponents' words are an earlier one's)
          bad = total > 0 && max(a0, b0) == kBadExp;
          x = to_double(H[c], L[c], a0 + b0);
          x = g.neg ? -x : x;
        } else {
          const int b1 = g.seg[1].eb[col];
          bad = max(max(a0, b0), max(a1, b1)) == kBadExp;
          const int e0 = a0 + b0, e1 = a1 + b1, d = e0 - e1;
          const long long sum = shift_down(X[0][c], d < 0 ? -d : 0) + shift_down(X[1][c], d > 0 ? d : 0);
          x = to_double(g.neg ? -sum : sum, max(e0, e1) - 55);
        }
        if (bad || lost) x = __longlong_as_double(0x7ff8000000000000ll);
        double* p = C + r + (long long)(g.c_nidx ? g.c_nidx[col] : col) * g.ldc;
        *p = g.add ? *p + x : x;
      }
    }
  }
  // teardown: a final commit, waited for with a bound, before TMEM is freed
  __syncthreads();
  if (wid == 1 && lane == 0) {
    oz::mma_commit(&fin_bar);
    for (long long it = 0; it < oz::kWaitLimit && !oz::mbar_try(&fin_bar, 0); it++) {
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (wid == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

template <int NSEG>
__global__ void __launch_bounds__(kThreads, 1) k_gemm(const Args g) {
  gemm_body<NSEG>(g, blockIdx.x, blockIdx.y);
}

// Products that differ by a step per grid row y (blocks of the
// back-transformation): pointers, extents and slab counts move by y times
// these (N is also cut at ncols - 128 y).
struct Step {
  long long A, B, C;  // bytes, bytes, elements
  int ea, eb, nks, M, ncols;
};
__global__ void __launch_bounds__(kThreads, 1) k_gemm_steps(const Args g0, const Step s) {
  Args g = g0;
  const int y = blockIdx.y;
  g.seg[0].A += y * s.A;
  g.seg[0].B += y * s.B;
  g.seg[0].ea += (long long)y * s.ea;
  g.seg[0].eb += (long long)y * s.eb;
  g.seg[0].nks += y * s.nks;
  g.M += y * s.M;
  g.N = min(g.N, s.ncols - kBM * y);
  g.C += y * s.C;
  gemm_body<1>(g, blockIdx.x, 0);
}

// ---- problems whose sizes are known on the device only (the eigenvector
// updates of a divide-and-conquer level): descriptor p of the SIMT GEMM's
// list, operands at p times a stride that holds the level's largest.
struct Group {
  const GemmDesc* d;
  unsigned char *A, *B;
  int *ea, *eb;        // exponents; the row maxima lie a_rows / b_rows words per problem further
  unsigned *ma, *mb;
  size_t a_stride, b_stride;  // bytes per problem
  int a_rows, b_rows;  // words per problem (multiples of 128)
  int* err;
};
GLA_DEV Source group_a(const GemmDesc& d) {
  return Source{(const double*)d.A, d.lda, d.m, d.k, d.a_kidx};
}
GLA_DEV Source group_b(const GemmDesc& d) {
  return Source{(const double*)d.B, d.ldb, d.n, d.k, d.b_kidx};
}
__global__ void __launch_bounds__(256) k_group_max_a(const Group g) {
  const Source s = group_a(g.d[blockIdx.z]);
  max_rows_body(s, g.ma + (size_t)blockIdx.z * g.a_rows);
}
__global__ void __launch_bounds__(256) k_group_max_b(const Group g) {
  const Source s = group_b(g.d[blockIdx.y]);
  max_cols_body(s, g.b_rows, g.mb + (size_t)blockIdx.y * g.b_rows);
}
template <bool LEFT>
__global__ void __launch_bounds__(256) k_group_tile(const Group g) {
  extern __shared__ __align__(16) unsigned char tsm[];
  const int p = blockIdx.z;
  const Source s = LEFT ? group_a(g.d[p]) : group_b(g.d[p]);
  const int nks = (s.len + kKS - 1) / kKS;
  if ((int)blockIdx.x * kBM >= s.count || (int)blockIdx.y >= nks) return;
  Operand o;
  o.base = LEFT ? g.A + p * g.a_stride : g.B + p * g.b_stride;
  o.exps = LEFT ? g.ea + (size_t)p * g.a_rows : g.eb + (size_t)p * g.b_rows;
  o.mx = LEFT ? g.ma + (size_t)p * g.a_rows : g.mb + (size_t)p * g.b_rows;
  tile_body<LEFT>(s, o, blockIdx.x, blockIdx.y, nks, tsm);
}
__global__ void __launch_bounds__(kThreads, 1) k_group_gemm(const Group g) {
  const int p = blockIdx.y;
  const GemmDesc d = g.d[p];
  if (d.m <= 0 || d.n <= 0) return;
  Args a{};
  a.seg[0].A = g.A + p * g.a_stride;
  a.seg[0].B = g.B + p * g.b_stride;
  a.seg[0].ea = g.ea + (size_t)p * g.a_rows;
  a.seg[0].eb = g.eb + (size_t)p * g.b_rows;
  a.seg[0].nks = a.seg[0].a_nks = a.seg[0].b_nks = (d.k + kKS - 1) / kKS;
  a.M = d.m;
  a.N = d.n;
  a.C = (double*)d.C;
  a.ldc = d.ldc;
  a.c_nidx = d.c_nidx;
  a.err = g.err;
  gemm_body<1>(a, blockIdx.x, 0);
}

// ---- compact-WY factors of the blocks of 128 reflectors: T (upper triangular,
// leading dimension 128) from the Gram matrices G = Y'Y and tau, T(i, i) =
// tau_i, T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i). The recurrence runs inside
// diagonal blocks of 32, one CTA each, eight lanes per dot product; two blocks
// a, b of equal order join by T_ab = -T_aa G_ab T_bb, a few columns per CTA.
// An SM does one FP64 warp instruction in 16 cycles, so it is the number of
// SMs that counts: one CTA per block of 128 took 200 us.
constexpr int kLeafT = 32;
// grid: (diagonal block, block of 128)
__global__ void __launch_bounds__(256) k_larft_leaf(const double* __restrict__ Gall, const double* __restrict__ tau,
                                                    double* __restrict__ Tall, int nref) {
  __shared__ double G[kLeafT][kLeafT + 1], T[kLeafT][kLeafT + 1], tv[kLeafT];  // [column][row]
  const int o = blockIdx.x * kLeafT, b = blockIdx.y, tid = threadIdx.x;
  const size_t off = (size_t)b * kBM * kBM + o + (size_t)o * kBM;
  for (int i = tid; i < kLeafT * kLeafT; i += 256) {
    const int r = i % kLeafT, c = i / kLeafT;
    G[c][r] = Gall[off + r + c * kBM];
    T[c][r] = 0.0;
  }
  if (tid < kLeafT) tv[tid] = b * kBM + o + tid < nref ? tau[b * kBM + o + tid] : 0.0;
  __syncthreads();
  const int r = tid >> 3, part = tid & 7;
  for (int i = 0; i < kLeafT; i++) {
    double s = 0.0;
    for (int q = r + part; q < i; q += 8) s = fma(T[q][r], G[i][q], s);
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (part == 0) {
      if (r < i) T[i][r] = -tv[i] * s;
      if (r == i) T[i][r] = tv[i];
    }
    __syncthreads();
  }
  for (int i = tid; i < kLeafT * kLeafT; i += 256) {
    const int rr = i % kLeafT, c = i / kLeafT;
    Tall[off + rr + c * kBM] = T[c][rr];
  }
}

// grid: (slice of the columns, pair, block of 128); H: order of the blocks joined
template <int H>
__global__ void __launch_bounds__(256) k_larft_merge(const double* __restrict__ Gall, double* __restrict__ Tall) {
  constexpr int kC = 256 / H;  // columns per CTA, one entry per thread
  __shared__ double M[kC][H + 1];
  const int tid = threadIdx.x, r = tid % H, cc = tid / H, c = blockIdx.x * kC + cc;
  const size_t aa = (size_t)blockIdx.z * kBM * kBM + (size_t)blockIdx.y * 2 * H * (kBM + 1);
  const size_t ab = aa + (size_t)H * kBM, bb = ab + H;
  double s = 0.0;
#pragma unroll 16
  for (int q = 0; q < H; q++) s = fma(Gall[ab + r + q * kBM], Tall[bb + q + c * kBM], s);  // G_ab T_bb
  M[cc][r] = s;
  __syncthreads();
  s = 0.0;
#pragma unroll 16
  for (int q = 0; q < H; q++) s = fma(Tall[aa + r + q * kBM], M[cc][q], s);
  Tall[ab + r + c * kBM] = -s;
  Tall[aa + H + r + c * kBM] = 0.0;
}

}  // namespace oz64
}  // namespace gla
