// Double-float products of the batched refinement (n <= 128) on the tcgen05
// tensor cores, run by the whole CTA that refines the matrix (no counterpart
// in GenericLinearAlgebra.jl).
//
//   C = P Q,  P (n x n) and Q (n x n) read through accessors returning float
//   pairs, C handed to a store functor as float pairs,
//
// by the Ozaki scheme of the large path's GEMM (ozaki.cuh; K. Ozaki,
// T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012)): every row i
// of P is scaled by 2^e_i >= max_k |p_ik| and every column j of Q by
// 2^f_j >= max_k |q_kj|, each scaled value is split into seven 7-bit integer
// slices (exact in bf16), and the 28 slice pairs with s + t <= 8 are
// multiplied by tcgen05.mma kind::f16 (bf16 in, FP32 out) into seven "level"
// accumulators in TMEM, L = s + t, each an exact integer sum (K <= 128: at
// most 128 x 37,895 < 2^24, see ozaki.cuh). C_ij = 2^(e_i + f_j) sum_L
// level_L(i, j) 2^(-7 L), summed in double-float: ~2^-47 relative to
// max_k |p_ik| max_k |q_kj| per term, as the double-float SIMT products.
//
// Shape: M = 128 rows of C per MMA (rows >= n are zero slices), N = 32
// columns per pass (7 levels x 32 = 224 of the CTA's 256 TMEM columns; two
// CTAs per SM share the 512), K in slabs of 32. Per pass and slab the CTA
// slices P's 128 x 32 block and Q's 32 x 32 block into shared memory in the
// MMA's canonical no-swizzle K-major layout (oz_prims.cuh), one thread
// issues the MMAs (per K = 16 step one per slice of P, see idesc_n) and
// commits to an mbarrier, and the CTA loads the next slab's values into
// registers while they run; after the last slab the eight warps drain the
// levels with tcgen05.ld (warp w reads TMEM lanes 32 (w % 4) .. +31,
// columns 16 (w / 4) .. +15), combine them and call the store functor.
//
// gemm() slices P again in every pass. The persistent kernel, whose CTA has a
// global scratch for three operands, slices each operand once
// (slice_operand) and multiplies by gemm_sliced(): slabs of K = 16 of both
// operands come by two bulk copies into one of two stages, so that a slab
// lands while the MMAs of the one before run, and no warp touches the values. At order
// 128 the products of one iteration took 260 us in gemm() (two CTAs per SM):
// the slicing of 12 x 4 slabs, each waited for in turn.
//
// Every mbarrier wait is bounded: a wait that runs out sets the error word
// and the CTA's abort flag, no further MMA is issued by the CTA, and the
// caller sees `false` (the matrix is then reported as not converged).
// teardown() waits (bounded) for every bulk copy and MMA the CTA issued
// before it frees the TMEM.
#pragma once
#include "df64.cuh"
#include "oz_prims.cuh"

namespace gla {
namespace tcs {

constexpr int kS = 7;                       // slices per operand
constexpr int kM = 128;                     // MMA M (rows of C per pass)
constexpr int kNT = 32;                     // columns of C per pass
constexpr int kTmemCols = 256;              // per CTA (two CTAs per SM)
constexpr int kKS = oz::kKS;                // k per slab
constexpr int kABlk = kM * kKS * 2;         // one slice of a P slab: 8 KB
constexpr int kBBlk = kNT * kKS * 2;        // one slice of a Q slab: 2 KB
constexpr int kSmem = kS * (kABlk + kBBlk);  // 70 KB of dynamic shared memory
// kind::f16 instruction descriptor: F32 accumulate (bit 4), bf16 A and B
// (bits 7, 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24. One MMA
// per A slice s multiplies it by Q's slices 1 .. 8 - s at once: those are
// adjacent 32-row blocks in shared memory (one operand of N = 32 (8 - s)
// rows in the same canonical layout) and their levels s + 1 .. 8 are
// adjacent 32-column accumulators in TMEM.
GLA_DEV constexpr uint32_t idesc_n(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}
static_assert(kS * kNT <= kTmemCols, "level accumulators exceed the CTA's TMEM columns");
// Slices of the operands in the scratch, K-major rows in slabs of K = 16. As
// P: [slab][8-row group][slice][2 core matrices], so that a slab's first rows,
// those that the upper triangle's pass needs, are one bulk copy; A at slot 0 and X' at slot 1. As Q: the columns of [X | Y], the 8-column
// groups of Y after those of X, [slab][4 groups][slice][group][2 core
// matrices], so that a pass's part of a slab is one bulk copy; slots 2 and 3.
constexpr int kRG = 256;                                     // one 8-row group of one slice of a slab
constexpr int kOpBytes = (128 / 16) * kS * (128 / 8) * kRG;  // order 128: 224 KB
constexpr int kScratchOps = 4;
constexpr int kStageP = kS * (kM / 8) * kRG, kStageQ = kS * (kNT / 8) * kRG, kStage = kStageP + kStageQ;  // 35 KB
static_assert(2 * kStage <= kSmem, "two stages of gemm_sliced in the slabs of gemm");
static_assert(kM <= 128, "one row of C per TMEM lane");

// Per-CTA state in static shared memory.
struct Shared {
  uint64_t bar;  // MMA completion (one phase per commit)
  uint64_t fin;  // teardown: every MMA of the CTA finished
  uint64_t full[2];   // gemm_sliced: the stage's slab has landed
  uint64_t empty[2];  // gemm_sliced: the MMAs that read the stage are done
  uint32_t tmem;
  int abort;
};

struct Ctx {
  Shared* sh;
  unsigned char* slabs;  // kSmem bytes of dynamic shared memory, 16-byte aligned
  unsigned char* ops;    // kScratchOps kOpBytes of global scratch of this CTA, or null (gemm only)
  int* err;              // error word in global memory
  uint32_t phase;        // parity of the next completion of sh->bar
  // (thread 0) slabs asked for and slabs seen to land, over the CTA's life: slab
  // g is in stage g % 2 and completes that stage's phase g / 2
  uint32_t asked, landed;
};

// All threads of the CTA (256); TMEM is held until teardown().
GLA_DEV void setup(Ctx& c, Shared* sh, unsigned char* slabs, int* err, unsigned char* ops = nullptr) {
  c.sh = sh;
  c.slabs = slabs;
  c.ops = ops;
  c.err = err;
  c.phase = 0;
  c.asked = c.landed = 0;
  if (threadIdx.x == 0) {
    oz::mbar_init(&sh->bar, 1);
    oz::mbar_init(&sh->fin, 1);
    for (int s = 0; s < 2; s++) {
      oz::mbar_init(&sh->full[s], 1);
      oz::mbar_init(&sh->empty[s], 1);
    }
    sh->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz::smem_u32(&sh->tmem)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
}

// All threads of the CTA, once, before it exits.
GLA_DEV void teardown(Ctx& c) {
  __syncthreads();
  if (threadIdx.x == 0) {     // the thread that issued every MMA of this CTA
    for (uint32_t g = c.landed; g != c.asked; g++)  // (abort path) the last bulk loads land before the CTA exits
      for (long long it = 0; it < oz::kWaitLimit && !oz::mbar_try(&c.sh->full[g & 1], (g >> 1) & 1); it++) {
      }
    oz::mma_commit(&c.sh->fin);
    for (long long it = 0; it < oz::kWaitLimit && !oz::mbar_try(&c.sh->fin, 0); it++) {
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.sh->tmem), "r"(kTmemCols));
}

GLA_DEV bool ok(const Ctx& c) { return !c.sh->abort; }

// Wait for the next commit (all threads); false once the CTA has aborted.
GLA_DEV bool wait_mma(Ctx& c) {
  if (!c.sh->abort && !oz::mbar_wait(&c.sh->bar, c.phase, c.err)) c.sh->abort = 1;
  c.phase ^= 1;
  __syncthreads();
  return !c.sh->abort;
}

// 2^e = f g for |e| <= 252 (beyond that x f g is 0 or infinite all the same,
// for the normal x of these sums).
struct Pow2 {
  float f, g;
};
GLA_DEV Pow2 pow2_of(int e) {
  const int a = min(max(e, -126), 126), b = min(max(e - a, -126), 126);
  return Pow2{__int_as_float((a + 127) << 23), __int_as_float((b + 127) << 23)};
}
GLA_DEV float scale2(float x, Pow2 p) { return x * p.f * p.g; }

// Seven slices of the pair (v0, v1) / 2^e as bf16x2 words, as k_oz_tile:
// d = rint(128 v), then the remainder times 128, kept exactly in
// double-float. th - d is a multiple of ulp(th) and |tl| <= ulp(th) / 2, so
// the remainder's (hi, lo) comes from a fast two-sum.
GLA_DEV void slices7(df64 v0, df64 v1, int e, uint32_t (&w)[kS]) {
  const Pow2 p = pow2_of(-e);
  float h0 = scale2(v0.hi, p), l0 = scale2(v0.lo, p);
  float h1 = scale2(v1.hi, p), l1 = scale2(v1.lo, p);
#pragma unroll
  for (int s = 0; s < kS; s++) {
    const float t0 = h0 * 128.f, u0 = l0 * 128.f, t1 = h1 * 128.f, u1 = l1 * 128.f;
    const float d0 = rintf(t0), d1 = rintf(t1);
    quick_two_sum(t0 - d0, u0, h0, l0);
    quick_two_sum(t1 - d1, u1, h1, l1);
    // |d| <= 128: the bf16 is the float's upper half, exactly
    w[s] = __byte_perm(__float_as_uint(d0), __float_as_uint(d1), 0x7632);
  }
}
// The same stored at dst + s * stride.
GLA_DEV void slice7x2(df64 v0, df64 v1, int e, unsigned char* dst, int stride) {
  uint32_t w[kS];
  slices7(v0, v1, e, w);
#pragma unroll
  for (int s = 0; s < kS; s++) *reinterpret_cast<uint32_t*>(dst + s * stride) = w[s];
}

GLA_DEV int exp_of(float m) { return m > 0.f ? ilogbf(m) + 1 : 0; }

// Scale exponents of the columns of an n x n column-major array: out[j] =
// exp_of(max_k |hi(M(k, j))|), one warp per column, four columns and all
// their loads in flight per warp (all threads of the CTA; ends with a barrier). A row of P whose
// exponent is given this way (P = X', or P = A symmetric) needs no pass of
// its own.
GLA_DEV void col_exps(int n, const df64* __restrict__ M, int* out) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int j0 = wid * 4; j0 < n; j0 += nw * 4) {
    float x[4][4], m[4];  // (n <= 128: a column is four loads; those past an end repeat the last entry)
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        x[u][q] = M[(size_t)min(j0 + u, n - 1) * n + min(lane + 32 * q, n - 1)].hi;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      m[u] = fmaxf(fmaxf(fabsf(x[u][0]), fabsf(x[u][1])), fmaxf(fabsf(x[u][2]), fabsf(x[u][3])));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m[u] = fmaxf(m[u], __shfl_xor_sync(0xffffffffu, m[u], o));
      if (lane == 0 && j0 + u < n) out[j0 + u] = exp_of(m[u]);
    }
  }
  __syncthreads();
}

// Scale exponents of the rows of an n x n column-major array: out[i] =
// exp_of(max_j |hi(M(i, j))|), two threads per row, eight loads in flight
// (consecutive threads read consecutive rows of a column); all 256 threads of
// the CTA, ends with a barrier.
GLA_DEV void row_exps(int n, const df64* __restrict__ M, int* out) {
  __shared__ float other[kM];
  const int i = threadIdx.x & (kM - 1), ic = min(i, n - 1), h = threadIdx.x >> 7;
  float m = 0.f;
  for (int j0 = h * 8; j0 < n; j0 += 16) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; u++) x[u] = M[(size_t)min(j0 + u, n - 1) * n + ic].hi;
#pragma unroll
    for (int u = 0; u < 8; u++) m = fmaxf(m, fabsf(x[u]));
  }
  if (h == 1) other[i] = m;
  __syncthreads();
  if (h == 0 && i < n) out[i] = exp_of(fmaxf(m, other[i]));
  __syncthreads();
}

// Slab staging: a warp fills whole 8 x 8 core matrices (each lane one row
// and two consecutive k: 128 contiguous bytes per warp and slice, free of
// bank conflicts). P's 128 x 32 slab is 64 core matrices (8 per warp), Q's
// 32 x 32 slab 16 (2 per warp). The values are loaded into registers first
// (all loads of a slab in flight together) and sliced after.
constexpr int kPPairs = kM * kKS / 2 / 256;   // pairs per thread: 8
constexpr int kQPairs = kNT * kKS / 2 / 256;  // 2
struct SlabRegs {
  df64 p[kPPairs][2];
  df64 q[kQPairs][2];
};

// core matrix cm of a slab with rows/8 row groups: rows 8 (cm / 4) + lane / 4,
// k 8 (cm % 4) + 2 (lane % 4)
GLA_DEV int cm_row(int cm, int lane) { return ((cm >> 2) << 3) + (lane >> 2); }
GLA_DEV int cm_k(int cm, int lane) { return ((cm & 3) << 3) + ((lane & 3) << 1); }

// rows: the rows of P this pass needs (the rest are zero slices); nc: the
// columns of Q.
template <class LP, class LQ>
GLA_DEV void slab_load(SlabRegs& g, int n, int nc, int rows, int k0, int j0, const LP& lp, const LQ& lq) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const df64 zero = df_make(0.f, 0.f);
#pragma unroll
  for (int t = 0; t < kPPairs; t++) {
    const int cm = wid + 8 * t;
    const int r = cm_row(cm, lane), k = k0 + cm_k(cm, lane);
    g.p[t][0] = (r < rows && k < n) ? lp(r, k) : zero;
    g.p[t][1] = (r < rows && k + 1 < n) ? lp(r, k + 1) : zero;
  }
#pragma unroll
  for (int t = 0; t < kQPairs; t++) {
    const int cm = wid + 8 * t;
    const int j = j0 + cm_row(cm, lane), k = k0 + cm_k(cm, lane);
    g.q[t][0] = (j < nc && k < n) ? lq(k, j) : zero;
    g.q[t][1] = (j < nc && k + 1 < n) ? lq(k + 1, j) : zero;
  }
}

GLA_DEV void slab_slice(const SlabRegs& g, const Ctx& c, int nc, int rows, int j0, const int* ea, const int* eb) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* sa = c.slabs;
  unsigned char* sb = c.slabs + kS * kABlk;
#pragma unroll
  for (int t = 0; t < kPPairs; t++) {
    const int cm = wid + 8 * t;
    const int r = cm_row(cm, lane), kk = cm_k(cm, lane);
    unsigned char* dst = sa + oz::tile_off(r, kk);
    if (r < rows) {
      slice7x2(g.p[t][0], g.p[t][1], ea[r], dst, kABlk);
    } else {  // rows of the M = 128 operand not needed (or beyond n)
#pragma unroll
      for (int q = 0; q < kS; q++) *reinterpret_cast<uint32_t*>(dst + q * kABlk) = 0u;
    }
  }
#pragma unroll
  for (int t = 0; t < kQPairs; t++) {
    const int cm = wid + 8 * t;
    const int cc = cm_row(cm, lane), kk = cm_k(cm, lane);
    const int j = j0 + cc;
    unsigned char* dst = sb + oz::tile_off(cc, kk);
    if (j < nc) {
      slice7x2(g.q[t][0], g.q[t][1], eb[j], dst, kBBlk);
    } else {
#pragma unroll
      for (int q = 0; q < kS; q++) *reinterpret_cast<uint32_t*>(dst + q * kBBlk) = 0u;
    }
  }
}

// The sums of the levels of the columns c0 .. c0 + 7 of the pass, rows 32
// (w % 4) + lane of warp w: (hi, lo) in 2^(e_i + f_j). All levels are loaded
// before the first is used.
GLA_DEV void levels8(const Ctx& c, int c0, float (&ph)[8], float (&pl)[8]) {
  const uint32_t t = c.sh->tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (uint32_t)c0;
  uint32_t v[kS][8];
#pragma unroll
  for (int L = 0; L < kS; L++) oz::tmem_ld8(t + (uint32_t)(L * kNT), v[L]);
  asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
  for (int u = 0; u < 8; u++) {
    float h = __uint_as_float(v[kS - 1][u]) * 0x1p-56f, l = 0.f;
#pragma unroll
    for (int L = kS; L >= 2; L--) {
      float sh, se;
      two_sum(h, __uint_as_float(v[L - 2][u]) * __int_as_float((127 - 7 * L) << 23), sh, se);
      h = sh;
      l += se;
    }
    two_sum(h, l, ph[u], pl[u]);
  }
}

// C = P Q for n <= 128 (all 256 threads of the CTA). ea[i] / eb[j]: scale
// exponents of row i of P and column j of Q (shared memory, i, j < n; any
// e with 2^e >= the row's or column's largest |hi| is exact, the smallest
// such is the most accurate). upper: only i <= j is stored. Returns false
// when the CTA has aborted (C is then incomplete).
template <class LP, class LQ, class ST>
GLA_DEV bool gemm(Ctx& c, int n, int nc, const int* ea, const int* eb, const LP& lp, const LQ& lq, const ST& store,
                  bool upper) {
  const int tid = threadIdx.x;
  if (c.sh->abort) return false;
  const int nks = (n + kKS - 1) / kKS;
  SlabRegs g;
  for (int j0 = 0; j0 < nc; j0 += kNT) {
    // P rows sliced: all; or (upper) the stored i <= j < j0 + 32
    const int rows = upper ? min(n, j0 + kNT) : n;
    slab_load(g, n, nc, rows, 0, j0, lp, lq);
    for (int q = 0; q < nks; q++) {
      // the MMAs of the previous slab read the buffers: wait for them
      if (q > 0 && !wait_mma(c)) return false;
      slab_slice(g, c, nc, rows, j0, ea, eb);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint64_t a0 = oz::make_desc(oz::smem_u32(c.slabs));
        const uint64_t b0 = oz::make_desc(oz::smem_u32(c.slabs + kS * kABlk));
#pragma unroll
        for (int ks = 0; ks < kKS / 16; ks++)
#pragma unroll
          for (int s = 1; s <= kS; s++) {
            // slice s of P times slices 1 .. 8 - s of Q into levels s + 1 .. 8;
            // s = 1 reaches every level first, so its MMA of the pass's first
            // k step starts the accumulators from zero
            const uint32_t acc = (q == 0 && ks == 0 && s == 1) ? 0u : 1u;
            oz::mma_f16(c.sh->tmem + (uint32_t)((s - 1) * kNT), a0 + (uint64_t)(((s - 1) * kABlk + ks * 256) >> 4),
                        b0 + (uint64_t)((ks * 256) >> 4), idesc_n(kNT * (kS + 1 - s)), acc);
          }
        oz::mma_commit(&c.sh->bar);
      }
      // the next slab's loads overlap these MMAs
      if (q + 1 < nks) slab_load(g, n, nc, rows, (q + 1) * kKS, j0, lp, lq);
    }
    if (!wait_mma(c)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;");
    const int wid = tid >> 5, r = (wid & 3) * 32 + (tid & 31);
    if ((wid & 3) * 32 < n) {
      const int er = ea[min(r, n - 1)];
#pragma unroll 1
      for (int c0 = (wid >> 2) * 16; c0 < (wid >> 2) * 16 + 16; c0 += 8) {
        float ph[8], pl[8];
        levels8(c, c0, ph, pl);
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int j = j0 + c0 + u;
          if (r >= n || j >= nc || (upper && r > j)) continue;
          const Pow2 p = pow2_of(er + eb[j]);
          store(r, j, df_make(scale2(ph[u], p), scale2(pl[u], p)));
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();  // the accumulators are free for the next pass
  }
  return true;
}

// C = P Q with Q square (nc = n).
template <class LP, class LQ, class ST>
GLA_DEV bool gemm(Ctx& c, int n, const int* ea, const int* eb, const LP& lp, const LQ& lq, const ST& store,
                  bool upper) {
  return gemm(c, n, n, ea, eb, lp, lq, store, upper);
}

// The slices of the order-n operand whose row r (of P; or column of Q) is
// column r of M, each scaled by ex[r] (shared memory): as P into slot opP
// unless negative, as Q from column group vq on unless negative. A warp takes
// core matrices, four at a time, 128 contiguous bytes per slice. All threads;
// one copy of the code for every operand.
static __device__ __noinline__ void slice_operand(unsigned char* ops, int opP, int vq, int n, const df64* M, const int* ex) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nrg = (n + 7) >> 3, nkc = 2 * ((n + 15) >> 4), per = (nkc + 3) >> 2, nblk = (2 * nrg + 3) >> 2;
  df64 nx[4][2];
  int ne = 0;
  auto fetch = [&](int it) {  // the values of work item it, on their way while the one before is sliced
    const int rg = it / per, kc0 = (it - rg * per) * 4, r = min(rg * 8 + (lane >> 2), n - 1);
    const df64* col = M + (size_t)r * n;
    ne = ex[r];
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
      for (int q = 0; q < 2; q++) nx[t][q] = col[min(8 * (kc0 + t) + 2 * (lane & 3) + q, n - 1)];
  };
  if (wid < nrg * per) fetch(wid);
#pragma unroll 1
  for (int it = wid; it < nrg * per; it += 8) {
    const int rg = it / per, kc0 = (it - rg * per) * 4, e = ne, v = vq + rg;
    df64 x[4][2];
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const bool in = 8 * (kc0 + t) + 2 * (lane & 3) + q < n;
        x[t][q].hi = in ? nx[t][q].hi : 0.f;
        x[t][q].lo = in ? nx[t][q].lo : 0.f;
      }
    if (it + 8 < nrg * per) fetch(it + 8);
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int kc = kc0 + t, ks = kc >> 1, in = (kc & 1) * 128 + lane * 4;
      if (kc >= nkc) break;
      unsigned char* dp = ops + (size_t)opP * kOpBytes + (size_t)(ks * nrg + rg) * (kS * kRG) + in;
      unsigned char* dq =
          ops + (size_t)2 * kOpBytes + (size_t)(ks * nblk + (v >> 2)) * kStageQ + (v & 3) * kRG + in;
      uint32_t w[kS];
      slices7(x[t][0], x[t][1], e, w);
      if (opP >= 0)
#pragma unroll
        for (int s = 0; s < kS; s++) *reinterpret_cast<uint32_t*>(dp + s * kRG) = w[s];
      if (vq >= 0)
#pragma unroll
        for (int s = 0; s < kS; s++) *reinterpret_cast<uint32_t*>(dq + s * (kNT / 8) * kRG) = w[s];
    }
  }
}

// Descriptor of a K = 16 slab: row groups sbo bytes apart.
GLA_DEV uint64_t desc_k16(uint32_t saddr, int sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(128u >> 4) << 16 | (uint64_t)((uint32_t)sbo >> 4) << 32 |
         (uint64_t)1 << 46;
}

// From the slices in the scratch, with P in slot opP and its exponents ea:
//   nq = 1: D1 = P X;   nq = 2 (P = X'): D0 = I - P X and D1 = P Y, entries
//   (i, j), i <= j, only.
// ex, ey: the exponents of X's and Y's columns. Four column groups of 8 per
// pass. What P's stage holds beyond its rows reaches only TMEM lanes that no
// one reads, and the column groups past the last only columns that no one
// reads. Returns false when the CTA has aborted (D is then incomplete).
static __device__ __noinline__ bool gemm_sliced(Ctx& c, int n, int nq, int opP, const int* ea, const int* ex, const int* ey,
                                         df64* D0, df64* D1) {
  const int tid = threadIdx.x, wid = tid >> 5;
  if (c.sh->abort) return false;
  const int nrg = (n + 7) >> 3, nks = (n + 15) >> 4, nv = nq * nrg, nblk = (2 * nrg + 3) >> 2;
  const unsigned char* srcP = c.ops + (size_t)opP * kOpBytes;
  const unsigned char* srcQ = c.ops + (size_t)2 * kOpBytes;
  // the slices, and what else was in the stages, before the copies' proxy
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  // (thread 0) the next slab of this call: pass av, slab ak
  int av = 0, ak = 0;
  auto ask_next = [&]() {
    if (4 * av >= nv) return true;
    const uint32_t g = c.asked;
    if (g >= 2 && !oz::mbar_wait(&c.sh->empty[g & 1], ((g >> 1) - 1) & 1, c.err)) return false;
    // the row groups that the pass's columns need (upper: up to the last column)
    const int v1 = min(4 * av + 4, nv);
    const int rows = nq == 1 || (4 * av < nrg && v1 > nrg) ? nrg : v1 <= nrg ? v1 : v1 - nrg;
    unsigned char* st = c.slabs + (g & 1) * kStage;
    oz::mbar_expect_tx(&c.sh->full[g & 1], (uint32_t)(rows * kS * kRG + kStageQ));
    oz::bulk_g2s(st, srcP + (size_t)ak * (kS * nrg * kRG), (uint32_t)(rows * kS * kRG), &c.sh->full[g & 1]);
    oz::bulk_g2s(st + kStageP, srcQ + (size_t)(ak * nblk + av) * kStageQ, (uint32_t)kStageQ, &c.sh->full[g & 1]);
    c.asked = g + 1;
    if (++ak == nks) {
      ak = 0;
      av++;
    }
    return true;
  };
  bool ok = true;
  if (tid == 0) ok = ask_next();
  for (int v0 = 0; v0 < nv; v0 += 4) {
    if (tid == 0) {
#pragma unroll 1
      for (int ks = 0; ks < nks && ok; ks++) {
        ok = ask_next();
        const uint32_t g = c.landed;
        ok = ok && oz::mbar_wait(&c.sh->full[g & 1], (g >> 1) & 1, c.err);
        if (!ok) break;
        c.landed = g + 1;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t st = oz::smem_u32(c.slabs + (g & 1) * kStage);
        const uint64_t a0 = desc_k16(st, kS * kRG), b0 = desc_k16(st + kStageP, kRG);
#pragma unroll
        for (int s = 1; s <= kS; s++)  // (see gemm)
          oz::mma_f16(c.sh->tmem + (uint32_t)((s - 1) * kNT), a0 + (uint64_t)(((s - 1) * kRG) >> 4), b0,
                      idesc_n(kNT * (kS + 1 - s)), (ks == 0 && s == 1) ? 0u : 1u);
        oz::mma_commit(&c.sh->empty[g & 1]);
        if (ks + 1 == nks) oz::mma_commit(&c.sh->bar);
      }
      if (!ok) c.sh->abort = 1;  // (the error word is set: the other warps' wait ends)
    }
    if (wid == 0) __syncwarp();
    if (!wait_mma(c)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;");
    const int r = (wid & 3) * 32 + (tid & 31);
#pragma unroll 1
    for (int h = 2 * (wid >> 2); h < 2 * (wid >> 2) + 2; h++) {
      const int v = v0 + h;
      const bool y = v >= nrg;                    // (uniform: a group of 8 columns lies in X or in Y)
      const int j0 = (y ? v - nrg : v) * 8;
      if (v >= nv || (wid & 3) * 32 >= n || (nq == 2 && (wid & 3) * 32 > j0 + 7)) continue;
      float ph[8], pl[8];
      levels8(c, 8 * h, ph, pl);
      const int er = ea[min(r, n - 1)];
      const int* eb = y ? ey : ex;
      df64* D = nq == 2 && !y ? D0 : D1;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int j = j0 + u;
        if (r >= n || j >= n || (nq == 2 && r > j)) continue;
        const Pow2 p = pow2_of(er + eb[j]);
        df64 x = df_make(scale2(ph[u], p), scale2(pl[u], p));
        if (nq == 2 && !y) x = df_add(df_make(r == j ? 1.f : 0.f, 0.f), df_neg(x));
        D[(size_t)j * n + r] = x;
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();  // the accumulators are free for the next pass
  }
  return true;
}

}  // namespace tcs
}  // namespace gla
