// Host side of the FP64-accurate tensor-core GEMM (ozaki64.cuh) and the three
// stages of the FP64 large-matrix path that run on it: the trailing update of
// the reduction, the eigenvector updates of divide and conquer, and the
// back-transformation.
#include <algorithm>
#include <mutex>
#include <new>

#include "gla_large.h"
#include "gla_status.h"
#include "ozaki64.cuh"

namespace gla {

struct Oz64 {
  int n = 0, nb = 0, nks = 0, splits = 1;
  int* err = nullptr;              // set when a bounded wait ran out (owned by the context)
  unsigned char* arena = nullptr;  // sliced operands, shared by the stages (they run one after another)
  size_t arena_bytes = 0;
  int* words = nullptr;            // exponents and row maxima, shared likewise
  size_t nwords = 0;
  double* G = nullptr;             // Gram matrices and T factors of the back-transformation's blocks
  double* T = nullptr;
  double* Wp = nullptr;            // split-K partials of Y'Z
  // divide and conquer: shapes of the largest level
  int dc_min = 0;
};

namespace {
using namespace oz64;

constexpr long long kSlab = (long long)kS * kBB;  // one row block's slab: 56 KB

int blocks(int rows) { return (rows + kBM - 1) / kBM; }
int slabs(int len) { return (len + kKS - 1) / kKS; }
int tiles(int M, int N) { return blocks(M) * ((N + kBN - 1) / kBN); }

cudaError_t set_attributes() {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    auto set = [](const void* f, size_t bytes) {
      if (attr == cudaSuccess) attr = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    set((const void*)k_gemm<1>, kSmem);
    set((const void*)k_gemm<2>, kSmem);
    set((const void*)k_gemm_steps, kSmem);
    set((const void*)k_group_gemm, kSmem);
    set((const void*)k_tile<false>, kSlab);
    set((const void*)k_tile<true>, kSlab);
    set((const void*)k_group_tile<false>, kSlab);
    set((const void*)k_group_tile<true>, kSlab);
    set((const void*)k_slice_vw, kSlab);
    set((const void*)k_slice_blockcol, kSlab);
    set((const void*)k_slice_w, kSlab);
  });
  return attr;
}
}  // namespace

namespace {
// Strides of a divide-and-conquer level of `nprob` products of up to m1max
// rows, mmax columns and mmax k.
struct GroupShape {
  size_t a_stride, b_stride, bytes, words;
  int a_rows, b_rows;
};
GroupShape group_shape(int nprob, int m1max, int mmax) {
  GroupShape s;
  s.a_rows = blocks(m1max) * kBM;
  s.b_rows = blocks(mmax) * kBM;
  s.a_stride = (size_t)blocks(m1max) * slabs(mmax) * kSlab;
  s.b_stride = (size_t)blocks(mmax) * slabs(mmax) * kSlab;
  s.bytes = nprob * (s.a_stride + s.b_stride);
  s.words = 2 * (size_t)nprob * (s.a_rows + s.b_rows);
  return s;
}
}  // namespace

int oz64_create(Oz64** out, int n, int* err) {
  *out = nullptr;
  Oz64* w = new (std::nothrow) Oz64();
  if (!w) return -1000 - (int)cudaErrorMemoryAllocation;
  w->n = n;
  w->err = err;
  const int nb = w->nb = blocks(n), nks = w->nks = slabs(n);
  const size_t nbp = (size_t)nb * kBM;
  // back-transformation: Y by columns, V by block columns, Z, W, T
  w->arena_bytes = kSlab * ((size_t)nb * nks + (size_t)nb * nb * 4 + (size_t)nb * nks + 2 * (size_t)nb * 4);
  w->nwords = 2 * nbp + (size_t)nb * nbp + 2 * nbp + nbp + 2 * nbp;
  // divide and conquer: every level of the balanced tree with merges of 256 or more
  for (int d = 0; ; d++) {
    const int m = (n + (1 << d) - 1) >> d;
    if (m < kOz64MinMerge) break;
    const GroupShape g = group_shape(2 << d, (m + 1) / 2, m);
    w->arena_bytes = std::max(w->arena_bytes, g.bytes);
    w->nwords = std::max(w->nwords, g.words);
  }
  w->splits = std::max(1, std::min(8, 152 / std::max(1, (n + kBN - 1) / kBN)));
  const int nblk = std::max(1, blocks(n - 1));
  cudaError_t e = cudaMalloc((void**)&w->arena, w->arena_bytes);
  if (e == cudaSuccess) e = cudaMalloc((void**)&w->words, sizeof(int) * w->nwords);
  if (e == cudaSuccess) e = cudaMalloc((void**)&w->G, sizeof(double) * nblk * kBM * kBM);
  if (e == cudaSuccess) e = cudaMalloc((void**)&w->T, sizeof(double) * nblk * kBM * kBM);
  if (e == cudaSuccess) e = cudaMalloc((void**)&w->Wp, sizeof(double) * w->splits * kBM * nbp);
  if (e == cudaSuccess) e = set_attributes();
  if (e != cudaSuccess) {
    oz64_destroy(w);
    return cuda_status(e);
  }
  *out = w;
  return 0;
}

void oz64_destroy(Oz64* w) {
  if (!w) return;
  cudaFree(w->arena);
  cudaFree(w->words);
  cudaFree(w->G);
  cudaFree(w->T);
  cudaFree(w->Wp);
  delete w;
}

size_t oz64_bytes(const Oz64* w) {
  return w->arena_bytes + 4 * w->nwords + sizeof(double) * (2 * (size_t)w->nb + (size_t)w->splits * w->nb) * kBM * kBM;
}

// A[t:, t:] -= V W' + W V' (lower triangle): two segments of one slab each.
cudaError_t oz64_rank2k(Oz64* w, const double* VW, int nbp, int t, double* A, long long lda, cudaStream_t st) {
  const int n = w->n, m = n - t, nb = blocks(m);
  VwArgs a;
  a.VW = VW;
  a.ld = n;
  a.t = t;
  a.m = m;
  a.nbp = nbp;
  for (int k = 0; k < 2; k++) {
    a.op[k].base = w->arena + (size_t)k * nb * kSlab;
    a.op[k].exps = w->words + (size_t)k * nb * kBM;
    a.op[k].mx = nullptr;
  }
  k_slice_vw<<<dim3(nb, 2), 256, kSlab, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  Args g{};
  for (int k = 0; k < 2; k++) {
    g.seg[k].A = a.op[k].base;
    g.seg[k].ea = a.op[k].exps;
    g.seg[k].B = a.op[1 - k].base;
    g.seg[k].eb = a.op[1 - k].exps;
    g.seg[k].nks = g.seg[k].a_nks = g.seg[k].b_nks = 1;
  }
  g.M = g.N = m;
  g.C = A + t + (long long)t * lda;
  g.ldc = lda;
  g.neg = g.add = g.lower = 1;
  g.err = w->err;
  k_gemm<2><<<tiles(m, m), kThreads, kSmem, st>>>(g);
  return cudaGetLastError();
}


// The eigenvector updates of one divide-and-conquer level: descriptors
// d[0 .. nprob) on the device, products of at most m1max x mmax with k <= mmax.
cudaError_t oz64_grouped(Oz64* w, const GemmDesc* d, int nprob, int m1max, int mmax, cudaStream_t st) {
  const GroupShape s = group_shape(nprob, m1max, mmax);
  if (s.bytes > w->arena_bytes || s.words > w->nwords) return cudaErrorInvalidValue;
  Group g;
  g.d = d;
  g.A = w->arena;
  g.B = w->arena + nprob * s.a_stride;
  g.a_stride = s.a_stride;
  g.b_stride = s.b_stride;
  g.a_rows = s.a_rows;
  g.b_rows = s.b_rows;
  int* p = w->words;
  g.ma = (unsigned*)p;
  p += (size_t)nprob * s.a_rows;
  g.mb = (unsigned*)p;
  p += (size_t)nprob * s.b_rows;
  g.ea = p;
  p += (size_t)nprob * s.a_rows;
  g.eb = p;
  g.err = w->err;
  cudaError_t e = cudaMemsetAsync(g.ma, 0, sizeof(int) * nprob * s.a_rows, st);
  if (e != cudaSuccess) return e;
  k_group_max_a<<<dim3((m1max + 255) / 256, (mmax + 63) / 64, nprob), 256, 0, st>>>(g);
  k_group_max_b<<<dim3((s.b_rows + 7) / 8, nprob), 256, 0, st>>>(g);
  k_group_tile<true><<<dim3(blocks(m1max), slabs(mmax), nprob), 256, kSlab, st>>>(g);
  k_group_tile<false><<<dim3(blocks(mmax), slabs(mmax), nprob), 256, kSlab, st>>>(g);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_group_gemm<<<dim3(tiles(m1max, mmax), nprob), kThreads, kSmem, st>>>(g);
  return cudaGetLastError();
}

// Z := Q Z, Q = B_0 B_1 ..., B_b = I - Y_b T_b Y_b' with 128 reflectors a
// block. Y: the reflectors as columns with their unit elements and zeros above
// (n x n; overwritten), tau their scalars. With V_b = Y_b T_b formed once, a
// block is W = Y_b' Z, Z -= V_b W. Block b touches rows 128 b .. only, and its
// operands start on a slab there.
cudaError_t oz64_backtr(Oz64* w, double* Y, const double* tau, double* Z, long long ldz, cudaStream_t st) {
  const int n = w->n, nb = w->nb, nks = w->nks, nref = n - 1, nblk = blocks(nref);
  const size_t nbp = (size_t)nb * kBM;
  unsigned char* p = w->arena;
  auto take = [&](size_t nslab) {
    unsigned char* q = p;
    p += nslab * kSlab;
    return q;
  };
  int* wd = w->words;
  auto words = [&](size_t k) {
    int* q = wd;
    wd += k;
    return q;
  };
  Operand yc{take((size_t)nb * nks), words(nbp), (unsigned*)words(nbp)};
  Operand zs{take((size_t)nb * nks), words(nbp), (unsigned*)words(nbp)};
  Operand ws{take((size_t)nb * 4), words(nbp), nullptr};
  Operand ts{take((size_t)nb * 4), words(nbp), (unsigned*)words(nbp)};
  unsigned char* vr = take((size_t)nb * nb * 4);
  int* vexp = words((size_t)nb * nbp);
  cudaError_t e;
  // Y by columns; G_b = Y_b' Y_b; T_b
  Source sy{Y, n, n, n, nullptr};
  k_max_cols<<<(int)((nbp + 7) / 8), 256, 0, st>>>(sy, (int)nbp, yc.mx);
  k_tile<false><<<dim3(nb, nks), 256, kSlab, st>>>(sy, yc);
  Args g{};
  g.seg[0] = Seg{yc.base, yc.base, yc.exps, yc.exps, nks, nks, nks};
  g.M = g.N = kBM;
  g.C = w->G;
  g.ldc = kBM;
  g.err = w->err;
  Step sg{};
  sg.A = sg.B = (long long)(nks + 4) * kSlab;
  sg.C = kBM * kBM;
  sg.ea = sg.eb = kBM;
  sg.nks = -4;
  sg.ncols = 1 << 30;
  k_gemm_steps<<<dim3(2, nblk), kThreads, kSmem, st>>>(g, sg);
  k_larft_leaf<<<dim3(kBM / kLeafT, nblk), 256, 0, st>>>(w->G, tau, w->T, nref);
  k_larft_merge<32><<<dim3(4, 2, nblk), 256, 0, st>>>(w->G, w->T);
  k_larft_merge<64><<<dim3(16, 1, nblk), 256, 0, st>>>(w->G, w->T);
  // V_b = Y_b T_b over Y, then V by block columns
  k_slice_blockcol<<<dim3(nb, nblk), 256, kSlab, st>>>(Y, n, n, (int)nbp, vr, vexp);
  const int trows = nblk * kBM;  // the T factors' columns, one after another
  Source sT{w->T, kBM, trows, kBM, nullptr};
  k_max_cols<<<(trows + 7) / 8, 256, 0, st>>>(sT, trows, ts.mx);
  k_tile<false><<<dim3(nblk, 4), 256, kSlab, st>>>(sT, ts);
  Args gv{};
  gv.seg[0] = Seg{vr, ts.base, vexp, ts.exps, 4, 4, 4};
  gv.M = n;
  gv.N = kBM;
  gv.C = Y;
  gv.ldc = n;
  gv.err = w->err;
  Step sv{};
  sv.A = (long long)(nb + 1) * 4 * kSlab;
  sv.B = (long long)4 * kSlab;
  sv.C = (long long)kBM * (n + 1);
  sv.ea = (int)nbp + kBM;
  sv.eb = kBM;
  sv.M = -kBM;
  sv.ncols = n;
  k_gemm_steps<<<dim3(2 * nb, nblk), kThreads, kSmem, st>>>(gv, sv);
  k_slice_blockcol<<<dim3(nb, nblk), 256, kSlab, st>>>(Y, n, n, (int)nbp, vr, vexp);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  for (int b = nblk - 1; b >= 0; b--) {
    const int r0 = b * kBM, len = n - r0, ks = slabs(len);
    Source sz{Z + r0, ldz, n, len, nullptr};
    k_max_cols<<<nb * kBM / 8, 256, 0, st>>>(sz, nb * kBM, zs.mx);
    k_tile<false><<<dim3(nb, ks), 256, kSlab, st>>>(sz, zs);
    int per = ks, splits = 1;
    if (w->splits > 1) {  // at least eight slabs a split
      splits = std::max(1, std::min(w->splits, ks / 8));
      per = (ks + splits - 1) / splits;
      splits = (ks + per - 1) / per;
    }
    Args h{};
    h.seg[0] = Seg{yc.base + ((size_t)b * nks + 4 * b) * kSlab, zs.base, yc.exps + r0, zs.exps, ks, nks, ks};
    h.M = kBM;
    h.N = n;
    h.C = w->Wp;
    h.ldc = kBM;
    h.ksplit = splits > 1 ? per : 0;
    h.split_stride = (long long)kBM * (long long)nbp;
    h.err = w->err;
    k_gemm<1><<<dim3(tiles(kBM, n), splits), kThreads, kSmem, st>>>(h);
    k_slice_w<<<dim3(nb, 4), 256, kSlab, st>>>(w->Wp, splits, h.split_stride, n, ws);
    Args u{};
    u.seg[0] = Seg{vr + ((size_t)b * nb + b) * 4 * kSlab, ws.base, vexp + (size_t)b * nbp + r0, ws.exps, 4, 4, 4};
    u.M = len;
    u.N = n;
    u.C = Z + r0;
    u.ldc = ldz;
    u.neg = u.add = 1;
    u.err = w->err;
    k_gemm<1><<<tiles(len, n), kThreads, kSmem, st>>>(u);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// ---- a single product of any shape, with operand buffers that grow
struct Oz64Gemm {
  unsigned char* buf = nullptr;
  int* words = nullptr;
  size_t bytes = 0, nwords = 0;
  int* err = nullptr;
};

namespace {
template <class P>
cudaError_t grow(P** p, size_t* cap, size_t need, size_t unit) {
  if (*cap >= need) return cudaSuccess;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMalloc((void**)p, unit * need);
  if (e == cudaSuccess) *cap = need;
  return e;
}
}  // namespace

void oz64_gemm_release(Oz64Gemm** w) {
  if (!*w) return;
  cudaFree((*w)->buf);
  cudaFree((*w)->words);
  cudaFree((*w)->err);
  delete *w;
  *w = nullptr;
}

int oz64_gemm_status(Oz64Gemm* w, cudaStream_t st) {
  int word = 0;
  cudaError_t e = cudaSuccess;
  if (w) e = cudaMemcpyAsync(&word, w->err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && word) {
    e = cudaMemsetAsync(w->err, 0, sizeof(int), st);
    if (e == cudaSuccess) e = cudaErrorLaunchTimeout;
  }
  return e == cudaSuccess ? 0 : cuda_status(e);
}

cudaError_t oz64_gemm_mark(Oz64Gemm* w) {
  const int word = 1;
  return cudaMemcpy(w->err, &word, sizeof(int), cudaMemcpyHostToDevice);
}

cudaError_t oz64_gemm(Oz64Gemm** wp, bool ta, int m, int n, int k, const double* A, long long lda, const double* B,
                      long long ldb, double* C, long long ldc, bool add, cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  if (m < kOz64MinGemm || n < kOz64MinGemm || k < kOz64MinGemm) {
    GemmDesc g{};
    g.m = m;
    g.n = n;
    g.k = k;
    g.A = A;
    g.lda = lda;
    g.B = B;
    g.ldb = ldb;
    g.C = C;
    g.ldc = ldc;
    g.alpha = 1.0;
    g.beta = add ? 1.0 : 0.0;
    return gemm_launch(true, ta, false, false, g, 1, st);
  }
  cudaError_t e;
  if (!*wp) {
    Oz64Gemm* w = new (std::nothrow) Oz64Gemm();
    if (!w) return cudaErrorMemoryAllocation;
    e = cudaMalloc((void**)&w->err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(w->err, 0, sizeof(int));
    if (e == cudaSuccess) e = set_attributes();
    if (e != cudaSuccess) {
      oz64_gemm_release(&w);
      return e;
    }
    *wp = w;
  }
  Oz64Gemm* w = *wp;
  const int ba = blocks(m), bb = blocks(n), ks = slabs(k);
  if ((e = grow(&w->buf, &w->bytes, (size_t)(ba + bb) * ks * kSlab, 1)) != cudaSuccess) return e;
  if ((e = grow(&w->words, &w->nwords, 2 * (size_t)(ba + bb) * kBM, sizeof(int))) != cudaSuccess) return e;
  Operand a{w->buf, w->words, (unsigned*)(w->words + ba * kBM)};
  Operand b{w->buf + (size_t)ba * ks * kSlab, w->words + 2 * ba * kBM, (unsigned*)(w->words + (2 * ba + bb) * kBM)};
  Source sa{A, lda, m, k, nullptr}, sb{B, ldb, n, k, nullptr};
  if (ta) {
    k_max_cols<<<ba * kBM / 8, 256, 0, st>>>(sa, ba * kBM, a.mx);
    k_tile<false><<<dim3(ba, ks), 256, kSlab, st>>>(sa, a);
  } else {
    if ((e = cudaMemsetAsync(a.mx, 0, sizeof(unsigned) * ba * kBM, st)) != cudaSuccess) return e;
    k_max_rows<<<dim3((m + 255) / 256, (k + 63) / 64), 256, 0, st>>>(sa, a.mx);
    k_tile<true><<<dim3(ba, ks), 256, kSlab, st>>>(sa, a);
  }
  k_max_cols<<<bb * kBM / 8, 256, 0, st>>>(sb, bb * kBM, b.mx);
  k_tile<false><<<dim3(bb, ks), 256, kSlab, st>>>(sb, b);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  Args g{};
  g.seg[0] = Seg{a.base, b.base, a.exps, b.exps, ks, ks, ks};
  g.M = m;
  g.N = n;
  g.C = C;
  g.ldc = ldc;
  g.add = add ? 1 : 0;
  g.err = w->err;
  k_gemm<1><<<tiles(m, n), kThreads, kSmem, st>>>(g);
  return cudaGetLastError();
}

}  // namespace gla
