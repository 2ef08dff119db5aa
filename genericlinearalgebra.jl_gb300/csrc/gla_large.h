// Internal interface of the large-matrix (n > 128) path: blocked
// tridiagonalisation, divide-and-conquer tridiagonal eigensolver,
// back-transformation and the drivers that chain them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm_simt.cuh"

struct gla_plan_s;

namespace gla {

constexpr int kLargeMaxN = 16384;
constexpr int kSytrdNB = 32;    // panel width of the tridiagonalisation
constexpr int kBacktrNB = 64;   // reflectors per compact-WY block of the back-transformation

// ---- GEMM launchers (gemm_simt.cuh). With splits > 1, g.ksplit and
// g.split_stride describe the split-K partial outputs written to g.C.
cudaError_t gemm_launch(bool f64, bool ta, bool tb, bool lower, const GemmDesc& g, int splits, cudaStream_t st);
// Problems whose sizes are only known on the device: one launch over
// nprob descriptors, grid sized for max_m x max_n outputs (A, B not transposed).
cudaError_t gemm_launch_grouped(bool f64, const GemmDesc* d_descs, int nprob, int max_m, int max_n, cudaStream_t st);

// ---- double-float GEMM (dfgemm.cu): C = op(A) B with A = Ahi + Alo and
// B = Bhi + Blo (Alo / Blo may be null), column-major; lower: write only the
// lower triangle of C.
struct DfGemmDesc {
  int m, n, k;
  int lower;
  const float* Ahi;
  const float* Alo;
  long long lda;
  const float* Bhi;
  const float* Blo;
  long long ldb;
  float* Chi;
  float* Clo;
  long long ldc;
};
cudaError_t dfgemm_launch(const DfGemmDesc& g, bool ta, cudaStream_t st);

// ---- tcgen05 Ozaki GEMM (ozaki.cuh / ozaki.cu): C = A B to double-float
// accuracy on the bf16 tensor cores. Operands are sliced first: the A operand
// from the columns of a float-pair matrix (its rows after transposition, or
// the rows of a symmetric matrix), the B operand from its columns; S = 7
// slices of 7 bits each (oz_create; the slice count must match the work
// object's), relative to the largest entry of the row or column:
// double-float accuracy whatever the spread of the entries. oz_create with
// m = 0 or n = 0 allocates only the other operand.
struct OzWork;
int oz_create(OzWork** out, int m, int n, int K);
// FP32-accuracy configuration: S = 4 slices (28 bits relative to the row and
// column maxima, pairs up to 2^-35), 128 x 128 tiles, C written in FP32 to
// Chi (Clo unused).
int oz_create_f32(OzWork** out, int m, int n, int K);
void oz_destroy(OzWork* w);
cudaError_t oz_slice(OzWork* w, bool a_operand, const float* hi, const float* lo, long long ld, int count, int len,
                     int S, cudaStream_t st);
cudaError_t oz_gemm(OzWork* w, int M, int N, int K, float* Chi, float* Clo, long long ldc, bool lower,
                    cudaStream_t st);
// A operand from wa, B operand from wb (error word of wa).
cudaError_t oz_gemm2(OzWork* wa, OzWork* wb, int M, int N, int K, float* Chi, float* Clo, long long ldc, bool lower,
                     cudaStream_t st);
int* oz_error_word(OzWork* w);
// A operand from the rows of a column-major matrix (element (r, k) at r + k ld).
cudaError_t oz_slice_rows(OzWork* w, const float* hi, const float* lo, long long ld, int rows, int len, int S,
                          cudaStream_t st);
bool oz_fits(const OzWork* w, int m, int n, int K);
size_t oz_bytes(const OzWork* w);

// cudaMalloc that adds what it got to *total (each object counts its own).
inline cudaError_t counted_malloc(void** p, size_t bytes, size_t* total) {
  const size_t b = bytes < 16 ? 16 : bytes;
  const cudaError_t e = cudaMalloc(p, b);
  if (e == cudaSuccess) *total += b;
  return e;
}

// ---- FP64-accurate tensor-core GEMM (ozaki64.cuh / ozaki64.cu) and the
// stages of the FP64 path that run on it. One object per large context of
// order n; err: the word its bounded waits set (the context's).
struct Oz64;
int oz64_create(Oz64** out, int n, int* err);
void oz64_destroy(Oz64* w);
size_t oz64_bytes(const Oz64* w);
// Smallest merge whose level runs on it: below, the FP64 loops' few tiles cost
// about what the slicing and its four launches do (tridiagonals of order 300,
// 500 and 1500 in 1.24, 1.65 and 2.47 ms; with 128 1.20, 1.58 and 2.42 and
// operands for another level; with 512 1.33, 1.75 and 2.56).
constexpr int kOz64MinMerge = 256;
// A[t:, t:] -= V W' + W V' (lower triangle of the order-n matrix A): V the
// first nbp <= 32 columns of VW (leading dimension n), W the next nbp.
cudaError_t oz64_rank2k(Oz64* w, const double* VW, int nbp, int t, double* A, long long lda, cudaStream_t st);
// Problems whose sizes are known on the device only: d[0 .. nprob), not
// transposed, at most m1max x mmax with k <= mmax (a level of the tree).
cudaError_t oz64_grouped(Oz64* w, const GemmDesc* d, int nprob, int m1max, int mmax, cudaStream_t st);
// Z := Q Z (n x n) from the reflectors Y (n x n columns with their unit
// elements, zeros above and in the last column; overwritten) and tau.
cudaError_t oz64_backtr(Oz64* w, double* Y, const double* tau, double* Z, long long ldz, cudaStream_t st);

// C = op(A) B (+ C when add), FP64, column-major, m x n x k: on the tensor
// cores when every extent reaches kOz64MinGemm, by the SIMT GEMM below that
// (there a tile of 128 rows is half empty or more: complex order 128 in 4.07 ms
// with the line at 128 and 4.48 at 256; order 96 3.58, and 3.30 with it at 64).
// *w, made by
// the first call, holds the operand buffers, which grow; calls that share it
// run on one stream after another. Should a bounded wait run out, C is NaN and
// oz64_gemm_status tells.
struct Oz64Gemm;
constexpr int kOz64MinGemm = 128;
cudaError_t oz64_gemm(Oz64Gemm** w, bool ta, int m, int n, int k, const double* A, long long lda, const double* B,
                      long long ldb, double* C, long long ldc, bool add, cudaStream_t st);
void oz64_gemm_release(Oz64Gemm** w);
// Waits for st; 0, or cudaErrorLaunchTimeout's status when a wait of a product
// since the last call ran out, whose mark it clears (w may be null: no product yet).
int oz64_gemm_status(Oz64Gemm* w, cudaStream_t st);
// For tests: leaves the mark such a wait would leave.
cudaError_t oz64_gemm_mark(Oz64Gemm* w);
// The products of gla_zheev and gla_qheev (null before their first call).
Oz64Gemm* complex_gemm();
Oz64Gemm* quaternion_gemm();

// ---- adjoint of one large eigen-decomposition (large_adjoint.cu):
// Abar = V (diag(wbar) + sym(F o (V' Vbar))) V' for orders up to nmax of
// the context (its tensor-core slice buffers and float-pair planes,
// ~70 n^2 bytes).
struct LargeAdjoint;
int large_adjoint_create(LargeAdjoint** out, int nmax);
void large_adjoint_destroy(LargeAdjoint* a);
size_t large_adjoint_bytes(const LargeAdjoint* a);
cudaError_t large_adjoint(LargeAdjoint* a, int n, const double* w, const double* V, long long ldv,
                          const double* wbar, const double* Vbar, long long ldvb, double* Abar, long long lda,
                          double gap_rel, cudaStream_t st);

// ---- stage plans (one order, one working precision)
struct SytrdPlan;
// tc (FP32 only): trailing updates on the tensor cores (3xTF32, tc_gemm.cuh).
cudaError_t sytrd_plan_create(SytrdPlan** out, int n, bool f64, bool tc = false);
void sytrd_plan_destroy(SytrdPlan* p);
cudaError_t sytrd_enqueue(SytrdPlan* p, void* A, long long lda, void* d, void* e, void* tau, cudaStream_t st);
int* sytrd_error_word(SytrdPlan* p);
void sytrd_set_oz64(SytrdPlan* p, Oz64* oz);
void sytrd_keep_entries(SytrdPlan* p);  // no fixed-point panels
// Every panel on one thread-block cluster, so that several reductions run on
// SMs of their own; false (and unchanged) above kSideBySideMaxN or where the
// device cannot hold the cluster.
// Eight matrices of order 1000 take 31 ms side by side in FP64 and two 24 ms,
// one after another 11 to 12 ms each. Beyond the line a cluster's 16 SMs no
// longer hold a column's work against the whole GPU's: two of order 1200 take
// 34.5 ms side by side and 32.8 one after another, though four 36.6 and 66.1.
constexpr int kSideBySideMaxN = 1024;
bool sytrd_set_cluster_only(SytrdPlan* p);
size_t sytrd_plan_bytes(const SytrdPlan* p);

struct DcPlan;
// bisect_leaves (FP32 only): the leaves go through the per-eigenvalue solver
// (GLA_FLAG_F32_BISECT) instead of the QL chase; for the FP32 stage of the
// FP32 + refinement path, whose refinement absorbs its ~1e-4 orthogonality.
int dc_plan_create(DcPlan** out, int n, bool f64, bool bisect_leaves = false);
void dc_plan_destroy(DcPlan* p);
// Z has leading dimension n; info gets one word per leaf.
int dc_enqueue(DcPlan* p, void* d, const void* e, void* Z, int* leaf_info, cudaStream_t st);
void dc_set_oz64(DcPlan* p, Oz64* oz);
int* dc_fail_word(DcPlan* p);
int dc_leaf_count(const DcPlan* p);
size_t dc_plan_bytes(const DcPlan* p);

struct BacktrPlan;
// tc (FP32 only): both GEMMs of every block on the tensor cores (3xTF32).
int backtr_plan_create(BacktrPlan** out, int n, bool f64, bool tc = false);
void backtr_plan_destroy(BacktrPlan* p);
size_t backtr_plan_bytes(const BacktrPlan* p);
// Error word the back-transformation's tensor-core GEMMs set when a bounded
// wait runs out (the large context passes its reduction's word).
void backtr_set_error_word(BacktrPlan* p, int* err);
void backtr_set_oz64(BacktrPlan* p, Oz64* oz);
// Z := Q Z, or Q' Z when trans, for Z of ncol columns (-1: n).
int backtr_enqueue(BacktrPlan* p, const void* A, long long lda, const void* tau, void* Z, long long ldz,
                   cudaStream_t st, int ncol = -1, bool trans = false);

// ---- large-path context: workspace for one order n and one working precision
struct LargeCtx;
// refine_stage (FP32 only): the context solves the FP32 stage of the FP32 +
// refinement path, whose refinement absorbs errors of ~1e-4: its
// divide-and-conquer leaves go through the per-eigenvalue solver and its
// trailing updates and back-transformation through the 3xTF32 tensor-core
// GEMM. Plain FP32 solves keep the QL leaves and the FP32 SIMT GEMMs.
// side: the context runs beside others of the same plan, on streams of their
// own: no launch of it may need the whole GPU at once (its panels run on one
// cluster; cudaErrorNotSupported where they cannot).
int large_create(LargeCtx** out, int n, bool f64, bool refine_stage = false, bool side = false);
void large_destroy(LargeCtx* c);
// For a context whose operands are the caller's own (gla_dsytrd, gla_dormtr):
// the reduction's products and Z := Q Z in FP64 throughout. Fixed-point
// operands are exact to 2^-57 of the largest entry of their unit or column,
// which is what an eigen-decomposition's accuracy is measured by; but where Q
// does not couple two groups of rows, the product on one of them owes nothing
// to the size of the other.
void large_keep_entries(LargeCtx* c);
size_t large_workspace_bytes(const LargeCtx* c);  // device memory of the context, in bytes
// Stage times of the last large_syev (ms): tridiagonalisation (with the
// load), divide and conquer, back-transformation (with the store).
void large_stage_ms(const LargeCtx* c, float* ms3);

// Householder tridiagonalisation of the lower triangle of A (n x n, leading
// dimension lda, working precision), in place: d, e, tau and the reflectors
// below the subdiagonal (symtri! layout, unit element implicit).
int large_sytrd(LargeCtx* c, void* A, long long lda, void* d, void* e, void* tau, cudaStream_t st);
// The context's n x n working matrix (leading dimension n).
void* large_work_matrix(LargeCtx* c);
// Scratch for the bits of a matrix's largest |entry|.
unsigned long long* large_amax(LargeCtx* c);
// Eigenpairs of the symmetric tridiagonal (d, e): d becomes the ascending
// eigenvalues, Z (ldz) the eigenvectors. info: 0, or > 0 if a subproblem
// did not converge.
int large_stedc(LargeCtx* c, void* d, const void* e, void* Z, long long ldz, int* info, cudaStream_t st);
// Z := Q Z with Q = H_0 H_1 ... H_{n-2} from large_sytrd.
int large_ormtr(LargeCtx* c, const void* A, long long lda, const void* tau, void* Z, long long ldz, cudaStream_t st,
                int ncol = -1, bool trans = false);
// Clears the word that bounded waits set (the reduction clears it itself):
// before a divide and conquer that does not follow a reduction.
int large_clear_error(LargeCtx* c, cudaStream_t st);
// Full eigen-decomposition of one matrix. tcode: kF64, kF32 or kF32FromF64
// (double input solved in FP32; outputs float). Ain has leading dimension
// lda and uplo 'L'/'U'; w gets the ascending eigenvalues, V (ldv) the
// eigenvectors when wantv. *info_host: 0, -1 (non-finite input), > 0
// unconverged. Synchronises st before returning.
int large_syev(LargeCtx* c, int tcode, bool wantv, bool lower, const void* Ain, long long lda, void* w, void* V,
               long long ldv, int* info_host, cudaStream_t st);

// SymTridiagonal (d, e) of the context's order (FP64 context): ascending
// eigenvalues into w, eigenvectors into Z (ldz, may be null). *info_host: 0,
// -1 (non-finite input), > 0 unconverged. Synchronises st.
int large_stev(LargeCtx* c, const double* d, const double* e, double* w, double* Z, long long ldz, int* info_host,
               cudaStream_t st);

// ---- refinement of FP32 eigenpairs of one large matrix (large_refine.cu)
struct RefineLarge;
int refine_large_create(RefineLarge** out, int n, bool side = false);
void refine_large_destroy(RefineLarge* r);
size_t refine_large_bytes(const RefineLarge* r);  // (with the clusters' contexts it has made so far)
// Buffers the FP32 solve can write straight into: eigenvectors (n x n,
// leading dimension n) and eigenvalues (n).
float* refine_large_xbuf(RefineLarge* r);
float* refine_large_wbuf(RefineLarge* r);
// A: FP64 input (uplo triangle, leading dimension lda); X32/w32: FP32
// eigenpairs (ascending); outputs w (FP64, ascending) and V (ldv, may be
// null). Synchronises st. Returns 0, -1 for non-finite input, or a status.
int refine_large_run(RefineLarge* r, const double* A, long long lda, bool lower, const float* X32, long long ldx,
                     const float* w32, double* w, double* V, long long ldv, cudaStream_t st);
int refine_large_iters(const RefineLarge* r);
int refine_large_rotations(const RefineLarge* r);  // cluster Rayleigh-Ritz steps of the last run

// ---- leaf solves of the divide and conquer: a batched small-matrix plan
// over the leaf orders, fed with tridiagonal (d, e) in its arena layout.
int plan_stev_batched(gla_plan_s* p, int tcode, const void* din, const void* ein, void* Q, void* w, int* info,
                      cudaStream_t st);

}  // namespace gla
