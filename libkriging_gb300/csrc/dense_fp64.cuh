// dense_fp64.cuh -- FP64 dense kernels for the blocked Cholesky, triangular inverse and R^-1 (sm_103a).
//
// Measured on GB300: DFMA peaks at ~1.19 TFLOP/s while DMMA (mma.sync f64) peaks at ~1.04 TFLOP/s, so the FP64
// tiles are register-blocked DFMA.  Every kernel takes a batch index from blockIdx.z and per-matrix strides so
// that multistart evaluations of one design run in the same launch.
#pragma once
#include "common.cuh"

namespace lkg {

constexpr int NB = 64;  // block size of the blocked factorisations (also the GEMM tile edge)

// Operand view for a tile GEMM: element (row r, col c) of the logical operand is p[r*sr + c*sc].
struct MatView {
  const double* p;
  int64_t sr, sc;      // element strides
  int64_t batch;       // element stride between batch entries (0 = shared)
};

// ---- launch helpers (implemented in dense_fp64.cu) ----
// C(M x N) = beta*C + alpha * A(M x K) * B(K x N)  with A, B generic views; C column-major (ldc) in place.
// lower_only: skip tiles strictly above the diagonal and write only r >= c (diagonal offset c_off - r_off).
void gemm_tiles(int M, int N, int K, double alpha, MatView A, MatView B, double beta, double* C, int64_t ldc,
                int64_t c_batch, int batch, bool lower_only, cudaStream_t st);

// One Cholesky step on the diagonal block at (k0, k0) of each batch matrix (lda, stride mstride):
// factors the nb x nb block in place and writes its inverse into Dinv (NB*NB per block, block index blk).
void potrf_diag(double* A, int64_t lda, int64_t mstride, int k0, int nb, double* Dinv, int64_t dinv_bstride,
                int blk, int* info, int batch, cudaStream_t st, bool chained = false);

// Full blocked lower Cholesky of each batch matrix (n x n, lower triangle referenced), keeping the inverses of
// the diagonal blocks in Dinv (nblk * NB * NB per matrix).  info[b] = 1-based column of the first non-positive
// pivot, 0 on success.
void potrf_blocked(double* A, int64_t lda, int64_t mstride, int n, double* Dinv, int* info, int batch,
                   cudaStream_t st);

// W = L^-1 (lower, out of place, zero above the diagonal) from L and the diagonal-block inverses.
void trtri_blocked(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* W,
                   int64_t ldw, int64_t wstride, int batch, cudaStream_t st);

// C = W^T W, lower triangle (= R^-1 when W = L^-1).
void wtw_lower(const double* W, int64_t ldw, int64_t wstride, int n, double* C, int64_t ldc, int64_t cstride,
               int batch, cudaStream_t st);

// W = 0 with the Dinv blocks (full NB x NB blocks with their zero upper parts) on its diagonal: what the triangular
// inverses start from (no later step of theirs writes a diagonal block).
void inverse_init(const double* Dinv, int n, double* W, int64_t ldw, int64_t wstride, int batch, cudaStream_t st);

// Digit-product variants: the O(n^3) products on the bf16 tensor cores by error-free splitting into 7-bit digits
// (ozaki7.cuh); the diagonal blocks stay FP64.  With 8 digits (57-bit operands with wide leading digits, 56-bit without, one rounding per 256 columns) they
// serve the FP64 path too: see digits_pay().
constexpr int FP64_DIGITS = 8;
struct MixedWorkspace {
  int digits = FP64_DIGITS;      // digits of the Cholesky's products (6 .. 8)
  int digits_inv = FP64_DIGITS;  // digits of the triangular inverse and W^T W, which feed only the gradient (5 .. 8)
  bool wide = true;              // 8-bit leading digits (ozaki7.cu)
  int* err = nullptr;            // status words of the products (OZ7_ERR_WORDS)
  void* panel = nullptr;  // bf16 planes, oz7_plane_elems(n, 256, 8) for each of panel_group entries
  int* panel_exp = nullptr;
  void* rowblk = nullptr;  // bf16 planes, same size
  int* rowblk_exp = nullptr;
  void* wchunk = nullptr;  // bf16 planes, oz7_plane_elems(n, wk, 8) for each of chunk_group entries
  int* wchunk_exp = nullptr;
  int panel_group = 1, chunk_group = 1;  // a batch's entries share the buffers, this many at a time
  int wk = 0;  // columns of a chunk of the long products (W^T W, square products): a multiple of 256, at least 512
  int n = 0;
  // look-ahead of the blocked Cholesky (single matrix): the next panel is factored on side_stream, on side_ctas SMs
  // kept free by the trailing update, with its splits in side / side_exp (the size of panel); off when null
  cudaStream_t side_stream = nullptr;
  cudaEvent_t ev_strip = nullptr, ev_panel = nullptr;
  void* side = nullptr;
  int* side_exp = nullptr;
  int side_ctas = 0;
};
void potrf_blocked_mixed(double* A, int64_t lda, int64_t mstride, int n, double* Dinv, int* info, int batch,
                         const MixedWorkspace& ws, cudaStream_t st);
void trtri_blocked_mixed(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* W,
                         int64_t ldw, int64_t wstride, int batch, const MixedWorkspace& ws, cudaStream_t st);
void wtw_lower_mixed(const double* W, int64_t ldw, int64_t wstride, int n, double* C, int64_t ldc, int64_t cstride,
                     int batch, const MixedWorkspace& ws, cudaStream_t st);

// C (n x n, ldc) = A B with A, B n x n column-major (lda, ldb), FP64_DIGITS digits, in chunks of ws.wk / 2 columns of A
void gemm_square_digits(int n, const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                        const MixedWorkspace& ws, cudaStream_t st);
// Bytes of scratch for trsm_lower_left_digits, and L X = B in place (B n x r column-major, ldb; one matrix); err: status
// words of the products (OZ7_ERR_WORDS)
size_t trsm_digits_bytes(int n, int r);
void trsm_lower_left_digits(const double* L, int64_t lda, int n, const double* Dinv, double* B, int64_t ldb, int r,
                            void* scratch, int* err, cudaStream_t st);
// Whether the FP64 path runs its products over n x n factors as 8-digit products (else as DFMA tiles).
bool digits_pay(int n);

// Dinv blocks (nblk * NB * NB per matrix) of an existing lower factor L: the inverses of its NB x NB diagonal
// blocks, computed exactly as potrf_diag computes them.
void trtri_diag_blocks(const double* L, int64_t lda, int64_t mstride, int n, double* Dinv, int batch,
                       cudaStream_t st);
// D(c, r) = S(r, c) for r < rows, c < cols (column-major, leading dimensions lds, ldd)
void transpose_copy(const double* S, int64_t lds, double* D, int64_t ldd, int rows, int cols, cudaStream_t st);
// A(i, i) += v for i < n
void add_diag(double* A, int64_t lda, int n, double v, cudaStream_t st);
// A(i, j) = 0 for i < j < n in every batch matrix
void zero_upper(double* A, int64_t lda, int64_t mstride, int n, int batch, cudaStream_t st);

// Solve L X = B in place (B n x r column-major, ldb, batch stride bstride).
void trsm_lower_left(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* B,
                     int64_t ldb, int64_t bstride, int r, int batch, cudaStream_t st);
// Solve L^T X = B in place.
void trsm_lower_left_t(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* B,
                       int64_t ldb, int64_t bstride, int r, int batch, cudaStream_t st);

}  // namespace lkg
