// dense_mixed.cu -- blocked Cholesky / triangular inverse / W^T W with the O(n^3) products on the bf16 tensor cores
// (error-free splitting into 7-bit digits, ozaki7.cuh).  The diagonal-block factorisations and inverses stay FP64.
#include "dense_fp64.cuh"
#include "ozaki7.cuh"

#include <algorithm>

namespace lkg {

namespace {

// Two-level blocked Cholesky: 256-wide panels factored in 64-wide steps (FP64 diagonal block; panel solve and the update
// of the panel's remaining columns as 64-deep digit products), then one rank-256 trailing update per panel.  Every
// product reads split copies of its operands, so the in-place ones (the panel solve) are safe.
//
// Look-ahead (single matrix, ws.side_stream set): the trailing update of panel p is cut into the strip of panel p + 1's
// columns and the rest.  After the strip, panel p + 1 is factored on the side stream -- its diagonal blocks, splits
// and small products on ws.side_ctas SMs -- while the rest of the update runs on the other SMs; the main stream
// waits for the panel before splitting it.  Every entry receives the same operations either way, so the factor is
// bit-identical with and without the look-ahead.
void factor_panel7(double* A, int64_t lda, int64_t mstride, int n, int K0, double* Dinv, int* info, int batch,
                   Split7& SA, Split7& SD, int max_ctas, cudaStream_t st) {
  const int nblk = ceil_div(n, NB);
  const int64_t dstride = (int64_t)nblk * NB * NB;
  const int W = std::min(OZ7_KB, n - K0);
  const bool chained = max_ctas == 0;  // beside the other stream's products, kernels that wait are in their way
  for (int k0 = K0; k0 < K0 + W; k0 += NB) {
    const int nb = std::min(NB, n - k0), k = k0 / NB;
    potrf_diag(A, lda, mstride, k0, nb, Dinv, dstride, k, info, batch, st, chained && k0 > K0);
    const int M = n - k0 - nb;
    if (M <= 0) continue;
    double* A21 = A + (k0 + nb) + (int64_t)k0 * lda;
    // L21 = A21 Dinv_k^T: B rows are the rows of Dinv_k
    oz7_split2(M, nb, A21, 1, lda, mstride, SA, nb, nb, Dinv + (int64_t)k * NB * NB, 1, NB, dstride, SD, batch, st,
               chained);
    oz7_gemm_ex(M, nb, 0, 1, 1.0, SA, 0, SD, 0, 0.0, A21, lda, mstride, batch, false, max_ctas, st);
    const int wr = K0 + W - (k0 + nb);  // panel columns right of this block
    if (wr > 0) {  // A(k0+nb:, k0+nb:K0+W) -= L21 L21(0:wr, :)^T (the strict upper part written is never read)
      oz7_split(M, nb, A21, 1, lda, mstride, batch, SA, st, chained);
      oz7_gemm_ex(M, wr, 0, 1, -1.0, SA, 0, SA, 0, 1.0, A21 + (int64_t)nb * lda, lda, mstride, batch, false,
                  max_ctas, st);
    }
  }
}

void potrf_blocked_mixed7(double* A, int64_t lda, int64_t mstride, int n, double* Dinv, int* info, int batch,
                          const MixedWorkspace& ws, cudaStream_t st) {
  LKG_CUDA(cudaMemsetAsync(info, 0, sizeof(int) * batch, st));
  const int S = ws.digits;
  Split7 P = oz7_buffer(ws.panel, ws.panel_exp, S, ws.n, OZ7_KB, OZ7_KB, ws.err, ws.wide);
  Split7 SA = oz7_buffer(ws.panel, ws.panel_exp, S, ws.n, NB, NB, ws.err, ws.wide);
  Split7 SD = oz7_buffer(ws.rowblk, ws.rowblk_exp, S, ws.n, NB, NB, ws.err, ws.wide);
  const bool ahead = ws.side_stream && batch == 1;
  if (!ahead) {
    for (int K0 = 0; K0 < n; K0 += OZ7_KB) {
      const int W = std::min(OZ7_KB, n - K0);
      factor_panel7(A, lda, mstride, n, K0, Dinv, info, batch, SA, SD, 0, st);
      const int M2 = n - K0 - W;
      if (M2 <= 0) continue;
      // A22 -= P2 P2^T, P2 = L(K0+W:, K0:K0+W), one 256-wide k block
      double* P2 = A + (K0 + W) + (int64_t)K0 * lda;
      oz7_split(M2, W, P2, 1, lda, mstride, batch, P, st, true);
      oz7_gemm(M2, M2, 0, 1, -1.0, P, P, 1.0, P2 + (int64_t)W * lda, lda, mstride, batch, true, st);
    }
    return;
  }
  // the side stream's panel splits have their own buffer: the main stream's trailing update still reads P (the
  // Dinv splits in rowblk are used by one stream at a time)
  Split7 SAs = oz7_buffer(ws.side, ws.side_exp, S, ws.n, NB, NB, ws.err, ws.wide);
  const int rest_ctas = std::max(1, oz7_sm_count() - ws.side_ctas);
  factor_panel7(A, lda, mstride, n, 0, Dinv, info, batch, SA, SD, 0, st);
  for (int K0 = 0; K0 < n; K0 += OZ7_KB) {
    const int W = std::min(OZ7_KB, n - K0);
    const int M2 = n - K0 - W;
    if (M2 <= 0) break;
    double* P2 = A + (K0 + W) + (int64_t)K0 * lda;
    oz7_split(M2, W, P2, 1, lda, mstride, batch, P, st);
    const int W1 = std::min(OZ7_KB, M2);  // the next panel's width
    // the strip of the next panel's columns: A(K0+W:, K0+W:K0+W+W1) -= P2 P2(0:W1, :)^T
    oz7_gemm_ex(M2, W1, 0, 1, -1.0, P, 0, P, 0, 1.0, P2 + (int64_t)W * lda, lda, mstride, batch, false, 0, st);
    const int M3 = M2 - W1;
    if (M3 <= 0) {  // the last panel: nothing left to overlap with
      factor_panel7(A, lda, mstride, n, K0 + W, Dinv, info, batch, SA, SD, 0, st);
      continue;
    }
    LKG_CUDA(cudaEventRecord(ws.ev_strip, st));
    LKG_CUDA(cudaStreamWaitEvent(ws.side_stream, ws.ev_strip, 0));
    factor_panel7(A, lda, mstride, n, K0 + W, Dinv, info, batch, SAs, SD, ws.side_ctas, ws.side_stream);
    LKG_CUDA(cudaEventRecord(ws.ev_panel, ws.side_stream));
    // the rest of the update, lower: A(K0+W+W1:, K0+W+W1:) -= P2(W1:, :) P2(W1:, :)^T
    oz7_gemm_ex(M3, M3, 0, 1, -1.0, P, W1, P, W1, 1.0, P2 + W1 + (int64_t)(W + W1) * lda, lda, mstride, batch, true,
                rest_ctas, st);
    LKG_CUDA(cudaStreamWaitEvent(st, ws.ev_panel, 0));
  }
}

// The 64-wide steps of one 256-row block of the triangular inverse (rows K0 .. K0 + Wd, the D^-1 blocks on the diagonal
// already): W(k0:k0+nb, 0:k0) = -Dinv_k Acc(k0:k0+nb, 0:k0), then the block's rows below accumulate
// L(k0+nb:, k0:k0+nb) W(k0:k0+nb, 0:k0+nb).
void trtri_block7(const double* L, int64_t lda, int64_t mstride, int n, int K0, int Wd, const double* Dinv,
                  int64_t dstride, double* W, int64_t ldw, int64_t wstride, int batch, Split7& SA, Split7& SB,
                  cudaStream_t st) {
  for (int k0 = K0; k0 < K0 + Wd; k0 += NB) {
    const int nb = std::min(NB, n - k0), k = k0 / NB;
    if (k0 > 0) {  // W(k0:k0+nb, 0:k0) = -Dinv_k Acc(k0:k0+nb, 0:k0): B rows are the columns of Acc
      oz7_split2(nb, nb, Dinv + (int64_t)k * NB * NB, 1, NB, dstride, SA, k0, nb, W + k0, ldw, 1, wstride, SB,
                 batch, st, true);
      oz7_gemm(nb, k0, 0, 1, -1.0, SA, SB, 0.0, W + k0, ldw, wstride, batch, false, st);
    }
    const int mr = K0 + Wd - (k0 + nb);  // rows of this 256-row block below the 64-row one
    if (mr > 0) {  // Acc(k0+nb:K0+Wd, 0:k0+nb) += L(k0+nb:K0+Wd, k0:k0+nb) W(k0:k0+nb, 0:k0+nb)
      oz7_split2(mr, nb, L + (k0 + nb) + (int64_t)k0 * lda, 1, lda, mstride, SA, k0 + nb, nb, W + k0, ldw, 1,
                 wstride, SB, batch, st, true);
      oz7_gemm(mr, k0 + nb, 0, 1, 1.0, SA, SB, 1.0, W + k0 + nb, ldw, wstride, batch, false, st);
    }
  }
}

// Two-level triangular inverse: inside a 256-row block the 64-wide steps, below it one rank-256 update of the
// accumulated rows; every product on the digit kernel.  (A look-ahead like the Cholesky's -- the next block's 64-wide
// steps on a side stream while the rest of the update runs -- measured 1.9 ms slower per n = 16384 evaluation: the
// steps' wide products need most of the SMs, so it is not used here.)
void trtri_blocked_mixed7(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* W,
                          int64_t ldw, int64_t wstride, int batch, const MixedWorkspace& ws, cudaStream_t st) {
  const int nblk = ceil_div(n, NB);
  const int64_t dstride = (int64_t)nblk * NB * NB;
  inverse_init(Dinv, n, W, ldw, wstride, batch, st);
  const int S = ws.digits_inv;
  Split7 SL = oz7_buffer(ws.panel, ws.panel_exp, S, ws.n, OZ7_KB, OZ7_KB, ws.err, ws.wide);
  Split7 SR = oz7_buffer(ws.rowblk, ws.rowblk_exp, S, ws.n, OZ7_KB, OZ7_KB, ws.err, ws.wide);
  Split7 SA = oz7_buffer(ws.panel, ws.panel_exp, S, ws.n, NB, NB, ws.err, ws.wide);
  Split7 SB = oz7_buffer(ws.rowblk, ws.rowblk_exp, S, ws.n, NB, NB, ws.err, ws.wide);
  for (int K0 = 0; K0 < n; K0 += OZ7_KB) {
    const int Wd = std::min(OZ7_KB, n - K0);
    trtri_block7(L, lda, mstride, n, K0, Wd, Dinv, dstride, W, ldw, wstride, batch, SA, SB, st);
    const int M2 = n - K0 - Wd;
    if (M2 <= 0) continue;
    // Acc(K0+Wd:, 0:N) += L(K0+Wd:, K0:K0+Wd) W(K0:K0+Wd, 0:N), N = K0 + Wd
    const int N = K0 + Wd;
    oz7_split2(M2, Wd, L + (K0 + Wd) + (int64_t)K0 * lda, 1, lda, mstride, SL, N, Wd, W + K0, ldw, 1, wstride, SR,
               batch, st, true);
    oz7_gemm(M2, N, 0, 1, 1.0, SL, SR, 1.0, W + K0 + Wd, ldw, wstride, batch, false, st);
  }
}

// R^-1 = W^T W in chunks of ws.wk rows of W: rows past the chunk's last hold no entry of it (W is lower triangular), so
// chunk c0 updates the leading c0 + kc block.  Every tile adds its 256-row blocks in ascending order, one rounding
// each, whatever the chunk, so the result does not depend on ws.wk.
void wtw_lower_mixed7(const double* W, int64_t ldw, int64_t wstride, int n, double* C, int64_t ldc, int64_t cstride,
                      int batch, const MixedWorkspace& ws, cudaStream_t st) {
  Split7 SW = oz7_buffer(ws.wchunk, ws.wchunk_exp, ws.digits_inv, ws.n, ws.wk, OZ7_KB, ws.err, ws.wide);
  for (int c0 = 0; c0 < n; c0 += ws.wk) {
    const int kc = std::min(ws.wk, n - c0);
    oz7_split(c0 + kc, kc, W + c0, ldw, 1, wstride, batch, SW, st);  // rows of the split = columns of W
    oz7_wtw(c0 + kc, c0, SW, C, ldc, cstride, batch, st);
  }
}

}  // namespace

void potrf_blocked_mixed(double* A, int64_t lda, int64_t mstride, int n, double* Dinv, int* info, int batch,
                         const MixedWorkspace& ws, cudaStream_t st) {
  const int64_t dstride = (int64_t)ceil_div(n, NB) * NB * NB;
  for (int b = 0; b < batch; b += ws.panel_group)
    potrf_blocked_mixed7(A + b * mstride, lda, mstride, n, Dinv + b * dstride, info + b, std::min(ws.panel_group, batch - b),
                         ws, st);
}

void trtri_blocked_mixed(const double* L, int64_t lda, int64_t mstride, int n, const double* Dinv, double* W,
                         int64_t ldw, int64_t wstride, int batch, const MixedWorkspace& ws, cudaStream_t st) {
  const int64_t dstride = (int64_t)ceil_div(n, NB) * NB * NB;
  for (int b = 0; b < batch; b += ws.panel_group)
    trtri_blocked_mixed7(L + b * mstride, lda, mstride, n, Dinv + b * dstride, W + b * wstride, ldw, wstride,
                         std::min(ws.panel_group, batch - b), ws, st);
}

void wtw_lower_mixed(const double* W, int64_t ldw, int64_t wstride, int n, double* C, int64_t ldc, int64_t cstride,
                     int batch, const MixedWorkspace& ws, cudaStream_t st) {
  for (int b = 0; b < batch; b += ws.chunk_group)
    wtw_lower_mixed7(W + b * wstride, ldw, wstride, n, C + b * cstride, ldc, cstride, std::min(ws.chunk_group, batch - b),
                     ws, st);
}

void gemm_square_digits(int n, const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                        const MixedWorkspace& ws, cudaStream_t st) {
  const int S = FP64_DIGITS, kh = ws.wk / 2 / OZ7_KB * OZ7_KB;  // half of the chunk buffer for each operand
  __nv_bfloat16* planes = static_cast<__nv_bfloat16*>(ws.wchunk);
  Split7 SA = oz7_buffer(planes, ws.wchunk_exp, S, ws.n, kh, OZ7_KB, ws.err, true);
  Split7 SB = oz7_buffer(planes + oz7_plane_elems(ws.n, kh, S), ws.wchunk_exp + oz7_exp_elems(ws.n, kh, OZ7_KB), S, ws.n,
                         kh, OZ7_KB, ws.err, true);
  for (int c0 = 0; c0 < n; c0 += kh) {
    const int kc = std::min(kh, n - c0);
    oz7_split2(n, kc, A + (int64_t)c0 * lda, 1, lda, 0, SA, n, kc, B + c0, ldb, 1, 0, SB, 1, st, c0 > 0);
    oz7_gemm(n, n, 0, SA.nblk, 1.0, SA, SB, c0 == 0 ? 0.0 : 1.0, C, ldc, 0, 1, false, st);
  }
}

size_t trsm_digits_bytes(int n, int r) {
  auto bytes = [](int rows) {
    return oz7_plane_elems(rows, OZ7_KB, FP64_DIGITS) * sizeof(__nv_bfloat16) +
           (oz7_exp_elems(rows, OZ7_KB, NB) * sizeof(int) + 255) / 256 * 256;
  };
  return bytes(n) + bytes(r);
}

// Two-level forward substitution with many right-hand sides, the structure of the digit Cholesky: inside a 256-row panel
// the 64-row steps X_k = Dinv_k B_k and the update of the panel's remaining rows, then one rank-256 update of the rows
// below.  A column's result depends on that column alone (its own exponents), so predictions do not depend on how the
// points are grouped.
void trsm_lower_left_digits(const double* L, int64_t lda, int n, const double* Dinv, double* B, int64_t ldb, int r,
                            void* scratch, int* err, cudaStream_t st) {
  const int S = FP64_DIGITS;
  char* at = static_cast<char*>(scratch);
  void* lp = at;
  at += oz7_plane_elems(n, OZ7_KB, S) * sizeof(__nv_bfloat16);
  void* xp = at;
  at += oz7_plane_elems(r, OZ7_KB, S) * sizeof(__nv_bfloat16);
  int* le = reinterpret_cast<int*>(at);
  int* xe = le + (oz7_exp_elems(n, OZ7_KB, NB) * sizeof(int) + 255) / 256 * 64;
  Split7 SL = oz7_buffer(lp, le, S, n, OZ7_KB, OZ7_KB, err, true);
  Split7 SX = oz7_buffer(xp, xe, S, r, OZ7_KB, OZ7_KB, err, true);
  Split7 sl = oz7_buffer(lp, le, S, n, NB, NB, err, true), sx = oz7_buffer(xp, xe, S, r, NB, NB, err, true);
  for (int K0 = 0; K0 < n; K0 += OZ7_KB) {
    const int Wd = std::min(OZ7_KB, n - K0);
    for (int k0 = K0; k0 < K0 + Wd; k0 += NB) {
      const int nb = std::min(NB, n - k0), k = k0 / NB;
      oz7_split2(nb, nb, Dinv + (int64_t)k * NB * NB, 1, NB, 0, sl, r, nb, B + k0, ldb, 1, 0, sx, 1, st, k > 0);
      oz7_gemm(nb, r, 0, 1, 1.0, sl, sx, 0.0, B + k0, ldb, 0, 1, false, st);
      const int mr = K0 + Wd - (k0 + nb);
      if (mr > 0) {
        oz7_split2(mr, nb, L + (k0 + nb) + (int64_t)k0 * lda, 1, lda, 0, sl, r, nb, B + k0, ldb, 1, 0, sx, 1, st,
                   true);
        oz7_gemm(mr, r, 0, 1, -1.0, sl, sx, 1.0, B + k0 + nb, ldb, 0, 1, false, st);
      }
    }
    const int M2 = n - K0 - Wd;
    if (M2 <= 0) continue;
    oz7_split2(M2, Wd, L + (K0 + Wd) + (int64_t)K0 * lda, 1, lda, 0, SL, r, Wd, B + K0, ldb, 1, 0, SX, 1, st,
               true);
    oz7_gemm(M2, r, 0, 1, -1.0, SL, SX, 1.0, B + K0 + Wd, ldb, 0, 1, false, st);
  }
}

// The FP64 path's products as digit products: GB300 issues one FP64 warp instruction per 19 clocks and SM (1.25 TFLOP/s
// over the chip), so 36 exact bf16 products of 7-bit digits are 10 to 30 times faster than one DFMA.  Their error is no
// larger: one rounding per 256 columns instead of one per column, on operands of 57 bits.  On the same matrices, 24 designs
// of n = 4096, d = 8 against 80-bit arithmetic (geometric means): LL 1.2e-11 here, 1.4e-11 with DFMA (absolute), gradient
// 1.1e-13 here, 1.7e-13 with DFMA (relative).  Measured, LL + gradient, d =
// 4, matern5_2 (us, DFMA / digits), one matrix: n = 192 434 / 475, 256 550 / 588, 448 906 / 946; 64 at once: n = 192
// 2756 / 1985, 256 4414 / 2792, 448 12184 / 5222; one matrix of 1024 8313 / 3394 (large DFMA tiles).  The rule looks at n
// alone, so that a matrix gives the same bits alone and in a batch: from 192 on a batch gains more than one matrix loses.
bool digits_pay(int n) { return n >= 192; }

}  // namespace lkg
