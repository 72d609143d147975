// dense_f64.cuh — blocked FP64 dense kernels and drivers (host API).
#pragma once

#include "common.cuh"
#include <vector>

#include "gemm_f64.cuh"
#include "pool.h"
#include "solve_class.h"

namespace gprx {

// Panel width of the blocked factor / inverse / solves.  The in-place GEMM
// steps need it ≤ the 128-wide GEMM tile.
constexpr int NB = 128;

// C = alpha·opA·opB + beta·C on DMMA tiles chosen by their number (see
// gemm_f64.cuh); C must not alias A or B.
cudaError_t dgemm(bool ta, bool tb, const GemmParams& p, cudaStream_t s, int batch = 1);

// Small helper building GemmParams.
GemmParams gemm_params(int M, int N, int K, const double* A, long long lda, const double* B, long long ldb,
                       double* C, long long ldc, double alpha, double beta, const DevStatus* st);

// Side streams and events of the look-ahead factorization (one per handle):
// aux carries the chain, aux2 the column update's rows below the diagonal
// block (concurrent with the diagonal block).  After the factor, aux is free
// for work beside the inverse's products (side: events for that).
struct FactorCtx {
  Lane& lane;  // of the handle: aux and aux2 are its side streams
  std::vector<cudaEvent_t> ev;
  cudaEvent_t side[4] = {nullptr, nullptr, nullptr, nullptr};
  explicit FactorCtx(Lane& l) : lane(l) {}
  FactorCtx(const FactorCtx&) = delete;
  FactorCtx& operator=(const FactorCtx&) = delete;
  ~FactorCtx();
  cudaError_t ensure(int nblk);
};

// In-place lower Cholesky of A (n×n, ld) by right-looking blocks of NB.
// linv receives the inverse of every diagonal block (ceil(n/NB) blocks of
// NB×NB, column-major, ld NB).  A non-positive pivot sets st (CHOLESKY_FAILED,
// info = global row) and every later kernel of the stream returns at once.
// With ctx, the chain column update → diagonal block → panel solve of step
// k+1 runs on ctx->aux (high priority) while the trailing update of step k
// runs on s; on return all work is ordered before later work on s.
cudaError_t potrf_blocked(double* A, long long ld, int n, double* linv, DevStatus* st, cudaStream_t s,
                          FactorCtx* ctx = nullptr);

// Inverses of the diagonal NB-blocks of a lower triangle (unit: unit diagonal).
cudaError_t tri_inv_blocks(const double* L, long long ld, int n, bool unit, double* linv, DevStatus* st,
                           cudaStream_t s);

// X = L⁻¹ into X (n×n, ldx), from L and its diagonal block inverses.  X's
// strict upper triangle must be zero on entry; scratch holds ceil(n/2)²
// doubles.
cudaError_t trtri_blocked(const double* L, long long ld, int n, const double* linv, double* X, long long ldx,
                          double* scratch, DevStatus* st, cudaStream_t s);

// C (lower) = Xᵀ X for lower-triangular X: K⁻¹ from X = L⁻¹.
cudaError_t lauum_lower(const double* X, long long ldx, int n, double* C, long long ldc, DevStatus* st,
                        cudaStream_t s);

struct EmuWork;

// B (n×q, ldb) := L⁻¹ B   /   := L⁻ᵀ B, with L's diagonal block inverses: by
// recursive halving (X1 from the top half, one update B2 −= L21 X1 with K = n/2,
// then the bottom half; the transpose bottom half first) down to blocks that
// tri_solve takes in one launch (SOLVE_BULK: to 128-row blocks).  The class
// (solve_class of the whole solve) fixes where the recursion stops, and with it the
// bits of a column: they do not depend on q within a class.
cudaError_t trsm_lower(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                       DevStatus* st, cudaStream_t s);
cudaError_t trsm_lower_t(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                         DevStatus* st, cudaStream_t s);
cudaError_t trsm_lower(SolveClass cls, const double* L, long long ld, int n, const double* linv, double* B, long long ldb,
                       int q, DevStatus* st, cudaStream_t s);
cudaError_t trsm_lower_t(SolveClass cls, const double* L, long long ld, int n, const double* linv, double* B, long long ldb,
                         int q, DevStatus* st, cudaStream_t s);

// The same two solves (trans: L⁻ᵀ) in one launch of thread-block clusters
// (tri_solve.cu); a column's bits do not depend on q.  Any q for n ≤ 8192,
// one right-hand side for every n.
cudaError_t tri_solve(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                      bool trans, const DevStatus* st, cudaStream_t s);
// One right-hand side in FP64 FMAs (other bits than tri_solve's).  prefix
// (forward only): prefix[i + s·ldp] receives the sum of L(i, :) x over the
// columns of the first s + 1 blocks, for the rows below block s.
cudaError_t tri_solve_vec(const double* L, long long ld, int n, const double* linv, double* b, bool trans,
                          const DevStatus* st, cudaStream_t s, double* prefix = nullptr, long long ldp = 0);

// out = log|det L|² contribution: 2 Σ ln L_ii (lower LLT) or Σ ln D_i (ldlt=true).
cudaError_t logdet_diag(const double* L, long long ld, int n, bool ldlt, double* out, DevStatus* st,
                        cudaStream_t s);

// z = X y for lower-triangular X (n×n, ld).
cudaError_t trmv_lower(const double* X, long long ld, int n, const double* y, double* z, DevStatus* st,
                       cudaStream_t s);
// out_j = Σ_{i ≥ (lower ? j : 0)} M(i,j) v_i  for j < ncols: one warp per
// column, or (block) one CTA, for few long columns: 12 → 4 µs for one of 1000,
// 36 → 8 µs for the squares over D of four of 2000.  The sums differ in bits.
cudaError_t gemv_t(const double* M, long long ld, int nrows, int ncols, bool lower, const double* v, double* out,
                   DevStatus* st, cudaStream_t s, bool block = false);
// out_j = Σ_i M(i,j)² (/ w_i when w != nullptr) for j < ncols.
// VarianceOf (on): the latent variance max(0, kss − sum) plus `add` instead.
struct VarianceOf {
  bool on = false;
  double kss = 0.0, add = 0.0;
};
cudaError_t col_sumsq(const double* M, long long ld, int nrows, int ncols, const double* w, double* out,
                      DevStatus* st, cudaStream_t s, bool block = false, VarianceOf var = {});

// out = Σ_i a_i b_i (single block, deterministic).
cudaError_t dot_dev(const double* a, const double* b, int n, double* out, DevStatus* st, cudaStream_t s);

// The same two products with the FP64 GEMMs emulated on the int8 tensor
// cores (emu_gemm.cuh) wherever the blocks are at least emu_min wide; the
// narrower levels stay on DMMA.  X's strict upper triangle must be zero.
cudaError_t trtri_blocked_emu(const double* L, long long ld, int n, const double* linv, double* X, long long ldx,
                              double* scratch, const EmuWork& w, int emu_min, DevStatus* st, cudaStream_t s);
cudaError_t lauum_lower_emu(const double* X, long long ldx, int n, double* C, long long ldc, const EmuWork& w,
                            DevStatus* st, cudaStream_t s);

// Lower LLT of A (n×n) and X = L⁻¹ together by recursive halving: A11 → (L11,
// X11) recursively, L21 = A21 X11ᵀ, A22 −= L21 L21ᵀ, A22 → (L22, X22),
// X21 = −X22 (L21 X11), the coupling products as emulated FP64 GEMMs; blocks
// of at most `leaf` rows use potrf_blocked and trtri_blocked_emu.  linv gets
// the diagonal-block inverses (block index = row / NB); scratch holds
// ceil(n/2)² doubles.  X's strict upper triangle must be zero.
cudaError_t potrf_trtri_rec(double* A, long long ld, int n, double* X, long long ldx, double* linv,
                            double* scratch, const EmuWork& w, int leaf, int emu_min, DevStatus* st,
                            cudaStream_t s, FactorCtx* ctx);

// Sets X (n×n, ld) to the identity (full columns, zero off the diagonal).
cudaError_t set_identity(double* X, long long ld, int n, cudaStream_t s);

}  // namespace gprx
