// diag_block.cuh — the diagonal-block step of the blocked Cholesky (LLT of an
// nb×nb block and its inverse, one CTA), shared by the blocked factor and the
// batched per-problem evaluation.
#pragma once

#include "gemm_f64.cuh"

namespace gprx {

constexpr int NB_DIAG = 128;

// ---------------------------------------------------------------------------
// Diagonal block (nb ≤ 128): LLT and the block's inverse X = L⁻¹ in shared
// memory, one CTA of a multiple of 128 and at least 256 threads (FD_THREADS:
// warp 0 and fifteen helper warps).  The block is padded to a multiple of 16
// with an identity tail.
//
// Left-looking by 16-column blocks p, two barriers per step:
//   warp 0   : the leaf (p, p) takes panel p−1 (its earlier panels are in),
//              then its 16×16 LLT and inverse in registers (lane = row);
//   helpers  : column block p below the leaf takes panel p−1; column block
//              p+1 takes panels 0..p−1 in one product; block row p−1 of X:
//              T = L_{p−1,<p−1} X_{<p−1,<p−1}, then X_{p−1,<p−1} = −X_{p−1,p−1} T;
//              and the stores of L column block p−1 and of X block row p−2 to
//              global memory;
//   all      : the panel below leaf p, A X_ppᵀ, refined once where the leaf's pivots
//              spread (leaf_spread).
// Column block q arrives by its own cp.async group, waited for one step
// before its first use, so the factor starts while the block still loads.
//
// Storage: L lower in s (ld FLS); X(i, j) for j < i in the transposed slot
// s[j + i·FLS] (the upper triangle), X(i, i) = 1/L_ii on the diagonal once
// block row i of X is formed (L's diagonal is kept in ldiag for the store).
// ---------------------------------------------------------------------------
constexpr int FD_THREADS = 512;
constexpr int LF = 16;                      // leaf / panel width
constexpr int FLS = NB_DIAG + 4;            // ld of the block (≡ 4 mod 16: conflict-free fragments)
constexpr int TLD = 20;                     // ld of T (16 rows; ≡ 4 mod 16)
constexpr int TMP_DOUBLES = TLD * NB_DIAG;  // T: 16 rows × up to 112 columns

// C(16×8) += A(16×K) · B(K×8) with A(i,k) = a[i·ai + k·ak], B(k,j) = b[k·bk + j·bj].
// AMASK: A(i,k) = 0 for k > i + moff;  BMASK: B(k,j) = 0 for k < j + moff.
template <bool AMASK = false, bool BMASK = false>
__device__ __forceinline__ void mma_tile_smem(double (&c)[4], const double* a, int ai, int ak, const double* b, int bk,
                                              int bj, int K, int moff = 0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 4
  for (int kk = 0; kk < K; kk += 4) {
    const int k = kk + t;
    double a0 = a[g * ai + k * ak];
    double a1 = a[(g + 8) * ai + k * ak];
    double b0 = b[k * bk + g * bj];
    if (AMASK) {
      if (k > g + moff) a0 = 0.0;
      if (k > g + 8 + moff) a1 = 0.0;
    }
    if (BMASK && k < g + moff) b0 = 0.0;
    dmma_16x8x4(c, a0, a1, b0);
  }
}

// Reciprocal of a positive normal number: the hardware's 20-bit estimate x0
// and one cubic step, 1/d = x0 (1 + e + e²) + O(e³) with e = 1 − d·x0 (the
// geometric series).  e + e² goes to *corr, x0 to *seed: 1/d = seed·(1 + corr).
__device__ __forceinline__ void rcp_parts(double d, double* seed, double* corr) {
  double x0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d));
  const double e = fma(-d, x0, 1.0);
  *seed = x0;
  *corr = fma(e, e, e);
}

// 16×16 leaf LLT and inverse, one warp: lane r < 16 holds row r of the block
// at (off, off) of s in registers, lane 16 + r row r of the identity, which the
// same elimination turns into row r of L⁻ᵀ.  Writes L (below the diagonal)
// back to s, X = L⁻¹ to the transposed slots (X(i, c) to s[c + i·FLS], the
// diagonal included), 1/L_jj to rinv[off + j] and L_jj to ldiag[off + j].
// Returns the failing column or −1 (uniform over the warp).
//
// Bound by the chain from pivot to pivot on one warp (an FP64 operation is 13
// cycles there).  The columns stay unscaled (Schur complements a_ij, so
// A −= a_j a_jᵀ / d_j) until the end: a pivot needs a reciprocal instead of a
// square root, column j is broadcast before its pivot's reciprocal is known
// (the entry of the next pivot by a shuffle, the rest through the block itself),
// and every lane forms the next pivot d' − a²·x0·(1 + corr), so a step is the
// estimate, four FMAs and one shuffle that overlaps them.  The square
// roots of all pivots follow in parallel.  2.9 K cycles a leaf alone, 4.3 K
// beside the helpers' shared-memory loads (5.4 K and 8.6 K with the rsqrt and
// the scaled column on the chain and no inverse; broadcasts by shuffles only:
// 3.6 K and 4.9 K; a loop over the pivots instead of straight code: 3.7 K, 5.0 K).
static __device__ __noinline__ int leaf16_factor(double* s, int off, double* rinv, double* ldiag) {
  const int lane = threadIdx.x & 31, r = lane & 15;
  const bool low = lane < 16;
  double* row = s + (off + r) + off * FLS;
  double d[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) d[c] = low ? (c <= r ? row[c * FLS] : 0.0) : (c == r ? 1.0 : 0.0);
  int bad = -1;
  double mine = 1.0;                     // this row's pivot
  double dg = low ? row[r * FLS] : 0.0;  // and its diagonal entry, updated by the row itself
  double piv = __shfl_sync(0xffffffffu, dg, 0);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const double v = d[j];
    const double b1 = __shfl_sync(0xffffffffu, v, j + 1);
    const double dn = __shfl_sync(0xffffffffu, dg, j + 1);
    if (low ? r > j : r <= j) row[j * FLS] = v;
    __syncwarp();
    double b[16];
#pragma unroll
    for (int c = j + 2; c < 16; ++c) b[c] = s[(off + c) + (off + j) * FLS];
    if (!(piv > 0.0) && bad < 0) bad = j;
    if (r == j) mine = piv;
    if (j + 1 < 16) {
      double x0, corr;
      rcp_parts(piv, &x0, &corr);
      const double q = b1 * b1 * x0;
      piv = fma(-q, corr, dn - q);
      const double u = v * fma(x0, corr, x0);
      d[j + 1] = fma(-u, b1, d[j + 1]);
      dg = fma(-u, v, dg);
#pragma unroll
      for (int c = j + 2; c < 16; ++c) d[c] = fma(-u, b[c], d[c]);  // rows above c: never read
    }
  }
  if (bad >= 0) return bad;
  const double rs = rsqrt(mine);
  __syncwarp();
  // column c of both triangles times 1/L_cc
#pragma unroll 4
  for (int k = 0; k < 8; ++k) {
    const int c = 2 * k + (lane >> 4);
    row[c * FLS] *= __shfl_sync(0xffffffffu, rs, c);
  }
  if (low) {
    rinv[off + r] = rs;
    ldiag[off + r] = mine * rs;
  }
  __syncwarp();
  return -1;
}

// Whether a leaf's pivots spread so far that its explicit inverse costs digits: the
// largest diagonal entry of L over the smallest is above 2^2.5 (the high words'
// difference is the ratio's logarithm, in steps of 2^-20 and linear between powers
// of two).  The error of A X_ppᵀ grows with the leaf's condition number.
__device__ __forceinline__ bool leaf_spread(const double* ldiag) {
  const unsigned h = (unsigned)__double2hiint(ldiag[threadIdx.x & 15]);
  return __reduce_max_sync(0xffffffffu, h) - __reduce_min_sync(0xffffffffu, h) > (5u << 19);
}

// c += A(16 rows from r0, c0..) X_ppᵀ (c0 = 16p), one warp.
__device__ __forceinline__ void panel_times_x(const double* s, int r0, int c0, double (&c)[2][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int kk = 0; kk < LF; kk += 4) {
    const int k = kk + t4;
    const double a0 = s[r0 + g + (c0 + k) * FLS], a1 = s[r0 + g + 8 + (c0 + k) * FLS];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // B(k, j) = X(j, k), zero for k > j
      const int j = 8 * h + g;
      dmma_16x8x4(c[h], a0, a1, k <= j ? s[c0 + k + (c0 + j) * FLS] : 0.0);
    }
  }
}
// Entry r of half h of the accumulator tile of those rows.
__device__ __forceinline__ double& panel_entry(double* s, int r0, int c0, int h, int r) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  return s[r0 + g + ((r & 2) ? 8 : 0) + (c0 + 8 * h + 2 * t4 + (r & 1)) * FLS];
}

// The 16 rows from r0 below leaf p, one warp: A(rows, c0..) X_ppᵀ.
__device__ __forceinline__ void panel_rows(double* s, int r0, int c0) {
  double c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
  panel_times_x(s, r0, c0, c);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) panel_entry(s, r0, c0, h, r) = c[h][r];
}

// The same with one step of refinement, P += (A − P L_ppᵀ) X_ppᵀ, which brings the
// residual back to that of a substitution.  Measured (rms error of one evaluation
// against 80-bit arithmetic, RBF, 64 points in ten lengthscales, noise 1e-5: NLML,
// gradient, α): substitution 5.0e-12, 1.6e-11, 3.0e-11; the product alone 4.6e-11,
// 1.0e-10, 4.9e-10; refined 5.7e-12, 1.2e-11, 3.3e-11; at noise 0.1 all three 1e-15.
// Out of line: few leaves take it, and the batched kernels have no registers for it.
static __device__ __noinline__ void panel_rows_refined(double* s, const double* ldiag, int r0, int c0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  double c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}}, a[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) a[h][r] = panel_entry(s, r0, c0, h, r);
  panel_times_x(s, r0, c0, c);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) panel_entry(s, r0, c0, h, r) = c[h][r];
  __syncwarp();
#pragma unroll
  for (int kk = 0; kk < LF; kk += 4) {  // a −= P L_ppᵀ
    const int k = kk + t4;
    const double a0 = -s[r0 + g + (c0 + k) * FLS], a1 = -s[r0 + g + 8 + (c0 + k) * FLS];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 8 * h + g;
      dmma_16x8x4(a[h], a0, a1, k < j ? s[c0 + j + (c0 + k) * FLS] : k == j ? ldiag[c0 + k] : 0.0);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) panel_entry(s, r0, c0, h, r) = a[h][r];
  __syncwarp();
  panel_times_x(s, r0, c0, c);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) panel_entry(s, r0, c0, h, r) = c[h][r];
}

// One lower 16×16 tile of A[rbeg.., cbeg..] −= Σ_{k<K} L[rbeg+i, k0+k] L[cbeg+j, k0+k]
// (entries above the diagonal are left alone; both column halves share the A
// fragments, so that the loads do not crowd out the leaf's).
__device__ __forceinline__ void syrk_tile(double* s, int rbeg, int cbeg, int k0, int K) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const double* a = s + rbeg + g + (k0 + t4) * FLS;
  const double* b = s + cbeg + g + (k0 + t4) * FLS;
  double c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll 4
  for (int kk = 0; kk < K; kk += 4) {
    const double a0 = a[kk * FLS], a1 = a[kk * FLS + 8];
    dmma_16x8x4(c[0], a0, a1, b[kk * FLS]);
    dmma_16x8x4(c[1], a0, a1, b[kk * FLS + 8]);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = rbeg + g + ((r & 2) ? 8 : 0), col = cbeg + 8 * h + 2 * t4 + (r & 1);
      if (row >= col) s[row + col * FLS] -= c[h][r];
    }
}

// 16×16 tiles of a 16-column block from row r0 to npad.
__device__ __forceinline__ int colblock_tiles(int r0, int npad) { return (npad - r0) / 16; }

// The 16×16 leaf inverse of block q (one warp): lane c computes column c of
// L_qq⁻¹ by substitution; X(i, c) goes to s[c + i·FLS] (i ≥ c: the diagonal
// and the transposed slot above it).
__device__ __forceinline__ void leaf16_inverse(double* s, int q, const double* rinv) {
  const int lane = threadIdx.x & 31, c = lane & 15, off = q * LF;
  double acc[LF];
#pragma unroll
  for (int i = 0; i < LF; ++i) acc[i] = (i == c) ? 1.0 : 0.0;
#pragma unroll
  for (int t = 0; t < LF; ++t) {
    const double x = acc[t] * rinv[off + t];
    acc[t] = x;
#pragma unroll
    for (int j = t + 1; j < LF; ++j) acc[j] = fma(-s[(off + j) + (off + t) * FLS], x, acc[j]);
  }
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < LF; ++i)
      if (i >= c) s[(off + c) + (off + i) * FLS] = acc[i];
  }
}

// T tile tn of block row q (a0 = 16q): T(:, j0..j0+7) = L_{q,<q}(:, kb..) X_{<q,<q}(kb.., j0..),
// k from kb = j0 rounded down to 4 (X(k, j) = 0 for k < j), T in tmp (ld TLD).
__device__ __forceinline__ void inv_t_tile(const double* s, double* tmp, int q, int tn) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int a0 = q * LF, j0 = 8 * tn, kb = j0 & ~3;
  double c[4] = {0, 0, 0, 0};
  // A(i, k) = L(a0 + i, kb + k);  B(k, j) = X(kb + k, j0 + j) = s[(j0 + j) + (kb + k)·FLS], 0 for kb + k < j0 + j
  mma_tile_smem<false, true>(c, s + a0 + kb * FLS, 1, FLS, s + j0 + kb * FLS, FLS, 1, a0 - kb, j0 - kb);
  const int row = g, col = j0 + 2 * t4;
  tmp[row + col * TLD] = c[0];
  tmp[row + (col + 1) * TLD] = c[1];
  tmp[(row + 8) + col * TLD] = c[2];
  tmp[(row + 8) + (col + 1) * TLD] = c[3];
}

// X tile tn of block row q: X(a0+i, j0+j) = −Σ_{k ≤ i} X_qq(i, k) T(k, j0+j), into the transposed slot.
__device__ __forceinline__ void inv_x_tile(double* s, const double* tmp, int q, int tn) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int a0 = q * LF, j0 = 8 * tn;
  double c[4] = {0, 0, 0, 0};
  // A(i, k) = X_qq(i, k) = s[(a0 + k) + (a0 + i)·FLS] for k ≤ i;  B(k, j) = T(k, j0 + j)
  mma_tile_smem<true, false>(c, s + a0 + a0 * FLS, FLS, 1, tmp + j0 * TLD, 1, TLD, LF, 0);
  const int row = a0 + g, col = j0 + 2 * t4;
  s[col + row * FLS] = -c[0];
  s[(col + 1) + row * FLS] = -c[1];
  s[col + (row + 8) * FLS] = -c[2];
  s[(col + 1) + (row + 8) * FLS] = -c[3];
}

// Stores of finished parts, one warp each.
// L column block q, columns q·16 + 8·half .. +8, rows from the diagonal (L_jj
// from ldiag; 16-byte stores from the first even row when vec).
__device__ __forceinline__ void store_l_part(const double* s, const double* ldiag, double* A, long long lda,
                                             long long k0, int nb, bool vec, int q, int half) {
  const int lane = threadIdx.x & 31;
  for (int j = q * LF + 8 * half; j < q * LF + 8 * half + 8 && j < nb; ++j) {
    double* col = A + k0 + (k0 + j) * lda;
    const double* sc = s + j * FLS;
    if (vec) {
      const int i0 = (j + 1) & ~1;
      if ((j & 1) && lane == 0) col[j] = ldiag[j];
      for (int i = i0 + 2 * lane; i + 1 < nb; i += 64)
        *reinterpret_cast<double2*>(col + i) = make_double2(i == j ? ldiag[j] : sc[i], sc[i + 1]);
      if (((nb - i0) & 1) && lane == 0) col[nb - 1] = (nb - 1 == j) ? ldiag[j] : sc[nb - 1];
    } else {
      for (int i = j + lane; i < nb; i += 32) col[i] = (i == j) ? ldiag[j] : sc[i];
    }
  }
}

// Block row q of X into linv (ld NB_DIAG, zero above the diagonal and in the
// padding), columns [part·cw, (part+1)·cw), cw = NB_DIAG / nparts.
__device__ __forceinline__ void store_x_part(const double* s, double* linv, int nb, int q, int part, int nparts) {
  const int lane = threadIdx.x & 31, cw = NB_DIAG / nparts;
  const int i = q * LF + 2 * (lane & 7);
  for (int jb = part * cw; jb < (part + 1) * cw; jb += 4) {
    const int j = jb + (lane >> 3);
    const double a = (i < nb && j < nb && j <= i) ? s[j + i * FLS] : 0.0;
    const double b = (i + 1 < nb && j < nb && j <= i + 1) ? s[j + (i + 1) * FLS] : 0.0;
    *reinterpret_cast<double2*>(linv + i + j * NB_DIAG) = make_double2(a, b);
  }
}

// cp.async.wait_group with a run-time count (0 ≤ n ≤ 7 groups left in flight)
__device__ __forceinline__ void cp_async_wait_n(int n) {
  switch (n < 0 ? 0 : n) {
    case 0: cp_async_wait<0>(); break;
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    case 4: cp_async_wait<4>(); break;
    case 5: cp_async_wait<5>(); break;
    case 6: cp_async_wait<6>(); break;
    default: cp_async_wait<7>(); break;
  }
}

// The work of step p that is off warp 0's chain.  Products (dealt over nh
// warps, h = this warp's index among them, −1: none): inverse block row
// q = p − 1 (T, then — after the barrier of the nh warps — X_{q,<q}) and the
// updates of column blocks p (panel p−1, below the leaf) and p+1 (panels
// 0..p−1).  Stores (over ns warps, index sh): L column block p−1
// and X block row p−2.  With tail, p = np and the whole CTA takes part in both
// (barriers are __syncthreads).
static __device__ void diag_helpers(double* s, double* tmp, const double* rinv, const double* ldiag, double* A, long long lda,
                             long long k0, int nb, double* linv, bool vec, int p, int np, int h, int nh, int sh, int ns,
                             bool tail) {
  const int npad = np * LF, c0 = p * LF, r1 = c0 + LF, q = p - 1;
  if (sh >= 0 && linv) {
    const int n_ls = p >= 1 ? 2 : 0, xs_parts = tail ? 4 : 2, n_xs = p >= 2 ? xs_parts : 0;
    for (int t = sh; t < n_ls + n_xs; t += ns) {
      if (t < n_ls) store_l_part(s, ldiag, A, lda, k0, nb, vec, q, t);
      else store_x_part(s, linv, nb, p - 2, t - n_ls, xs_parts);
    }
  }
  if (h < 0) return;
  const int n_t = p >= 2 ? 2 * q : 0;
  const int n_next = (!tail && p >= 1 && p + 1 < np) ? colblock_tiles(r1, npad) : 0;
  const int n_cur = (!tail && p >= 1 && r1 < npad) ? colblock_tiles(r1, npad) : 0;
  const int total = n_t + n_next + n_cur;
  for (int t = h; t < total; t += nh) {
    int u = t;
    if (u < n_t) { inv_t_tile(s, tmp, q, u); continue; }
    u -= n_t;
    if (u < n_next) {  // column block p+1, rows from r1, panels 0..p−1
      syrk_tile(s, r1 + 16 * u, r1, 0, c0);
      continue;
    }
    u -= n_next;  // column block p below the leaf, panel p−1
    syrk_tile(s, r1 + 16 * u, c0, c0 - LF, LF);
  }
  if (p < 2) return;
  if (tail) __syncthreads();
  else asm volatile("bar.sync 1, %0;" ::"r"(32 * nh) : "memory");
  for (int t = h; t < 2 * q; t += nh) inv_x_tile(s, tmp, q, t);
}

// Identity padding of the block's lower part up to a multiple of 16.
static __device__ __forceinline__ void diag_block_pad(double* s, int nb) {
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int npad = (nb + LF - 1) / LF * LF;
  if (nb < npad)
    for (int j = warp; j < npad; j += nw)
      for (int i = j + lane; i < npad; i += 32)
        if (i >= nb || j >= nb) s[i + j * FLS] = (i == j) ? 1.0 : 0.0;
}

// Factor and inverse of the nb×nb lower block in s (its column blocks possibly
// still arriving, one cp.async group each; padded with the identity): L below
// the diagonal of s, X in the transposed slots, and — unless linv is null — L
// back to (k0, k0) of A and X to linv (ld NB_DIAG, zero above the diagonal).
// smem: diag_block_smem() bytes from s on; fail_sh a shared int.  Returns the
// failing column (uniform over the CTA) or −1.
static __device__ int diag_block_core(double* A, long long lda, long long k0, int nb, double* linv, bool vec,
                                      double* smem, int* fail_sh) {
  int& fail = *fail_sh;
  double* s = smem;                  // NB_DIAG × FLS
  double* tmp = s + NB_DIAG * FLS;   // TMP_DOUBLES
  double* rinv = tmp + TMP_DOUBLES;  // NB_DIAG reciprocal pivots
  double* ldiag = rinv + NB_DIAG;    // NB_DIAG diagonal entries of L
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int npad = (nb + LF - 1) / LF * LF, np = npad / LF;
  if (threadIdx.x == 0) fail = -1;
  cp_async_wait_n(np - 2);  // column blocks 0 and 1
  __syncthreads();
  for (int p = 0; p < np; ++p) {
    const int c0 = p * LF, r1 = c0 + LF;
    if (warp == 0) {
      if (p > 0) {  // the leaf's last update: panel p−1
        syrk_tile(s, c0, c0, c0 - LF, LF);
        __syncwarp();
      }
      const int f = leaf16_factor(s, c0, rinv, ldiag);
      if (f >= 0 && lane == 0) fail = c0 + f;
    } else {
      // the warps that share warp 0's scheduler (and its FP64 pipe, which a
      // DMMA holds for 32 cycles) store; the others multiply
      const bool store = (warp & 3) == 0;
      diag_helpers(s, tmp, rinv, ldiag, A, lda, k0, nb, linv, vec, p, np, store ? -1 : warp - 1 - warp / 4,
                   nw - nw / 4, store ? warp / 4 - 1 : -1, nw / 4 - 1, false);
    }
    __syncthreads();
    if (fail >= 0) break;
    // panel: 16 rows below the leaf per warp
    if (r1 + 16 * warp < npad) {
      const bool fix = leaf_spread(ldiag + c0);
      for (int r0 = r1 + 16 * warp; r0 < npad; r0 += 16 * nw) {
        if (fix) panel_rows_refined(s, ldiag, r0, c0);
        else panel_rows(s, r0, c0);
      }
    }
    cp_async_wait_n(np - 3 - p);  // column block p+2, used by the next step's helpers
    __syncthreads();
  }
  if (fail >= 0) {
    cp_async_wait<0>();
    __syncthreads();
    return fail;
  }
  // the last block row of X, the last column block of L, the last two block
  // rows of X into linv (all warps)
  diag_helpers(s, tmp, rinv, ldiag, A, lda, k0, nb, linv, vec, np, np, warp, nw, warp, nw, true);
  __syncthreads();
  if (!linv) return -1;
  // block rows np−1 .. NB_DIAG/16 − 1 (those past the block are zeros)
  for (int t = warp; t < (NB_DIAG / LF - np + 1) * 4; t += nw) store_x_part(s, linv, nb, np - 1 + t / 4, t % 4, 4);
  __syncthreads();
  return -1;
}

// The whole diagonal-block step for one CTA: load the nb×nb lower block at
// (k0, k0) of A, factor it (L back into A), invert it (L⁻¹ into linv).  Returns
// as diag_block_core; either way no copy into shared memory is in flight on
// return.
static __device__ int diag_block_factor_inv(double* A, long long lda, long long k0, int nb, double* linv, double* smem,
                                            int* fail_sh) {
  double* s = smem;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, np = (nb + LF - 1) / LF;
  // column block q is cp.async group q of every thread (16-byte copies from
  // the even row at or above the diagonal): blocks 0 and 1 are waited for, the
  // rest arrives during the first steps
  const bool vec = ((lda & 1) == 0) && ((((unsigned long long)(A + k0 + k0 * lda)) & 15) == 0);
  for (int q = 0; q < np; ++q) {
    for (int j = q * LF + warp; j < q * LF + LF && j < nb; j += nw) {
      if (vec) {
        for (int i = (j & ~1) + 2 * lane; i < nb; i += 64) {
          if (i + 1 < nb) {
            unsigned sa = (unsigned)__cvta_generic_to_shared(s + i + j * FLS);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(A + (k0 + i) + (k0 + j) * lda));
          } else {
            cp_async8(s + i + j * FLS, A + (k0 + i) + (k0 + j) * lda, true);
          }
        }
      } else {
        for (int i = j + lane; i < nb; i += 32) cp_async8(s + i + j * FLS, A + (k0 + i) + (k0 + j) * lda, true);
      }
    }
    cp_async_commit();
  }
  diag_block_pad(s, nb);  // the copies never reach these entries
  return diag_block_core(A, lda, k0, nb, linv, vec, smem, fail_sh);
}

inline size_t diag_block_smem() { return (size_t)(NB_DIAG * FLS + TMP_DOUBLES + 2 * NB_DIAG) * sizeof(double); }

}  // namespace gprx
