// dense_f64.cu — blocked FP64 Cholesky, triangular inverse, Xᵀ X and
// triangular solves on the DMMA GEMM (gemm_f64.cuh).
//
// Replaces faer's llt::factor::cholesky_in_place (gprx src/linalg/chol.rs:141-167),
// llt::solve (chol.rs:334-339, src/workspace.rs:395-425) and
// solve_lower_triangular_in_place (src/gpr/shared.rs:831-842).
//
// Layout: column-major, element (i, j) at i + j·ld, lower triangle.  A panel
// width NB = 128 matches the GEMM tile so the panel solve and the diagonal
// block applications can run in place (one CTA covers a whole panel row /
// column strip and reads it fully before writing).

#include <algorithm>

#include "dense_f64.cuh"
#include "emu_gemm.cuh"
#include "diag_block.cuh"

namespace gprx {

// 64×64 tiles of four warps (32×32 each, 57 KB, three to four CTAs a SM): one
// CTA's barriers and epilogue hide behind the others' DMMAs.  Measured against
// the 128×128 tile of eight warps (one CTA a SM), TF/s: 4096³ 29.7 / 28.0,
// 512 × 65536 with K = 512 28.8 / 26.2 (A transposed 29.1 / 26.5), A·Aᵀ of
// 1024 × 65536 split over K 31.1 / 27.7, K = 128 22.3 / 17.3; the sums run over
// k in the same order for every tile shape.
template <bool TA, bool TB>
static cudaError_t dgemm_wide(const GemmParams& p, cudaStream_t s, int batch) {
  return launch_dgemm<64, 64, 16, 32, 32, 3, TA, TB>(p, batch, s);
}

// Output tiles of a product (LOWER_TILES: those not strictly above the diagonal).
static long long gemm_tiles(const GemmParams& p, int bm, int bn) {
  const int tm = ceil_div(p.M, bm), tn = ceil_div(p.N, bn);
  if (!(p.mode & GEMM_LOWER_TILES)) return (long long)tm * tn;
  long long c = 0;
  for (int j = 0; j < tn; ++j) {
    const long long need = p.col0 + (long long)j * bn - p.row0 - (bm - 1);
    c += std::max(0LL, tm - (need <= 0 ? 0 : (need + bm - 1) / bm));
  }
  return c;
}

// The tile by how many the product has: few tiles leave SMs idle, and the
// longest k range decides when triangular operands give the tiles different
// lengths, so below four 64×64 tiles a SM the tile is 32×64 (k chunks of 32 in
// four stages, eight warps of 16×16: one memory latency a product).  Measured
// (µs, 128×128 / 64×64 / 32×64): Xᵀ X of n = 512 92 / 37 / 21, n = 1537
// 264 / 115 / 80, n = 2048 347 / 178 / 153, n = 3000 506 / 377 / 429; a
// triangular product of n = 256 49 / 21 / 13, n = 1000 176 / 88 / 83, n = 2048
// 555 / 414 / 443, n = 3000 1390 / 1079 / 1281.
template <bool TA, bool TB>
static cudaError_t dgemm_fill(const GemmParams& p, cudaStream_t s, int batch) {
  const int z = (p.mode & GEMM_SPLIT_K) ? p.splits : batch;
  if (gemm_tiles(p, 64, 64) * z >= 4 * B200_SMS) return dgemm_wide<TA, TB>(p, s, batch);
  return launch_dgemm<32, 64, 32, 16, 16, 4, TA, TB>(p, batch, s);
}

cudaError_t dgemm(bool ta, bool tb, const GemmParams& p, cudaStream_t s, int batch) {
  if (!ta && !tb) return dgemm_fill<false, false>(p, s, batch);
  if (!ta && tb) return dgemm_fill<false, true>(p, s, batch);
  if (ta && !tb) return dgemm_fill<true, false>(p, s, batch);
  return dgemm_fill<true, true>(p, s, batch);
}

// B := A·B or Aᵀ·B in place (M, K ≤ 128): one tile holds every row of its
// columns and reads them all before it writes.
static cudaError_t dgemm_inplace(bool ta, const GemmParams& p, cudaStream_t s) {
  if (p.M > 128) return cudaErrorInvalidValue;
  if (ta) return launch_dgemm<128, 64, 32, 64, 16, 2, true, false>(p, 1, s);
  return launch_dgemm<128, 64, 32, 64, 16, 2, false, false>(p, 1, s);
}

GemmParams gemm_params(int M, int N, int K, const double* A, long long lda, const double* B, long long ldb,
                       double* C, long long ldc, double alpha, double beta, const DevStatus* st) {
  GemmParams p{};
  p.M = M;
  p.N = N;
  p.K = K;
  p.A = A;
  p.lda = lda;
  p.B = B;
  p.ldb = ldb;
  p.C = C;
  p.ldc = ldc;
  p.alpha = alpha;
  p.beta = beta;
  p.mode = 0;
  p.row0 = p.col0 = p.krow0 = 0;
  p.splits = 1;
  p.split_stride = 0;
  p.status = st;
  p.strideA = p.strideB = p.strideC = 0;
  p.tiles = 0;
  return p;
}

// ---------------------------------------------------------------------------
// diagonal block: factor and invert in shared memory
// ---------------------------------------------------------------------------
// Programmatic dependent launch on the factor's chain: a chain kernel first
// waits for its predecessor in the stream to complete (its writes visible),
// then lets its own dependent start launching, so the launch of the next
// chain kernel overlaps this one instead of following its completion.  Both
// instructions are no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void chain_dependency_wait_and_release() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__global__ void __launch_bounds__(FD_THREADS) potrf_diag_kernel(double* A, long long lda, long long k0, int nb,
                                                                 double* linv, DevStatus* st) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int fail;
  chain_dependency_wait_and_release();
  if (dev_failed(st)) return;
  int f = diag_block_factor_inv(A, lda, k0, nb, linv, smem, &fail);
  if (f >= 0 && threadIdx.x == 0) dev_fail(st, GPRX_CHOLESKY_FAILED, k0 + f);
}

// Inverse of one diagonal block per CTA, in the layout and with the tiles of
// the factor's diagonal step: the 16×16 leaf inverses in parallel, then block
// row q of X as X_qq (−L_{q,<q} X_{<q,<q}) on DMMA, two barriers a row.
// Latency-bound (eight rows in sequence, one CTA a block); the column by
// column form it replaces took 233 µs for the 16 blocks of n = 2000.
__global__ void __launch_bounds__(FD_THREADS) tri_inv_blocks_kernel(const double* L, long long ld, int n, bool unit,
                                                                    double* linv, DevStatus* st) {
  extern __shared__ __align__(16) double smem[];
  if (dev_failed(st)) return;
  double* s = smem;
  double* tmp = s + NB_DIAG * FLS;
  double* rinv = tmp + TMP_DOUBLES;
  const int tid = threadIdx.x, warp = tid >> 5, nw = FD_THREADS >> 5;
  const long long k0 = (long long)blockIdx.x * NB;
  const int nb = (int)min((long long)NB, n - k0), np = (nb + LF - 1) / LF, npad = np * LF;
  for (int e = tid; e < npad * npad; e += FD_THREADS) {
    const int i = e % npad, j = e / npad;
    if (i < j) continue;
    const bool in = i < nb;  // j ≤ i
    cp_async8(s + i + j * FLS, in ? L + (k0 + i) + (k0 + j) * ld : L, in);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  for (int i = tid; i < npad; i += FD_THREADS) rinv[i] = (unit || i >= nb) ? 1.0 : 1.0 / s[i + i * FLS];
  __syncthreads();
  for (int q = warp; q < np; q += nw) leaf16_inverse(s, q, rinv);
  __syncthreads();
  for (int q = 1; q < np; ++q) {
    for (int t = warp; t < 2 * q; t += nw) inv_t_tile(s, tmp, q, t);
    __syncthreads();
    for (int t = warp; t < 2 * q; t += nw) inv_x_tile(s, tmp, q, t);
    __syncthreads();
  }
  double* out = linv + (long long)blockIdx.x * NB * NB;
  for (int t = warp; t < (NB_DIAG / LF) * 4; t += nw) store_x_part(s, out, nb, t / 4, t % 4, 4);
}

static size_t fast_diag_smem(int nb) { (void)nb; return diag_block_smem(); }

static cudaError_t diag_attrs() {
  static SmemAllowed factor, inverse;
  const cudaError_t e = factor((const void*)potrf_diag_kernel, fast_diag_smem(NB));
  return e != cudaSuccess ? e : inverse((const void*)tri_inv_blocks_kernel, fast_diag_smem(NB));
}

#define CK(x)                                \
  do {                                       \
    cudaError_t e_ = (x);                    \
    if (e_ != cudaSuccess) return e_;        \
  } while (0)

FactorCtx::~FactorCtx() {
  for (auto e : ev) cudaEventDestroy(e);
  for (auto e : side)
    if (e) cudaEventDestroy(e);
}

cudaError_t FactorCtx::ensure(int nblk) {
  CK(lane.open_sides());
  for (auto& e : side)
    if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  while ((int)ev.size() < 3 * nblk + 2) {
    cudaEvent_t e;
    CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ev.push_back(e);
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// the chain's panel products: K ≤ NB, N ≤ NB
// ---------------------------------------------------------------------------
// C(M×N) = alpha · A(M×K) · B(N×K)ᵀ + beta · C with A(i,k) = A[i + k·lda],
// B(j,k) = B[j + k·ldb], C column-major; lower: only i ≥ j is written; tri: B is
// lower triangular (B(j,k) = 0 for k > j), so a warp's k range ends at its last
// column.  One CTA of 256 threads per TM-row strip stages the strip of A and all
// of B in shared memory in one go (K is one panel: no k pipeline, one memory
// latency instead of one per k chunk), prefetches its C values meanwhile,
// then runs the DMMA k steps.  A strip is read whole before it is written,
// so C may be A's rows when beta = 0 (the in-place panel solve).
//
// TM = 16 while the strips fit one wave of SMs (M ≤ 16·148), else 32: a strip of
// 32 rows holds its SM's DMMA pipe for 8192 cycles (4.2 µs), one of 16 rows for
// 4096, for 2304 with a triangular B.  Each scheduler gets two warps whose column
// blocks add up to the same k steps.
constexpr int PG_TM = 32;
constexpr int PG_LDB = NB + 4;
template <int TM>
constexpr int pg_lda() { return TM + 4; }  // ≡ 4 mod 16 doubles: conflict-free fragments
template <int TM>
inline size_t panel_gemm_smem() { return (size_t)(NB * pg_lda<TM>() + NB * PG_LDB) * sizeof(double); }

struct PanelGemmArgs {
  int M, N, K;
  const double* A;
  long long lda;
  const double* B;
  long long ldb;
  double* C;
  long long ldc;
  double alpha, beta;
  int lower, tri;
  const DevStatus* st;
};

template <int TM>
__global__ void __launch_bounds__(256) panel_gemm_kernel(PanelGemmArgs g) {
  constexpr int LDA = pg_lda<TM>(), NJ = TM / 8;  // warps: 16 rows × 8·NJ columns
  extern __shared__ __align__(16) double smem[];
  chain_dependency_wait_and_release();
  if (dev_failed(g.st)) return;
  double* sA = smem;             // [k][i], ld LDA
  double* sB = smem + NB * LDA;  // [k][j], ld PG_LDB
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t4 = lane & 3;
  const int m0 = blockIdx.x * TM;
  const int KP = (g.K + 3) & ~3;
  const bool a16 = ((g.lda & 1) == 0) && ((reinterpret_cast<unsigned long long>(g.A) & 15) == 0);
  const bool b16 = ((g.ldb & 1) == 0) && ((reinterpret_cast<unsigned long long>(g.B) & 15) == 0);
  // A strip: TM × KP (zero past M and K)
  if (a16) {
    for (int e = tid; e < (TM / 2) * KP; e += 256) {
      const int i = 2 * (e % (TM / 2)), k = e / (TM / 2), gi = m0 + i;
      const int bytes = (gi < g.M && k < g.K) ? (gi + 1 < g.M ? 16 : 8) : 0;
      const unsigned d = (unsigned)__cvta_generic_to_shared(sA + k * LDA + i);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d),
                   "l"(bytes ? g.A + gi + (long long)k * g.lda : g.A), "r"(bytes));
    }
  } else {
    for (int e = tid; e < TM * KP; e += 256) {
      const int i = e % TM, k = e / TM, gi = m0 + i;
      const bool ok = gi < g.M && k < g.K;
      cp_async8(sA + k * LDA + i, ok ? g.A + gi + (long long)k * g.lda : g.A, ok);
    }
  }
  // B: NB × KP (zero past N and K)
  if (b16) {
    for (int e = tid; e < (NB / 2) * KP; e += 256) {
      const int j = 2 * (e % (NB / 2)), k = e / (NB / 2);
      const int bytes = (j < g.N && k < g.K) ? (j + 1 < g.N ? 16 : 8) : 0;
      const unsigned d = (unsigned)__cvta_generic_to_shared(sB + k * PG_LDB + j);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d),
                   "l"(bytes ? g.B + j + (long long)k * g.ldb : g.B), "r"(bytes));
    }
  } else {
    for (int e = tid; e < NB * KP; e += 256) {
      const int j = e % NB, k = e / NB;
      const bool ok = j < g.N && k < g.K;
      cp_async8(sB + k * PG_LDB + j, ok ? g.B + j + (long long)k * g.ldb : g.B, ok);
    }
  }
  cp_async_commit();
  // TM = 32: a 2 × 4 grid of 16 × 32 blocks, columns 0 1 3 2; TM = 16: eight
  // blocks of 16 × 16, columns 0 1 2 3 7 6 5 4 (warps w and w + 4 share a scheduler)
  const int wm = TM == 32 ? warp & 1 : 0, w = TM == 32 ? warp >> 1 : warp;
  const int wn = TM == 32 ? (w < 2 ? w : 5 - w) : (w < 4 ? w : 11 - w);
  const int rb = wm * 16, cb = wn * 8 * NJ;
  const bool wskip = (cb >= g.N) || (g.lower && m0 + rb + 15 < cb);
  double cv[NJ][4];
#pragma unroll
  for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = m0 + rb + gq + ((r & 2) ? 8 : 0), col = cb + nj * 8 + 2 * t4 + (r & 1);
      const bool ok = !wskip && g.beta != 0.0 && row < g.M && col < g.N && !(g.lower && row < col);
      cv[nj][r] = ok ? g.C[row + (long long)col * g.ldc] : 0.0;
    }
  cp_async_wait<0>();
  __syncthreads();
  if (wskip) return;
  double acc[NJ][4];
#pragma unroll
  for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[nj][r] = 0.0;
  const int ke = g.tri ? min(KP, cb + 8 * NJ) : KP;
#pragma unroll 4
  for (int kk = 0; kk < ke; kk += 4) {
    const double a0 = sA[(kk + t4) * LDA + rb + gq];
    const double a1 = sA[(kk + t4) * LDA + rb + gq + 8];
    double b[NJ];
#pragma unroll
    for (int nj = 0; nj < NJ; ++nj) b[nj] = sB[(kk + t4) * PG_LDB + cb + nj * 8 + gq];
#pragma unroll
    for (int nj = 0; nj < NJ; ++nj) dmma_16x8x4(acc[nj], a0, a1, b[nj]);
  }
#pragma unroll
  for (int nj = 0; nj < NJ; ++nj)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = m0 + rb + gq + ((r & 2) ? 8 : 0), col = cb + nj * 8 + 2 * t4 + (r & 1);
      if (row < g.M && col < g.N && !(g.lower && row < col)) {
        double v = g.alpha * acc[nj][r];
        if (g.beta != 0.0) v = fma(g.beta, cv[nj][r], v);
        g.C[row + (long long)col * g.ldc] = v;
      }
    }
}

// launch with programmatic stream serialization (the kernel waits for its
// predecessor itself: chain_dependency_wait_and_release)
template <typename... Params, typename... Args>
static cudaError_t launch_chain(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int TM>
static cudaError_t panel_gemm_launch(const PanelGemmArgs& g, cudaStream_t s, bool chained) {
  static SmemAllowed allowed;
  CK(allowed((const void*)panel_gemm_kernel<TM>, panel_gemm_smem<TM>()));
  if (chained)
    return launch_chain(panel_gemm_kernel<TM>, dim3(ceil_div(g.M, TM)), dim3(256), panel_gemm_smem<TM>(), s, g);
  GPRX_LAUNCH(panel_gemm_kernel<TM>, ceil_div(g.M, TM), 256, panel_gemm_smem<TM>(), s, g);
  return cudaGetLastError();
}

static cudaError_t panel_gemm(int M, int N, int K, const double* A, long long lda, const double* B, long long ldb,
                              double* C, long long ldc, double alpha, double beta, bool lower, bool tri,
                              const DevStatus* st, cudaStream_t s, bool chained = false) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  if (N > NB || K > NB || K < 0) return cudaErrorInvalidValue;
  const PanelGemmArgs g{M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, lower ? 1 : 0, tri ? 1 : 0, st};
  return M <= 16 * B200_SMS ? panel_gemm_launch<16>(g, s, chained) : panel_gemm_launch<PG_TM>(g, s, chained);
}

// rows below the diagonal block up to which the chain uses dependent launch
// (at larger trailing blocks the bulk update fills the GPU, and panel CTAs
// launched early would sit waiting on SMs it could use)
constexpr int CHAIN_PDL_ROWS = 4096;

// The diagonal block at k0 and the panel below it.  before_panel: an event
// the panel waits for (the rest of the column update on another stream).
static cudaError_t diag_and_panel(double* A, long long ld, int n, int k0, double* linv, DevStatus* st,
                                  cudaStream_t s, cudaEvent_t before_panel = nullptr) {
  int nbk = min(NB, n - k0);
  double* lk = linv + (long long)(k0 / NB) * NB * NB;
  int rest = n - k0 - nbk;
  const bool chained = rest <= CHAIN_PDL_ROWS;
  if (chained) {
    CK(launch_chain(potrf_diag_kernel, dim3(1), dim3(FD_THREADS), fast_diag_smem(nbk), s, A, ld, (long long)k0, nbk,
                    lk, st));
  } else {
    GPRX_LAUNCH(potrf_diag_kernel, 1, FD_THREADS, fast_diag_smem(nbk), s, A, ld, (long long)k0, nbk, lk, st);
  }
  if (rest > 0) {
    double* P = A + (k0 + nbk) + (long long)k0 * ld;
    // panel: P := P · L_kk⁻ᵀ, i.e. P(i,j) = Σ_k P(i,k) L_kk⁻¹(j,k) (in place:
    // a strip is staged whole before it is written); after an event wait the
    // launch is a plain one
    if (before_panel) CK(cudaStreamWaitEvent(s, before_panel, 0));
    CK(panel_gemm(rest, nbk, nbk, P, ld, lk, NB, P, ld, 1.0, 0.0, false, true, st, s, chained && !before_panel));
  }
  return cudaGetLastError();
}

// The bulk trailing update of the look-ahead factor (K = NB) runs on 64×64
// tiles of four warps: CTAs short enough that the chain's high-priority kernels
// get SMs as they retire (no SM is held back).  Measured (evaluation, n = 1537
// / 8192): 1.04 / 24.0 ms, against 1.03 / 24.2 ms on 64×128 tiles of eight
// warps; 128×128 tiles capped at 132 CTAs took 11.67 ms for the n = 8192 factor
// where the 64×128 tiles took 10.35 ms.

cudaError_t potrf_blocked(double* A, long long ld, int n, double* linv, DevStatus* st, cudaStream_t s,
                          FactorCtx* ctx) {
  CK(diag_attrs());
  const int nblk = ceil_div(n, NB);
  if (!ctx) {
    for (int k0 = 0; k0 < n; k0 += NB) {
      CK(diag_and_panel(A, ld, n, k0, linv, st, s));
      int nbk = min(NB, n - k0), rest = n - k0 - nbk;
      if (rest <= 0) break;
      double* P = A + (k0 + nbk) + (long long)k0 * ld;
      double* A22 = A + (k0 + nbk) + (long long)(k0 + nbk) * ld;
      GemmParams ps = gemm_params(rest, rest, nbk, P, ld, P, ld, A22, ld, -1.0, 1.0, st);
      ps.mode = GEMM_LOWER_TILES;
      CK(dgemm(false, true, ps, s));
    }
    return cudaGetLastError();
  }
  CK(ctx->ensure(nblk));
  cudaStream_t X = ctx->lane.aux();
  cudaEvent_t* Ep = ctx->ev.data();          // panel k done (on X)
  cudaEvent_t* Es = ctx->ev.data() + nblk;   // trailing update of step k done (on s)
  cudaEvent_t* Ec = ctx->ev.data() + 2 * nblk + 2;  // column update's lower rows of step k done (on aux2)
  cudaEvent_t Ein = ctx->ev[2 * nblk];
  cudaStream_t X2 = ctx->lane.aux2();
  CK(cudaEventRecord(Ein, s));
  CK(cudaStreamWaitEvent(X, Ein, 0));
  CK(diag_and_panel(A, ld, n, 0, linv, st, X));
  CK(cudaEventRecord(Ep[0], X));
  int last = 0;
  for (int k = 0; k < nblk; ++k) {
    const int c1 = (k + 1) * NB;  // first column of block k+1
    if (c1 >= n) break;
    const int k0 = k * NB;
    const double* Pk = A + c1 + (long long)k0 * ld;  // panel k, rows from c1
    // critical chain of block k+1 (side stream): column block k+1 −= panel
    // k · (its top rows)ᵀ — the diagonal block's rows on the chain, the rows
    // below on aux2 while the diagonal block is factored; the panel solve
    // waits for both
    if (k >= 1) CK(cudaStreamWaitEvent(X, Es[k - 1], 0));
    const int m = n - c1, w = min(NB, n - c1);
    cudaEvent_t lower_done = nullptr;
    if (m > NB) {
      if (k >= 1) CK(cudaStreamWaitEvent(X2, Es[k - 1], 0));
      CK(cudaStreamWaitEvent(X2, Ep[k], 0));
      CK(panel_gemm(m - NB, w, NB, Pk + NB, ld, Pk, ld, A + (c1 + NB) + (long long)c1 * ld, ld, -1.0, 1.0, false,
                    false, st, X2));
      CK(cudaEventRecord(Ec[k], X2));
      lower_done = Ec[k];
    }
    CK(panel_gemm(min(m, NB), w, NB, Pk, ld, Pk, ld, A + c1 + (long long)c1 * ld, ld, -1.0, 1.0, true, false, st,
                  X));
    CK(diag_and_panel(A, ld, n, c1, linv, st, X, lower_done));
    CK(cudaEventRecord(Ep[k + 1], X));
    last = k + 1;
    // bulk trailing update of step k (main stream): columns from c2
    CK(cudaStreamWaitEvent(s, Ep[k], 0));
    const int c2 = c1 + NB;
    if (c2 < n) {
      int m = n - c2;
      const double* Pk2 = A + c2 + (long long)k0 * ld;
      GemmParams ps = gemm_params(m, m, NB, Pk2, ld, Pk2, ld, A + c2 + (long long)c2 * ld, ld, -1.0, 1.0, st);
      ps.mode = GEMM_LOWER_TILES;
      CK((launch_dgemm<64, 64, 16, 32, 32, 3, false, true>(ps, 1, s)));
    }
    CK(cudaEventRecord(Es[k], s));
  }
  CK(cudaStreamWaitEvent(s, Ep[last], 0));
  return cudaGetLastError();
}

cudaError_t tri_inv_blocks(const double* L, long long ld, int n, bool unit, double* linv, DevStatus* st,
                           cudaStream_t s) {
  CK(diag_attrs());
  int nblk = ceil_div(n, NB);
  if (nblk == 0) return cudaSuccess;
  GPRX_LAUNCH(tri_inv_blocks_kernel, nblk, FD_THREADS, fast_diag_smem(NB), s, L, ld, n, unit, linv, st);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// identity / triangular inverse / Xᵀ X
// ---------------------------------------------------------------------------
__global__ void set_identity_kernel(double* X, long long ld, int n) {
  long long total = (long long)n * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    int i = (int)(e % n), j = (int)(e / n);
    X[i + j * ld] = (i == j) ? 1.0 : 0.0;
  }
}

cudaError_t set_identity(double* X, long long ld, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  long long total = (long long)n * n;
  int blocks = (int)std::min<long long>((total + 255) / 256, (long long)B200_SMS * 16);
  GPRX_LAUNCH(set_identity_kernel, blocks, 256, 0, s, X, ld, n);
  return cudaGetLastError();
}

// X = L⁻¹ by recursive doubling over the NB-blocks: the diagonal blocks are
// the inverses the factor left in linv; at each level every pair of sibling
// blocks gets X21 = −X22 (L21 X11), two batched triangular products with the
// k-ranges cut to the nonzero triangles.  X's strict upper triangle must be
// zero on entry (it is never written).  scratch holds ceil(n/2)² doubles.
// One CTA per 16 columns of a block (one CTA per block took 35 µs).
constexpr int CDB_COLS = 16;
__global__ void __launch_bounds__(NB) copy_diag_blocks_kernel(const double* linv, int n, double* X, long long ldx) {
  const long long k0 = (long long)blockIdx.x * NB;
  const int nb = (int)min((long long)NB, n - k0), i = threadIdx.x, j0 = blockIdx.y * CDB_COLS;
  if (i >= nb) return;
  const double* src = linv + (long long)blockIdx.x * NB * NB + i;
  double* dst = X + (k0 + i) + k0 * ldx;
#pragma unroll
  for (int j = j0; j < j0 + CDB_COLS; ++j)
    if (j < nb) dst[j * ldx] = src[j * NB];
}

static cudaError_t copy_diag_blocks(const double* linv, int n, double* X, long long ldx, cudaStream_t s) {
  GPRX_LAUNCH(copy_diag_blocks_kernel, dim3(ceil_div(n, NB), NB / CDB_COLS), NB, 0, s, linv, n, X, ldx);
  return cudaGetLastError();
}

cudaError_t trtri_blocked(const double* L, long long ld, int n, const double* linv, double* X, long long ldx,
                          double* scratch, DevStatus* st, cudaStream_t s) {
  CK(copy_diag_blocks(linv, n, X, ldx, s));
  for (long long b = 2LL * NB; b < 2LL * n; b *= 2) {
    long long h = b / 2;
    if (h >= n) break;
    long long full = n / b;            // pairs with both halves of size h
    long long r = n - full * b;        // tail: a pair when it reaches past h
    for (int part = 0; part < 2; ++part) {
      long long s0, cnt, h2;
      if (part == 0) {
        if (full == 0) continue;
        s0 = 0;
        cnt = full;
        h2 = h;
      } else {
        if (r <= h) continue;
        s0 = full * b;
        cnt = 1;
        h2 = r - h;
      }
      // T = L21 · X11   (h2 × h, K = h; X11 lower → k from the column)
      GemmParams p1 = gemm_params((int)h2, (int)h, (int)h, L + (s0 + h) + s0 * ld, ld, X + s0 + s0 * ldx, ldx,
                                  scratch, h2, 1.0, 0.0, st);
      p1.mode = GEMM_K_FROM_COL;
      p1.strideA = b + b * ld;
      p1.strideB = b + b * ldx;
      p1.strideC = h2 * h;
      CK(dgemm(false, false, p1, s, (int)cnt));
      // X21 = −X22 · T   (h2 × h, K = h2; X22 lower → k up to the row)
      GemmParams p2 = gemm_params((int)h2, (int)h, (int)h2, X + (s0 + h) + (s0 + h) * ldx, ldx, scratch, h2,
                                  X + (s0 + h) + s0 * ldx, ldx, -1.0, 0.0, st);
      p2.mode = GEMM_K_TO_ROW;
      p2.strideA = b + b * ldx;
      p2.strideB = h2 * h;
      p2.strideC = b + b * ldx;
      CK(dgemm(false, false, p2, s, (int)cnt));
    }
  }
  return cudaGetLastError();
}

cudaError_t trtri_blocked_emu(const double* L, long long ld, int n, const double* linv, double* X, long long ldx,
                              double* scratch, const EmuWork& w, int emu_min, DevStatus* st, cudaStream_t s) {
  CK(copy_diag_blocks(linv, n, X, ldx, s));
  for (long long b = 2LL * NB; b < 2LL * n; b *= 2) {
    long long h = b / 2;
    if (h >= n) break;
    long long full = n / b;
    long long r = n - full * b;
    for (int part = 0; part < 2; ++part) {
      long long s0, cnt, h2;
      if (part == 0) {
        if (full == 0) continue;
        s0 = 0;
        cnt = full;
        h2 = h;
      } else {
        if (r <= h) continue;
        s0 = full * b;
        cnt = 1;
        h2 = r - h;
      }
      if (h < emu_min) {
        GemmParams p1 = gemm_params((int)h2, (int)h, (int)h, L + (s0 + h) + s0 * ld, ld, X + s0 + s0 * ldx, ldx,
                                    scratch, h2, 1.0, 0.0, st);
        p1.mode = GEMM_K_FROM_COL;
        p1.strideA = b + b * ld;
        p1.strideB = b + b * ldx;
        p1.strideC = h2 * h;
        CK(dgemm(false, false, p1, s, (int)cnt));
        GemmParams p2 = gemm_params((int)h2, (int)h, (int)h2, X + (s0 + h) + (s0 + h) * ldx, ldx, scratch, h2,
                                    X + (s0 + h) + s0 * ldx, ldx, -1.0, 0.0, st);
        p2.mode = GEMM_K_TO_ROW;
        p2.strideA = b + b * ldx;
        p2.strideB = h2 * h;
        p2.strideC = b + b * ldx;
        CK(dgemm(false, false, p2, s, (int)cnt));
        continue;
      }
      for (long long c = 0; c < cnt; ++c) {
        const long long o = s0 + c * b;
        // T = L21 · X11 (rows of L21 against the columns of X11; X11 lower:
        // k from the tile's first column)
        EmuOperand a = w.op_a((int)h2, (int)h), bo = w.op_b((int)h, (int)h);
        CK(emu_slice(L + (o + h) + o * ld, ld, false, a, s));
        CK(emu_slice(X + o + o * ldx, ldx, true, bo, s));
        CK(emu_gemm(a, bo, scratch, h2, 1.0, 0.0, false, 0, 0, 2, w.err, s));
        // X21 = −X22 · T (X22 lower: k up to the tile's last row)
        EmuOperand a2 = w.op_a((int)h2, (int)h2), b2 = w.op_b((int)h, (int)h2);
        CK(emu_slice(X + (o + h) + (o + h) * ldx, ldx, false, a2, s));
        CK(emu_slice(scratch, h2, true, b2, s));
        CK(emu_gemm(a2, b2, X + (o + h) + o * ldx, ldx, -1.0, 0.0, false, 0, 0, 3, w.err, s));
      }
    }
  }
  return cudaGetLastError();
}

cudaError_t potrf_trtri_rec(double* A, long long ld, int n, double* X, long long ldx, double* linv,
                            double* scratch, const EmuWork& w, int leaf, int emu_min, DevStatus* st,
                            cudaStream_t s, FactorCtx* ctx) {
  if (n <= leaf) {
    CK(potrf_blocked(A, ld, n, linv, st, s, ctx));
    return trtri_blocked_emu(A, ld, n, linv, X, ldx, scratch, w, emu_min, st, s);
  }
  const int n1 = (n / 2 + NB - 1) / NB * NB, n2 = n - n1;
  CK(potrf_trtri_rec(A, ld, n1, X, ldx, linv, scratch, w, leaf, emu_min, st, s, ctx));
  double* A21 = A + n1;
  double* A22 = A + n1 + (long long)n1 * ld;
  // L21 = A21 X11ᵀ (rows of A21 against the rows of X11, k ≤ j), written over A21
  {
    EmuOperand a = w.op_a(n2, n1), b = w.op_b(n1, n1);
    CK(emu_slice(A21, ld, false, a, s));
    CK(emu_slice(X, ldx, false, b, s));
    CK(emu_gemm(a, b, A21, ld, 1.0, 0.0, false, 0, 0, 4, w.err, s));
  }
  // A22 −= L21 L21ᵀ (lower)
  {
    EmuOperand l = w.op_a(n2, n1);
    CK(emu_slice(A21, ld, false, l, s));
    CK(emu_gemm(l, l, A22, ld, -1.0, 1.0, true, 0, 0, 0, w.err, s));
  }
  CK(potrf_trtri_rec(A22, ld, n2, X + n1 + (long long)n1 * ldx, ldx, linv + (long long)(n1 / NB) * NB * NB, scratch,
                     w, leaf, emu_min, st, s, ctx));
  // T = L21 X11 (X11 lower: k from the tile's first column), X21 = −X22 T
  // (X22 lower: k up to the tile's last row)
  {
    EmuOperand a = w.op_a(n2, n1), b = w.op_b(n1, n1);
    CK(emu_slice(A21, ld, false, a, s));
    CK(emu_slice(X, ldx, true, b, s));
    CK(emu_gemm(a, b, scratch, n2, 1.0, 0.0, false, 0, 0, 2, w.err, s));
    EmuOperand a2 = w.op_a(n2, n2), b2 = w.op_b(n1, n2);
    CK(emu_slice(X + n1 + (long long)n1 * ldx, ldx, false, a2, s));
    CK(emu_slice(scratch, n2, true, b2, s));
    CK(emu_gemm(a2, b2, X + n1, ldx, -1.0, 0.0, false, 0, 0, 3, w.err, s));
  }
  return cudaGetLastError();
}

cudaError_t lauum_lower_emu(const double* X, long long ldx, int n, double* C, long long ldc, const EmuWork& w,
                            DevStatus* st, cudaStream_t s) {
  (void)st;
  // C(i, j) = Σ_k X(k,i) X(k,j): both operands are the rows of Xᵀ; lower,
  // k from the tile's first row
  EmuOperand a = w.op_a(n, n);
  CK(emu_slice(X, ldx, true, a, s));
  return emu_gemm(a, a, C, ldc, 1.0, 0.0, true, 0, 0, 1, w.err, s);
}

cudaError_t lauum_lower(const double* X, long long ldx, int n, double* C, long long ldc, DevStatus* st,
                        cudaStream_t s) {
  GemmParams p = gemm_params(n, n, n, X, ldx, X, ldx, C, ldc, 1.0, 0.0, st);
  p.mode = GEMM_LOWER_TILES | GEMM_K_FROM_ROW;
  return dgemm_fill<true, false>(p, s, 1);
}

// split point of a recursive solve: half of n rounded up to whole NB blocks
// (the diagonal-block inverses are indexed by row / NB)
static int rec_split(int n) { return ceil_div(ceil_div(n, 2), NB) * NB; }

// The block a class's recursion ends with: one tri_solve launch up to so many
// rows, or (SOLVE_BULK) one 128-row block times its inverse, in place.
static int solve_leaf(SolveClass cls, int n) {
  return cls == SOLVE_FEW ? n : cls == SOLVE_MID ? 512 : cls == SOLVE_WIDE ? 256 : NB;
}
static cudaError_t solve_block(SolveClass cls, const double* L, long long ld, int n, const double* linv, double* B,
                               long long ldb, int q, bool trans, DevStatus* st, cudaStream_t s) {
  if (cls != SOLVE_BULK) return tri_solve(L, ld, n, linv, B, ldb, q, trans, st, s);
  return dgemm_inplace(trans, gemm_params(n, q, n, linv, NB, B, ldb, B, ldb, 1.0, 0.0, st), s);
}

cudaError_t trsm_lower(SolveClass cls, const double* L, long long ld, int n, const double* linv, double* B, long long ldb,
                       int q, DevStatus* st, cudaStream_t s) {
  const int n1 = rec_split(n);
  if (n <= solve_leaf(cls, n) || n1 >= n) return solve_block(cls, L, ld, n, linv, B, ldb, q, false, st, s);
  const int n2 = n - n1;
  CK(trsm_lower(cls, L, ld, n1, linv, B, ldb, q, st, s));
  GemmParams p = gemm_params(n2, q, n1, L + n1, ld, B, ldb, B + n1, ldb, -1.0, 1.0, st);
  CK(dgemm(false, false, p, s));
  return trsm_lower(cls, L + n1 + (long long)n1 * ld, ld, n2, linv + (long long)(n1 / NB) * NB * NB, B + n1, ldb, q,
                    st, s);
}

cudaError_t trsm_lower_t(SolveClass cls, const double* L, long long ld, int n, const double* linv, double* B, long long ldb,
                         int q, DevStatus* st, cudaStream_t s) {
  const int n1 = rec_split(n);
  if (n <= solve_leaf(cls, n) || n1 >= n) return solve_block(cls, L, ld, n, linv, B, ldb, q, true, st, s);
  const int n2 = n - n1;
  CK(trsm_lower_t(cls, L + n1 + (long long)n1 * ld, ld, n2, linv + (long long)(n1 / NB) * NB * NB, B + n1, ldb, q, st,
                  s));
  GemmParams p = gemm_params(n1, q, n2, L + n1, ld, B + n1, ldb, B, ldb, -1.0, 1.0, st);
  CK(dgemm(true, false, p, s));
  return trsm_lower_t(cls, L, ld, n1, linv, B, ldb, q, st, s);
}

cudaError_t trsm_lower(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                       DevStatus* st, cudaStream_t s) {
  if (q == 1) return tri_solve_vec(L, ld, n, linv, B, false, st, s);
  return trsm_lower(solve_class(n, q), L, ld, n, linv, B, ldb, q, st, s);
}

cudaError_t trsm_lower_t(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                         DevStatus* st, cudaStream_t s) {
  if (q == 1) return tri_solve_vec(L, ld, n, linv, B, true, st, s);
  return trsm_lower_t(solve_class(n, q), L, ld, n, linv, B, ldb, q, st, s);
}

// ---------------------------------------------------------------------------
// reductions and matrix-vector products (HBM-bound)
// ---------------------------------------------------------------------------
__global__ void logdet_kernel(const double* L, long long ld, int n, bool ldlt, double* out, const DevStatus* st) {
  __shared__ double red[32];
  if (dev_failed(st)) return;
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += log(L[i + (long long)i * ld]);
  double s = block_sum(acc, red);
  if (threadIdx.x == 0) *out = ldlt ? s : 2.0 * s;
}

cudaError_t logdet_diag(const double* L, long long ld, int n, bool ldlt, double* out, DevStatus* st,
                        cudaStream_t s) {
  GPRX_LAUNCH(logdet_kernel, 1, 1024, 0, s, L, ld, n, ldlt, out, st);
  return cudaGetLastError();
}

// z_i = Σ_{j ≤ i} X_ij y_j: a block owns 32 rows and walks the columns.
constexpr int TRMV_ROWS = 32;
__global__ void __launch_bounds__(1024) trmv_lower_kernel(const double* X, long long ld, int n, const double* y,
                                                            double* z, const DevStatus* st) {
  constexpr int CG = 32;  // column groups: 32 rows × 32 groups, four loads in flight per thread
  __shared__ double part[CG][TRMV_ROWS + 1];
  if (dev_failed(st)) return;
  const int r = threadIdx.x % TRMV_ROWS, cg = threadIdx.x / TRMV_ROWS;
  const int i = blockIdx.x * TRMV_ROWS + r;
  const int jmax = min(n, (blockIdx.x + 1) * TRMV_ROWS);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (i < n) {
    int j = cg;
    for (; j + 3 * CG < jmax; j += 4 * CG) {
      const double x0 = j <= i ? X[i + (long long)j * ld] : 0.0;
      const double x1 = j + CG <= i ? X[i + (long long)(j + CG) * ld] : 0.0;
      const double x2 = j + 2 * CG <= i ? X[i + (long long)(j + 2 * CG) * ld] : 0.0;
      const double x3 = j + 3 * CG <= i ? X[i + (long long)(j + 3 * CG) * ld] : 0.0;
      a0 = fma(x0, y[j], a0);
      a1 = fma(x1, y[j + CG], a1);
      a2 = fma(x2, y[j + 2 * CG], a2);
      a3 = fma(x3, y[j + 3 * CG], a3);
    }
    for (; j < jmax; j += CG)
      if (j <= i) a0 = fma(X[i + (long long)j * ld], y[j], a0);
  }
  part[cg][r] = (a0 + a1) + (a2 + a3);
  __syncthreads();
  if (cg == 0 && i < n) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < CG; ++c) s += part[c][r];
    z[i] = s;
  }
}

cudaError_t trmv_lower(const double* X, long long ld, int n, const double* y, double* z, DevStatus* st,
                       cudaStream_t s) {
  GPRX_LAUNCH(trmv_lower_kernel, ceil_div(n, TRMV_ROWS), TRMV_ROWS * 32, 0, s, X, ld, n, y, z, st);
  return cudaGetLastError();
}

// Sum over one column: a warp's lanes or (BLOCK) a whole CTA of 256 threads;
// the first thread of the group gets it.
template <bool BLOCK>
__device__ __forceinline__ double column_sum(double acc) {
  __shared__ double red[32];
  return BLOCK ? block_sum(acc, red) : warp_sum(acc);
}

template <bool BLOCK>
__global__ void __launch_bounds__(256) gemv_t_kernel(const double* M, long long ld, int nrows, int ncols, bool lower,
                                                     const double* v, double* out, const DevStatus* st) {
  constexpr int G = BLOCK ? 256 : 32;
  if (dev_failed(st)) return;
  const int c = (blockIdx.x * 256 + threadIdx.x) / G, t = threadIdx.x % G;
  if (c >= ncols) return;
  const double* col = M + (long long)c * ld;
  double acc = 0.0;
  for (int i = (lower ? c : 0) + t; i < nrows; i += G) acc = fma(col[i], v[i], acc);
  acc = column_sum<BLOCK>(acc);
  if (t == 0) out[c] = acc;
}

cudaError_t gemv_t(const double* M, long long ld, int nrows, int ncols, bool lower, const double* v, double* out,
                   DevStatus* st, cudaStream_t s, bool block) {
  if (ncols <= 0) return cudaSuccess;
  if (block) GPRX_LAUNCH(gemv_t_kernel<true>, ncols, 256, 0, s, M, ld, nrows, ncols, lower, v, out, st);
  else GPRX_LAUNCH(gemv_t_kernel<false>, ceil_div((long long)ncols * 32, 256), 256, 0, s, M, ld, nrows, ncols, lower, v, out, st);
  return cudaGetLastError();
}

template <bool BLOCK>
__global__ void __launch_bounds__(256) col_sumsq_kernel(const double* M, long long ld, int nrows, int ncols,
                                                        const double* w, double* out, VarianceOf var,
                                                        const DevStatus* st) {
  constexpr int G = BLOCK ? 256 : 32;
  if (dev_failed(st)) return;
  const int c = (blockIdx.x * 256 + threadIdx.x) / G, t = threadIdx.x % G;
  if (c >= ncols) return;
  const double* col = M + (long long)c * ld;
  double acc = 0.0;
  for (int i = t; i < nrows; i += G) {
    const double v = col[i];
    acc = w ? fma(v, v / w[i], acc) : fma(v, v, acc);
  }
  acc = column_sum<BLOCK>(acc);
  if (t != 0) return;
  const double lat = var.kss - acc;
  out[c] = var.on ? (lat < 0.0 ? 0.0 : lat) + var.add : acc;  // a NaN stays one
}

cudaError_t col_sumsq(const double* M, long long ld, int nrows, int ncols, const double* w, double* out,
                      DevStatus* st, cudaStream_t s, bool block, VarianceOf var) {
  if (ncols <= 0) return cudaSuccess;
  const int grid = block ? ncols : ceil_div((long long)ncols * 32, 256);
  if (block) GPRX_LAUNCH(col_sumsq_kernel<true>, grid, 256, 0, s, M, ld, nrows, ncols, w, out, var, st);
  else GPRX_LAUNCH(col_sumsq_kernel<false>, grid, 256, 0, s, M, ld, nrows, ncols, w, out, var, st);
  return cudaGetLastError();
}

__global__ void dot_kernel(const double* a, const double* b, int n, double* out, const DevStatus* st) {
  __shared__ double red[32];
  if (dev_failed(st)) return;
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc = fma(a[i], b[i], acc);
  double s = block_sum(acc, red);
  if (threadIdx.x == 0) *out = s;
}

cudaError_t dot_dev(const double* a, const double* b, int n, double* out, DevStatus* st, cudaStream_t s) {
  GPRX_LAUNCH(dot_kernel, 1, 1024, 0, s, a, b, n, out, st);
  return cudaGetLastError();
}

}  // namespace gprx
