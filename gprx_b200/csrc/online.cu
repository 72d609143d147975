// online.cu — OnlineGpr on the device: LLT → LDLT, bordered append, row /
// column delete, lazy α.
//
// Reference: FittedGpr::into_online / LdltStore::fill_ld_from_llt
// (gprx src/gpr/fitted.rs:757-765, src/gpr/factor_store.rs:157-179),
// OnlineGpr::insert_with + LdltStore::append_border (src/gpr/online.rs:794-900,
// factor_store.rs:210-237), OnlineGpr::delete + LdltStore::delete_index →
// faer ldlt::update::delete_rows_and_cols_clobber (online.rs:564-611,
// factor_store.rs:239-255, src/linalg/ldlt.rs:113-122), the stale α solve
// (src/linalg/ldlt.rs:146-204) and IdRegistry (src/points.rs:76-190).
//
// The row/column delete is restated as the rank-1 LDLT update of the
// trailing block by D_k l_k l_kᵀ (Gill, Golub, Murray & Saunders 1974, C1):
// p = L⁻¹ w, the scalars in closed form from one running sum, then every entry
// from the sum of its own row up to its column block.

#include <algorithm>
#include <cmath>

#include "exact.cuh"

namespace gprx {

__global__ void llt_to_ldlt_kernel(double* A, long long ld, int n) {
  // column j: D_j = L_jj², L_ij ← L_ij / L_jj (i > j)
  int j = blockIdx.x;
  if (j >= n) return;
  double ljj = A[j + (long long)j * ld];
  for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) A[i + (long long)j * ld] /= ljj;
  __syncthreads();
  if (threadIdx.x == 0) A[j + (long long)j * ld] = ljj * ljj;
}

// Border of one appended point: w (in place in `w`) holds L⁻¹ k; writes
// v = D⁻¹ w into row n of A and δ = k_new − Σ w_i v_i onto the diagonal.
__global__ void ldlt_border_kernel(double* A, long long ld, int n, const double* w, double k_new, DevStatus* st) {
  __shared__ double red[32];
  if (dev_failed(st)) return;
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double di = A[i + (long long)i * ld];
    double vi = w[i] / di;
    A[n + (long long)i * ld] = vi;
    acc = fma(vi * vi, di, acc);
  }
  double vtdv = block_sum(acc, red);
  if (threadIdx.x == 0) {
    double delta = k_new - vtdv;
    if (!(delta > 0.0) || !isfinite(delta)) dev_fail(st, GPRX_CHOLESKY_FAILED, n);
    else A[n + (long long)n * ld] = delta;
  }
}

// Rank-1 update L D Lᵀ + a·w wᵀ of the trailing block (rows r0 .. n−1, w =
// L[r0.., idx], a = D_idx) with p = L⁻¹ w: the recurrence
//   D'_j = D_j + a_j p_j²,  β_j = a_j p_j / D'_j,  a_{j+1} = a_j D_j / D'_j
// has 1/a_{j+1} = 1/a_j + p_j²/D_j, so every a_j comes from one running sum of
// non-negative terms.  Rows count from row0 (a multiple of the block width;
// p is zero before r0).  One CTA: a thread sums a run of rows, the runs are
// scanned in shared memory.
constexpr int R1_THREADS = 1024;
__global__ void __launch_bounds__(R1_THREADS) ldlt_rank1_scan_kernel(const double* A, long long ld, int row0, int r0,
                                                                     int n, int idx, const double* p, double* beta,
                                                                     double* dnew, const DevStatus* st) {
  __shared__ double run[R1_THREADS];
  if (dev_failed(st)) return;
  const int tid = threadIdx.x, per = (n - r0 + R1_THREADS - 1) / R1_THREADS;
  const int lo = min(n, r0 + tid * per), hi = min(n, lo + per);
  double acc = 0.0;
  for (int i = lo; i < hi; ++i) acc += p[i - row0] * p[i - row0] / A[i + (long long)i * ld];
  run[tid] = acc;
  __syncthreads();
  for (int o = 1; o < R1_THREADS; o *= 2) {
    const double v = tid >= o ? run[tid - o] : 0.0;
    __syncthreads();
    run[tid] += v;
    __syncthreads();
  }
  double t = 1.0 / A[idx + (long long)idx * ld] + (tid > 0 ? run[tid - 1] : 0.0);
  for (int i = lo; i < hi; ++i) {
    const double pi = p[i - row0], di = A[i + (long long)i * ld], a = 1.0 / t;
    const double dn = fma(a * pi, pi, di);
    beta[i - row0] = a * pi / dn;
    dnew[i - row0] = dn;
    t += pi * pi / di;
  }
}

// The same update in place for at most 32 trailing rows (m from r0): one warp, a row a
// lane.  One launch instead of the block inverse, the solve and the scan: a delete
// from a model of 8 to 32 points takes 41 to 44 µs, 46 to 54 by way of those.
constexpr int DEL_ROWS = 128;
constexpr int DEL_SHORT = 32;
__global__ void __launch_bounds__(DEL_SHORT) ldlt_rank1_short_kernel(double* A, long long ld, int r0, int m, int idx,
                                                                     const DevStatus* st) {
  if (dev_failed(st)) return;
  const int lane = threadIdx.x, r = r0 + lane;
  const bool live = lane < m;
  double w = live ? A[r + (long long)idx * ld] : 0.0;
  double d = live ? A[r + (long long)r * ld] : 1.0;
  double a = A[idx + (long long)idx * ld];
  double l[DEL_SHORT];
#pragma unroll
  for (int c = 0; c < DEL_SHORT; ++c) l[c] = (live && c < lane) ? A[r + (long long)(r0 + c) * ld] : 0.0;
#pragma unroll
  for (int c = 0; c < DEL_SHORT; ++c) {
    if (c >= m) break;
    const double p = __shfl_sync(0xffffffffu, w, c), dc = __shfl_sync(0xffffffffu, d, c);
    const double dn = fma(a * p, p, dc), beta = a * p / dn;
    a = a * dc / dn;
    if (lane == c) d = dn;
    if (lane > c) {
      w = fma(-p, l[c], w);
      l[c] = fma(beta, w, l[c]);
    }
  }
  if (!live) return;
  A[r + (long long)r * ld] = d;
#pragma unroll
  for (int c = 0; c < DEL_SHORT; ++c)
    if (c < lane) A[r + (long long)(r0 + c) * ld] = l[c];
}

// B = A without row and column idx, the trailing block updated on the way (p null:
// it is up to date): thread = row, a CTA walks one 128-column block.  Row r enters the block
// with w_r less the sum over the blocks before it (prefix) and leaves behind
// L'_rc = L_rc + β_c w_r column by column.  HBM/L2-bound: the lower triangle
// is read once and written once (6 µs of 32 MB at n = 2000 out of L2); the
// single-CTA form took 4.5 ms there, every column through one SM.
__global__ void __launch_bounds__(DEL_ROWS) ldlt_delete_kernel(const double* A, long long ld, int n, int idx, int row0,
                                                               const double* p, const double* beta,
                                                               const double* dnew, const double* prefix,
                                                               long long ldp, double* B, long long ldb,
                                                               const DevStatus* st) {
  if (dev_failed(st)) return;
  const int r = blockIdx.x * DEL_ROWS + threadIdx.x, c0 = blockIdx.y * NB;
  if (r >= n || r == idx || r < c0) return;
  const int c1 = min(min(n, c0 + NB), r + 1);  // columns [c0, c1) of this row
  const double* a = A + r;
  const int rb = r > idx ? r - 1 : r;
  for (int c = c0; c < min(c1, idx); ++c) B[rb + (long long)c * ldb] = a[(long long)c * ld];
  if (r < idx) return;
  int c = max(c0, idx + 1);
  if (c >= c1) return;
  if (!p) {
    for (; c < c1; ++c) B[rb + (long long)(c - 1) * ldb] = a[(long long)c * ld];
    return;
  }
  double w = a[(long long)idx * ld];
  if (c0 > row0) w -= prefix[(r - row0) + (long long)((c0 - row0) / NB - 1) * ldp];
  const int last = min(c1, r);  // strictly below the diagonal
  for (; c + 8 <= last; c += 8) {
    double l[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) l[u] = a[(long long)(c + u) * ld];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      w = fma(-p[c + u - row0], l[u], w);
      B[rb + (long long)(c + u - 1) * ldb] = fma(beta[c + u - row0], w, l[u]);
    }
  }
  for (; c < last; ++c) {
    const double l = a[(long long)c * ld];
    w = fma(-p[c - row0], l, w);
    B[rb + (long long)(c - 1) * ldb] = fma(beta[c - row0], w, l);
  }
  if (c1 == r + 1) B[rb + (long long)(r - 1) * ldb] = dnew[r - row0];
}

__global__ void drop_row_kernel(const double* x, long long ldx, int n, int d, int idx, double* out, long long ldo) {
  long long total = (long long)(n - 1) * d;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    int i = (int)(e % (n - 1)), f = (int)(e / (n - 1));
    int si = i >= idx ? i + 1 : i;
    out[i + (long long)f * ldo] = x[si + (long long)f * ldx];
  }
}

__global__ void div_by_diag_kernel(double* v, const double* A, long long ld, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] /= A[i + (long long)i * ld];
}

gprx_status ExactState::online_begin() {
  gprx_status st;
  if (online) return GPRX_OK;
  if (!factor_ok || !alpha_ok) {
    if ((st = factor_current()) != GPRX_OK) return st;
  }
  llt_to_ldlt_kernel<<<n, 256, 0, stream>>>(A.p, ld, n);
  count_launch();
  GPRX_CUDA_TRY(cudaGetLastError());
  online = true;
  factor_ok = false;
  linv_ok = false;
  GPRX_CUDA_TRY(cudaStreamSynchronize(stream));
  return GPRX_OK;
}

gprx_status ExactState::with_llt_view(const std::function<gprx_status()>& op) {
  if (!online) return op();
  // keep the LDLT: a failed operation leaves the online model as it was
  const size_t keep = (size_t)ld * n;
  if (ldlt_keep.ensure(std::max<size_t>(keep, 1)) != cudaSuccess || alpha_keep.ensure(std::max(n, 1)) != cudaSuccess)
    return set_error(GPRX_OUT_OF_MEMORY, "device allocation of the online factor copy failed");
  GPRX_CUDA_TRY(cudaMemcpyAsync(ldlt_keep.p, A.p, sizeof(double) * keep, cudaMemcpyDeviceToDevice, stream));
  GPRX_CUDA_TRY(cudaMemcpyAsync(alpha_keep.p, alpha.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, stream));
  const bool alpha_was_ok = alpha_ok;
  const double jitter_was = jitter;
  std::vector<double> theta_was(num_params());
  get_params(theta_was.data());
  online = false;
  factor_ok = false;
  linv_ok = false;
  alpha_ok = false;
  gprx_status st = op();
  if (st == GPRX_OK && (!factor_ok || !alpha_ok)) st = factor_current();
  if (st == GPRX_OK) {
    llt_to_ldlt_kernel<<<n, 256, 0, stream>>>(A.p, ld, n);
    count_launch();
    GPRX_CUDA_TRY(cudaGetLastError());
  } else {
    gprx_error_info saved = last_error();
    write_params(theta_was.data());
    GPRX_CUDA_TRY(cudaMemcpyAsync(A.p, ldlt_keep.p, sizeof(double) * keep, cudaMemcpyDeviceToDevice, stream));
    GPRX_CUDA_TRY(cudaMemcpyAsync(alpha.p, alpha_keep.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, stream));
    alpha_ok = alpha_was_ok;
    jitter = jitter_was;
    last_error() = saved;
  }
  online = true;
  factor_ok = false;
  linv_ok = false;
  GPRX_CUDA_TRY(cudaStreamSynchronize(stream));
  return st;
}

gprx_status ExactState::grow(int needed) {
  if (needed <= cap) return GPRX_OK;
  int new_cap = std::max(needed, std::max(cap, 1) * 2);
  long long new_ld = round_ld(new_cap);
  DevBuf<double> nA{lane}, nx{lane}, ny{lane};
  if (nA.alloc((size_t)new_ld * new_cap) != cudaSuccess || nx.alloc((size_t)new_cap * d) != cudaSuccess ||
      ny.alloc(new_cap) != cudaSuccess)
    return set_error(GPRX_OUT_OF_MEMORY, "online capacity growth");
  GPRX_CUDA_TRY(cudaMemcpy2DAsync(nA.p, sizeof(double) * new_ld, A.p, sizeof(double) * ld, sizeof(double) * n, n,
                                  cudaMemcpyDeviceToDevice, stream));
  GPRX_CUDA_TRY(cudaMemcpy2DAsync(nx.p, sizeof(double) * new_cap, x.p, sizeof(double) * cap, sizeof(double) * n, d,
                                  cudaMemcpyDeviceToDevice, stream));
  GPRX_CUDA_TRY(cudaMemcpyAsync(ny.p, y.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, stream));
  GPRX_CUDA_TRY(cudaStreamSynchronize(stream));
  std::swap(A.p, nA.p);
  std::swap(A.n, nA.n);
  std::swap(x.p, nx.p);
  std::swap(x.n, nx.n);
  std::swap(y.p, ny.p);
  std::swap(y.n, ny.n);
  int nblk = ceil_div(new_cap, NB);
  if (linv.alloc((size_t)nblk * NB * NB) != cudaSuccess || alpha.alloc(new_cap) != cudaSuccess ||
      z.alloc(new_cap) != cudaSuccess || tmpv.alloc(new_cap) != cudaSuccess)
    return set_error(GPRX_OUT_OF_MEMORY, "online capacity growth");
  Xinv.reset();
  qbuf.reset();
  cap = new_cap;
  ld = new_ld;
  linv_ok = false;
  alpha_ok = false;
  return GPRX_OK;
}

gprx_status ExactState::online_insert(const double* xnew, double ynew, uint64_t* id) {
  if (!online) return set_error(GPRX_INVALID_CONFIG, "call gprx_online_begin first");
  if (!xnew || !id) return set_error(GPRX_INVALID_ARGUMENT, "null pointer");
  if (!all_finite(xnew, d) || !std::isfinite(ynew)) return set_error(GPRX_NONFINITE_INPUT, "non-finite point");
  gprx_status st;
  if ((st = grow(n + 1)) != GPRX_OK) return st;
  if (qx.ensure((size_t)d + 8) != cudaSuccess) return set_error(GPRX_OUT_OF_MEMORY, "insert scratch");
  if ((st = reset_status()) != GPRX_OK) return st;
  if (!linv_ok) {
    GPRX_CUDA_TRY(tri_inv_blocks(A.p, ld, n, true, linv.p, status.p, stream));
    linv_ok = true;
  }
  GPRX_CUDA_TRY(cudaMemcpyAsync(qx.p, xnew, sizeof(double) * d, cudaMemcpyHostToDevice, stream));
  // k = K(X, x_new) into tmpv (n×1), then w = L⁻¹ k (unit lower)
  GPRX_CUDA_TRY(fill_cross(kern, x.p, cap, n, qx.p, 1, 1, tmpv.p, n, status.p, stream));
  GPRX_CUDA_TRY(trsm_lower(A.p, ld, n, linv.p, tmpv.p, n, 1, status.p, stream));
  double k_new = kern.diag_value() + noise() + jitter;  // online.rs:855-862
  ldlt_border_kernel<<<1, 1024, 0, stream>>>(A.p, ld, n, tmpv.p, k_new, status.p);
  count_launch();
  DevStatus ds;
  if ((st = read_status(&ds)) != GPRX_OK) return st;
  if (ds.code != GPRX_OK) return status_to_error(ds, 0.0, n + 1, GPRX_STAGE_ONLINE_INSERT);
  // append x, y (the store keeps them in buffer order)
  GPRX_CUDA_TRY(cudaMemcpy2DAsync(x.p + n, sizeof(double) * cap, xnew, sizeof(double), sizeof(double), d,
                                  cudaMemcpyHostToDevice, stream));
  GPRX_CUDA_TRY(cudaMemcpyAsync(y.p + n, &ynew, sizeof(double), cudaMemcpyHostToDevice, stream));
  GPRX_CUDA_TRY(cudaStreamSynchronize(stream));
  y_host.push_back(ynew);
  n += 1;
  *id = next_id++;
  ids.push_back(*id);
  alpha_ok = false;
  // the appended row changes only the last diagonal block
  linv_ok = false;
  return GPRX_OK;
}

gprx_status ExactState::online_delete(uint64_t id) {
  if (!online) return set_error(GPRX_INVALID_CONFIG, "call gprx_online_begin first");
  if (n <= 1) return set_error(GPRX_INSUFFICIENT_DATA, "an online model keeps at least one point");
  auto it = std::lower_bound(ids.begin(), ids.end(), id);
  if (it == ids.end() || *it != id) return set_error(GPRX_INVALID_POINT_ID, "unknown point id");
  int idx = (int)(it - ids.begin());
  gprx_status st;
  if ((st = reset_status()) != GPRX_OK) return st;
  const int row0 = (idx + 1) / NB * NB, len = n - row0;  // whole blocks from the first trailing row
  DevBuf<double> nA{lane};  // the compacted factor, in the last delete's spare if it is still there
  if (nA.take_spare(this, (size_t)ld * cap) != cudaSuccess || spare_x.ensure((size_t)cap * d) != cudaSuccess ||
      spare_y.ensure(cap) != cudaSuccess ||
      r1.ensure((size_t)std::max(len, 1) * (3 + ceil_div(std::max(len, 1), NB))) != cudaSuccess)
    return set_error(GPRX_OUT_OF_MEMORY, "online delete scratch");
  double* p = r1.p;
  double* beta = p + std::max(len, 0);
  double* dnew = beta + std::max(len, 0);
  double* prefix = dnew + std::max(len, 0);
  const int m = n - idx - 1;
  if (m > 0 && m <= DEL_SHORT) {
    GPRX_LAUNCH(ldlt_rank1_short_kernel, 1, DEL_SHORT, 0, stream, A.p, ld, idx + 1, m, idx, status.p);
    p = nullptr;
    linv_ok = false;
  } else if (m > 0) {
    if (!linv_ok) {
      GPRX_CUDA_TRY(tri_inv_blocks(A.p, ld, n, true, linv.p, status.p, stream));
      linv_ok = true;
    }
    // p = L⁻¹ w over the blocks that hold trailing rows, zero before them
    const int lead = idx + 1 - row0;
    if (lead > 0) GPRX_CUDA_TRY(cudaMemsetAsync(p, 0, sizeof(double) * lead, stream));
    GPRX_CUDA_TRY(cudaMemcpyAsync(p + lead, A.p + (idx + 1) + (long long)idx * ld, sizeof(double) * (n - idx - 1),
                                  cudaMemcpyDeviceToDevice, stream));
    GPRX_CUDA_TRY(tri_solve_vec(A.p + row0 + (long long)row0 * ld, ld, len, linv.p + (long long)(row0 / NB) * NB * NB,
                                p, false, status.p, stream, prefix, len));
    GPRX_LAUNCH(ldlt_rank1_scan_kernel, 1, R1_THREADS, 0, stream, A.p, ld, row0, idx + 1, n, idx, p, beta, dnew,
                status.p);
  }
  GPRX_LAUNCH(ldlt_delete_kernel, dim3(ceil_div(n, DEL_ROWS), ceil_div(n, NB)), DEL_ROWS, 0, stream, A.p, ld, n, idx,
              row0, p, beta, dnew, prefix, (long long)len, nA.p, ld, status.p);
  GPRX_LAUNCH(drop_row_kernel, ceil_div((long long)(n - 1) * d, 256) + 1, 256, 0, stream, x.p, cap, n, d, idx,
              spare_x.p, cap);
  GPRX_LAUNCH(drop_row_kernel, ceil_div(n, 256) + 1, 256, 0, stream, y.p, cap, n, 1, idx, spare_y.p, cap);
  DevStatus ds;
  if ((st = read_status(&ds)) != GPRX_OK) return st;
  if (ds.code != GPRX_OK) return status_to_error(ds, 0.0, n, GPRX_STAGE_ONLINE_DELETE);
  std::swap(A.p, nA.p);
  std::swap(A.n, nA.n);
  nA.keep_spare(this);
  std::swap(x.p, spare_x.p);
  std::swap(x.n, spare_x.n);
  std::swap(y.p, spare_y.p);
  std::swap(y.n, spare_y.n);
  y_host.erase(y_host.begin() + idx);
  ids.erase(it);
  n -= 1;
  alpha_ok = false;
  linv_ok = false;
  return GPRX_OK;
}

gprx_status ExactState::online_alpha() {
  gprx_status st;
  if ((st = reset_status()) != GPRX_OK) return st;
  if (!linv_ok) {
    GPRX_CUDA_TRY(tri_inv_blocks(A.p, ld, n, true, linv.p, status.p, stream));
    linv_ok = true;
  }
  GPRX_CUDA_TRY(cudaMemcpyAsync(alpha.p, y.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, stream));
  GPRX_CUDA_TRY(trsm_lower(A.p, ld, n, linv.p, alpha.p, n, 1, status.p, stream));
  div_by_diag_kernel<<<ceil_div(n, 256), 256, 0, stream>>>(alpha.p, A.p, ld, n);
  count_launch();
  GPRX_CUDA_TRY(trsm_lower_t(A.p, ld, n, linv.p, alpha.p, n, 1, status.p, stream));
  DevStatus ds;
  if ((st = read_status(&ds)) != GPRX_OK) return st;
  if (ds.code != GPRX_OK) return status_to_error(ds, 0.0, n, GPRX_STAGE_ONLINE_INSERT);
  alpha_ok = true;
  return GPRX_OK;
}

}  // namespace gprx
