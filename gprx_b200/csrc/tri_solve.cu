// tri_solve.cu — triangular solves with few right-hand sides, one launch.
//
// B := L⁻¹ B or L⁻ᵀ B for a strip of 8·NT columns is a chain over the 128-row
// blocks of L: x_s = L_ss⁻¹ (b_s − Σ_{t<s} L_st x_t).  A thread-block cluster
// of C CTAs owns one strip; block s belongs to CTA s mod C.  At step s every
// CTA reads x_s (written to B by its owner) and folds L_ts x_s into the sums
// of its own later blocks, the owner of block s+1 first: its tile L_{s+1,s}
// and the inverse of its diagonal block were staged in shared memory and
// registers beforehand, so the chain from x_s to x_{s+1} is one barrier, two
// 128×128 products on DMMA and one store.  The cluster barrier orders the
// steps: CTAs of one cluster are co-resident, so nothing spins.
//
// What bounds it: for one strip the chain (about 2 µs a block); for many
// strips the reads of L, n²/2 values per strip out of L2.  The two-product
// form it replaces took two launches of one to n/128 tiles of 128×128 for
// every block: 33 µs each with one right-hand side, 16 blocks = 1.05 ms at
// n = 2000.
//
// A column's result does not depend on q, on its place in a strip, on NT or
// on C: the sums over s ascend and each tile adds its even and odd k steps in
// two accumulators, whichever CTA does it.

#include <algorithm>

#include "dense_f64.cuh"

namespace gprx {

namespace {

constexpr int TS_THREADS = 256;
constexpr int TS_LD = NB + 4;  // ≡ 4 mod 16 doubles: conflict-free fragments
constexpr int TS_MAX_CLUSTER = 16;
constexpr int TS_SMEM_MAX = 227 * 1024;

struct TriSolveArgs {
  const double* L;
  long long ld;
  int n;
  const double* linv;
  double* B;
  long long ldb;
  int q;
  int C;
  double* prefix;
  long long ldp;
  const DevStatus* st;
};

// one: a single right-hand side keeps only its own column's sums, so that
// every n whose matrix fits in memory has a plan
inline size_t ts_smem(int NT, int own, bool one) {
  return sizeof(double) * ((size_t)NB * TS_LD + 2 * (size_t)8 * NT * TS_LD +
                           (size_t)own * (one ? NB : NT * 4 * TS_THREADS));
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <bool TRANS, int NT>
__global__ void __launch_bounds__(TS_THREADS, 1) tri_solve_kernel(TriSolveArgs g) {
  extern __shared__ __align__(16) double ts_sm[];
  if (dev_failed(g.st)) return;  // the same word for the whole cluster
  double* tile = ts_sm;                   // L_{s+1,s}: [k][i], transposed solve [i][k]
  double* xs = tile + NB * TS_LD;         // x_s: [column][k]
  double* bs = xs + 8 * NT * TS_LD;       // right-hand side of the owned block
  double* sums = bs + 8 * NT * TS_LD;     // [owned block][accumulator][thread], one column: [owned block][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t4 = lane & 3;
  const int n = g.n, C = g.C, rank = blockIdx.x % C, j0 = (blockIdx.x / C) * 8 * NT;
  const int ncol = min(8 * NT, g.q - j0);
  const int nblk = (n + NB - 1) / NB;
  double* const B = g.B + (long long)j0 * g.ldb;
  const int r0 = 16 * warp + gq;  // this lane's rows of a block: r0 and r0 + 8
  auto first = [&](int s) { return (TRANS ? nblk - 1 - s : s) * NB; };

  double lf[32][2];    // A fragments of the owned diagonal block's inverse
  double cb[NT][4];    // the owned block's rows of B
  const int own = (nblk - rank + C - 1) / C;
  const bool one = g.q == 1, keep = !one || t4 == 0;
  auto slot = [&](int o, int t, int r) {
    return one ? o * NB + r0 + 4 * r : (o * NT * 4 + t * 4 + r) * TS_THREADS + tid;
  };
  auto sum_of = [&](int o, int t, int r) { return keep && !(one && (r & 1)) ? sums[slot(o, t, r)] : 0.0; };
  auto set_sum = [&](int o, int t, int r, double v) {
    if (keep && !(one && (r & 1))) sums[slot(o, t, r)] = v;
  };
  for (int o = 0; o < own; ++o)
#pragma unroll
    for (int e = 0; e < NT * 4; ++e) set_sum(o, e / 4, e % 4, 0.0);

  // Stages everything the owner of block s needs: L_{s,s−1}, the inverse of
  // the diagonal block (zero outside its triangle, so only the k steps of a
  // warp's rows that meet it), its rows of B.
  auto prefetch = [&](int s) {
    const int i0 = first(s);
    if (s > 0) {
      const int k0 = first(s - 1);
      for (int e = tid; e < NB * NB; e += TS_THREADS) {
        const int u = e % NB, v = e / NB;  // u runs along the column of L
        const int i = TRANS ? v : u, k = TRANS ? u : v;
        const bool ok = i0 + i < n && k0 + k < n;
        const double* src = TRANS ? g.L + (k0 + k) + (long long)(i0 + i) * g.ld
                                  : g.L + (i0 + i) + (long long)(k0 + k) * g.ld;
        cp_async8(tile + v * TS_LD + u, ok ? src : g.L, ok);
      }
      cp_async_commit();
    }
    const double* li = g.linv + (long long)(i0 / NB) * NB * NB;
    const int nb = min(NB, n - i0);
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) {
      const int k = 4 * kk + t4;
      const bool in = TRANS ? kk >= 4 * warp : kk < 4 * warp + 4;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = r0 + 8 * h;
        const bool ok = in && i < nb && k < nb && (TRANS ? k >= i : k <= i);
        lf[kk][h] = ok ? (TRANS ? li[k + i * NB] : li[i + k * NB]) : 0.0;
      }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = i0 + r0 + ((r & 2) ? 8 : 0), col = 8 * t + 2 * t4 + (r & 1);
        cb[t][r] = (row < n && col < ncol) ? B[row + (long long)col * g.ldb] : 0.0;
      }
  };
  // x_s = L_ss⁻¹ (b_s − sums) for the prefetched block, stored to B.
  auto solve = [&](int s) {
    const int i0 = first(s), o = s / C;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        bs[(8 * t + 2 * t4 + (r & 1)) * TS_LD + r0 + ((r & 2) ? 8 : 0)] =
            cb[t][r] - sum_of(o, t, r);
    __syncthreads();
    double a[NT][2][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 4; ++r) a[t][h][r] = 0.0;
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) {
      const bool in = TRANS ? kk >= 4 * warp : kk < 4 * warp + 4;
      if (!in) continue;
#pragma unroll
      for (int t = 0; t < NT; ++t)
        dmma_16x8x4(a[t][kk & 1], lf[kk][0], lf[kk][1], bs[(8 * t + gq) * TS_LD + 4 * kk + t4]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = i0 + r0 + ((r & 2) ? 8 : 0), col = 8 * t + 2 * t4 + (r & 1);
        if (row < n && col < ncol) B[row + (long long)col * g.ldb] = a[t][0][r] + a[t][1][r];
      }
  };
  // sums of owned block index o += (tile at i0, k0) · x; from shared memory
  // when staged, else from global in batches of eight k steps, one ahead.
  auto fold = [&](int o, int i0, int k0, int s, bool staged) {
    double a[NT][2][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        a[t][0][r] = sum_of(o, t, r);
        a[t][1][r] = 0.0;
      }
    if (staged) {
#pragma unroll 4
      for (int kk = 0; kk < 32; kk += 2)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = 4 * (kk + h) + t4;
          const double a0 = TRANS ? tile[r0 * TS_LD + k] : tile[k * TS_LD + r0];
          const double a1 = TRANS ? tile[(r0 + 8) * TS_LD + k] : tile[k * TS_LD + r0 + 8];
#pragma unroll
          for (int t = 0; t < NT; ++t) dmma_16x8x4(a[t][h], a0, a1, xs[(8 * t + gq) * TS_LD + k]);
        }
    } else {
      const int ia = i0 + r0, ib = ia + 8;
      double f[2][8][2];
      auto load = [&](int b, double (&d)[8][2]) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int k = k0 + 32 * b + 4 * u + t4;
          const bool kin = k < n;
          d[u][0] = (kin && ia < n) ? (TRANS ? g.L[k + (long long)ia * g.ld] : g.L[ia + (long long)k * g.ld]) : 0.0;
          d[u][1] = (kin && ib < n) ? (TRANS ? g.L[k + (long long)ib * g.ld] : g.L[ib + (long long)k * g.ld]) : 0.0;
        }
      };
      load(0, f[0]);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        if (b < 3) load(b + 1, f[(b + 1) & 1]);
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int t = 0; t < NT; ++t)
            dmma_16x8x4(a[t][u & 1], f[b & 1][u][0], f[b & 1][u][1], xs[(8 * t + gq) * TS_LD + 32 * b + 4 * u + t4]);
      }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int r = 0; r < 4; ++r) set_sum(o, t, r, a[t][0][r] + a[t][1][r]);
    if (NT == 1 && g.prefix && t4 == 0)
#pragma unroll
      for (int r = 0; r < 4; r += 2)
        if (i0 + r0 + 4 * r < n) g.prefix[(i0 + r0 + 4 * r) + s * g.ldp] = a[0][0][r] + a[0][1][r];
  };

  if (rank == 0) {
    prefetch(0);
    solve(0);
  }
  cluster_arrive();
  if (rank == 1 % C && nblk > 1) prefetch(1);
  cluster_wait();
  for (int s = 0; s + 1 < nblk; ++s) {
    const int k0 = first(s);
    __syncthreads();  // the previous step's reads of xs are done
    for (int e = tid; e < 8 * NT * NB; e += TS_THREADS) {
      const int k = e % NB, c = e / NB;
      xs[c * TS_LD + k] = (k0 + k < n && c < ncol) ? __ldcg(B + (k0 + k) + (long long)c * g.ldb) : 0.0;
    }
    const bool mine = (s + 1) % C == rank;
    if (mine) cp_async_wait<0>();
    __syncthreads();
    if (mine) {
      fold((s + 1) / C, first(s + 1), k0, s, true);
      solve(s + 1);
    }
    cluster_arrive();
    for (int t = s + 2 + (rank - (s + 2) % C + C) % C; t < nblk; t += C) fold(t / C, first(t), k0, s, false);
    if ((s + 2) % C == rank && s + 2 < nblk) {
      if (C == 1) __syncthreads();  // this CTA also used the tile at this step
      prefetch(s + 2);
    }
    cluster_wait();
  }
}

template <bool TRANS, int NT>
cudaError_t ts_launch(const TriSolveArgs& g, int strips, size_t smem, cudaStream_t s) {
  auto kern = tri_solve_kernel<TRANS, NT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX);
  if (e != cudaSuccess) return e;
  if (g.C > 8 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
    return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(strips * g.C));
  cfg.blockDim = dim3(TS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, kern, g);
}

// Whether the device can hold a cluster of 16 CTAs of one SM each (non-portable).
bool ts_cluster16() {
  static int cached[64] = {0};  // 0 unknown, 1 yes, 2 no; the same answer from every thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (cached[dev] == 0) {
    auto kern = tri_solve_kernel<false, 1>;
    int clusters = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(TS_THREADS);
    cfg.dynamicSmemBytes = TS_SMEM_MAX;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0;
    if (!ok) (void)cudaGetLastError();
    cached[dev] = ok ? 1 : 2;
  }
  return cached[dev] == 1;
}

// (NT, C) of a solve: 16-column strips from nine columns on; the largest
// cluster that keeps every strip resident at once (148 SMs) and has a block
// for every CTA, as far as the owned blocks' sums fit in shared memory.
bool ts_plan(int n, int q, int* NT, int* C) {
  const int nblk = ceil_div(n, NB);
  const int cmax = ts_cluster16() ? TS_MAX_CLUSTER : 8;
  for (int nt = q > 8 ? 2 : 1; nt >= 1; --nt) {
    const int strips = ceil_div(q, 8 * nt);
    int c = 1;
    while (c * 2 <= cmax && c * 2 <= nblk && (long long)c * 2 * strips <= 148) c *= 2;
    while (c < cmax && ts_smem(nt, ceil_div(nblk, c), q == 1) > TS_SMEM_MAX) c *= 2;
    if (ts_smem(nt, ceil_div(nblk, c), q == 1) <= TS_SMEM_MAX) {
      *NT = nt;
      *C = c;
      return true;
    }
  }
  return false;
}

}  // namespace

// Few right-hand sides: n·q ≤ 3·2²⁰.  Measured against trsm_lower_wide (µs):
// n = 512: q = 256 33 / 205, 4000 128 / 211, 10000 285 / 268; n = 1000:
// q = 256 117 / 435, 2000 253 / 443, 4000 501 / 529; n = 2000: q = 1 80 / 851,
// 256 263 / 894, 1000 644 / 898, 2000 1162 / 1080; n = 4096: q = 1 193 / 1747,
// 500 1574 / 1871, 1000 2850 / 2235.
bool tri_solve_few(long long n, long long q) {
  int nt, c;
  return n > 0 && q > 0 && n * q <= (3LL << 20) && ts_plan((int)n, (int)q, &nt, &c);
}

cudaError_t tri_solve(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                      bool trans, const DevStatus* st, cudaStream_t s, double* prefix, long long ldp) {
  if (n <= 0 || q <= 0) return cudaSuccess;
  int nt, c;
  if (!ts_plan(n, q, &nt, &c) || (prefix && q != 1)) return cudaErrorInvalidValue;
  TriSolveArgs g{L, ld, n, linv, B, ldb, q, c, prefix, ldp, st};
  const int strips = ceil_div(q, 8 * nt);
  const size_t smem = ts_smem(nt, ceil_div(ceil_div(n, NB), c), q == 1);
  if (trans) return nt == 1 ? ts_launch<true, 1>(g, strips, smem, s) : ts_launch<true, 2>(g, strips, smem, s);
  return nt == 1 ? ts_launch<false, 1>(g, strips, smem, s) : ts_launch<false, 2>(g, strips, smem, s);
}

}  // namespace gprx
