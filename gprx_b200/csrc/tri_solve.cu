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
// What bounds it: for one strip the chain and the tile that each CTA folds a step
// (5 µs a block measured; a 128×128 tile alone is 2048 cycles of DMMA); for many
// strips the reads of L, n²/2 values per strip out of L2.  The two-product
// form it replaces took two launches of one to n/128 tiles of 128×128 for
// every block: 33 µs each with one right-hand side, 16 blocks = 1.05 ms at
// n = 2000.
//
// A column's result does not depend on q, on its place in a strip, on NT or
// on C: the sums over s ascend and each tile adds its even and odd k steps in
// two accumulators, whichever CTA does it.

#include <algorithm>
#include <atomic>

#include "dense_f64.cuh"

namespace gprx {

namespace {

constexpr int TS_THREADS = 256;
constexpr int TS_LD = NB + 4;  // ≡ 4 mod 16 doubles: conflict-free fragments
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
  const DevStatus* st;
};

// one: a single right-hand side keeps only its own column's sums, so that
// every n whose matrix fits in memory has a plan
inline size_t ts_smem(int NT, int own, bool one) {
  return sizeof(double) * ((size_t)NB * TS_LD + 2 * (size_t)8 * NT * TS_LD +
                           (size_t)own * (one ? NB : NT * 4 * TS_THREADS));
}

// v to CTA `rank` of the cluster at shared address `addr` (of this CTA's layout)
__device__ __forceinline__ void cluster_store(unsigned addr, int rank, double v) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
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
  auto fold = [&](int o, int i0, int k0, bool staged) {
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
      fold((s + 1) / C, first(s + 1), k0, true);
      solve(s + 1);
    }
    cluster_arrive();
    for (int t = s + 2 + (rank - (s + 2) % C + C) % C; t < nblk; t += C) fold(t / C, first(t), k0, false);
    if ((s + 2) % C == rank && s + 2 < nblk) {
      if (C == 1) __syncthreads();  // this CTA also used the tile at this step
      prefetch(s + 2);
    }
    cluster_wait();
  }
}

// ---------------------------------------------------------------------------
// one right-hand side that is a vector of its own (α, the online updates)
// ---------------------------------------------------------------------------
// The same steps on FP64 FMAs: a DMMA spends seven eighths of its columns on
// one right-hand side (2 K cycles a 128×128 tile, 16 FMA a cycle and scheduler
// either way), here a tile costs 64 FMAs a thread.  L_{s+1,s} waits in
// registers, the diagonal block's inverse in shared memory, and the owner writes
// x_s into every CTA's shared memory (a read back from L2 and the store's way
// there were a third of the step).  Forward, a thread
// owns a row and half of the k range (column-major L: coalesced over rows);
// transposed, a warp owns 16 rows of Lᵀ, its lanes run along k, and a
// reduce-scatter of 16 shuffles leaves row ii in lanes 2·ii, 2·ii + 1.
// Bound by the reads of L at 16 SMs' rate and the chain.  Measured (forward /
// transposed, µs, on DMMA → here): n = 512 23 / 23 → 17 / 17, n = 2000 82 / 82 →
// 53 / 46, n = 4096 227 / 201 → 151 / 110.
struct TriVecArgs {
  const double* L;
  long long ld;
  int n;
  const double* linv;
  double* b;
  int C;
  double* prefix;
  long long ldp;
  const DevStatus* st;
};

inline size_t tv_smem(int own) { return sizeof(double) * ((size_t)NB * NB + 6 * NB + (size_t)own * NB); }

// v[ii] of 32 lanes summed; lane l returns row l / 2.
__device__ __forceinline__ double scatter16(double (&v)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int m = 8; m >= 1; m /= 2) {
    const bool up = lane & (2 * m);
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const double send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * m);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <bool TRANS>
__global__ void __launch_bounds__(TS_THREADS, 1) tri_vec_kernel(TriVecArgs g) {
  extern __shared__ __align__(16) double ts_sm[];
  if (dev_failed(g.st)) return;  // the same word for the whole cluster
  double* li = ts_sm;           // the owned diagonal block's inverse, ld NB
  double* xbuf = li + NB * NB;  // x_s in slot s mod 3, written by the owner into every CTA
  double* bs = xbuf + 3 * NB;   // right-hand side of the owned block
  double* part = bs + NB;       // [half][row]
  double* sums = part + 2 * NB;  // [owned block][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = g.n, C = g.C, rank = blockIdx.x % C, nblk = (n + NB - 1) / NB;
  const int row = tid & (NB - 1), half = tid >> 7, kb = 64 * half;  // forward
  auto first = [&](int s) { return (TRANS ? nblk - 1 - s : s) * NB; };
  const int own = (nblk - rank + C - 1) / C;
  for (int e = tid; e < own * NB; e += TS_THREADS) sums[e] = 0.0;
  double f[64];
  double bown = 0.0;  // row tid of the owned block's right-hand side
  auto load_tile = [&](int i0, int k0) {
#pragma unroll
    for (int u = 0; u < 64; ++u) {
      if (TRANS) {
        const int k = k0 + lane + 32 * (u & 3);
        f[u] = k < n ? g.L[k + (long long)(i0 + 16 * warp + (u >> 2)) * g.ld] : 0.0;
      } else {
        f[u] = i0 + row < n ? g.L[(i0 + row) + (long long)(k0 + kb + u) * g.ld] : 0.0;
      }
    }
  };
  // the inverse and the right-hand side of the CTA's next block, as soon as the
  // one before is solved (they depend on nobody)
  auto stage_block = [&](int s) {
    if (s >= nblk) return;
    const double* src = g.linv + (long long)(first(s) / NB) * NB * NB;
    for (int e = 2 * tid; e < NB * NB; e += 2 * TS_THREADS) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(li + e);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + e));
    }
    cp_async_commit();
    bown = tid < NB && first(s) + tid < n ? g.b[first(s) + tid] : 0.0;
  };
  // (tile in f) · x into the sums of owned block o
  auto fold = [&](int o, int i0, int s) {
    const double* xs = xbuf + (s % 3) * NB;
    if (TRANS) {
      double v[16], x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = xs[lane + 32 * u];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        v[i] = fma(f[4 * i], x[0], f[4 * i + 1] * x[1]) + fma(f[4 * i + 2], x[2], f[4 * i + 3] * x[3]);
      const double t = scatter16(v);
      if (!(lane & 1)) sums[o * NB + 16 * warp + (lane >> 1)] += t;
    } else {
      double a[4] = {0, 0, 0, 0};
#pragma unroll
      for (int u = 0; u < 64; u += 2) {
        const double2 x = *reinterpret_cast<const double2*>(xs + kb + u);
        a[u & 2] = fma(f[u], x.x, a[u & 2]);
        a[(u & 2) + 1] = fma(f[u + 1], x.y, a[(u & 2) + 1]);
      }
      __syncthreads();  // the previous fold's reads of part are done
      part[tid] = (a[0] + a[1]) + (a[2] + a[3]);
      __syncthreads();
      if (tid < NB) {
        const double t = sums[o * NB + tid] + (part[tid] + part[NB + tid]);
        sums[o * NB + tid] = t;
        if (g.prefix && i0 + tid < n) g.prefix[(i0 + tid) + s * g.ldp] = t;
      }
    }
  };
  auto solve = [&](int s) {
    const int i0 = first(s), o = s / C;
    cp_async_wait<0>();
    __syncthreads();
    if (tid < NB) bs[tid] = bown - sums[o * NB + tid];  // zero past n: both terms are
    __syncthreads();
    if (TRANS) {  // Σ_{k ≥ i} X(k, i) b_k
      double v[16], x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = bs[lane + 32 * u];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (32 * u + 31 >= 16 * warp) v[i] = fma(li[(16 * warp + i) * NB + lane + 32 * u], x[u], v[i]);
      }
      const double t = scatter16(v);
      if (!(lane & 1)) part[16 * warp + (lane >> 1)] = t;
      __syncthreads();
    } else {  // Σ_{k ≤ i} X(i, k) b_k
      double a[4] = {0, 0, 0, 0};
      const int end = min(64, (row | 31) + 1 - kb);
#pragma unroll 8
      for (int u = 0; u < end; u += 4) {
        const double2 x0 = *reinterpret_cast<const double2*>(bs + kb + u);
        const double2 x1 = *reinterpret_cast<const double2*>(bs + kb + u + 2);
        a[0] = fma(li[(kb + u) * NB + row], x0.x, a[0]);
        a[1] = fma(li[(kb + u + 1) * NB + row], x0.y, a[1]);
        a[2] = fma(li[(kb + u + 2) * NB + row], x1.x, a[2]);
        a[3] = fma(li[(kb + u + 3) * NB + row], x1.y, a[3]);
      }
      part[tid] = (a[0] + a[1]) + (a[2] + a[3]);
      __syncthreads();
      if (tid < NB) part[tid] += part[NB + tid];
    }
    // x_s into every CTA's buffer
    if (tid < NB) {
      const unsigned at = (unsigned)__cvta_generic_to_shared(xbuf + (s % 3) * NB + tid);
      if (s + 1 < nblk)
        for (int c = 0; c < C; ++c) cluster_store(at, c, part[tid]);
    }
  };
  auto store = [&](int s) {
    if (tid < NB && first(s) + tid < n) g.b[first(s) + tid] = part[tid];
  };

  cluster_arrive();  // every CTA has started: its shared memory may be written
  stage_block(rank);
  if (rank == 1 % C && nblk > 1) load_tile(first(1), first(0));
  cluster_wait();
  if (rank == 0) solve(0);
  cluster_arrive();
  if (rank == 0) {
    store(0);
    __syncthreads();  // the inverse has been read
    stage_block(C);
  }
  cluster_wait();
  for (int s = 0; s + 1 < nblk; ++s) {
    const int k0 = first(s);
    const bool mine = (s + 1) % C == rank;
    if (mine) {
      fold((s + 1) / C, first(s + 1), s);
      solve(s + 1);
    }
    // slot (s + 1) mod 3 held x_{s−2}: a CTA behind this one is folding x_{s−1}
    // at the latest (it has arrived at the barrier before), so nobody reads it
    cluster_arrive();
    if (mine) {
      store(s + 1);
      __syncthreads();  // the inverse has been read
      stage_block(s + 1 + C);
    }
    for (int t = s + 2 + (rank - (s + 2) % C + C) % C; t < nblk; t += C) {
      load_tile(first(t), k0);
      fold(t / C, first(t), s);
    }
    if ((s + 2) % C == rank && s + 2 < nblk) load_tile(first(s + 2), first(s + 1));
    cluster_wait();
  }
}

template <typename Args>
cudaError_t ts_launch(void (*kern)(Args), const Args& g, int ctas, size_t smem, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX);
  if (e != cudaSuccess) return e;
  if (g.C > 8 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
    return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
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

// Clusters of 2^lc CTAs that the current device holds at once (one CTA takes an SM;
// a cluster lies in one GPC, so there are fewer than SMs / CTAs of them: 16 of 8 and
// 7 of 16).  0: no such cluster.
int ts_resident(int lc) {
  static std::atomic<int> cached[64][5];  // the count plus one; the same answer from every thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::atomic<int>& known = cached[dev][lc];
  if (known.load(std::memory_order_relaxed) == 0) {
    auto kern = tri_solve_kernel<false, 1>;
    int clusters = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << lc);
    cfg.blockDim = dim3(TS_THREADS);
    cfg.dynamicSmemBytes = TS_SMEM_MAX;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1u << lc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX) == cudaSuccess &&
                    (lc < 4 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess;
    if (!ok) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    known.store(clusters + 1, std::memory_order_relaxed);
  }
  return known.load(std::memory_order_relaxed) - 1;
}

// (NT, C) of a solve: 16-column strips from nine columns on; the largest
// cluster of which the device holds one for every strip at once and that has a
// block for every CTA, as far as the owned blocks' sums fit in shared memory.
// *held: every strip is resident.
bool ts_plan(int n, int q, int* NT, int* C, bool* held) {
  const int nblk = ceil_div(n, NB);
  for (int nt = q > 8 ? 2 : 1; nt >= 1; --nt) {
    const int strips = ceil_div(q, 8 * nt);
    int lc = 0;
    while (lc < 4 && (2 << lc) <= nblk && ts_resident(lc + 1) >= strips) ++lc;
    while (lc < 4 && ts_smem(nt, ceil_div(nblk, 1 << lc), q == 1) > TS_SMEM_MAX && ts_resident(lc + 1) > 0) ++lc;
    if (ts_smem(nt, ceil_div(nblk, 1 << lc), q == 1) <= TS_SMEM_MAX) {
      *NT = nt;
      *C = 1 << lc;
      *held = ts_resident(lc) >= strips;
      return true;
    }
  }
  return false;
}

}  // namespace

// One launch while the device holds every strip's cluster at once and a CTA's own
// blocks fold at most six 8-column tiles a step (SOLVE_OWN: then the chain of blocks,
// not the folds, sets the pace), and one right-hand side always.  Else recursion
// with blocks of 512 rows up to q = 1200 and of 256 rows from there on.  Measured
// (a prediction, µs, one launch / 512): n = 1000, q = 64 112 / 134, 400 116 / 138;
// n = 2000, q = 64 172 / 254, 200 186 / 261, 320 (eight tiles) 312 / 283; n = 4096,
// q = 112 397 / 557, 160 (eight) 735 / 615; n = 8192, q = 48 844 / 1256, 64 (not held)
// 1691 / 1255; n = 16384, q = 8 (eight) 3150 / 2739.  Up to 512 rows both are the one
// launch, and the line lies where a prediction's sums by a CTA a column stop paying
// (n = 256, q = 1200 78 / 67).  The solve alone (512 / 256 / two
// GEMMs per 128 rows): n = 1000, q = 1000 104 / 122 / 232, 2000 192 / 176 / 281;
// n = 4096, q = 1500 1627 / 1546 / 1881, 10000 6887 / 6785 / 7763.  From q = 16384 on
// the launch's L2 reads (n²/2 values for every 16 columns) cost more than products of
// 128-row blocks with their inverses: an Sgpr evaluation (m = 1024, q = 10⁶) takes
// 344 ms with blocks of 256, 307 ms so.  One block of at most 128 rows goes there from
// q = 6000 on: the launch stages the block and its inverse for every 16 columns, the
// product for every 64 (a sparse prediction with two solves, m = 64, µs, launch /
// product: q = 4096 107 / 107, 8000 144 / 129, 16384 209 / 174; m = 16 107 / 103,
// 143 / 120, 202 / 160).
constexpr int SOLVE_OWN = 6;
constexpr int SOLVE_ONE_BLOCK_Q = 6000;
SolveClass solve_class(long long n, long long q) {
  int nt, c;
  bool held;
  if (q == 1) return SOLVE_FEW;
  if (q <= 1200 && (n > 512 || n * q <= 200000) && ts_plan((int)n, (int)q, &nt, &c, &held) && held &&
      nt * ceil_div(ceil_div((int)n, NB), c) <= SOLVE_OWN)
    return SOLVE_FEW;
  if (n <= NB && q > SOLVE_ONE_BLOCK_Q) return SOLVE_BULK;
  return q <= 1200 ? SOLVE_MID : q <= 16384 ? SOLVE_WIDE : SOLVE_BULK;
}

cudaError_t tri_solve(const double* L, long long ld, int n, const double* linv, double* B, long long ldb, int q,
                      bool trans, const DevStatus* st, cudaStream_t s) {
  if (n <= 0 || q <= 0) return cudaSuccess;
  int nt, c;
  bool held;
  if (!ts_plan(n, q, &nt, &c, &held)) return cudaErrorInvalidValue;
  const TriSolveArgs g{L, ld, n, linv, B, ldb, q, c, st};
  const int strips = ceil_div(q, 8 * nt);
  const size_t smem = ts_smem(nt, ceil_div(ceil_div(n, NB), c), q == 1);
  void (*kern)(TriSolveArgs) = trans ? (nt == 1 ? tri_solve_kernel<true, 1> : tri_solve_kernel<true, 2>)
                                     : (nt == 1 ? tri_solve_kernel<false, 1> : tri_solve_kernel<false, 2>);
  return ts_launch(kern, g, strips * c, smem, s);
}

cudaError_t tri_solve_vec(const double* L, long long ld, int n, const double* linv, double* b, bool trans,
                          const DevStatus* st, cudaStream_t s, double* prefix, long long ldp) {
  if (n <= 0) return cudaSuccess;
  const int nblk = ceil_div(n, NB);
  int c = 1;
  for (int lc = 1; lc <= 4 && (1 << lc) <= nblk && ts_resident(lc) > 0; ++lc) c = 1 << lc;
  const size_t smem = tv_smem(ceil_div(nblk, c));
  if (smem > TS_SMEM_MAX || (prefix && trans)) return cudaErrorInvalidValue;
  const TriVecArgs g{L, ld, n, linv, b, c, prefix, ldp, st};
  return ts_launch(trans ? tri_vec_kernel<true> : tri_vec_kernel<false>, g, c, smem, s);
}

}  // namespace gprx
