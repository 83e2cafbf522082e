// Kernels of the H-LU's tile schedule on dense diagonal tiles (hm_lu.cu): the
// tile's LU with leaf-local pivoting, the panel solves and the inverses of its
// triangles, the loads and trailing updates of the diagonal tiles.
#pragma once
#include "hm_internal.h"
#include "hm_lowrank.cuh"

#include <cooperative_groups.h>

namespace hm {

// ---------------------------------------------------------------------------
// diagonal tiles: load
// ---------------------------------------------------------------------------
// One stored leaf of a diagonal tile: dense (C) or low-rank (A B') elements of
// the storage format, written as FP64 into dst (column stride ldd)
struct DiagLoad {
  const void *C, *A, *B;
  int64_t ldc, lda, ldb, ldd;
  double* dst;
  int m, n, k, dense;      // dense: C holds the leaf
  int ctype, rtype;        // HM_F64 / HM_F32 / HM_BF16 of C, of A and B
};
__device__ __forceinline__ double diag_elem(const void* p, int64_t e, int type) {
  if (type == HM_F64) return ((const double*)p)[e];
  if (type == HM_F32) return (double)((const float*)p)[e];
  return (double)__bfloat162float(((const __nv_bfloat16*)p)[e]);
}
static __global__ void __launch_bounds__(256) lu_diag_load_kernel(const DiagLoad* __restrict__ jobs) {
  const DiagLoad J = jobs[blockIdx.x];
  for (int j = blockIdx.y; j < J.n; j += gridDim.y)
    for (int i = threadIdx.x; i < J.m; i += blockDim.x) {
      double v = 0.0;
      if (J.dense) v = diag_elem(J.C, i + j * J.ldc, J.ctype);
      else
        for (int q = 0; q < J.k; ++q)
          v = fma(diag_elem(J.A, i + q * J.lda, J.rtype), diag_elem(J.B, j + q * J.ldb, J.rtype), v);
      J.dst[i + j * J.ldd] = v;
    }
}

// ---------------------------------------------------------------------------
// diagonal tiles: LU with partial pivoting inside each diagonal leaf
// ---------------------------------------------------------------------------
// The S x S tile A (column-major, ld S), diagonal leaves [leaf[p], leaf[p+1]):
// leaf by leaf the leaf's own LU, the solves of its row and column panels and
// the update of what remains, as lu! does on the tile's blocks
// (src/hlu.jl:465-515); P[goff + i] receives the pivots.  One cluster of eight
// CTAs: the leaf's LU runs in one CTA's shared memory, the panels and the
// update (32 x 32 blocks on FP64 matrix instructions) on all 64 warps, cluster
// barriers between.  Bound: the latency of the leaves' LU, one column after
// another.  The tile lives in L2; it is read with .cg loads, since the CTAs of
// other SMs write it.
constexpr int DL_CTAS = 8, DL_WARPS = 8;

struct DiagLu {
  double* A;
  int S, nleaf;
  const int32_t* leaf;
  int64_t* P;
  int64_t goff;
  int* flags;
};

// LU of the m x m block D (column stride ld) by one CTA; perm[i] = the row of
// the block that ends up in row i.  First maximum as pivot, whole-row swaps.
static __device__ __forceinline__ int leaf_pivot(const double* col, int j, int m, int lane, int* flags) {
  double best = -1.0;
  int bi = INT32_MAX;
  for (int i = j + lane; i < m; i += 32) {
    const double a = fabs(col[i]);
    if (a > best) { best = a; bi = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double a2 = __shfl_xor_sync(0xffffffffu, best, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
    if (a2 > best || (a2 == best && i2 < bi)) { best = a2; bi = i2; }
  }
  // every candidate NaN: no maximum was found; keep the row
  const bool none = bi == INT32_MAX;
  if (lane == 0 && (none || !(best != 0.0))) atomicOr(flags, none ? 6 : 4);   // exactly zero (or NaN) pivot
  return none ? j : bi;
}
static __device__ void leaf_getrf(double* D, int ld, int m, int* perm, int* flags) {
  __shared__ int s_piv;
  __shared__ double mult[160];                           // column j's multipliers
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int i = threadIdx.x; i < m; i += blockDim.x) perm[i] = i;
  if (warp == 0) {
    const int p = leaf_pivot(D, 0, m, lane, flags);
    if (lane == 0) s_piv = p;
  }
  __syncthreads();
  for (int j = 0; j < m; ++j) {
    // column j: swapped and divided by warp 0, the other columns swapped
    const int p = s_piv;
    if (warp == 0) {
      double* col = D + j * ld;
      const double piv = col[p], old = col[j];
      __syncwarp();
      for (int i = j + 1 + lane; i < m; i += 32) {
        double l = i == p ? old : col[i];
        if (piv != 0.0) l /= piv;
        col[i] = l;
        mult[i] = l;
      }
      if (lane == 0) {
        col[j] = piv;
        const int t = perm[j];
        perm[j] = perm[p];
        perm[p] = t;
      }
    }
    if (p != j)
      for (int c = threadIdx.x - 32; c < m; c += blockDim.x - 32)
        if (c >= 0 && c != j) {
          const double t = D[j + c * ld];
          D[j + c * ld] = D[p + c * ld];
          D[p + c * ld] = t;
        }
    __syncthreads();
    // the other columns, a warp each: column j + 1 first, whose pivot warp 0
    // finds before the barrier
    for (int c = j + 1 + warp; c < m; c += nwarp) {
      double* col = D + c * ld;
      const double u = col[j];
      for (int i = j + 1 + lane; i < m; i += 32) col[i] = fma(-mult[i], u, col[i]);
    }
    if (warp == 0 && j + 1 < m) {
      __syncwarp();
      const int pn = leaf_pivot(D + (j + 1) * ld, j + 1, m, lane, flags);
      if (lane == 0) s_piv = pn;
    }
    __syncthreads();
  }
}

// The kernels below run a sequence of short solves, each by a few warps once: a
// solve unrolled over its 32 steps is 500 to 4000 instructions that are fetched
// from L2 for one use (12,000 cycles for a 32 x 32 solve).  So the loops over
// the steps stay loops: the register window slides instead, x[i - 1] = x[i] -
// (factor) x[0].

// Columns [jb, jb + 32) of the block, rows jb .. m - 1 (at most 32 RPL), by one
// warp with its rows in registers: a pivot costs three warp reductions of the
// values' bit patterns, a division and the broadcasts of the pivot row, and no
// barrier.  Rows are not moved until the end: pos is the place a row has
// reached, and ends as where it goes (dst[i] = place of row jb + i); a column
// is stored when it is finished, in the rows' old places.
template <int RPL>
static __device__ __forceinline__ void leaf_panel(double* D, int ld, int m, int jb, int* dst, int* flags) {
  const int lane = threadIdx.x & 31;
  const int nb = min(32, m - jb);
  double x[RPL][32];
  int pos[RPL];
#pragma unroll
  for (int u = 0; u < RPL; ++u) {
    const int i = jb + lane + 32 * u;
    pos[u] = i < m ? i : INT32_MAX;
#pragma unroll
    for (int c = 0; c < 32; ++c) x[u][c] = D[min(i, m - 1) + (jb + min(c, nb - 1)) * ld];
  }
#pragma unroll 1
  for (int j = jb; j < jb + nb; ++j) {
    // largest magnitude among the rows from place j on (NaN: none), the first
    // place on ties
    unsigned hi = 0, lo = 0;
    int at = INT32_MAX;
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      const double v = fabs(x[u][0]);
      if (pos[u] >= j && pos[u] != INT32_MAX && v == v) {
        const unsigned h = (unsigned)__double2hiint(v) + 1u, l = (unsigned)__double2loint(v);
        if (h > hi || (h == hi && (l > lo || (l == lo && pos[u] < at)))) { hi = h; lo = l; at = pos[u]; }
      }
    }
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    int pp = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml && mh ? at : INT32_MAX);
    if (mh == 0u) pp = j;                                  // every candidate NaN: keep the row
    if (lane == 0 && (mh == 0u || (mh == 1u && ml == 0u))) atomicOr(flags, mh == 0u ? 6 : 4);   // or a zero pivot
    bool mine = false;
    int slot = 0;
#pragma unroll
    for (int u = 0; u < RPL; ++u)
      if (pos[u] == pp) { mine = true; slot = u; }
    const int pl = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
    const int ps = RPL > 1 ? __shfl_sync(0xffffffffu, slot, pl) : 0;
#pragma unroll
    for (int u = 0; u < RPL; ++u) {                        // rows pp and j trade places
      if (pos[u] == pp) pos[u] = j;
      else if (pos[u] == j) pos[u] = pp;
    }
    auto from_pivot = [&](int c) {
      double v = x[0][c];
      if (RPL > 1 && ps) v = x[RPL - 1][c];
      return __shfl_sync(0xffffffffu, v, pl);
    };
    const double piv = from_pivot(0);
    double f[RPL];                                         // multipliers (of the rows not placed yet)
#pragma unroll
    for (int u = 0; u < RPL; ++u) {
      double l = x[u][0];
      if (pos[u] > j && piv != 0.0) l /= piv;
      f[u] = l;
      if (jb + lane + 32 * u < m) D[jb + lane + 32 * u + j * ld] = l;
    }
#pragma unroll
    for (int c = 1; c < 32; ++c) {
      const double w = from_pivot(c);
#pragma unroll
      for (int u = 0; u < RPL; ++u) x[u][c - 1] = pos[u] > j ? fma(-f[u], w, x[u][c]) : x[u][c];
    }
  }
  __syncwarp();
  // the rows of the panel to their places, column by column
#pragma unroll 1
  for (int c = jb; c < jb + nb; ++c) {
    double v[RPL];
#pragma unroll
    for (int u = 0; u < RPL; ++u) v[u] = D[min(jb + lane + 32 * u, m - 1) + c * ld];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < RPL; ++u)
      if (jb + lane + 32 * u < m) D[pos[u] + c * ld] = v[u];
    __syncwarp();
  }
#pragma unroll
  for (int u = 0; u < RPL; ++u)
    if (jb + lane + 32 * u < m) dst[lane + 32 * u] = pos[u];
  __syncwarp();
}

// The same LU for blocks of at most 64 rows: one or two warp panels, between
// them the row exchanges, the solve and the update of the other half by all
// warps.
template <int M>
static __device__ void leaf_getrf_small(double* D, int ld, int m, int* perm, int* flags) {
  __shared__ int dst[64];
  __shared__ int old[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int i = threadIdx.x; i < m; i += blockDim.x) perm[i] = i;
  __syncthreads();
  for (int jb = 0; jb < m; jb += 32) {
    if (warp == 0) {
      if (M > 32 && m - jb > 32) leaf_panel<2>(D, ld, m, jb, dst, flags);
      else leaf_panel<1>(D, ld, m, jb, dst, flags);
    }
    __syncthreads();
    const int nr = m - jb, nb = min(32, nr);
    // the other columns' rows, and the permutation, go the same way
    if (threadIdx.x < nr) old[threadIdx.x] = perm[jb + threadIdx.x];
    for (int c = warp; c < m; c += nwarp) {
      if (c >= jb && c < jb + nb) continue;
      double* col = D + c * ld + jb;
      const double v0 = lane < nr ? col[lane] : 0.0, v1 = lane + 32 < nr ? col[lane + 32] : 0.0;
      __syncwarp();
      if (lane < nr) D[c * ld + dst[lane]] = v0;
      if (lane + 32 < nr) D[c * ld + dst[lane + 32]] = v1;
    }
    __syncthreads();
    if (threadIdx.x < nr) perm[dst[threadIdx.x]] = old[threadIdx.x];
    if (M > 32 && nr > 32) {                               // nb = 32: the columns right of the panel
      if (warp == 0 && jb + 32 + lane < m) {
        double* col = D + (jb + 32 + lane) * ld + jb;
        double x[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = col[i];
        // (entries whose row lies past the panel's 32 are never used)
#pragma unroll 1
        for (int l = 0; l < 32; ++l) {
          const double xl = x[0];
          const double* f = D + jb + l + (jb + l) * ld;
          col[l] = xl;
#pragma unroll
          for (int i = 1; i < 32; ++i) x[i - 1] = fma(-f[i], xl, x[i]);
        }
      }
      __syncthreads();
      const int rem = nr - 32;
      for (int e = threadIdx.x; e < 32 * rem; e += blockDim.x) {
        const int i = e & 31, c = jb + 32 + (e >> 5);
        if (i < rem) {
          double v = D[jb + 32 + i + c * ld];
#pragma unroll 8
          for (int l = 0; l < 32; ++l) v = fma(-D[jb + 32 + i + (jb + l) * ld], D[jb + l + c * ld], v);
          D[jb + 32 + i + c * ld] = v;
        }
      }
    }
    __syncthreads();
  }
}

// M: rows of a leaf at most (32, 64: panel columns in registers; 160: in place)
template <int M>
__global__ void __cluster_dims__(DL_CTAS, 1, 1) __launch_bounds__(32 * DL_WARPS, 1) lu_diag_kernel(DiagLu a) {
  namespace cg = cooperative_groups;
  auto cluster = cg::this_cluster();
  extern __shared__ double sm[];
  constexpr int LD = M + 1;
  double* D = sm;                                        // the leaf's block
  double* rinv = D + M * LD;                             // 1 / its pivots
  double* stage = rinv + M;                              // a warp's 32 columns (M <= 64)
  __shared__ int perm[M];
  const int rank = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int gw = rank * DL_WARPS + warp, nw = DL_CTAS * DL_WARPS;
  const int S = a.S;
  double* A = a.A;
  // leaf [j0, j0 + m) in rank 0's D: its LU, written back with the pivots
  auto leaf_lu = [&](int j0, int m) {
    {
      if constexpr (M <= 64) leaf_getrf_small<M>(D, LD, m, perm, a.flags);
      else leaf_getrf(D, LD, m, perm, a.flags);
      for (int e = threadIdx.x; e < m * m; e += blockDim.x)
        A[(j0 + e % m) + (int64_t)(j0 + e / m) * S] = D[e % m + e / m * LD];
      for (int i = threadIdx.x; i < m; i += blockDim.x) a.P[a.goff + j0 + i] = a.goff + j0 + perm[i];
    }
  };
  if (rank == 0) {
    const int m = a.leaf[1];
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) D[e % m + e / m * LD] = __ldcg(A + e % m + (int64_t)(e / m) * S);
    __syncthreads();
    leaf_lu(0, m);
  }
  for (int p = 0; p < a.nleaf; ++p) {
    const int j0 = a.leaf[p], j1 = a.leaf[p + 1], m = j1 - j0;
    cluster.sync();
    if (rank != 0) {
#pragma unroll 4
      for (int e = threadIdx.x; e < m * m; e += 32 * DL_WARPS)
        D[e % m + e / m * LD] = __ldcg(A + (j0 + e % m) + (int64_t)(j0 + e / m) * S);
      for (int i = threadIdx.x; i < m; i += blockDim.x) perm[i] = (int)(__ldcg(a.P + a.goff + j0 + i) - a.goff - j0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) rinv[i] = i < m ? 1.0 / D[i + i * LD] : 1.0;
    __syncthreads();
    // row panel: rows [j0, j1) of every other column, permuted, and solved
    // with the unit lower triangle right of the leaf
    const int nc = S - m;
    if constexpr (M <= 64) {
      double* T = stage + warp * 32 * LD;
      for (int it = gw; it * 32 < nc; it += nw) {
        // (past the last column: the last again, not stored; loads in flight
        // together, one column after another they cost an L2 latency each)
#pragma unroll
        for (int i0 = 0; i0 < M; i0 += 32) {
          const double* row = A + j0 + perm[min(i0 + lane, m - 1)];
#pragma unroll
          for (int cc0 = 0; cc0 < 32; cc0 += 16) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
              const int c = min(it * 32 + cc0 + u, nc - 1);
              v[u] = __ldcg(row + (int64_t)(c < j0 ? c : c + m) * S);
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) T[(cc0 + u) * LD + i0 + lane] = v[u];
          }
        }
        __syncwarp();
        const int c = it * 32 + lane;
        if (c < nc && c >= j0) {
          double x[M];
#pragma unroll
          for (int i = 0; i < M; ++i) x[i] = T[lane * LD + i];
#pragma unroll 1
          for (int l = 0; l < m; ++l) {
            const double xl = x[0];
            const double* f = D + l + l * LD;                // (what lies past the leaf is never used)
            T[lane * LD + l] = xl;
#pragma unroll
            for (int i = 1; i < M; ++i) x[i - 1] = fma(-f[i], xl, x[i]);
          }
        }
        __syncwarp();
        for (int cc = 0; cc < 32 && it * 32 + cc < nc; ++cc) {
          const int c2 = it * 32 + cc, col = c2 < j0 ? c2 : c2 + m;
          for (int i = lane; i < m; i += 32) A[(j0 + i) + (int64_t)col * S] = T[cc * LD + i];
        }
        __syncwarp();
      }
    } else {
      for (int c = gw * 32 + lane; c < nc; c += nw * 32) {
        const int col = c < j0 ? c : c + m;
        double* x = A + j0 + (int64_t)col * S;
        double t[M];
        for (int i = 0; i < m; ++i) t[i] = __ldcg(x + perm[i]);
        if (c >= j0)
          for (int l = 0; l < m; ++l)
            for (int i = l + 1; i < m; ++i) t[i] = fma(-D[i + l * LD], t[l], t[i]);
        for (int i = 0; i < m; ++i) x[i] = t[i];
      }
    }
    // column panel: columns [j0, j1) of the rows below, times the inverse of
    // the leaf's upper triangle
    // (from the last warp down: the first ones have a row panel)
    for (int r = j1 + (nw - 1 - gw) * 32 + lane; r < S; r += nw * 32) {
      double* xr = A + r + (int64_t)j0 * S;
      double x[M];
      if constexpr (M <= 64) {
#pragma unroll
        for (int l = 0; l < M; ++l) x[l] = __ldcg(xr + (int64_t)min(l, m - 1) * S);
#pragma unroll 1
        for (int l = 0; l < m; ++l) {
          const double xl = x[0] * rinv[l];
          const double* f = D + l + l * LD;
          xr[(int64_t)l * S] = xl;
#pragma unroll
          for (int c = 1; c < M; ++c) x[c - 1] = fma(-f[c * LD], xl, x[c]);
        }
      } else {
        for (int l = 0; l < m; ++l) x[l] = __ldcg(xr + (int64_t)l * S);
        for (int l = 0; l < m; ++l) {
          x[l] *= rinv[l];
          for (int c = l + 1; c < m; ++c) x[c] = fma(-x[l], D[l + c * LD], x[c]);
        }
        for (int l = 0; l < m; ++l) xr[(int64_t)l * S] = x[l];
      }
    }
    cluster.sync();
    if (p + 1 == a.nleaf) break;
    // the rest: A -= (column panel) (row panel).  Rank 0 updates the next leaf's
    // block into its D and factorises it, the others meanwhile everything else
    const int j2 = a.leaf[p + 2], m2 = j2 - j1;
    if (rank == 0) {
      // an 8 x 8 block a warp, 16 K values' operands in flight
      const int n8 = (m2 + 7) / 8;
      for (int it = warp; it < n8 * n8; it += DL_WARPS) {
        const int r0 = j1 + it % n8 * 8, c0 = j1 + it / n8 * 8;
        const int ra = min(r0 + g, S - 1), cb = min(c0 + g, S - 1);
        double acc[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) acc[h] = __ldcg(A + ra + (int64_t)min(c0 + 2 * q + h, S - 1) * S);
#pragma unroll 1
        for (int k = 0; k < m; k += 32) {
          double x[8], y[8];
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const int kk = min(k + 4 * s + q, m - 1);
            x[s] = __ldcg(A + ra + (int64_t)(j0 + kk) * S);
            y[s] = __ldcg(A + (j0 + kk) + (int64_t)cb * S);
          }
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const bool in = k + 4 * s + q < m;
            dmma(acc, in ? -x[s] : 0.0, in ? y[s] : 0.0);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 - j1 + g, c = c0 - j1 + 2 * q + h;
          if (r < m2 && c < m2) D[r + c * LD] = acc[h];
        }
      }
      __syncthreads();
      leaf_lu(j1, m2);
    } else if constexpr (M <= 64) {
      // strips of 32 rows: the strip's column panel and the row panel, 256
      // columns at a time, go through shared memory (over the panels'
      // staging), then a 32 x 32 block a warp
      constexpr int LL = 36, LU_ = M + 4;                    // strides: 4 modulo 16
      double* Ls = stage;                                    // [k][32 rows]
      double* Us = Ls + M * LL;                              // [column][k]
      const int mk = (m + 3) / 4 * 4;
      for (int r0 = j1 + 32 * (rank - 1); r0 < S; r0 += 32 * (DL_CTAS - 1)) {
        __syncthreads();
        for (int e = threadIdx.x; e < mk * 32; e += 32 * DL_WARPS) {
          const int r = e & 31, k = e >> 5;
          Ls[k * LL + r] = k < m && r0 + r < S ? -__ldcg(A + r0 + r + (int64_t)(j0 + k) * S) : 0.0;
        }
        for (int c0 = j1; c0 < S; c0 += 32 * DL_WARPS) {
          __syncthreads();
          const int ncol = min(32 * DL_WARPS, S - c0);
#pragma unroll 8
          for (int e = threadIdx.x; e < mk * ncol; e += 32 * DL_WARPS) {
            const int k = e % mk, c = e / mk;
            Us[c * LU_ + k] = k < m ? __ldcg(A + j0 + k + (int64_t)(c0 + c) * S) : 0.0;
          }
          const int cw = c0 + 32 * warp;                     // this warp's columns
          double acc[4][4][2];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                acc[i][j][h] = __ldcg(A + min(r0 + 8 * i + g, S - 1) + (int64_t)min(cw + 8 * j + 2 * q + h, S - 1) * S);
          __syncthreads();
          if (cw < S) {
#pragma unroll 1
            for (int k = 0; k < mk; k += 4) {
              double x[4], y[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) x[i] = Ls[(k + q) * LL + 8 * i + g];
#pragma unroll
              for (int j = 0; j < 4; ++j) y[j] = Us[(32 * warp + 8 * j + g) * LU_ + k + q];
#pragma unroll
              for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j], x[i], y[j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const int r = r0 + 8 * i + g, c = cw + 8 * j + 2 * q + h;
                  if (r < S && c < S && (r >= j2 || c >= j2)) A[r + (int64_t)c * S] = acc[i][j][h];
                }
          }
        }
      }
    } else {
      for (int c = j1 + gw - DL_WARPS; c < S; c += nw - DL_WARPS)
        for (int r = j1 + lane; r < S; r += 32) {
          if (r < j2 && c < j2) continue;
          double v = __ldcg(A + r + (int64_t)c * S);
          for (int k = 0; k < m; ++k)
            v = fma(-__ldcg(A + r + (int64_t)(j0 + k) * S), __ldcg(A + (j0 + k) + (int64_t)c * S), v);
          A[r + (int64_t)c * S] = v;
        }
    }
  }
}

// shared memory: the leaf, the reciprocals, then the row panels' staging or the
// operands of the update; the solves read up to M columns past the leaf
template <int M> constexpr size_t diag_lu_smem() {
  const size_t base = (size_t)M * (M + 1) + M;
  if (M > 64) return sizeof(double) * base;
  const size_t panel = (size_t)DL_WARPS * 32 * (M + 1);
  const size_t upd = (size_t)M * 36 + (size_t)32 * DL_WARPS * (M + 4);
  return sizeof(double) * (base + (panel > upd ? panel : upd));
}

// ---------------------------------------------------------------------------
// triangular solves with a factored tile
// ---------------------------------------------------------------------------
// X <- T^-1 X for up to 32 columns in shared memory (column stride ldx, a
// multiple of 16 plus 4: the matrix operands then read 16 banks at a time), T
// lower triangular with element (i, l) at T[i rs + l cs], unit or not, from row
// block b0 on.  By blocks of 32 rows: what the finished rows contribute on FP64
// matrix instructions (8 warps: 8 rows x 16 columns each), then the block's own
// triangle by substitution, one column a lane.
constexpr int TP_COLS = 32;
static inline __host__ __device__ int tp_ldx(int S) { return (S + 11) / 16 * 16 + 4; }

static __device__ void tile_trsm(const double* __restrict__ T, int64_t rs, int64_t cs, int S, bool unit, double* X,
                                 int ldx, int nc, int b0, double* L, double* rinv) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int mt = warp & 3, nh = warp >> 2;
  for (int r0 = b0; r0 < S; r0 += 32) {
    const int nr = min(32, S - r0);
    // the block's triangle, column-major with stride 33
    for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
      int i, l;
      if (rs == 1 || rs == -1) { i = e & 31; l = e >> 5; } else { l = e & 31; i = e >> 5; }
      // skewed: row l + d of column l at d + 32 l, zeros past the end
      if (l <= i) {
        const double v = i < nr ? __ldg(T + (r0 + i) * rs + (r0 + l) * cs) : 0.0;
        L[i - l + l * 32] = v;
        if (i == l) rinv[i] = unit || i >= nr ? 1.0 : 1.0 / v;
      } else {
        L[32 - l + i + l * 32] = 0.0;
      }
    }
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    const double* tp = T + min(r0 + 8 * mt + g, S - 1) * rs;
    const double* x0 = X + (16 * nh + g) * ldx;
    const double* x1 = x0 + 8 * ldx;
#pragma unroll 8
    for (int k = b0; k < r0; k += 4) {
      const double t = __ldg(tp + (k + q) * cs);
      dmma(acc[0], t, x0[k + q]);
      dmma(acc[1], t, x1[k + q]);
    }
    if (8 * mt + g < nr) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < 2; ++u) X[(16 * nh + 8 * h + 2 * q + u) * ldx + r0 + 8 * mt + g] -= acc[h][u];
    }
    __syncthreads();
    if (warp == 0 && lane < nc) {
      double* xp = X + lane * ldx + r0;
      double x[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) x[i] = xp[min(i, nr - 1)];
#pragma unroll 1
      for (int l = 0; l < nr; ++l) {
        const double xl = x[0] * rinv[l];
        const double* f = L + l * 32;
        xp[l] = xl;
#pragma unroll
        for (int i = 1; i < 32; ++i) x[i - 1] = fma(-f[i], xl, x[i]);
      }
    }
    __syncthreads();
  }
}

static inline size_t tp_smem(int S) { return sizeof(double) * ((size_t)TP_COLS * tp_ldx(S) + 32 * 33 + 32); }

// The panels of step k: blockIdx.y = 0: the A factors of tiles (k, j > k), rows
// permuted, times L^-1; 1: the B factors of tiles (i > k, k) times U^-T.  A CTA
// takes TP_TILES tiles and solves their columns below the rank, 32 at a time.
constexpr int TP_TILES = 4;
struct PanelArgs {
  const double* D;         // the factored tile, S x S
  int S, T, k, cap;
  const int64_t* P;        // + goff: its pivots
  int64_t goff;
  double *Ap, *Bp;         // panels of tile k
  const int32_t* kmat;
};
static __global__ void __launch_bounds__(256) lu_panel_kernel(PanelArgs a) {
  extern __shared__ double sm[];
  const int S = a.S, ldx = tp_ldx(S);
  double* X = sm;
  double* L = X + TP_COLS * ldx;
  double* rinv = L + 32 * 33;
  __shared__ double* col[TP_COLS];
  __shared__ int s_n, s_tile, s_col;
  const bool up = blockIdx.y == 0;
  const int t0 = a.k + 1 + (int)blockIdx.x * TP_TILES, t1 = min(a.T, t0 + TP_TILES);
  int tile = t0, c = 0;                                  // next column: c of `tile`
  for (;;) {
    if (threadIdx.x == 0) {
      int n = 0;
      while (tile < t1 && n < TP_COLS) {
        const int r = up ? a.kmat[a.k * a.T + tile] : a.kmat[tile * a.T + a.k];
        double* base = (up ? a.Ap : a.Bp) + (int64_t)tile * a.cap * S;
        while (c < r && n < TP_COLS) col[n++] = base + (int64_t)c++ * S;
        if (c >= r) { ++tile; c = 0; }
      }
      s_n = n; s_tile = tile; s_col = c;
    }
    __syncthreads();
    const int n = s_n;
    tile = s_tile;
    c = s_col;
    if (n == 0) return;
    for (int e = threadIdx.x; e < TP_COLS * S; e += blockDim.x) {
      const int cc = e / S, i = e % S;
      double v = 0.0;
      if (cc < n) v = col[cc][up ? (int)(a.P[a.goff + i] - a.goff) : i];
      X[cc * ldx + i] = v;
    }
    __syncthreads();
    if (up) tile_trsm(a.D, 1, S, S, true, X, ldx, n, 0, L, rinv);
    else tile_trsm(a.D, S, 1, S, false, X, ldx, n, 0, L, rinv);
    for (int e = threadIdx.x; e < n * S; e += blockDim.x) col[e / S][e % S] = X[(e / S) * ldx + e % S];
    __syncthreads();
  }
}

// Inverses of the unit lower L (blockIdx.z = 0) and the upper U (1) of the
// packed tiles D, 32 columns a CTA: column-major into C, row-major into R
// (zeros in the other triangle included).
struct InverseArgs {
  const double* const* D;
  double* const* C[2];
  double* const* R[2];
  const int32_t* size;
};
static __global__ void __launch_bounds__(256) lu_inverse_kernel(InverseArgs a) {
  extern __shared__ double sm[];
  const int tile = blockIdx.y, S = a.size[tile], c0 = (int)blockIdx.x * TP_COLS;
  if (c0 >= S) return;
  const int ldx = tp_ldx(S), n = min(TP_COLS, S - c0);
  double* X = sm;
  double* L = X + TP_COLS * ldx;
  double* rinv = L + 32 * 33;
  const double* D = a.D[tile];
  for (int e = threadIdx.x; e < TP_COLS * S; e += blockDim.x) X[(e / S) * ldx + e % S] = e % S == c0 + e / S ? 1.0 : 0.0;
  __syncthreads();
  // columns c0 .. of the identity: the rows above c0 stay zero
  const bool up = blockIdx.z == 1;
  if (!up) tile_trsm(D, 1, S, S, true, X, ldx, n, c0, L, rinv);
  else tile_trsm(D, S, 1, S, false, X, ldx, n, c0, L, rinv);
  // X holds columns c0 .. of L^-1, or of U^-T (rows c0 .. of U^-1)
  double* major = (up ? a.R[1] : a.C[0])[tile];
  double* minor = (up ? a.C[1] : a.R[0])[tile];
  for (int e = threadIdx.x; e < n * S; e += blockDim.x) major[(int64_t)(c0 + e / S) * S + e % S] = X[(e / S) * ldx + e % S];
  for (int e = threadIdx.x; e < n * S; e += blockDim.x) minor[(int64_t)(e / n) * S + c0 + e % n] = X[(e % n) * ldx + e / n];
}

// ---------------------------------------------------------------------------
// trailing diagonal tiles: D_i -= A_ik (B_ik' A_ki) B_ki'
// ---------------------------------------------------------------------------
struct DiagUpdate {
  const double* const* Ap;
  const double* const* Bp;
  double* const* D;
  const int32_t* size;
  const int32_t* kmat;
  int T, cap, k, i0;       // tiles i0 + blockIdx.y
};
// A CTA updates 32 rows of a tile: W = B_ik' A_ki (every CTA its own copy, a
// few dot products), its rows of A_ik W, then the rank-k update.  Bound: the
// tile's bytes, read and written once.
static __global__ void __launch_bounds__(256) lu_diag_update_kernel(DiagUpdate a) {
  extern __shared__ double sm[];
  const int i = a.i0 + (int)blockIdx.y, k = a.k, S = a.size[i], Sk = a.size[k], r0 = (int)blockIdx.x * 32;
  const int ka = a.kmat[i * a.T + k], kb = a.kmat[k * a.T + i];
  if (r0 >= S || ka == 0 || kb == 0) return;
  double* W = sm;                                        // ka x kb
  double* Q = W + a.cap * a.cap;                         // 32 x kb, row-major
  const double* Bik = a.Bp[k] + (int64_t)i * a.cap * Sk;
  const double* Aki = a.Ap[k] + (int64_t)i * a.cap * Sk;
  const double* Aik = a.Ap[i] + (int64_t)k * a.cap * S;
  const double* Bki = a.Bp[i] + (int64_t)k * a.cap * S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = warp; e < ka * kb; e += 8) {
    const double *x = Bik + (int64_t)(e % ka) * Sk, *y = Aki + (int64_t)(e / ka) * Sk;
    double s = 0.0;
#pragma unroll 4
    for (int t = lane; t < Sk; t += 32) s = fma(x[t], y[t], s);
    s = warp_sum(s);
    if (lane == 0) W[e] = s;
  }
  __syncthreads();
  const int nr = min(32, S - r0);
  for (int e = threadIdx.x; e < 32 * kb; e += 256) {
    const int r = e & 31, c = e >> 5;
    double s = 0.0;
    if (r < nr)
      for (int l = 0; l < ka; ++l) s = fma(Aik[r0 + r + (int64_t)l * S], W[l + c * ka], s);
    Q[r * a.cap + c] = s;
  }
  __syncthreads();
  if (lane >= nr) return;
  double* d = a.D[i] + r0 + lane;
  for (int j0 = warp * 8; j0 < S; j0 += 64) {            // eight columns in flight
    double s[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) s[u] = j0 + u < S ? d[(int64_t)(j0 + u) * S] : 0.0;
    for (int c = 0; c < kb; ++c) {
      const double x = -Q[lane * a.cap + c];
#pragma unroll
      for (int u = 0; u < 8; ++u) s[u] = fma(x, __ldg(Bki + min(j0 + u, S - 1) + (int64_t)c * S), s[u]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + u < S) d[(int64_t)(j0 + u) * S] = s[u];
  }
}

}  // namespace hm
