// Multi-RHS H-matvec (K5) with FP64 arithmetic: Y = H X and Y = H' X for an
// n x c block of right-hand sides, the device form of *(Hmat, Matrix)
// (src/harithm.jl:323-329), which the reference evaluates one column at a
// time.  Every factor is streamed from HBM once per block of at most 32
// columns.  This is the path of FP64 factors (tcgen05 has no FP64 kind); the
// low-rank part of FP32/BF16 handles runs on the tensor cores in FP32
// (hm_matvec_tc.cu), their dense leaves here (mvm_dense_kernel).
//
// Both phases are chains of FP64 tensor-core MMAs (mma.sync m8n8k4, the one
// FP64 matrix instruction) with the factors read straight from global memory
// in the operand layout: lane (g, q) = (lane / 4, lane % 4) holds A(g, q),
// B(q, g) and C(g, 2 q), C(g, 2 q + 1).  An 8 x 4 block of a column-major
// factor is four runs of 64 bytes (phase 2), its transpose eight runs of 64
// bytes for two MMAs (phase 1), so no staging in shared memory is needed.
// Bound: HBM up to 16 columns (an MMA's 256 FMAs take 4 cycles of an SM: 32
// bytes of factor a cycle against the 23 that HBM delivers), FP64 beyond.
//
// Phase 1: Z = F1' X_seg, a warp per tile of 32 factor columns that share an
//          input segment (K = segment rows, N = right-hand sides).
// Phase 2: Y = F2 Z + C X, a CTA per row slab (the slabs of the single-column
//          phase 2): its warps are groups of 32 rows times a split of the
//          slab's entries, whose partial sums meet in shared memory.
#include "hm_internal.h"
#include "hm_lowrank.cuh"

#include <algorithm>
#include <type_traits>
#include <vector>

namespace hm {

// One factor column of F1 and a tile of up to 32 of them (one input segment)
struct MbCol {
  uint64_t off;            // pool element offset of the column
  uint64_t z;              // its row of Z
};
struct MbTile {
  uint32_t col0, ncol, seg0, len;
};

namespace {

// two consecutive elements of a factor column as FP64 (the pair starts on an
// even element; columns are padded to 4 elements and 16 bytes)
__device__ __forceinline__ double2 ld_pair(const double* p) { return __ldcs(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ double2 ld_pair(const float* p) {
  const float2 v = __ldcs(reinterpret_cast<const float2*>(p));
  return make_double2(v.x, v.y);
}
__device__ __forceinline__ double2 ld_pair(const __nv_bfloat16* p) {
  const uint32_t w = __ldcs(reinterpret_cast<const unsigned int*>(p));
  return make_double2((double)__uint_as_float(w << 16), (double)__uint_as_float(w & 0xffff0000u));
}
__device__ __forceinline__ double ld_one(const double* p) { return __ldcs(p); }
__device__ __forceinline__ double ld_one(const float* p) { return (double)__ldcs(p); }
__device__ __forceinline__ double ld_one(const __nv_bfloat16* p) {
  return (double)__uint_as_float((uint32_t)__ldcs(reinterpret_cast<const unsigned short*>(p)) << 16);
}

constexpr int MB_MT = 4;                    // M tiles (of 8) a warp owns: 32 factor columns, 32 output rows
constexpr int MB_WARPS = 8;

// ---------------------------------------------------------------------------
// phase 1
// ---------------------------------------------------------------------------
template <typename T, int NT>
__global__ void __launch_bounds__(MB_WARPS * 32, NT <= 2 ? 2 : 1)
    mb_phase1_kernel(const MbTile* __restrict__ tiles, int64_t ntile, const MbCol* __restrict__ cols,
                     const T* __restrict__ pool, const double* __restrict__ X, int64_t ldx, int ncols, int ncb,
                     double* __restrict__ Z, int ldz) {
  constexpr int PD = sizeof(T) == 2 ? 8 : 4;              // columns are padded to PD elements (col_pad_elems)
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int64_t gw = (int64_t)blockIdx.x * MB_WARPS + (threadIdx.x >> 5);
  const int64_t nw = (int64_t)gridDim.x * MB_WARPS;
  for (int64_t w = gw; w < ntile * ncb; w += nw) {
    const MbTile tl = tiles[w / ncb];
    const int cb = (int)(w % ncb) * 8 * NT;
    const T* F[MB_MT];
#pragma unroll
    for (int i = 0; i < MB_MT; ++i)
      F[i] = pool + cols[tl.col0 + min((uint32_t)(8 * i + g), tl.ncol - 1)].off;
    const int mt = (int)((tl.ncol + 7) / 8);
    const int len = (int)tl.len, plen = (len + PD - 1) / PD * PD;
    const double* xb[NT];                                // X's columns of this lane (past the last: the last, into unused columns of Z)
#pragma unroll
    for (int j = 0; j < NT; ++j) xb[j] = X + tl.seg0 + (int64_t)min(cb + 8 * j + g, ncols - 1) * ldx;
    // pairs of X in one load where every column's segment is 16-byte aligned
    const bool pair = !(len & 1) && !((reinterpret_cast<uintptr_t>(X) >> 3 | tl.seg0 | (uint64_t)ldx) & 1);
    double acc[MB_MT][NT][2];
#pragma unroll
    for (int i = 0; i < MB_MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    // 16 rows a step (K index 8 h + 2 q + s -> MMA s of half h), the operands
    // of the next D steps in flight
    constexpr int D = 1;
    double2 a[D][MB_MT][2], x[D][NT][2];
    auto load = [&](int r0, double2 (&A)[MB_MT][2], double2 (&B)[NT][2]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // unconditional loads (a branch would put each beside its use): past
        // the end the last rows are read again and zeros multiplied
        const int r = r0 + 8 * h + 2 * q;
#pragma unroll
        for (int i = 0; i < MB_MT; ++i) {
          A[i][h] = ld_pair(F[i] + min(r, plen - 2));
          if (r >= plen) A[i][h] = make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          if (pair) {
            B[j][h] = __ldg(reinterpret_cast<const double2*>(xb[j] + min(r, len - 2)));
          } else {
            B[j][h].x = __ldg(xb[j] + min(r, len - 1));
            B[j][h].y = __ldg(xb[j] + min(r + 1, len - 1));
          }
          if (r >= len) B[j][h].x = 0.0;
          if (r + 1 >= len) B[j][h].y = 0.0;
        }
      }
    };
#pragma unroll
    for (int d = 0; d < D; ++d) load(16 * d, a[d], x[d]);
    for (int r0 = 0; r0 < len; r0 += 16 * D) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        double2 an[MB_MT][2], xn[NT][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int i = 0; i < MB_MT; ++i) an[i][h] = a[d][i][h];
#pragma unroll
          for (int j = 0; j < NT; ++j) xn[j][h] = x[d][j][h];
        }
        load(r0 + 16 * (d + D), a[d], x[d]);             // past the end: zeros
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < MB_MT; ++i)
            if (i < mt) {
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                dmma(acc[i][j], an[i][h].x, xn[j][h].x);
                dmma(acc[i][j], an[i][h].y, xn[j][h].y);
              }
            }
      }
    }
#pragma unroll
    for (int i = 0; i < MB_MT; ++i)
      if ((uint32_t)(8 * i + g) < tl.ncol) {
        double* zp = Z + cols[tl.col0 + 8 * i + g].z * ldz + cb + 2 * q;
#pragma unroll
        for (int j = 0; j < NT; ++j)
          *reinterpret_cast<double2*>(zp + 8 * j) = make_double2(acc[i][j][0], acc[i][j][1]);
      }
  }
}

// ---------------------------------------------------------------------------
// phase 2
// ---------------------------------------------------------------------------
// acc += the entries [e0, e1) of one kind: A(row, entry) = the entry's value in
// the row, B = row zi of V (V(zi, col) at V[zi vr + col vc], columns < vcols).
// 32 entries (8 steps of K = 4) make a batch; a step's operand registers are
// refilled from the next batch as soon as the step is consumed.  Batches whose
// entries all cover this warp's rows (most: leaves end where slabs end) take
// loads at constant offsets from one pointer; the others clamp and mask.
template <typename E, int NT>
__device__ __forceinline__ void mb_entries(const SlabEnt* __restrict__ ents, uint32_t e0, uint32_t e1,
                                           const E* __restrict__ pool, const double* __restrict__ V, int64_t vr,
                                           int64_t vc, int vcols, int cb, int row0, int mt, int lane,
                                           double (&acc)[MB_MT][NT][2]) {
  if (e0 >= e1) return;
  const int g = lane >> 2, q = lane & 3;
  constexpr int D = 8;
  double a[D][MB_MT], b[D][NT];
  uint64_t mask = 0;                                     // step d, bits 5 d ..: A values 0 .. 3 and the B row to be zeroed
  int64_t vo[NT];                                        // columns past the last: the last, into unused columns
#pragma unroll
  for (int j = 0; j < NT; ++j) vo[j] = min(cb + 8 * j + g, vcols - 1) * vc;
  const int nb = (int)((e1 - e0 + 31) / 32);
  const SlabEnt none{0, 0, 255u | 255u << 8};            // row 255: in no slab
  auto fetch = [&](int t) {
    const uint32_t e = e0 + 32 * t + lane;
    return e < e1 ? ents[e] : none;
  };
  // the operands of step d of the batch whose entries the lanes hold in N
  auto refill = [&](const SlabEnt& N, bool full, int d) {
    const int src = 4 * d + q;
    const uint64_t off = __shfl_sync(0xffffffffu, (unsigned long long)(N.off & SLAB_OFF_MASK), src);
    const uint32_t meta = __shfl_sync(0xffffffffu, N.meta, src), zi = __shfl_sync(0xffffffffu, N.zi, src);
    const uint32_t lo = meta & 255u, span = (meta >> 8 & 255u) - lo;
    const E* p = pool + off;
    const double* v = V + zi * vr;
#pragma unroll
    for (int j = 0; j < NT; ++j) b[d][j] = __ldg(v + vo[j]);
    if (full) {
      p += row0 + g - (int)lo;
#pragma unroll
      for (int i = 0; i < MB_MT; ++i) a[d][i] = ld_one(p + 8 * i);
    } else {
      // a row not covered reads the entry's last one (past the entries the
      // pool's first); its zero replaces the value when the step is consumed
      // (here it would wait for the load)
      uint32_t m = lo == 255u ? 16u : 0u;
#pragma unroll
      for (int i = 0; i < MB_MT; ++i) {
        const uint32_t r = (uint32_t)(row0 + 8 * i + g) - lo;
        if (i < mt) a[d][i] = ld_one(p + min(r, span));
        m |= (r > span ? 1u : 0u) << i;
      }
      mask = (mask & ~((uint64_t)31 << 5 * d)) | (uint64_t)m << 5 * d;
    }
  };
  auto covers = [&](const SlabEnt& N) {
    return __all_sync(0xffffffffu, (int)(N.meta & 255u) <= row0 &&
                                       (int)(N.meta >> 8 & 255u) >= row0 + 8 * MB_MT - 1 && (N.meta & 255u) != 255u) != 0;
  };
  SlabEnt N = fetch(0);
  bool was_full = covers(N);                             // of the batch being consumed
#pragma unroll
  for (int d = 0; d < D; ++d) refill(N, was_full, d);
  N = fetch(1);
  for (int t = 0; t < nb; ++t) {
    const SlabEnt N2 = fetch(t + 2);
    const bool full = covers(N), more = t + 1 < nb;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      double an[MB_MT], bn[NT];
#pragma unroll
      for (int i = 0; i < MB_MT; ++i) an[i] = a[d][i];
#pragma unroll
      for (int j = 0; j < NT; ++j) bn[j] = b[d][j];
      const uint32_t m = (uint32_t)(mask >> 5 * d) & 31u;
      if (more) refill(N, full, d);
      if (!was_full) {
#pragma unroll
        for (int i = 0; i < MB_MT; ++i)
          if (m >> i & 1u) an[i] = 0.0;
        if (m & 16u) {
#pragma unroll
          for (int j = 0; j < NT; ++j) bn[j] = 0.0;
        }
      }
#pragma unroll
      for (int i = 0; i < MB_MT; ++i)
        if (i < mt) {
#pragma unroll
          for (int j = 0; j < NT; ++j) dmma(acc[i][j], an[i], bn[j]);
        }
    }
    N = N2;
    was_full = full;
  }
}

template <typename T, typename TD, int NT>
__global__ void __launch_bounds__(MB_WARPS * 32, 1)
    mb_phase2_kernel(const Slab* __restrict__ slabs, const SlabEnt* __restrict__ ents, const T* __restrict__ rk,
                     const TD* __restrict__ dn, const double* __restrict__ Z, int ldz, const double* __restrict__ X,
                     int64_t ldx, int ncols, int ncb, double* __restrict__ Y, int64_t ldy) {
  __shared__ double part[MB_WARPS / 2][32][8 * NT + 1];  // the splits' sums, half the warps' at a time
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const Slab S = slabs[blockIdx.x / ncb];
  const int cb = (int)(blockIdx.x % ncb) * 8 * NT;
  // row groups of at most 32 rows (whole M tiles), ks splits of the entries
  const int ngrp = ((int)S.nrows + 31) / 32;             // at most 7
  const int ks = ngrp > 4 ? 1 : ngrp > 2 ? 2 : ngrp == 2 ? 4 : 8;
  const int grp = warp / ks, sp = warp % ks;
  const int grows = (((int)S.nrows + ngrp - 1) / ngrp + 7) / 8 * 8;
  const int row0 = grp * grows, mt = grp < ngrp ? min(grows, max(0, (int)S.nrows - row0) + 7) / 8 : 0;
  double acc[MB_MT][NT][2];
#pragma unroll
  for (int i = 0; i < MB_MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  if (mt > 0) {
    auto share = [&](uint32_t b, uint32_t e, uint32_t& s0, uint32_t& s1) {
      const uint32_t n = e - b, per = (n + 4 * ks - 1) / (4 * ks) * 4;
      s0 = b + min(n, sp * per);
      s1 = b + min(n, (sp + 1) * per);
    };
    uint32_t s0, s1;
    share(S.begin, S.dense, s0, s1);
    mb_entries<T, NT>(ents, s0, s1, rk, Z, ldz, 1, ldz, cb, row0, mt, lane, acc);
    share(S.dense, S.mid, s0, s1);
    mb_entries<TD, NT>(ents, s0, s1, dn, X, 1, ldx, ncols, cb, row0, mt, lane, acc);
    // dense leaves read along their rows (H'x): 32 input indices an entry
    for (uint32_t e = S.mid + sp; e < S.end; e += ks) {
      const SlabEnt E = ents[e];
      const uint32_t lo = E.meta & 255u, span = (E.meta >> 8 & 255u) - lo;
      const int cnt = (int)(E.meta >> 24);
      const int64_t ld = (int64_t)(E.off >> 40);
      const TD* p = dn + (E.off & SLAB_OFF_MASK);
      double a[8][MB_MT], b[8][NT];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int k = 4 * s + q;
#pragma unroll
        for (int i = 0; i < MB_MT; ++i) {
          const uint32_t r = (uint32_t)(row0 + 8 * i + g) - lo;
          a[s][i] = ld_one(p + min(r, span) * ld + min(k, cnt - 1));
          if (k >= cnt || r > span) a[s][i] = 0.0;
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          b[s][j] = __ldg(X + E.zi + min(k, cnt - 1) + min(cb + 8 * j + g, ncols - 1) * ldx);
          if (k >= cnt) b[s][j] = 0.0;
        }
      }
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int i = 0; i < MB_MT; ++i)
          if (i < mt) {
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma(acc[i][j], a[s][i], b[s][j]);
          }
    }
  }
  // the splits of a row group, summed pairwise: upper half into the lower half
  for (int half = ks / 2; half >= 1; half /= 2) {
    __syncthreads();
    const int slot = grp * half + (sp >= half ? sp - half : sp);
    if (mt > 0 && sp >= half && sp < 2 * half) {
#pragma unroll
      for (int i = 0; i < MB_MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          part[slot][8 * i + g][8 * j + 2 * q] = acc[i][j][0];
          part[slot][8 * i + g][8 * j + 2 * q + 1] = acc[i][j][1];
        }
    }
    __syncthreads();
    if (mt > 0 && sp < half) {
#pragma unroll
      for (int i = 0; i < MB_MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          acc[i][j][0] += part[slot][8 * i + g][8 * j + 2 * q];
          acc[i][j][1] += part[slot][8 * i + g][8 * j + 2 * q + 1];
        }
    }
  }
  if (mt == 0 || sp != 0) return;
#pragma unroll
  for (int i = 0; i < MB_MT; ++i) {
    const int r = row0 + 8 * i + g;
    if (i < mt && r < (int)S.nrows) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = cb + 8 * j + 2 * q + c;
          if (col < ncols) Y[(int64_t)(S.row0 + r) + col * ldy] = acc[i][j][c];
        }
    }
  }
}

// The dense leaves' part of Y = H X alone (the tensor-core kernels add the
// low-rank part afterwards): a warp per 32 output rows and block of 8 NT
// columns walks its window's dense leaves, 4 x NT MMAs for every four input
// indices, with A (the leaf) and B (X) read straight from global memory, the
// next batch of D steps in flight while one is consumed.  Bound: FP64 from 16
// columns on (a warp's step of 4 + NT loads feeds 4 NT MMAs), the loads'
// latency below.  One FMA per row and column with X staged in shared memory
// (a 16-byte shared load for two FMAs) took, with the transposed copy of X it
// needed, 853 us against 239 (n = 2^18, 64 columns; n = 200000, 16
// columns: 194 against 79).
template <int NT>
struct DensePass {
  static constexpr int D = NT >= 8 ? 1 : NT >= 4 ? 2 : 4;       // steps of a batch
  static constexpr int CTAS = NT >= 8 ? 2 : NT >= 4 ? 3 : 4;
};

template <typename TD, int NT>
__global__ void __launch_bounds__(128, DensePass<NT>::CTAS)
    mvm_dense_kernel(const MvWin* __restrict__ win, const P2Desc* __restrict__ d, const TD* __restrict__ dn,
                     const double* __restrict__ X, int64_t n, int64_t ldx, int ncols, int ncb, double* __restrict__ Y,
                     int64_t ldy) {
  constexpr int D = DensePass<NT>::D;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int cb = (int)(blockIdx.x % ncb) * 8 * NT;
  const int64_t grow = ((int64_t)(blockIdx.x / ncb) * 4 + warp) * 32;   // the warp's first output row
  if (grow >= n) return;
  const MvWin W = win[grow / MV_WROWS];
  const int w0 = (int)(grow - W.row0);
  int64_t xc[NT];                                        // this lane's columns of X (a repeated one past the last)
#pragma unroll
  for (int j = 0; j < NT; ++j) xc[j] = (int64_t)min(cb + 8 * j + g, ncols - 1) * ldx;
  double acc[4][NT][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (uint32_t b0 = W.begin; b0 < W.end; b0 += 32) {
    P2Desc E{};
    if (b0 + lane < W.end) E = d[b0 + lane];
    unsigned todo = __ballot_sync(0xffffffffu, E.cnt > 0 && E.row_off < w0 + 32 && E.row_off + (int)E.m > w0);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint64_t off = __shfl_sync(0xffffffffu, (unsigned long long)E.off, src);
      const int ro = __shfl_sync(0xffffffffu, E.row_off, src), m = (int)__shfl_sync(0xffffffffu, E.m, src);
      const int ld = (int)__shfl_sync(0xffffffffu, E.ld, src), cnt = (int)__shfl_sync(0xffffffffu, E.cnt, src);
      const uint32_t in0 = __shfl_sync(0xffffffffu, E.aux, src);
      const bool tr = __shfl_sync(0xffffffffu, (int)E.type, src) == P2_DENSE_T;
      const int64_t rs = tr ? ld : 1, cs = tr ? 1 : ld;   // strides of a row and of an input index
      const TD* ap[4];
      unsigned in = 0;                                    // bit i: row w0 + 8 i + g belongs to the leaf
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int lr = w0 + 8 * i + g - ro;
        in |= (lr >= 0 && lr < m ? 1u : 0u) << i;
        ap[i] = dn + off + min(max(lr, 0), m - 1) * rs;
      }
      const double* xp = X + in0;
      const bool rows = __all_sync(0xffffffffu, in == 15u);
      float an[D][4];
      double bn[D][NT];
      // loads are always in range (clamped); what lies outside is masked when used
      auto fetch = [&](int c, float (&a)[D][4], double (&b)[D][NT]) {
#pragma unroll
        for (int e = 0; e < D; ++e) {
          const int k = min(c + 4 * e + q, cnt - 1);
#pragma unroll
          for (int i = 0; i < 4; ++i) a[e][i] = (float)__ldg(ap[i] + k * cs);
#pragma unroll
          for (int j = 0; j < NT; ++j) b[e][j] = __ldg(xp + k + xc[j]);
        }
      };
      fetch(0, an, bn);
      for (int c = 0; c < cnt; c += 4 * D) {
        float a[D][4];
        double b[D][NT];
#pragma unroll
        for (int e = 0; e < D; ++e) {
#pragma unroll
          for (int i = 0; i < 4; ++i) a[e][i] = an[e][i];
#pragma unroll
          for (int j = 0; j < NT; ++j) b[e][j] = bn[e][j];
        }
        fetch(c + 4 * D, an, bn);
        if (!rows || c + 4 * D > cnt) {
#pragma unroll
          for (int e = 0; e < D; ++e) {
            const bool k = c + 4 * e + q < cnt;
#pragma unroll
            for (int i = 0; i < 4; ++i) a[e][i] = k && (in >> i & 1u) ? a[e][i] : 0.f;
#pragma unroll
            for (int j = 0; j < NT; ++j) b[e][j] = k ? b[e][j] : 0.0;
          }
        }
#pragma unroll
        for (int e = 0; e < D; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const double av = (double)a[e][i];
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma(acc[i][j], av, b[e][j]);
          }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t r = grow + 8 * i + g;
    if (r < n) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = cb + 8 * j + 2 * q + c;
          if (col < ncols) Y[r + col * ldy] = acc[i][j][c];
        }
    }
  }
}

// the block products' scratch in the handle (Z, or the transposed input)
int block_scratch(hm_handle* h, size_t bytes, double** out) {
  if (h->xm_bytes < bytes) {
    if (h->d_xm) cudaFree(h->d_xm);
    h->d_xm = nullptr;
    h->xm_bytes = 0;
    HM_CUDA_TRY(cudaMalloc(&h->d_xm, bytes));
    h->xm_bytes = bytes;
  }
  *out = (double*)h->d_xm;
  return HM_OK;
}

// The factor columns of phase 1 by input segment (one per cluster), 32 to a tile,
// from the descriptors of the single-column phase 1: columns counted per cluster,
// the clusters' ranges and tiles by one CTA, then each leaf's columns put in its
// cluster's range.  Which of a cluster's leaves comes first is left to the atomics:
// every column's sums are its own.  Made on the host from the leaves the table took
// 2.1 ms of a first product's 4.7 (n = 2^17).
struct MbSeg {
  uint32_t seg0, len, cnt, next;         // columns; next free one
};
__global__ void __launch_bounds__(256) mb_count_kernel(const P1Desc* __restrict__ d, int64_t nd, MbSeg* __restrict__ seg) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  const P1Desc D = d[i];
  seg[D.cl].seg0 = D.seg0;               // the same value from every leaf of the cluster
  seg[D.cl].len = D.len;
  atomicAdd(&seg[D.cl].cnt, (uint32_t)D.k);
}
__global__ void __launch_bounds__(1024) mb_tiles_kernel(MbSeg* __restrict__ seg, int64_t ncl, MbTile* __restrict__ tile,
                                                        uint32_t* __restrict__ ntile) {
  __shared__ uint32_t sum[2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t base[2] = {0, 0};             // columns, tiles
  for (int64_t b = 0; b < ncl; b += 1024) {
    const int64_t i = b + threadIdx.x;
    MbSeg S{};
    if (i < ncl) S = seg[i];
    const uint32_t own[2] = {S.cnt, (S.cnt + 8 * MB_MT - 1) / (8 * MB_MT)};
    uint32_t at[2];
    __syncthreads();                     // the last round's sums
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t incl = own[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) sum[q][warp] = incl;
      at[q] = base[q] + incl - own[q];
    }
    __syncthreads();
    for (int w = 0; w < 32; ++w)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (w < warp) at[q] += sum[q][w];
        base[q] += sum[q][w];
      }
    if (i < ncl && S.cnt > 0) {
      seg[i].next = at[0];
      for (uint32_t c = 0, t = at[1]; c < S.cnt; c += 8 * MB_MT, ++t)
        tile[t] = MbTile{at[0] + c, min(8u * MB_MT, S.cnt - c), S.seg0, S.len};
    }
  }
  if (threadIdx.x == 0) *ntile = base[1];
}
__global__ void __launch_bounds__(256) mb_column_kernel(const P1Desc* __restrict__ d, int64_t nd, MbSeg* __restrict__ seg,
                                                        MbCol* __restrict__ col) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 8;   // eight threads a leaf
  P1Desc D{};
  uint32_t at = 0;
  if (i < nd) {
    D = d[i];
    if (threadIdx.x % 8 == 0) at = atomicAdd(&seg[D.cl].next, (uint32_t)D.k);
  }
  at = __shfl_sync(0xffffffffu, at, threadIdx.x & 24);
  for (uint32_t r = threadIdx.x % 8; r < D.k; r += 8)
    col[(uint64_t)at + r] = MbCol{D.off + (uint64_t)r * D.stride, (uint64_t)D.zoff + r};
}

int ensure_columns(hm_handle* h, MvPlan& P) {
  if (P.d_mbcol || P.np1 == 0) return HM_OK;
  const int64_t ncl = (int64_t)h->cl_s.size();
  const size_t cb = pad_to((int64_t)sizeof(MbCol) * h->zlen, 256);
  const size_t tb = pad_to((int64_t)sizeof(MbTile) * (h->zlen / (8 * MB_MT) + std::min(ncl, P.np1)), 256);
  // the segments, needed to make the table only, behind it if they are small
  const size_t gb = sizeof(MbSeg) * (size_t)ncl + 16;
  char* d = nullptr;
  char* tmp = nullptr;
  const bool behind = gb <= (size_t)1 << 20;
  cudaError_t e = cudaMalloc((void**)&d, cb + tb + (behind ? gb : 0));
  if (e == cudaSuccess && behind) {
    tmp = d + cb + tb;
  } else if (e == cudaSuccess && cudaMalloc((void**)&tmp, gb) != cudaSuccess) {
    cudaFree(d);
    e = cudaErrorMemoryAllocation;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(HM_ERR_OOM, std::string("block product columns: ") + cudaGetErrorString(e));
  }
  uint32_t* d_n = (uint32_t*)tmp;
  MbSeg* seg = (MbSeg*)(tmp + 16);
  uint32_t ntile = 0;
  e = cudaMemsetAsync(tmp, 0, gb, h->stream);
  if (e == cudaSuccess) {
    mb_count_kernel<<<(unsigned)((P.np1 + 255) / 256), 256, 0, h->stream>>>(P.d_p1, P.np1, seg);
    mb_tiles_kernel<<<1, 1024, 0, h->stream>>>(seg, ncl, (MbTile*)(d + cb), d_n);
    mb_column_kernel<<<(unsigned)((P.np1 + 31) / 32), 256, 0, h->stream>>>(P.d_p1, P.np1, seg, (MbCol*)d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&ntile, d_n, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);   // the caller's stream reads the table next
  if (!behind) cudaFree(tmp);
  if (e != cudaSuccess) {
    cudaFree(d);
    return fail(HM_ERR_CUDA, std::string("block product columns: ") + cudaGetErrorString(e));
  }
  P.d_mbcol = (MbCol*)d;
  P.d_mbtile = (MbTile*)(d + cb);
  P.nmbtile = (int64_t)ntile;
  return HM_OK;
}

template <typename T, int NT>
int launch_multi(hm_handle* h, const double* d_x, double* d_y, int64_t ncols, int trans, cudaStream_t st) {
  using TD = typename std::conditional<std::is_same<T, double>::value, double, float>::type;
  MvPlan& P = trans ? h->bwd : h->fwd;
  bool slabs = false;
  HM_TRY(ensure_slabs(h, trans, st, &slabs));
  if (!slabs) {                                          // no lists: column by column
    for (int64_t c = 0; c < ncols; ++c) HM_TRY(matvec_device(h, d_x + c * h->n, d_y + c * h->n, trans, st));
    return HM_OK;
  }
  HM_TRY(ensure_columns(h, P));
  const int ld = (int)pad_to(ncols, 8 * NT);
  const int ncb = ld / (8 * NT);
  double* z = nullptr;
  HM_TRY(block_scratch(h, sizeof(double) * (size_t)std::max<int64_t>(h->zlen, 1) * ld, &z));
  const int64_t nblk = (int64_t)P.nslab * ncb;
  if (nblk > (int64_t)INT32_MAX) return fail(HM_ERR_UNSUPPORTED, "too many phase-2 blocks");
  if (P.nmbtile > 0) {
    const int64_t blocks = std::min<int64_t>((P.nmbtile * ncb + MB_WARPS - 1) / MB_WARPS, 148 * 64);
    mb_phase1_kernel<T, NT><<<(unsigned)blocks, MB_WARPS * 32, 0, st>>>(
        P.d_mbtile, P.nmbtile, P.d_mbcol, (const T*)h->d_rk, d_x, h->n, (int)ncols, ncb, z, ld);
  }
  mb_phase2_kernel<T, TD, NT><<<(unsigned)nblk, MB_WARPS * 32, 0, st>>>(
      P.d_slab, P.d_ent, (const T*)h->d_rk, (const TD*)h->d_dense, z, ld, d_x, h->n, (int)ncols, ncb, d_y, h->n);
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

template <typename T>
int multi_t(hm_handle* h, const double* d_x, double* d_y, int64_t ncols, int trans, cudaStream_t st) {
  if (ncols <= 8) return launch_multi<T, 1>(h, d_x, d_y, ncols, trans, st);
  if (ncols <= 16) return launch_multi<T, 2>(h, d_x, d_y, ncols, trans, st);
  return launch_multi<T, 4>(h, d_x, d_y, ncols, trans, st);
}

// the dense leaves (FP32) of a tensor-core call, written into Y
template <int NT>
int launch_dense(hm_handle* h, const double* d_x, double* d_y, int64_t ncols, int trans, cudaStream_t st) {
  MvPlan& P = trans ? h->bwd : h->fwd;
  HM_TRY(split_p2(P));
  const int64_t ncb = (ncols + 8 * NT - 1) / (8 * NT), blocks = (h->n + 127) / 128 * ncb;
  if (blocks > (int64_t)INT32_MAX) return fail(HM_ERR_UNSUPPORTED, "too many dense-pass blocks");
  mvm_dense_kernel<float, NT><<<(unsigned)blocks, 128, 0, st>>>(P.d_wind, P.d_p2d, (const float*)h->d_dense, d_x, h->n,
                                                              h->n, (int)ncols, (int)ncb, d_y, h->n);
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

// the narrowest column block that holds the columns: a step's loads of the leaf
// serve the whole block, and MMAs on columns that are not there cost as much
int dense_pass(hm_handle* h, const double* d_x, double* d_y, int64_t ncols, int trans, cudaStream_t st) {
  if (ncols <= 8) return launch_dense<1>(h, d_x, d_y, ncols, trans, st);
  if (ncols <= 16) return launch_dense<2>(h, d_x, d_y, ncols, trans, st);
  if (ncols <= 32) return launch_dense<4>(h, d_x, d_y, ncols, trans, st);
  return launch_dense<8>(h, d_x, d_y, ncols, trans, st);
}

}  // namespace

// FP64 factors (no tensor-core kind for FP64), simt, or factors beyond the
// tensor-core path's range (2^100): the FP64 block kernels for the whole
// product.  FP32/BF16 factors: the dense leaves in FP64 (written into every
// row of Y), then the low-rank part on the tensor cores (added into Y).
int matvec_multi_device(hm_handle* h, const double* d_x, double* d_y, int64_t ncols, int trans, cudaStream_t st,
                        bool simt) {
  if (ncols <= 0) return HM_OK;
  if ((h->n + 2) * pad_to(ncols, 16) > (int64_t)1 << 40) return fail(HM_ERR_UNSUPPORTED, "right-hand side block too large");
  switch (h->storage) {
    case HM_F64: return multi_t<double>(h, d_x, d_y, ncols, trans, st);
    case HM_F32: {
      bool tc = false;
      if (!simt) HM_TRY(tc_prepare(h, trans, &tc));
      if (!tc) return multi_t<float>(h, d_x, d_y, ncols, trans, st);
      HM_TRY(dense_pass(h, d_x, d_y, ncols, trans, st));
      return matvec_multi_tc(h, d_x, d_y, ncols, trans, st);
    }
    default: {
      bool tc = false;
      if (!simt) HM_TRY(tc_prepare(h, trans, &tc));
      if (!tc) return multi_t<__nv_bfloat16>(h, d_x, d_y, ncols, trans, st);
      HM_TRY(dense_pass(h, d_x, d_y, ncols, trans, st));
      return matvec_multi_tc(h, d_x, d_y, ncols, trans, st);
    }
  }
}

}  // namespace hm
