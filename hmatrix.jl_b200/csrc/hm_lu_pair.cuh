// The trailing update of the H-LU's tile schedule: for every pair i != j of
// trailing tiles, A_ij B_ij' - A_ik (B_ik' A_kj) B_kj' recompressed into A_ij,
// B_ij (hm_lu.cu).  Included by hm_lu.cu after hm_core.cuh.
#pragma once
#include "hm_core.cuh"

namespace hm {

// Pair q of the trailing update of step k: mode 0 every pair i != j of the
// tiles (k, T); mode 1 the pairs of tile row and tile column k+1; mode 2 the
// pairs among the tiles (k+1, T).
__device__ __forceinline__ void tile_pair(int T, int k, int mode, int64_t gq, int& i, int& j) {
  if (mode == 1) {
    const int n1 = T - k - 2;
    if (gq < n1) { i = k + 1; j = k + 2 + (int)gq; }
    else { i = k + 2 + (int)(gq - n1); j = k + 1; }
    return;
  }
  const int base = mode == 2 ? k + 2 : k + 1;
  const int Tr = T - base;
  const int ii = (int)(gq / (Tr - 1));
  int jj = (int)(gq % (Tr - 1));
  if (jj >= ii) ++jj;
  i = base + ii;
  j = base + jj;
}
static int64_t tile_pair_count(int T, int k, int mode) {
  const int64_t Tr = T - k - 1;
  if (mode == 0) return Tr * (Tr - 1);
  if (mode == 1) return Tr >= 2 ? 2 * (Tr - 1) : 0;
  return Tr >= 2 ? (Tr - 1) * (Tr - 2) : 0;
}

struct PairArgs {
  double* const* Ap;         // row panels: A_ij at Ap[i] + j cap m_i
  double* const* Bp;         // column panels: B_ij at Bp[j] + i cap n_j
  const int32_t* size;
  int32_t* kmat;
  int T, cap, k, mode;
  double eps;
  int* flags;
  // pairs this kernel leaves to the next one: their indices and count
  const int32_t* in;         // the pairs to do (NULL: all, one a block)
  const int* nin;
  int32_t* out;
  int* nout;
};

// one pair's operands
struct PairView {
  double *A, *B;                       // A_ij (m x k1), B_ij (n x k1)
  const double *Aik, *Bik, *Akj, *Bkj; // (m x ka), (s x ka), (s x kb), (n x kb)
  int32_t* rank;
  int i, j, m, n, s, k1, ka, kb;
};
__device__ __forceinline__ PairView pair_view(const PairArgs& a, int64_t q) {
  PairView v;
  tile_pair(a.T, a.k, a.mode, q, v.i, v.j);
  v.m = a.size[v.i];
  v.n = a.size[v.j];
  v.s = a.size[a.k];
  const int64_t cap = a.cap;
  v.A = a.Ap[v.i] + v.j * cap * v.m;
  v.B = a.Bp[v.j] + v.i * cap * v.n;
  v.Aik = a.Ap[v.i] + a.k * cap * v.m;
  v.Bik = a.Bp[a.k] + v.i * cap * v.s;
  v.Akj = a.Ap[a.k] + v.j * cap * v.s;
  v.Bkj = a.Bp[v.j] + a.k * cap * v.n;
  v.rank = a.kmat + v.i * a.T + v.j;
  v.k1 = *v.rank;
  v.ka = a.kmat[v.i * a.T + a.k];
  v.kb = a.kmat[a.k * a.T + v.j];
  return v;
}

// ---------------------------------------------------------------------------
// small pairs: both tall factors in registers
// ---------------------------------------------------------------------------
// One CTA per pair: WPS warps hold [A_ij | -A_ik W] (the A side), WPS warps
// [B_ij | B_kj], eight rows a lane, up to RMAX columns (tiles of up to 256 WPS
// rows).  W = B_ik' A_kj comes from the B side's warps, so no panel product is
// stored between kernels.  Gram-Schmidt (twice per column) needs only warp
// reductions on either side, the core's SVD runs in one warp.  Bound: latency,
// so what counts is how many pairs an SM holds; staged in shared memory at 16
// columns a pair took 71,000 cycles with three pairs an SM (15,000 of them
// reading A_ik W from memory, 23,000 in block-wide Gram-Schmidt, 19,000 in the
// SVD).  Ranks here are 3 to 5 at n = 65536 (eps 1e-10).
template <int WPS>
struct SideSum {                       // sums over a side's threads
  double (*red)[WPS][16];              // [parity][warp][value]
  int side, warp, lane, par;
  // the values [from, to)
  template <typename V, int NV>
  __device__ __forceinline__ void operator()(V (&v)[NV], int from, int to) {
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i >= from && i < to) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
      }
    if constexpr (WPS > 1) {
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (i >= from && i < to && lane == i) red[par][warp][i] = v[i];
      asm volatile("bar.sync %0, %1;" ::"r"(side + 1), "n"(32 * WPS) : "memory");
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (i >= from && i < to) {
          V s = (V)red[par][0][i];
#pragma unroll
          for (int w = 1; w < WPS; ++w) s += (V)red[par][w][i];
          v[i] = s;
        }
      par ^= 1;
    }
  }
};

template <typename TS, int WPS, int RMAX>
__global__ void __launch_bounds__(64 * WPS) lu_pair_kernel(PairArgs a) {
  constexpr int ROWS = 8, CAPW = 48;   // rows a lane; rank capacity (RCORE_MAX / 2)
  // W and A_ik W are FP64 sums of FP64 factors whatever TS is: what is subtracted
  // from A_ij must not carry the core's rounding.  FP64 cores form them in x's
  // registers, FP32 ones a column at a time in registers of its own (n = 65536,
  // truncation 1e-6: 191 ms; two columns at a time, 30 registers more, 211).  In
  // FP32 the factors of a mixed LU were 22 % further from the FP64 ones (8 tiles of
  // 250 rows, l = 40: 2.4e-6 against 2.0e-6 of the norm) and no faster (200 ms).
  constexpr int WC = sizeof(TS) == 8 ? RMAX : 1;
  __shared__ double sW[CAPW * RMAX];   // W, ka x kb
  __shared__ TS sR[2][RMAX * RMAX];    // R of either side, then the coefficients of either output
  __shared__ TS sC[RMAX * (RMAX | 1)], sV[RMAX * (RMAX | 1)];
  __shared__ double sred[2][2][WPS][16];
  __shared__ TS sig[RMAX];
  __shared__ int ord[RMAX], s_k;
  const int side = threadIdx.x / (32 * WPS), st = threadIdx.x % (32 * WPS), lane = threadIdx.x & 31;
  const int nin = a.in ? *a.nin : 0;
  for (int64_t b = blockIdx.x; a.in ? b < nin : b == blockIdx.x; b += gridDim.x) {
    const int64_t pq = a.in ? a.in[b] : b;
    const PairView v = pair_view(a, pq);
    // nothing to subtract: the tile stays (from step 1 on it is a recompressed
    // one already)
    if (a.k > 0 && (v.ka == 0 || v.kb == 0)) continue;
    const int k1 = v.k1, r = k1 + v.kb, ka = v.ka;
    if (r == 0) {
      if (threadIdx.x == 0) *v.rank = 0;
      continue;
    }
    if (r > RMAX || max(max(v.m, v.n), v.s) > 32 * WPS * ROWS) {
      if (threadIdx.x == 0) {
        if (a.out) a.out[atomicAdd(a.nout, 1)] = (int32_t)pq;
        else atomicOr(a.flags, 1);     // nobody is left to take it (the host launches a kernel for every size)
      }
      continue;
    }
    __syncthreads();                   // the previous pair's shared memory
    SideSum<WPS> sum{sred[side], side, st >> 5, lane, 0};
    TS x[RMAX][ROWS];
    const int len = side ? v.n : v.m;
    auto load = [&](const double* p, int rows, auto (&c)[ROWS]) {
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        const int t = st + 32 * WPS * u;
        c[u] = t < rows ? p[t] : 0.0;
      }
    };
    if (side == 0) {
#pragma unroll
      for (int c = 0; c < RMAX; ++c) {
        if (c < k1) load(v.A + (int64_t)c * v.m, v.m, x[c]);
        else
#pragma unroll
          for (int u = 0; u < ROWS; ++u) x[c][u] = (TS)0;
      }
    } else {
      // W[l][c] = B_ik(:, l) . A_kj(:, c), NC columns from c0 on, which y holds
      auto dots = [&](auto& y, int c0) {
        constexpr int NC = (int)(sizeof(y) / sizeof(y[0]));
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (c0 + c < v.kb) load(v.Akj + (int64_t)(c0 + c) * v.s, v.s, y[c]);
#pragma unroll 1
        for (int l = 0; l < ka; ++l) {
          double t[ROWS], d[NC];
          load(v.Bik + (int64_t)l * v.s, v.s, t);
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            d[c] = 0.0;
            if (c0 + c < v.kb) {
#pragma unroll
              for (int u = 0; u < ROWS; ++u) d[c] = fma(t[u], y[c][u], d[c]);
            }
          }
          sum(d, 0, v.kb - c0);
          if (st == 0) {
#pragma unroll
            for (int c = 0; c < NC; ++c)
              if (c0 + c < v.kb) sW[l * RMAX + c0 + c] = d[c];
          }
        }
      };
      if constexpr (WC == RMAX) {
        dots(x, 0);
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < v.kb; c0 += WC) {
          double y[WC][ROWS];
          dots(y, c0);
        }
      }
#pragma unroll
      for (int c = 0; c < RMAX; ++c)
        if (c < r) load(c < k1 ? v.B + (int64_t)c * v.n : v.Bkj + (int64_t)(c - k1) * v.n, v.n, x[c]);
    }
    __syncthreads();
    if (side == 0) {
      // columns k1 .. r - 1: -A_ik W
      if constexpr (WC == RMAX) {
#pragma unroll 1
        for (int l = 0; l < ka; ++l) {
          double t[ROWS];
          load(v.Aik + (int64_t)l * v.m, v.m, t);
#pragma unroll
          for (int c = 0; c < RMAX; ++c)
            if (c >= k1 && c < r) {
              const double w = -sW[l * RMAX + c - k1];
#pragma unroll
              for (int u = 0; u < ROWS; ++u) x[c][u] = fma(t[u], w, x[c][u]);
            }
        }
      } else {
#pragma unroll 1
        for (int c0 = 0; c0 < v.kb; c0 += WC) {
          double y[WC][ROWS];
#pragma unroll
          for (int c = 0; c < WC; ++c)
#pragma unroll
            for (int u = 0; u < ROWS; ++u) y[c][u] = 0.0;
#pragma unroll 1
          for (int l = 0; l < ka; ++l) {
            double t[ROWS];
            load(v.Aik + (int64_t)l * v.m, v.m, t);
#pragma unroll
            for (int c = 0; c < WC; ++c) {
              const double w = c0 + c < v.kb ? -sW[l * RMAX + c0 + c] : 0.0;
#pragma unroll
              for (int u = 0; u < ROWS; ++u) y[c][u] = fma(t[u], w, y[c][u]);
            }
          }
#pragma unroll
          for (int c = 0; c < RMAX; ++c)
#pragma unroll
            for (int q = 0; q < WC; ++q)
              if (c == k1 + c0 + q && c < r) {
#pragma unroll
                for (int u = 0; u < ROWS; ++u) x[c][u] = (TS)y[q][u];
              }
        }
      }
    }
    // Gram-Schmidt, twice per column; once for the columns of A_ij and B_ij,
    // which from step 1 on are a previous core's output: orthogonal up to that
    // core's threshold (taken as exactly orthogonal they lose the digits that
    // cancel in the difference, and ranks grow from step to step)
    const int ok = a.k >= 1 ? k1 : 0;
    TS* R = sR[side];
    for (int e = st; e < r * r; e += 32 * WPS) R[e] = (TS)0;
    if constexpr (WPS > 1) asm volatile("bar.sync %0, %1;" ::"r"(side + 1), "n"(32 * WPS) : "memory");
    else __syncwarp();
    // (unrolled over the columns: rotating the slots through one loop body took
    // 13 % longer)
#pragma unroll
    for (int c = 0; c < RMAX; ++c)
      if (c < r) {
        TS tot[RMAX];
#pragma unroll
        for (int i = 0; i < RMAX; ++i) tot[i] = (TS)0;
#pragma unroll 1
        for (int pass = c < ok ? 1 : 0; pass < 2; ++pass) {
          TS d[RMAX];
#pragma unroll
          for (int i = 0; i < c; ++i) {
            d[i] = (TS)0;
#pragma unroll
            for (int u = 0; u < ROWS; ++u) d[i] = fma(x[i][u], x[c][u], d[i]);
          }
          sum(d, 0, c);
#pragma unroll
          for (int i = 0; i < c; ++i) {
            tot[i] += d[i];
#pragma unroll
            for (int u = 0; u < ROWS; ++u) x[c][u] = fma(-d[i], x[i][u], x[c][u]);
          }
        }
        TS nn[1] = {(TS)0};
#pragma unroll
        for (int u = 0; u < ROWS; ++u) nn[0] = fma(x[c][u], x[c][u], nn[0]);
        sum(nn, 0, 1);
        const TS nrm = sqrt(nn[0]), inv = nrm > (TS)0 ? (TS)1 / nrm : (TS)0;
#pragma unroll
        for (int u = 0; u < ROWS; ++u) x[c][u] *= inv;
        if (st == 0) {
#pragma unroll
          for (int i = 0; i < c; ++i) R[i + c * r] = tot[i];
          R[c + c * r] = nrm;
        }
      }
    __syncthreads();
    // core W = R_A R_B', V = I
    const int lw = r | 1;
    double sabs = 0.0;
    for (int e = threadIdx.x; e < r * r; e += 64 * WPS) {
      const int i = e % r, c = e / r;
      TS s = (TS)0;
      for (int q = max(i, c); q < r; ++q) s = fma(sR[0][i + q * r], sR[1][c + q * r], s);
      sC[i + c * lw] = s;
      sV[i + c * lw] = i == c ? (TS)1 : (TS)0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      for (int e = lane; e < r * r; e += 32) sabs += fabs((double)sC[e % r + e / r * lw]);
      sabs = warp_sum(sabs);
      int k = 0;
      if (sabs < 1e-5) {
        // compress(): an (absolutely) tiny core becomes rank-1 zeros (src/hlu.jl:163-167)
        k = -1;
      } else {
        const TS thr = (TS)fmax(sizeof(TS) == 8 ? 1e-15 : 1e-7, 1e-3 * a.eps);
        jacobi_warp16(sC, sV, r, lw, thr, (TS)(1e-3 * a.eps));
        // singular values, their stable descending order, findlast(S/S[1] > eps)
        TS s = (TS)0;
        if (lane < r) {
          for (int t = 0; t < r; ++t) s = fma(sC[t + lane * lw], sC[t + lane * lw], s);
          s = sqrt(s);
          sig[lane] = s;
          ord[lane] = lane;            // every entry a valid column even if a non-finite value breaks the order
        }
        __syncwarp();
        if (lane < r) {
          int pos = 0;
          for (int c = 0; c < r; ++c) pos += (sig[c] > s) || (sig[c] == s && c < lane);
          if (pos < r) ord[pos] = lane;
        }
        __syncwarp();
        const double s1 = r > 0 ? (double)sig[ord[0]] : 0.0;
        k = __popc(__ballot_sync(0xffffffffu, lane < r && (double)s / s1 > a.eps));
        if (!(s1 > 0.0)) k = 0;
        if (k > a.cap) {
          if (lane == 0) atomicOr(a.flags, 1);
          k = a.cap;
        }
        if (lane == 0 && !isfinite(sabs)) atomicOr(a.flags, 2);
      }
      if (lane == 0) s_k = k;
    }
    __syncthreads();
    const bool zero = s_k < 0;
    const int k = zero ? 0 : s_k;
    // coefficients: A' = Q_A (W / s), B' = Q_B (V s)
    for (int e = threadIdx.x; e < r * k; e += 64 * WPS) {
      const int t = e % r, o = ord[e / r];
      const TS s = sig[o];
      sR[0][e] = s > (TS)0 ? sC[t + o * lw] / s : (TS)0;
      sR[1][e] = sV[t + o * lw] * s;
    }
    __syncthreads();
    double* out = side ? v.B : v.A;
#pragma unroll 1
    for (int c = 0; c < k; ++c) {
      TS s[ROWS];
#pragma unroll
      for (int u = 0; u < ROWS; ++u) s[u] = (TS)0;
#pragma unroll
      for (int q = 0; q < RMAX; ++q)
        if (q < r) {
          const TS f = R[q + c * r];
#pragma unroll
          for (int u = 0; u < ROWS; ++u) s[u] = fma(x[q][u], f, s[u]);
        }
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        const int t = st + 32 * WPS * u;
        if (t < len) out[t + (int64_t)c * len] = (double)s[u];
      }
    }
    // columns beyond the old rank are zero already: only those a smaller rank
    // frees (and the zero column of a zero block)
    for (int c = k; c < (zero ? max(k1, 1) : k1); ++c)
      for (int t = st; t < len; t += 32 * WPS) out[t + (int64_t)c * len] = 0.0;
    if (threadIdx.x == 0) *v.rank = zero ? 1 : k;
  }
}

// ---------------------------------------------------------------------------
// the others: factors staged in shared memory (up to rl columns of at most smax
// rows) or in the block's own part of a global scratch
// ---------------------------------------------------------------------------
// TS: the precision of the staged factors and of the QR + SVD core (FP32 when
// the truncation tolerance is loose: the mixed-precision factorisation).  Bound:
// the latency of the QR's columns, so what counts is the warps an SM holds: the
// 2-D cloud, n = 65536, 128 tiles of 512 rows, cores of up to 52 columns in
// scratch, 2.45 s with 2 CTAs of 128 threads an SM, 1.79 with 2 of 256, 1.38 with
// the 3 of 256 that are resident (4: 1.69, in two waves).
constexpr int TC_THREADS = 256;
template <typename TS>
__global__ void __launch_bounds__(TC_THREADS) lu_tile_core_kernel(PairArgs a, int rl, int smax, TS* scratch) {
  extern __shared__ double sm_raw[];
  TS* sm = reinterpret_cast<TS*>(sm_raw);
  // W (cap x cap, FP64 as in the register kernel), then the factors
  const int64_t cw = (int64_t)a.cap * a.cap * (8 / sizeof(TS));
  TS* base = scratch ? scratch + (int64_t)blockIdx.x * (2 * smax * rl + cw) : sm + 3 * rl * (rl + 1);   // both even
  double* sw = reinterpret_cast<double*>(base);
  TS* XA = base + cw;
  TS* XB = XA + (int64_t)smax * rl;
  const int nin = *a.nin;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  for (int b = blockIdx.x; b < nin; b += gridDim.x) {
    const PairView v = pair_view(a, a.in[b]);
    const int k1 = v.k1, kb = v.kb, ka = v.ka, r = k1 + kb;
    if (r > rl) {
      if (threadIdx.x == 0) {
        if (a.out) a.out[atomicAdd(a.nout, 1)] = a.in[b];
        else atomicOr(a.flags, 1);     // nobody is left to take it (the last kernel holds 2 cap columns)
      }
      continue;
    }
    __syncthreads();
    for (int e = warp; e < ka * kb; e += nwarp) {
      const double *x = v.Bik + (int64_t)(e % ka) * v.s, *y = v.Akj + (int64_t)(e / ka) * v.s;
      double s = 0.0;
#pragma unroll 4
      for (int t = lane; t < v.s; t += 32) s = fma(x[t], y[t], s);
      s = warp_sum(s);
      if (lane == 0) sw[e] = s;
    }
    __syncthreads();
    for (int q = 0; q < r; ++q)
      for (int t = threadIdx.x; t < v.m; t += blockDim.x) {
        double s = 0.0;
        if (q < k1) s = v.A[t + (int64_t)q * v.m];
        else
          for (int l = 0; l < ka; ++l) s = fma(v.Aik[t + (int64_t)l * v.m], -sw[l + (q - k1) * ka], s);
        XA[t + q * v.m] = (TS)s;
      }
    for (int q = 0; q < r; ++q)
      for (int t = threadIdx.x; t < v.n; t += blockDim.x)
        XB[t + q * v.n] = (TS)(q < k1 ? v.B[t + (int64_t)q * v.n] : v.Bkj[t + (int64_t)(q - k1) * v.n]);
    __syncthreads();
    CoreJob J{};
    J.outA = v.A; J.outB = v.B;
    J.m = v.m; J.n = v.n; J.r = r; J.lda = max(v.m, 1); J.ldb = max(v.n, 1);
    J.ldoa = v.m; J.ldob = v.n; J.kcap = a.cap;
    J.zero_test = 1; J.rank = v.rank; J.zero_fill = 1;
    // the tile's columns at and beyond its previous rank k1 are zero: only the
    // columns [k, k1) a smaller new rank frees need zeros
    J.known_zero = 1; J.zero_from = k1;
    core_body_t<TS, true>(J, XA, XB, rl, a.eps, a.flags);
    __syncthreads();
  }
}

}  // namespace hm
