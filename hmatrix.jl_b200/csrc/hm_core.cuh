// Recompression core shared by the construction and the H-LU kernels (one
// CTA per job): CGS2 QR of the two tall factors, SVD of the small core by
// one-sided Jacobi, truncation, and the products that form the new factors.
// The tall factors may live in global or shared memory.
#pragma once
#include "hm_lowrank.cuh"

namespace hm {

// ===========================================================================
// Recompression core (K3): CGS2 QR of A and B in place, W = R_A R_B^T, one
// sided Jacobi SVD of W, truncation k = #{s_i/s_1 > eps_trunc}, and
// A' = Q_A U_k, B' = Q_B V_k S_k.  One CTA per job; smem 3 rmax (rmax + 1)
// doubles.
// ===========================================================================
template <typename TS>
static __device__ void cgs2_qr(TS* X, int len, int ld, int r, TS* Rm /* r x r, col-major */,
                        TS* proj /* r */, double* red) {
  for (int e = threadIdx.x; e < r * r; e += blockDim.x) Rm[e] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j = 0; j < r; ++j) {
    TS* xj = X + (int64_t)j * ld;
    for (int pass = 0; pass < 2; ++pass) {
      for (int i = w; i < j; i += nw) {
        const TS* qi = X + (int64_t)i * ld;
        TS s = 0;
        for (int t = lane; t < len; t += 32) s = fma(qi[t], xj[t], s);
        s = warp_sum(s);
        if (lane == 0) proj[i] = s;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < len; t += blockDim.x) {
        TS s = 0;
        for (int i = 0; i < j; ++i) s = fma(X[t + (int64_t)i * ld], proj[i], s);
        xj[t] -= s;
      }
      if (threadIdx.x < j) Rm[threadIdx.x + j * r] += proj[threadIdx.x];
      // after the second pass no barrier: the norm reads only this thread's
      // rows, and proj is rewritten only after the norm's barrier
      if (pass == 0) __syncthreads();
    }
    TS ss = 0;
    for (int t = threadIdx.x; t < len; t += blockDim.x) ss = fma(xj[t], xj[t], ss);
    // block_sum without its leading barrier: red was last read before the
    // previous column's closing barrier
    double sd = warp_sum((double)ss);
    if (lane == 0) red[w] = sd;
    __syncthreads();
    sd = 0.0;
    for (int q = 0; q < ((blockDim.x + 31) >> 5); ++q) sd += red[q];
    const TS nrm = sqrt((TS)sd);
    const TS inv = nrm > (TS)0 ? (TS)1 / nrm : (TS)0;
    for (int t = threadIdx.x; t < len; t += blockDim.x) xj[t] *= inv;
    if (threadIdx.x == 0) Rm[j + j * r] = nrm;
    __syncthreads();
  }
}

// Jacobi rotation of a column pair with squared norms al, be and dot product
// ga != 0: t = tan of the angle, c = cos, s = c t.  t only has to be near the
// angle that zeroes ga (20 bits: ga shrinks a millionfold instead of vanishing,
// and the pair is met again), so it comes from the approximate reciprocal and
// reciprocal square root; c is Newton-refined to full precision, which keeps
// the rotation orthogonal whatever t is.  Divisions and square roots in full
// precision made a round of rotations a chain of about 600 cycles.
__device__ __forceinline__ double rcp_fast(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ void jacobi_angle(double al, double be, double ga, double& c, double& s) {
  const double zeta = 0.5 * (be - al) * rcp_fast(ga);
  const double az = fmin(fabs(zeta), 1e150);               // its square stays finite
  const double q = fma(az, az, 1.0);
  double t = rcp_fast(az + q * rsqrt_fast(q));
  if (zeta < 0.0) t = -t;
  const double v = fma(t, t, 1.0);                         // in [1, 2]
  double y = rsqrt_fast(v);
  y = y * fma(-0.5 * v * y, y, 1.5);                       // Newton for v^(-1/2): 20, 40, full bits
  y = y * fma(-0.5 * v * y, y, 1.5);
  c = y;
  s = y * t;
}
__device__ __forceinline__ void jacobi_angle(float al, float be, float ga, float& c, float& s) {
  const float zeta = (be - al) / (2.f * ga);
  const float t = (zeta >= 0.f ? 1.f : -1.f) / (fabsf(zeta) + sqrtf(1.f + zeta * zeta));
  c = 1.f / sqrtf(1.f + t * t);
  s = c * t;
}

// One-sided Jacobi on the r <= 16 columns of W (r x r, column stride lw) and
// of V by ONE warp: 4 lanes a column pair, 4 rows a lane in registers, so that
// a round is eight pairs at once and needs no block barrier.  A pair is rotated
// while its cosine exceeds thr, unless one of its columns is below neg times
// the largest column of W: what that column holds is truncated and moves the
// singular values by less than neg.  (A core has about as many such columns as
// it keeps, rounding noise that takes twice the sweeps to put in order.)  Ends
// when a whole sweep's rounds in a row rotated nothing.
template <typename TS>
static __device__ void jacobi_warp16(TS* W, TS* V, int r, int lw, TS thr, TS neg) {
  const int lane = threadIdx.x & 31, sg = lane >> 2, sl = lane & 3;
  const int rr = (r + 1) & ~1, np = rr - 1;              // columns (even), rounds of a sweep
  const TS thr2 = thr * thr;
  TS big = 0;                                            // the largest squared column norm, times neg^2
  if (lane < r)
    for (int t = 0; t < r; ++t) big = fma(W[t + lane * lw], W[t + lane * lw], big);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  big *= neg * neg;
  // tournament pairing: place 0 stays, the others move one on every round
  int a = sg, b = np - sg;
  const bool in_play = sg < rr / 2;
  for (int round = 0, quiet = 0; round < 60 * np && quiet < np; ++round) {
    const int p = min(a, b), q = max(a, b);
    const bool act = in_play && q < r;
    TS *wp = W + p * lw, *wq = W + q * lw;
    TS x[4], y[4];
    TS al = 0, be = 0, ga = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = sl + 4 * i;
      const bool in = act && t < r;
      x[i] = in ? wp[t] : (TS)0;
      y[i] = in ? wq[t] : (TS)0;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      al = fma(x[i], x[i], al);
      be = fma(y[i], y[i], be);
      ga = fma(x[i], y[i], ga);
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
      al += __shfl_xor_sync(0xffffffffu, al, o);
      be += __shfl_xor_sync(0xffffffffu, be, o);
      ga += __shfl_xor_sync(0xffffffffu, ga, o);
    }
    const bool rot = act && fmin(al, be) > big && ga * ga > thr2 * al * be;
    if (__any_sync(0xffffffffu, rot)) {
      quiet = 0;
      if (rot) {
        TS *vp = V + p * lw, *vq = V + q * lw;
        TS u[4], v[4], c, s;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = min(sl + 4 * i, r - 1);
          u[i] = vp[t];
          v[i] = vq[t];
        }
        jacobi_angle(al, be, ga, c, s);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = sl + 4 * i;
          if (t < r) {
            wp[t] = c * x[i] - s * y[i];
            wq[t] = s * x[i] + c * y[i];
            vp[t] = c * u[i] - s * v[i];
            vq[t] = s * u[i] + c * v[i];
          }
        }
      }
      __syncwarp();
    } else {
      ++quiet;
    }
    if (a != 0) a = a == np ? 1 : a + 1;
    b = b == np ? 1 : b + 1;
  }
}

static __device__ void zero_cols(double* X, int len, int64_t ld, int c0, int c1) {
  for (int c = c0; c < c1; ++c)
    for (int i = threadIdx.x; i < len; i += blockDim.x) X[i + (int64_t)c * ld] = 0.0;
}

// TS: the working precision (double; float for a loose truncation, where
// FP32 Gram-Schmidt and Jacobi keep far more accuracy than the truncation
// discards).  A, B: the tall factors (in TS), J's other fields as for
// core_body; the new factors are written in FP64.
// JAC8 (the H-LU tile kernel): cores of up to 16 columns by jacobi_warp16, larger
// ones in Jacobi rounds with 8 lanes per column pair, so that a round's pairs run
// at once instead of one after another per warp, and the singular values ordered
// by a parallel rank count instead of one thread's selection sort.
template <typename TS, bool JAC8 = false>
static __device__ void core_body_t(const CoreJob& J, TS* __restrict__ JA, TS* __restrict__ JB, int rmax,
                                   double eps_trunc, int* __restrict__ flags) {
  extern __shared__ double sm_raw[];
  TS* sm = reinterpret_cast<TS*>(sm_raw);
  __shared__ double red[32];
  __shared__ TS proj[RCORE_MAX];
  __shared__ TS sig[RCORE_MAX];
  __shared__ int ord[RCORE_MAX];
  __shared__ int s_rot;
  __shared__ int s_k;
  int r = J.r_dev ? *J.r_dev : J.r;
  TS* b0 = sm;                           // R_A, later V (Jacobi right vectors)
  TS* b1 = sm + rmax * (rmax + 1);       // R_B, later U-coefficients
  TS* b2 = sm + 2 * rmax * (rmax + 1);   // W, later V-coefficients
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int pre = J.pre_status ? *J.pre_status : 0;
  if (pre != 0 || r > rmax) {
    // pre == 3: compress() of an absolutely tiny block -> rank-1 zeros;
    // otherwise the input could not be reduced (not converged / too large)
    if (threadIdx.x == 0 && pre != 3) atomicOr(flags, pre == 2 ? 2 : 1);
    zero_cols(J.outA, J.m, J.ldoa, 0, J.kcap);
    zero_cols(J.outB, J.n, J.ldob, 0, J.kcap);
    if (threadIdx.x == 0) *J.rank = (pre == 3) ? 1 : 0;
    return;
  }
  // zero_fill writes zeros up to zlim only: beyond it the columns are zero
  const int zlim = J.known_zero ? min(max(J.zero_from, 0), J.kcap) : J.kcap;
  if (r == 0) {
    if (J.zero_fill) {
      zero_cols(J.outA, J.m, J.ldoa, 0, zlim);
      zero_cols(J.outB, J.n, J.ldob, 0, zlim);
    }
    if (threadIdx.x == 0) *J.rank = 0;
    return;
  }
  cgs2_qr(JA, J.m, J.lda, r, b0, proj, red);
  cgs2_qr(JB, J.n, J.ldb, r, b1, proj, red);
  // W = R_A R_B^T  (r x r, column-major; JAC8: an odd column stride, whose
  // columns start in different banks)
  const int lw = JAC8 ? r | 1 : r;
  double sabs = 0.0;
  for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
    const int i = e % r, j = e / r;
    TS s = 0;
    for (int q = max(i, j); q < r; ++q) s = fma(b0[i + q * r], b1[j + q * r], s);
    b2[i + j * lw] = s;
    sabs += fabs((double)s);
  }
  sabs = block_sum(sabs, red);
  bool nonfinite = !isfinite(sabs);
  if (J.zero_test && sabs < 1e-5) {
    // compress(): an (absolutely) tiny core becomes rank-1 zeros (src/hlu.jl:163-167)
    const int kz = J.zero_fill ? max(zlim, 1) : 1;
    zero_cols(J.outA, J.m, J.ldoa, 0, kz);
    zero_cols(J.outB, J.n, J.ldob, 0, kz);
    if (threadIdx.x == 0) *J.rank = 1;
    return;
  }
  // V = I
  for (int e = threadIdx.x; e < r * r; e += blockDim.x) b0[e % r + e / r * lw] = (e % r == e / r) ? (TS)1 : (TS)0;
  __syncthreads();
  // one-sided Jacobi on the columns of W, round-robin pairing.  A pair is
  // rotated while its cosine exceeds thr; the truncation only needs the
  // singular values far below eps_trunc, so thr follows it (at least 1e-15)
  const int rr = (r + 1) & ~1;
  const TS thr = (TS)fmax(sizeof(TS) == 8 ? 1e-15 : 1e-7, 1e-3 * eps_trunc);
  if (JAC8 && r <= 16) {
    if (w == 0) jacobi_warp16(b2, b0, r, lw, thr, (TS)(1e-3 * eps_trunc));
    __syncthreads();
  } else
  for (int sweep = 0; sweep < 60; ++sweep) {
    if (threadIdx.x == 0) s_rot = 0;
    __syncthreads();
    for (int round = 0; round < rr - 1; ++round) {
      // tournament pairing: position 0 fixed, others rotate
      auto posv = [&](int q) { return q == 0 ? 0 : 1 + (q - 1 + round) % (rr - 1); };
      if constexpr (JAC8) {
        // 8 lanes per pair (4 pairs a warp at once, rows strided by 8): a
        // round's pairs run concurrently instead of one after another per warp
        const int sg = lane >> 3, sl = lane & 7;
        for (int base = w * 4; base < rr / 2; base += nw * 4) {
          const int pidx = base + sg;
          int p = 0, q = 0;
          bool act = pidx < rr / 2;
          if (act) {
            p = posv(pidx); q = posv(rr - 1 - pidx);
            if (p > q) { int t = p; p = q; q = t; }
            act = q < r;
          }
          TS* wp = b2 + p * lw;
          TS* wq = b2 + q * lw;
          TS al = 0, be = 0, ga = 0;
          if (act)
            for (int t = sl; t < r; t += 8) {
              al = fma(wp[t], wp[t], al);
              be = fma(wq[t], wq[t], be);
              ga = fma(wp[t], wq[t], ga);
            }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            al += __shfl_xor_sync(0xffffffffu, al, o);
            be += __shfl_xor_sync(0xffffffffu, be, o);
            ga += __shfl_xor_sync(0xffffffffu, ga, o);
          }
          if (act && ga != (TS)0 && ga * ga > thr * thr * al * be) {
            TS c, s;
            jacobi_angle(al, be, ga, c, s);
            TS* vp = b0 + p * lw;
            TS* vq = b0 + q * lw;
            for (int t2 = sl; t2 < r; t2 += 8) {
              const TS x = wp[t2], y = wq[t2];
              wp[t2] = c * x - s * y;
              wq[t2] = s * x + c * y;
              const TS u = vp[t2], v = vq[t2];
              vp[t2] = c * u - s * v;
              vq[t2] = s * u + c * v;
            }
            if (sl == 0) atomicAdd(&s_rot, 1);
          }
        }
      } else {
      for (int pidx = w; pidx < rr / 2; pidx += nw) {
        int p = posv(pidx), q = posv(rr - 1 - pidx);
        if (p > q) { int t = p; p = q; q = t; }
        if (q >= r) continue;
        TS* wp = b2 + p * r;
        TS* wq = b2 + q * r;
        TS al = 0, be = 0, ga = 0;
        for (int t = lane; t < r; t += 32) {
          al = fma(wp[t], wp[t], al);
          be = fma(wq[t], wq[t], be);
          ga = fma(wp[t], wq[t], ga);
        }
        al = warp_sum(al); be = warp_sum(be); ga = warp_sum(ga);
        if (ga != (TS)0 && fabs(ga) > thr * sqrt(al * be)) {
          const TS zeta = (be - al) / ((TS)2 * ga);
          const TS t = (zeta >= (TS)0 ? (TS)1 : (TS)-1) / (fabs(zeta) + sqrt((TS)1 + zeta * zeta));
          const TS c = (TS)1 / sqrt((TS)1 + t * t), s = c * t;
          TS* vp = b0 + p * r;
          TS* vq = b0 + q * r;
          for (int t2 = lane; t2 < r; t2 += 32) {
            const TS x = wp[t2], y = wq[t2];
            wp[t2] = c * x - s * y;
            wq[t2] = s * x + c * y;
            const TS u = vp[t2], v = vq[t2];
            vp[t2] = c * u - s * v;
            vq[t2] = s * u + c * v;
          }
          if (lane == 0) atomicAdd(&s_rot, 1);
        }
      }
      }
      __syncthreads();
    }
    if (s_rot == 0) break;
    __syncthreads();
  }
  // singular values = column norms of W; sort descending
  for (int j = w; j < r; j += nw) {
    TS s = 0;
    for (int t = lane; t < r; t += 32) s = fma(b2[t + j * lw], b2[t + j * lw], s);
    s = warp_sum(s);
    if (lane == 0) sig[j] = sqrt(s);
  }
  __syncthreads();
  if constexpr (JAC8) {
    // the same stable descending order in parallel (r <= RCORE_MAX < 128
    // threads): column j goes to the place of the values above it and of the
    // equal values before it; ord starts as the identity, so every entry
    // stays a valid column even if a non-finite value breaks the order.  k:
    // on the sorted values the findlast below is the count of ratios > eps.
    if ((int)threadIdx.x < r) ord[threadIdx.x] = threadIdx.x;
    __syncthreads();
    if ((int)threadIdx.x < r) {
      const TS sj = sig[threadIdx.x];
      int pos = 0;
      for (int c = 0; c < r; ++c) pos += (sig[c] > sj) || (sig[c] == sj && c < (int)threadIdx.x);
      if (pos < r) ord[pos] = threadIdx.x;
    }
    __syncthreads();
    const double s1 = sig[ord[0]];
    const int kc = __syncthreads_count((int)threadIdx.x < r && (double)sig[threadIdx.x] / s1 > eps_trunc);
    if (threadIdx.x == 0) s_k = (s1 > 0.0) ? kc : 0;
  } else if (threadIdx.x == 0) {
    for (int j = 0; j < r; ++j) ord[j] = j;
    for (int a = 0; a < r; ++a) {             // stable selection sort, descending
      int b = a;
      for (int c = a + 1; c < r; ++c)
        if (sig[ord[c]] > sig[ord[b]]) b = c;
      int t = ord[b];
      for (int c = b; c > a; --c) ord[c] = ord[c - 1];
      ord[a] = t;
    }
    const double s1 = sig[ord[0]];
    int k = 0;
    for (int j = 0; j < r; ++j)
      if ((double)sig[ord[j]] / s1 > eps_trunc) k = j + 1;   // findlast(S/S[1] .> εTrunc)
    if (!(s1 > 0.0)) k = 0;
    s_k = k;
  }
  __syncthreads();
  int k = s_k;
  if (k > J.kcap) {
    if (threadIdx.x == 0) atomicOr(flags, 1);
    k = J.kcap;
  }
  if (nonfinite && threadIdx.x == 0) atomicOr(flags, 2);
  // coefficients: CU[j][c] = W[j, ord c] / s ; CV[j][c] = V[j, ord c] * s
  for (int e = threadIdx.x; e < r * k; e += blockDim.x) {
    const int j = e % r, c = e / r;
    const int o = ord[c];
    const TS s = sig[o];
    b1[e] = s > (TS)0 ? b2[j + o * lw] / s : (TS)0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < r * k; e += blockDim.x) {
    const int j = e % r, c = e / r;
    const int o = ord[c];
    b2[e] = b0[j + o * lw] * sig[o];
  }
  __syncthreads();
  // (column, row) loops without a division per element; the same sums
  for (int c = 0; c < k; ++c)
    for (int i = threadIdx.x; i < J.m; i += blockDim.x) {
      TS s = 0;
      for (int j = 0; j < r; ++j) s = fma(JA[i + (int64_t)j * J.lda], b1[j + c * r], s);
      J.outA[i + (int64_t)c * J.ldoa] = (double)s;
    }
  for (int c = 0; c < k; ++c)
    for (int i = threadIdx.x; i < J.n; i += blockDim.x) {
      TS s = 0;
      for (int j = 0; j < r; ++j) s = fma(JB[i + (int64_t)j * J.ldb], b2[j + c * r], s);
      J.outB[i + (int64_t)c * J.ldob] = (double)s;
    }
  if (J.zero_fill && k < zlim) {
    zero_cols(J.outA, J.m, J.ldoa, k, zlim);
    zero_cols(J.outB, J.n, J.ldob, k, zlim);
  }
  if (threadIdx.x == 0) *J.rank = k;
}

static __device__ void core_body(const CoreJob& J, int rmax, double eps_trunc, int* __restrict__ flags) {
  core_body_t<double>(J, J.A, J.B, rmax, eps_trunc, flags);
}


}  // namespace hm
