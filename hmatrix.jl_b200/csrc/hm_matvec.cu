// H-matvec on sm_100a (K4): y = H x and y = H' x over the flattened leaf
// list, the device form of hmat_matvec! (src/harithm.jl:340-354) and
// transpose_hmat_mat_mul (src/harithm.jl:243-260).
//
// Phase 1: one warp per low-rank leaf streams its F1 factor (B for H*x)
//          with 16-byte loads and writes z = F1' x_seg (k values) to z[].
// Phase 2: y = sum_r F2[:,r] z_r over the low-rank leaves + C x_seg over the
//          dense leaves, by row slabs cut at clusters (the default; the lists
//          are made on first use), or by windows of 1024 output rows with 4
//          rows a lane (the lists that every plan has).
// FP64 factors are accumulated in FP64.  FP32 and BF16 factors are
// multiplied and summed in FP32 over the few vectors (phase 1) or entries
// (phase 2) a lane has in flight, and those FP32 partial sums are added in
// FP64: one conversion per group instead of one per element.
// For FP32 and BF16 factors the input is staged as 16-byte aligned shifted
// copies in FP32, so that every x-segment load in phase 1 is a vector load,
// whatever the segment start; with FP64 factors phase 1 reads x itself.
#include "hm_internal.h"
#include "hm_lowrank.cuh"

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cstring>

namespace hm {

// ---------------------------------------------------------------------------
// storage traits: 16-byte vector of factors + matching x vector
// ---------------------------------------------------------------------------
template <typename T> struct MvT;
template <> struct MvT<double> {
  static constexpr int VW = 2, U = 2;
  using X = double;
  using R = double2;
  struct XV { double2 a; };
  __device__ static R ld(const double* p) { return __ldcs(reinterpret_cast<const double2*>(p)); }
  __device__ static double dot(const R& f, const XV& x, double s) {
    s = fma(f.x, x.a.x, s);
    return fma(f.y, x.a.y, s);
  }
};
template <> struct MvT<float> {
  static constexpr int VW = 4, U = 2;
  using X = float;
  using R = float4;
  struct XV { float4 a; };
  __device__ static R ld(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
  __device__ static XV ldx(const float* p) { return XV{__ldg(reinterpret_cast<const float4*>(p))}; }
  // FP32 partial sum of one vector (the caller folds it into its FP64 sum)
  __device__ static float dotf(const R& f, const XV& x, float s) {
    s = fmaf(f.x, x.a.x, s);
    s = fmaf(f.y, x.a.y, s);
    s = fmaf(f.z, x.a.z, s);
    return fmaf(f.w, x.a.w, s);
  }
};
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
template <> struct MvT<__nv_bfloat16> {
  static constexpr int VW = 8, U = 2;
  using X = float;
  using R = uint4;
  struct XV { float4 a, b; };
  __device__ static R ld(const __nv_bfloat16* p) { return __ldcs(reinterpret_cast<const uint4*>(p)); }
  __device__ static XV ldx(const float* p) {
    return XV{__ldg(reinterpret_cast<const float4*>(p)), __ldg(reinterpret_cast<const float4*>(p) + 1)};
  }
  // BF16 -> FP32 is a shift of the bits; FP32 partial sum of one vector
  __device__ static float dotf(const R& f, const XV& x, float s) {
    s = fmaf(bf_lo(f.x), x.a.x, s);
    s = fmaf(bf_hi(f.x), x.a.y, s);
    s = fmaf(bf_lo(f.y), x.a.z, s);
    s = fmaf(bf_hi(f.y), x.a.w, s);
    s = fmaf(bf_lo(f.z), x.b.x, s);
    s = fmaf(bf_hi(f.z), x.b.y, s);
    s = fmaf(bf_lo(f.w), x.b.z, s);
    return fmaf(bf_hi(f.w), x.b.w, s);
  }
};

// shifted copies: copy q holds x[t - q] at index t (zero outside [q, n+q))
template <typename TX>
__global__ void xcopy_kernel(const double* __restrict__ x, int64_t n, TX* __restrict__ xs, int64_t stride, int ncopy) {
  const int64_t tot = stride * ncopy;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = e / stride, t = e % stride;
    const int64_t s = t - q;
    xs[e] = (s >= 0 && s < n) ? (TX)x[s] : (TX)0;
  }
}

// ---------------------------------------------------------------------------
// phase 1: z = F1' x_seg, one warp per low-rank leaf
// ---------------------------------------------------------------------------
// A leaf's columns r .. r + NR - 1 (1 to 4 of them, all in flight together).
// z of the NR columns is summed over the warp by one reduce-scatter.
template <typename T, int NR>
__device__ __forceinline__ void p1_columns(const T* __restrict__ F, uint32_t stride, uint32_t len,
                                           const typename MvT<T>::X* __restrict__ xb, double* __restrict__ z,
                                           int lane) {
  using Tr = MvT<T>;
  constexpr int VW = Tr::VW, U = Tr::U, NV = NR == 3 ? 4 : NR;
  const int nvec = (int)(stride / VW);
  double sc[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) sc[j] = 0.0;
  for (int v0 = lane; v0 < nvec; v0 += 32 * U) {
    typename Tr::R a[NR][U];
    typename Tr::XV xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = min(v0 + 32 * u, nvec - 1);          // past the end: the last vector, not summed
#pragma unroll
      for (int j = 0; j < NR; ++j) a[j][u] = Tr::ld(F + (int64_t)j * stride + (int64_t)v * VW);
      if constexpr (std::is_same<T, double>::value) {
        // the padding elements multiply no x (there may be none behind the last)
        xv[u].a.x = 2 * v < (int)len ? __ldg(xb + 2 * v) : 0.0;
        xv[u].a.y = 2 * v + 1 < (int)len ? __ldg(xb + 2 * v + 1) : 0.0;
      } else {
        xv[u] = Tr::ldx(xb + (int64_t)v * VW);
      }
    }
    if constexpr (std::is_same<T, double>::value) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + 32 * u < nvec) {
#pragma unroll
          for (int j = 0; j < NR; ++j) sc[j] = Tr::dot(a[j][u], xv[u], sc[j]);
        }
    } else {
      // FP32 products and partial sums over the U vectors in flight, folded
      // into the FP64 sums once per group
#pragma unroll
      for (int j = 0; j < NR; ++j) {
        float fp = 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < nvec) fp = Tr::dotf(a[j][u], xv[u], fp);
        sc[j] += (double)fp;
      }
    }
  }
  int idx;
  const double sum = warp_reduce_scatter<NV>(sc, lane, idx);
  if ((lane & (32 / NV - 1)) == 0 && idx < NR) z[idx] = sum;
}

// One warp per low-rank leaf, the next leaf's descriptor fetched while this
// one's columns stream; columns in groups of 4 or less, as even as they go.
// Bound: HBM.  Three columns at a time instead of two and one repeated column,
// and a third of the shuffles: the FP32 kernel had 16 warps an SM waiting on
// 2 x 4 vectors each and spent as many instructions reducing as loading.
template <typename T>
__global__ void __launch_bounds__(256, 3) mv_phase1_kernel(const P1Desc* __restrict__ d, int64_t nd,
                                                        const T* __restrict__ pool,
                                                        const typename MvT<T>::X* __restrict__ xs,
                                                        int64_t xs_stride, double* __restrict__ z) {
  using TX = typename MvT<T>::X;
  constexpr int XA = 16 / (int)sizeof(TX);
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  P1Desc N{};
  if (gw < nd) N = d[gw];
  for (int64_t b = gw; b < nd; b += nw) {
    const P1Desc D = N;
    if (b + nw < nd) N = d[b + nw];
    const TX* xb = xs + D.seg0;
    if constexpr (!std::is_same<T, double>::value) {
      const int q = (XA - (int)(D.seg0 % XA)) % XA;
      xb += q * xs_stride + q;
    }
    const T* F = pool + D.off;
    double* zp = z + D.zoff;
    for (int left = D.k; left > 0;) {
      const int ng = (left + 3) / 4, nr = (left + ng - 1) / ng;
      if (nr == 4) p1_columns<T, 4>(F, D.stride, D.len, xb, zp, lane);
      else if (nr == 3) p1_columns<T, 3>(F, D.stride, D.len, xb, zp, lane);
      else if (nr == 2) p1_columns<T, 2>(F, D.stride, D.len, xb, zp, lane);
      else p1_columns<T, 1>(F, D.stride, D.len, xb, zp, lane);
      F += (int64_t)nr * D.stride;
      zp += nr;
      left -= nr;
    }
  }
}

// ---------------------------------------------------------------------------
// phase 2: y(window) = sum over leaves covering the window.  Each lane owns 4
// consecutive output rows; when a leaf starts on a 4-row boundary of the
// window its 4 values come in one vector load (columns are padded to a
// multiple of 4 elements and 16 bytes, padding rows hold zeros).
// ---------------------------------------------------------------------------
constexpr int P2_NB = 32;      // descriptors staged per round
// SPLIT (2, 4 or 8 CTAs per 1024-row window) is chosen per handle by the
// autotuner (hm_autotune); 4 until then
template <int SPLIT> struct P2Shape {
  static constexpr int CROWS = MV_WROWS / SPLIT;   // rows of one CTA
  static constexpr int WARPS = CROWS / 128;        // 32 lanes x 4 rows a warp
  static constexpr int EMAX = 1024 / SPLIT;        // expanded (leaf, column) entries per sub-round
};
constexpr uint64_t P2_DENSE_FLAG = 1ull << 63;

// 4 consecutive rows of one column are loaded as raw words and converted to
// FP64 only when they are multiplied: a conversion next to its load would
// make the warp wait for that load before issuing the next entry's loads.
template <typename T> struct Row4;
template <> struct Row4<double> {               // dense leaves: double as well
  static constexpr int U = 4;
  struct Raw { double2 a, b; };
  __device__ static Raw zero() { return Raw{make_double2(0.0, 0.0), make_double2(0.0, 0.0)}; }
  __device__ static Raw ld(const double* p) {
    return Raw{__ldcs(reinterpret_cast<const double2*>(p)), __ldcs(reinterpret_cast<const double2*>(p) + 1)};
  }
  __device__ static Raw ldd(const double* p) { return ld(p); }
  __device__ static void put(Raw& r, int q, double v) {
    if (q == 0) r.a.x = v; else if (q == 1) r.a.y = v; else if (q == 2) r.b.x = v; else r.b.y = v;
  }
  __device__ static void cvt(const Raw& r, bool, double (&v)[4]) { v[0] = r.a.x; v[1] = r.a.y; v[2] = r.b.x; v[3] = r.b.y; }
};
template <> struct Row4<float> {                // dense leaves: float
  static constexpr int U = 8;
  using Raw = float4;
  __device__ static Raw zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ static Raw ld(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
  __device__ static Raw ldd(const float* p) { return ld(p); }
  __device__ static void put(Raw& r, int q, float v) {
    if (q == 0) r.x = v; else if (q == 1) r.y = v; else if (q == 2) r.z = v; else r.w = v;
  }
  __device__ static void cvt(const Raw& r, bool, double (&v)[4]) { v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w; }
  __device__ static void cvtf(const Raw& r, bool, float (&v)[4]) { v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w; }
};
template <> struct Row4<__nv_bfloat16> {        // dense leaves: float (raw float bits)
  static constexpr int U = 8;
  using Raw = uint4;
  __device__ static Raw zero() { return make_uint4(0u, 0u, 0u, 0u); }
  __device__ static Raw ld(const __nv_bfloat16* p) {
    const uint2 a = __ldcs(reinterpret_cast<const uint2*>(p));
    return make_uint4(a.x, a.y, 0u, 0u);
  }
  __device__ static Raw ldd(const float* p) {
    return __ldcs(reinterpret_cast<const uint4*>(p));
  }
  __device__ static void put(Raw& r, int q, float v) {
    const uint32_t b = __float_as_uint(v);
    if (q == 0) r.x = b; else if (q == 1) r.y = b; else if (q == 2) r.z = b; else r.w = b;
  }
  __device__ static void put(Raw& r, int q, __nv_bfloat16 v) {
    const uint32_t b = (uint32_t)__bfloat16_as_ushort(v);
    if (q == 0) r.x = (r.x & 0xffff0000u) | b;
    else if (q == 1) r.x = (r.x & 0x0000ffffu) | (b << 16);
    else if (q == 2) r.y = (r.y & 0xffff0000u) | b;
    else r.y = (r.y & 0x0000ffffu) | (b << 16);
  }
  __device__ static void cvt(const Raw& r, bool dense, double (&v)[4]) {
    if (dense) {
      v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y);
      v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
    } else {
      v[0] = bf_lo(r.x); v[1] = bf_hi(r.x); v[2] = bf_lo(r.y); v[3] = bf_hi(r.y);
    }
  }
  __device__ static void cvtf(const Raw& r, bool dense, float (&v)[4]) {
    if (dense) {
      v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y);
      v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
    } else {
      v[0] = bf_lo(r.x); v[1] = bf_hi(r.x); v[2] = bf_lo(r.y); v[3] = bf_hi(r.y);
    }
  }
};

template <typename T, typename TD, int SPLIT>
__global__ void __launch_bounds__(P2Shape<SPLIT>::WARPS * 32) mv_phase2_kernel(const MvWin* __restrict__ win,
                                                                  const P2Desc* __restrict__ d,
                                                                  const T* __restrict__ rk, const TD* __restrict__ dn,
                                                                  const double* __restrict__ z,
                                                                  const double* __restrict__ x,
                                                                  double* __restrict__ y) {
  constexpr int U = Row4<T>::U;
  constexpr int P2_SPLIT = SPLIT, P2_CROWS = P2Shape<SPLIT>::CROWS, P2_EMAX = P2Shape<SPLIT>::EMAX;
  __shared__ P2Desc sd[P2_NB];
  __shared__ int spre[P2_NB + 1];
  __shared__ uint64_t e_off[P2_EMAX];
  __shared__ int32_t e_ro[P2_EMAX];
  __shared__ uint32_t e_m[P2_EMAX];
  __shared__ uint32_t e_rs[P2_EMAX];
  __shared__ double e_z[P2_EMAX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MvWin W = win[blockIdx.x / P2_SPLIT];
  const int h0 = (int)(blockIdx.x % P2_SPLIT) * P2_CROWS;   // this CTA's rows of the window
  const int base = h0 + 4 * (warp * 32 + lane);  // first of this lane's rows in the window
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t b0 = W.begin; b0 < W.end; b0 += P2_NB) {
    const int nb = (int)min((uint32_t)P2_NB, W.end - b0);
    __syncthreads();
    if (warp == 0) {
      int cnt = 0;
      if (lane < nb) {
        sd[lane] = d[b0 + lane];
        // only leaves with rows in this CTA's part of the window are expanded
        const int r0 = sd[lane].row_off, r1 = r0 + (int)sd[lane].m;
        cnt = (r1 > h0 && r0 < h0 + P2_CROWS) ? (int)sd[lane].cnt : 0;
      }
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      spre[lane + 1] = incl;
      if (lane == 0) spre[0] = 0;
    }
    __syncthreads();
    const int total = spre[nb];
    for (int e0 = 0; e0 < total; e0 += P2_EMAX) {
      const int ne = min(P2_EMAX, total - e0);
      if (e0 > 0) __syncthreads();
      for (int e = threadIdx.x; e < ne; e += blockDim.x) {
        const int ge = e0 + e;
        int lo = 0, hi = nb - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (spre[mid] <= ge) lo = mid; else hi = mid - 1;
        }
        const P2Desc& D = sd[lo];
        const int c = ge - spre[lo];
        if (D.type == P2_RK) {
          e_off[e] = D.off + (uint64_t)c * D.ld;
          e_rs[e] = 1;
          e_z[e] = z[D.aux + c];
        } else if (D.type == P2_DENSE) {
          e_off[e] = (D.off + (uint64_t)c * D.ld) | P2_DENSE_FLAG;
          e_rs[e] = 1;
          e_z[e] = x[D.aux + c];
        } else {
          e_off[e] = (D.off + (uint64_t)c) | P2_DENSE_FLAG;
          e_rs[e] = D.ld;
          e_z[e] = x[D.aux + c];
        }
        e_ro[e] = D.row_off;
        e_m[e] = D.m;
      }
      __syncthreads();
      for (int e = 0; e < ne; e += U) {
        typename Row4<T>::Raw raw[U];
        double zz[U];
        bool isd[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          raw[u] = Row4<T>::zero();
          zz[u] = 0.0;
          isd[u] = false;
          const int ee = e + u;
          if (ee < ne) {
            const int ro = e_ro[ee];
            const int mm = (int)e_m[ee];
            const uint64_t o = e_off[ee];
            const uint32_t rs = e_rs[ee];
            const int lr = base - ro;
            const bool dense = (o & P2_DENSE_FLAG) != 0;
            zz[u] = e_z[ee];
            isd[u] = dense;
            if (((ro & 3) == 0) && rs == 1) {
              if (lr >= 0 && lr < mm) {
                if (dense) raw[u] = Row4<T>::ldd(dn + (o & ~P2_DENSE_FLAG) + lr);
                else raw[u] = Row4<T>::ld(rk + o + lr);
              }
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int r = lr + q;
                if (r >= 0 && r < mm) {
                  if (dense) Row4<T>::put(raw[u], q, __ldg(dn + (o & ~P2_DENSE_FLAG) + (uint64_t)r * rs));
                  else Row4<T>::put(raw[u], q, rk[o + (uint64_t)r]);
                }
              }
            }
          }
        }
        if constexpr (std::is_same<T, double>::value) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            double v[4];
            Row4<T>::cvt(raw[u], isd[u], v);
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = fma(v[q], zz[u], acc[q]);
          }
        } else {
          // FP32 products and partial sums over the U entries in flight,
          // folded into the FP64 row sums once per group
          float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int u = 0; u < U; ++u) {
            float v[4];
            Row4<T>::cvtf(raw[u], isd[u], v);
            const float zf = (float)zz[u];
#pragma unroll
            for (int q = 0; q < 4; ++q) part[q] = fmaf(v[q], zf, part[q]);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[q] += (double)part[q];
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (base + q < (int)W.nrows) y[W.row0 + base + q] = acc[q];
}

// ---------------------------------------------------------------------------
// phase 2 by row slabs: the output rows are cut at cluster boundaries into
// slabs of at most 224 rows; one CTA per slab, R = ceil(rows / 32) rows a lane
// (32 apart), its 8 warps splitting the slab's entries (one entry: one column
// of a leaf over the slab's rows) and adding their sums in shared memory, in
// one launch that writes every row once.  A lane reads single elements, 32
// consecutive rows per warp load, so a leaf may start at any row: no alignment
// to honour, and few idle lanes since leaves end where slabs end.  The next 32
// entries and their z values are fetched while the current ones are summed.
// Bound: HBM (R x 32 elements per entry).  Why slabs: grouped by tree cluster
// (one warp per 128 rows of a cluster, a launch per tree level) a level of
// n = 100003 has about 1000 warps with 760 dependent entries each, a fifth of
// what the SMs hold, and the levels run one after another.
// ---------------------------------------------------------------------------
constexpr int SL_WARPS = 8;
constexpr int SL_RMAX = 7;                     // rows a lane at most

// one element of a factor or dense leaf: how it is loaded and its value
template <typename E> struct SlT {
  using Raw = E;
  __device__ static Raw ld(const E* p) { return __ldcs(p); }
  __device__ static E val(Raw r) { return r; }
};
template <> struct SlT<__nv_bfloat16> {
  using Raw = unsigned short;
  __device__ static Raw ld(const __nv_bfloat16* p) { return __ldcs(reinterpret_cast<const unsigned short*>(p)); }
  __device__ static float val(Raw r) { return __uint_as_float((uint32_t)r << 16); }
};

// acc[q] += the entries [begin, begin + ne) of one kind, this warp's share of
// them in whole groups of 8: E the element type, v the array zi indexes
template <typename E, typename A, int R>
__device__ __forceinline__ void slab_sum(const SlabEnt* __restrict__ ents, uint32_t begin, uint32_t ne,
                                         const E* __restrict__ pool, const double* __restrict__ v, int warp, int lane,
                                         double (&acc)[R]) {
  // entries whose loads are in flight together: 16 to 56 loads, 64 registers at most
  constexpr int U = (sizeof(A) == 8 ? 32 : 64) / R >= 16 ? 16 : (sizeof(A) == 8 ? 32 : 64) / R >= 8 ? 8 : 4;
  const uint32_t per = (ne + SL_WARPS * 8 - 1) / (SL_WARPS * 8) * 8;
  const uint32_t e0 = begin + min(ne, warp * per), e1 = begin + min(ne, (warp + 1) * per);
  const SlabEnt none{0, 0, 255u | 255u << 8};            // row 255: in no slab
  SlabEnt cur = e0 + lane < e1 ? ents[e0 + lane] : none;
  A zc = e0 + lane < e1 ? (A)__ldg(v + cur.zi) : A(0);
  for (uint32_t e = e0; e < e1; e += 32) {
    const bool more = e + 32 + lane < e1;
    const SlabEnt nxt = more ? ents[e + 32 + lane] : none;
    const int n32 = (int)min(32u, e1 - e);
    const E* mine = pool + (cur.off & SLAB_OFF_MASK);
    A zn = A(0);
    for (int u0 = 0; u0 < n32; u0 += U) {
      typename SlT<E>::Raw raw[U][R];
      uint32_t first[U], span[U];                        // lane - lo, last - lo
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const E* p = reinterpret_cast<const E*>(__shfl_sync(0xffffffffu, (unsigned long long)mine, u0 + u));
        const uint32_t mt = __shfl_sync(0xffffffffu, cur.meta, u0 + u);
        first[u] = lane - (mt & 255u);
        span[u] = (mt >> 8 & 255u) - (mt & 255u);
        // no branch around the loads, or the compiler moves each beside its use:
        // rows not covered read the entry's last row
#pragma unroll
        for (int q = 0; q < R; ++q) raw[u][q] = SlT<E>::ld(p + min(first[u] + 32 * q, span[u]));
      }
      if (u0 == 0 && more) zn = (A)__ldg(v + nxt.zi);     // behind this group's loads
      A part[R];
#pragma unroll
      for (int q = 0; q < R; ++q) part[q] = A(0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const A zz = __shfl_sync(0xffffffffu, zc, u0 + u);
#pragma unroll
        for (int q = 0; q < R; ++q)
          if (first[u] + 32 * q <= span[u]) {            // rows not covered: an infinite z stays out
            if constexpr (std::is_same<A, double>::value) acc[q] = fma((A)SlT<E>::val(raw[u][q]), zz, acc[q]);
            else part[q] = fmaf(SlT<E>::val(raw[u][q]), zz, part[q]);
          }
        // FP32 products and partial sums over 8 entries, folded into the FP64
        // row sums
        if (!std::is_same<A, double>::value && u % 8 == 7) {
#pragma unroll
          for (int q = 0; q < R; ++q) {
            acc[q] += (double)part[q];
            part[q] = A(0);
          }
        }
      }
    }
    cur = nxt;
    zc = zn;
  }
}

// one slab's sums over this warp's entries, into its rows of part_sh
template <typename T, typename TD, int R>
__device__ __forceinline__ void slab_rows(const Slab& S, const SlabEnt* __restrict__ ents, const T* __restrict__ rk,
                                          const TD* __restrict__ dn, const double* __restrict__ z,
                                          const double* __restrict__ x, double* __restrict__ part_sh, int warp, int lane) {
  // the dense leaves of BF16 factors (near field, FP32) are FP64 products, as
  // they are in every other shape and direction
  using A = typename std::conditional<std::is_same<T, double>::value, double, float>::type;
  using AD = typename std::conditional<std::is_same<T, float>::value, float, double>::type;
  double acc[R];
#pragma unroll
  for (int q = 0; q < R; ++q) acc[q] = 0.0;
  slab_sum<T, A, R>(ents, S.begin, S.dense - S.begin, rk, z, warp, lane, acc);
  slab_sum<TD, AD, R>(ents, S.dense, S.mid - S.dense, dn, x, warp, lane, acc);
  // dense leaves read along their rows (H'x): an entry is 32 input indices of
  // one leaf; lane = input index (coalesced), 16 rows at a time, whose sums
  // over the lanes a reduce-scatter leaves in lanes 2 i and 2 i + 1
  for (uint32_t e = S.mid + warp; e < S.end; e += SL_WARPS) {
    const SlabEnt E = ents[e];
    const int lo = (int)(E.meta & 255u), last = (int)(E.meta >> 8 & 255u), cnt = (int)(E.meta >> 24);
    const int64_t ld = (int64_t)(E.off >> 40);
    const TD* base = dn + (E.off & SLAB_OFF_MASK) + lane;
    const double xv = lane < cnt ? __ldg(x + E.zi + lane) : 0.0;
#pragma unroll
    for (int g = 0; g < 2 * R; ++g) {
      const int g0 = 16 * g;                             // rows g0 .. g0 + 15
      if (g0 > last || g0 + 15 < lo) continue;
      double v[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const bool in = lane < cnt && g0 + r >= lo && g0 + r <= last;
        v[r] = in ? (double)__ldcs(base + (g0 + r - lo) * ld) : 0.0;
      }
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (lane < cnt && g0 + r >= lo && g0 + r <= last) v[r] *= xv;
      int idx;
      const double sum = warp_reduce_scatter<16>(v, lane, idx);
      const double got = __shfl_sync(0xffffffffu, sum, 2 * (lane & 15));
      if ((lane >> 4) == (g & 1)) acc[g >> 1] += got;
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q) part_sh[warp * 32 * SL_RMAX + lane + 32 * q] = acc[q];
}

template <typename T, typename TD>
__global__ void __launch_bounds__(SL_WARPS * 32, 2) mv_slab_kernel(const Slab* __restrict__ slabs,
                                                                const SlabEnt* __restrict__ ents,
                                                                const T* __restrict__ rk, const TD* __restrict__ dn,
                                                                const double* __restrict__ z,
                                                                const double* __restrict__ x,
                                                                double* __restrict__ y) {
  __shared__ double part_sh[SL_WARPS * 32 * SL_RMAX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Slab S = slabs[blockIdx.x];
  switch ((S.nrows + 31) / 32) {
    case 1: slab_rows<T, TD, 1>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    case 2: slab_rows<T, TD, 2>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    case 3: slab_rows<T, TD, 3>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    case 4: slab_rows<T, TD, 4>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    case 5: slab_rows<T, TD, 5>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    case 6: slab_rows<T, TD, 6>(S, ents, rk, dn, z, x, part_sh, warp, lane); break;
    default: slab_rows<T, TD, 7>(S, ents, rk, dn, z, x, part_sh, warp, lane);
  }
  __syncthreads();
  for (int r = threadIdx.x; r < (int)S.nrows; r += SL_WARPS * 32) {
    double s = part_sh[r];
#pragma unroll
    for (int w = 1; w < SL_WARPS; ++w) s += part_sh[w * 32 * SL_RMAX + r];
    y[S.row0 + r] = s;
  }
}

// ---------------------------------------------------------------------------
// plan construction
// ---------------------------------------------------------------------------
void free_mv_plan(MvPlan& p) {
  if (p.d_desc) cudaFree(p.d_desc);
  if (p.d_mbcol) cudaFree(p.d_mbcol);
  if (p.d_p2d) cudaFree(p.d_p2d);
  if (p.d_wind) cudaFree(p.d_wind);
  if (p.d_p2r) cudaFree(p.d_p2r);
  if (p.d_winr) cudaFree(p.d_winr);
  if (p.d_slab) cudaFree(p.d_slab);
  if (p.d_ent) cudaFree(p.d_ent);
  p = MvPlan{};
}

// The entries of the slabs, from the window lists that every plan has on the
// device: a warp per slab walks the leaves of its one or two windows (a leaf that
// reaches back before the second one was met in the first) and counts, or writes,
// an entry per column of those with rows in the slab; low-rank leaves first, those
// read along their rows (dense, H'x) last, each kind in list order.  Made by the
// host from the leaves, a first product waited 3.2 ms for the lists at n = 131072
// (70912 leaves), most of it in the host's caches, and for their upload.
struct SlabTotal {
  unsigned long long entries;
  unsigned long long narrow;             // a row stride too large for its field
};
template <bool FILL>
__global__ void __launch_bounds__(256) slab_lists_kernel(Slab* __restrict__ slabs, int64_t nslab,
                                                         const MvWin* __restrict__ win, const P2Desc* __restrict__ d,
                                                         SlabEnt* __restrict__ ent, SlabTotal* __restrict__ total) {
  const int lane = threadIdx.x & 31;
  const int64_t sl = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (sl >= nslab) return;
  const Slab S = slabs[sl];
  const int64_t s0 = S.row0, s1 = s0 + S.nrows;
  // next entry (FILL), or this lane's counts: low-rank, dense, along rows
  uint32_t at[3] = {FILL ? S.begin : 0u, FILL ? S.dense : 0u, FILL ? S.mid : 0u};
  bool narrow = false;
  const int64_t w0 = s0 / MV_WROWS, w1 = (s1 - 1) / MV_WROWS;
  for (int64_t w = w0; w <= w1; ++w) {
    const MvWin W = win[w];
    for (uint32_t b0 = W.begin; b0 < W.end; b0 += 32) {
      P2Desc D{};
      if (b0 + lane < W.end) D = d[b0 + lane];
      const int64_t o0 = w * MV_WROWS + D.row_off;
      const bool in = D.m > 0 && o0 < s1 && o0 + D.m > s0 && (w == w0 || D.row_off >= 0);
      const uint32_t ne = D.type == P2_DENSE_T ? (D.cnt + 31) / 32 : D.cnt;
      if constexpr (!FILL) {
        if (in) {
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if ((D.type == P2_RK ? 0 : D.type == P2_DENSE ? 1 : 2) == k) at[k] += ne;
          narrow = narrow || (D.type == P2_DENSE_T && D.ld >= 1u << 24);
        }
      } else {
        for (unsigned todo = __ballot_sync(0xffffffffu, in); todo; todo &= todo - 1) {
          const int src = __ffs(todo) - 1;
          const uint64_t off = __shfl_sync(0xffffffffu, (unsigned long long)D.off, src);
          const int64_t r0 = __shfl_sync(0xffffffffu, (long long)o0, src);
          const int64_t r1 = r0 + __shfl_sync(0xffffffffu, D.m, src);
          const uint32_t ld = __shfl_sync(0xffffffffu, D.ld, src), zi = __shfl_sync(0xffffffffu, D.aux, src);
          const uint32_t cnt = __shfl_sync(0xffffffffu, D.cnt, src), n = __shfl_sync(0xffffffffu, ne, src);
          const uint32_t type = __shfl_sync(0xffffffffu, (uint32_t)D.type, src);
          const int64_t a = r0 > s0 ? r0 : s0, b = r1 < s1 ? r1 : s1;
          const uint32_t meta = (uint32_t)(a - s0) | (uint32_t)(b - 1 - s0) << 8 | type << 16;
          uint32_t& p = type == P2_RK ? at[0] : type == P2_DENSE ? at[1] : at[2];
          for (uint32_t c = lane; c < n; c += 32) {
            SlabEnt E;
            if (type == P2_DENSE_T) {
              E.off = (off + (uint64_t)(a - r0) * ld + 32 * c) | (uint64_t)ld << 40;
              E.zi = zi + 32 * c;
              E.meta = meta | min(32u, cnt - 32 * c) << 24;
            } else {
              E.off = off + (uint64_t)c * ld + (uint64_t)(a - r0);
              E.zi = zi + c;
              E.meta = meta;
            }
            ent[p + c] = E;
          }
          p += n;
        }
      }
    }
  }
  if constexpr (!FILL) {
#pragma unroll
    for (int k = 0; k < 3; ++k) at[k] = __reduce_add_sync(0xffffffffu, at[k]);
    if (lane == 0) {
      slabs[sl].begin = at[0];
      slabs[sl].dense = at[1];
      slabs[sl].mid = at[2];
    }
    if (narrow) atomicOr(&total->narrow, 1ull);
  }
}

// counts -> entry ranges, slab after slab, by one CTA
__global__ void __launch_bounds__(1024) slab_scan_kernel(Slab* __restrict__ slabs, int64_t nslab,
                                                         SlabTotal* __restrict__ total) {
  __shared__ unsigned long long sum[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long base = 0;
  for (int64_t b = 0; b < nslab; b += 1024) {
    const int64_t i = b + threadIdx.x;
    Slab S{};
    if (i < nslab) S = slabs[i];
    const unsigned long long own = (unsigned long long)S.begin + S.dense + S.mid;
    unsigned long long incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();                                     // the last round's sums
    if (lane == 31) sum[warp] = incl;
    __syncthreads();
    unsigned long long first = base + incl - own;
    for (int q = 0; q < 32; ++q) {
      if (q < warp) first += sum[q];
      base += sum[q];
    }
    if (i < nslab) {
      S.end = (uint32_t)(first + own);
      S.mid = (uint32_t)(first + S.begin + S.dense);
      S.dense = (uint32_t)(first + S.begin);
      S.begin = (uint32_t)first;
      slabs[i] = S;
    }
  }
  if (threadIdx.x == 0) total->entries = base;
}

// The slab boundaries for slabs of at most `most` rows: the highest clusters
// that small, a leaf cluster above that size in equal pieces.  Leaves of the
// block tree sit on clusters, so they end where slabs do.
static void slab_cuts(const hm_handle* h, int64_t most, std::vector<Slab>& out) {
  out.clear();
  std::vector<int64_t> todo(1, 0);
  while (!todo.empty()) {
    const int64_t c = todo.back();
    todo.pop_back();
    const int64_t s = h->cl_s[c], m = h->cl_e[c] - s;
    if (m > most && h->cl_left[c] >= 0) {
      todo.push_back(h->cl_right[c]);
      todo.push_back(h->cl_left[c]);
      continue;
    }
    const int64_t np = (m + most - 1) / most;
    for (int64_t i = 0; i < np; ++i) {
      Slab S{};
      S.row0 = (uint32_t)(s + m * i / np);
      S.nrows = (uint32_t)(s + m * (i + 1) / np - S.row0);
      out.push_back(S);
    }
  }
}

// The slab size: of 32, 64, .. 224 rows at most, the one whose slabs leave the
// fewest lanes idle (the larger one on a tie: fewer entries per factor byte),
// among those that give every SM four slabs; 32 rows for matrices too small
// for that.  No slab above MaxBlock rows: a row shard is cut at clusters of at
// most that size, and its slabs are then the whole matrix's.
static void choose_slabs(const hm_handle* h, std::vector<Slab>& best) {
  slab_cuts(h, 32, best);
  double eff = 0.0;
  std::vector<Slab> v;
  for (int r = 1; r <= SL_RMAX; ++r) {
    if (r > 1 && h->prm.max_block > 0 && 32 * r > h->prm.max_block) break;
    slab_cuts(h, 32 * r, v);
    if (v.size() < 4 * 148) break;
    int64_t lanes = 0;
    for (const Slab& S : v) lanes += (S.nrows + 31) / 32 * 32;
    const double e = (double)h->n / (double)lanes;
    if (e >= eff * 0.999) {
      eff = std::max(eff, e);
      best = v;
    }
  }
}

// The slab lists of one direction.
static int build_slab_plan(hm_handle* h, MvPlan& P) {
  std::vector<Slab> slab;
  choose_slabs(h, slab);
  const int64_t nslab = (int64_t)slab.size();
  if (nslab > INT32_MAX) return HM_ERR_UNSUPPORTED;
  const size_t sb = sizeof(Slab) * slab.size(), so = pad_to((int64_t)sb, 256);
  struct Mem {                                           // given back unless the plan takes it
    void* p = nullptr;
    ~Mem() { if (p) cudaFree(p); }
  } lists, ents;
  auto no_memory = [] {
    cudaGetLastError();
    return HM_ERR_OOM;
  };
  if (cudaMalloc(&lists.p, so + sizeof(SlabTotal)) != cudaSuccess) return no_memory();
  Slab* d_slab = (Slab*)lists.p;
  SlabTotal* d_total = (SlabTotal*)((char*)lists.p + so);
  SlabTotal total{};
  const unsigned grid = (unsigned)((nslab + 7) / 8);
  HM_CUDA_TRY(cudaMemcpyAsync(d_slab, slab.data(), sb, cudaMemcpyHostToDevice, h->stream));
  HM_CUDA_TRY(cudaMemsetAsync(d_total, 0, sizeof(SlabTotal), h->stream));
  slab_lists_kernel<false><<<grid, 256, 0, h->stream>>>(d_slab, nslab, P.d_win, P.d_p2, nullptr, d_total);
  slab_scan_kernel<<<1, 1024, 0, h->stream>>>(d_slab, nslab, d_total);
  HM_CUDA_TRY(cudaGetLastError());
  HM_CUDA_TRY(cudaMemcpyAsync(&total, d_total, sizeof(SlabTotal), cudaMemcpyDeviceToHost, h->stream));
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  if (total.narrow || total.entries > (unsigned long long)UINT32_MAX) return HM_ERR_UNSUPPORTED;
  // a plain allocation is cheap up to 2 MB (a part of a block the driver holds) and
  // takes 0.2 ms longer than one from the stream-ordered pool above (first product
  // n = 32768 0.62 and 0.44 ms, n = 131072 1.08 and 0.81; n = 2000 0.13 and 0.36);
  // large lists stay out of a pool that may keep what is given back
  const size_t eb = sizeof(SlabEnt) * std::max<size_t>(total.entries, 1);
  const bool pooled = eb > (size_t)2 << 20 && eb <= (size_t)64 << 20;
  if ((pooled ? cudaMallocAsync(&ents.p, eb, h->stream) : cudaMalloc(&ents.p, eb)) != cudaSuccess) return no_memory();
  slab_lists_kernel<true><<<grid, 256, 0, h->stream>>>(d_slab, nslab, P.d_win, P.d_p2, (SlabEnt*)ents.p, d_total);
  HM_CUDA_TRY(cudaGetLastError());
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));         // the caller's stream reads the entries next
  P.d_slab = d_slab;
  P.d_ent = (SlabEnt*)ents.p;
  P.nslab = (int32_t)nslab;
  lists.p = ents.p = nullptr;
  return HM_OK;
}

// Builds the slab lists on first use; false: this plan cannot have them (no
// memory left for them, or an entry field too narrow), or not now (st is being
// captured, which forbids allocations), and the caller takes the window lists,
// which every plan has.
int ensure_slabs(hm_handle* h, int trans, cudaStream_t st, bool* usable) {
  MvPlan& P = trans ? h->bwd : h->fwd;
  if (!P.d_slab && !P.no_slab) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();   // the legacy stream beside a capture
    else if (cap != cudaStreamCaptureStatusNone) {
      *usable = false;
      return HM_OK;
    }
    const int s = build_slab_plan(h, P);
    if (s == HM_ERR_OOM || s == HM_ERR_UNSUPPORTED) P.no_slab = true;
    else if (s != HM_OK) return s;
  }
  *usable = P.d_slab != nullptr;
  return HM_OK;
}

int build_mv_descriptors(hm_handle* h, const std::vector<int64_t>& order, int trans) {
  const int eb = elem_bytes(h->storage), deb = dense_elem_bytes(h->storage);
  const int64_t n = h->n;
  MvPlan& P = trans ? h->bwd : h->fwd;
  free_mv_plan(P);
  if (n > (int64_t)UINT32_MAX / 2) return fail(HM_ERR_UNSUPPORTED, "n above 2^31");
  // z slots in pool order (shared by both directions)
  std::vector<uint32_t> zoff(h->leaves.size(), 0);
  int64_t z = 0;
  for (int64_t li : order)
    if (h->leaves[li].type == T_RK) { zoff[li] = (uint32_t)z; z += h->leaves[li].k; }
  if (z > (int64_t)UINT32_MAX) return fail(HM_ERR_UNSUPPORTED, "too many low-rank terms");
  if (!trans) {
    if (h->d_z) cudaFree(h->d_z);
    h->d_z = nullptr;
    h->zlen = z;
    if (z) HM_CUDA_TRY(cudaMalloc(&h->d_z, sizeof(double) * z));
  }
  std::vector<P1Desc> p1;
  p1.reserve(order.size());
  for (int64_t li : order) {
    const Leaf& L = h->leaves[li];
    if (L.type != T_RK || L.k == 0) continue;
    P1Desc D{};
    const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
    if (!trans) { D.off = L.off; D.seg0 = (uint32_t)L.col0; D.len = L.n; D.stride = (uint32_t)npad; }
    else { D.off = L.off + npad * L.k; D.seg0 = (uint32_t)L.row0; D.len = L.m; D.stride = (uint32_t)mpad; }
    D.zoff = zoff[li];
    D.k = (uint16_t)L.k;
    D.cl = (uint32_t)(trans ? L.s : L.t);
    p1.push_back(D);
  }
  const int64_t nwin = (n + MV_WROWS - 1) / MV_WROWS;
  // the windows' descriptors in pool order: count, then place
  std::vector<int64_t> at((size_t)nwin + 1, 0);
  for (const Leaf& L : h->leaves) {
    if (L.type == T_RK && L.k == 0) continue;
    const int64_t o0 = trans ? L.col0 : L.row0, oe = o0 + (trans ? L.n : L.m);
    for (int64_t w = o0 / MV_WROWS; w * MV_WROWS < oe; ++w) ++at[w + 1];
  }
  for (int64_t w = 0; w < nwin; ++w) at[w + 1] += at[w];
  if (at[nwin] > (int64_t)UINT32_MAX) return fail(HM_ERR_UNSUPPORTED, "too many matvec descriptors");
  std::vector<MvWin> wins(nwin);
  for (int64_t w = 0; w < nwin; ++w)
    wins[w] = MvWin{(uint32_t)(w * MV_WROWS), (uint32_t)std::min<int64_t>(MV_WROWS, n - w * MV_WROWS), (uint32_t)at[w],
                    (uint32_t)at[w + 1]};
  std::vector<P2Desc> p2((size_t)at[nwin]);
  for (int64_t li : order) {
    const Leaf& L = h->leaves[li];
    if (L.type == T_RK && L.k == 0) continue;
    const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
    const int64_t o0 = trans ? L.col0 : L.row0;
    const int64_t oe = o0 + (trans ? L.n : L.m);
    P2Desc D{};
    D.m = (uint32_t)(oe - o0);
    if (L.type == T_RK) {
      D.type = P2_RK;
      D.off = trans ? L.off : L.off + npad * L.k;
      D.ld = (uint32_t)(trans ? npad : mpad);
      D.aux = zoff[li];
      D.cnt = (uint32_t)L.k;
    } else {
      const int64_t ldc = col_pad(L.m, deb);
      D.type = trans ? P2_DENSE_T : P2_DENSE;
      D.off = L.off;
      D.ld = (uint32_t)ldc;
      D.aux = (uint32_t)(trans ? L.row0 : L.col0);
      D.cnt = (uint32_t)(trans ? L.m : L.n);
    }
    for (int64_t w = o0 / MV_WROWS; w * MV_WROWS < oe; ++w) {
      P2Desc E = D;
      E.row_off = (int32_t)(o0 - w * MV_WROWS);
      p2[at[w]++] = E;
    }
  }
  P.np1 = (int64_t)p1.size();
  P.np2 = (int64_t)p2.size();
  P.nwin = (int32_t)nwin;
  // one allocation for the three lists: each takes a third of a millisecond, and
  // as long again to free
  const size_t b1 = sizeof(P1Desc) * p1.size(), b2 = sizeof(P2Desc) * p2.size(), bw = sizeof(MvWin) * nwin;
  HM_CUDA_TRY(cudaMalloc(&P.d_desc, b1 + b2 + bw));
  P.desc_bytes = b1 + b2 + bw;
  P.d_p1 = (P1Desc*)P.d_desc;
  P.d_p2 = (P2Desc*)((char*)P.d_desc + b1);
  P.d_win = (MvWin*)((char*)P.d_desc + b1 + b2);
  if (b1) HM_CUDA_TRY(h2d_sync(P.d_p1, p1.data(), b1));
  if (b2) HM_CUDA_TRY(h2d_sync(P.d_p2, p2.data(), b2));
  HM_CUDA_TRY(h2d_sync(P.d_win, wins.data(), bw));
  return HM_OK;
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
static int ensure_xs(hm_handle* h, size_t bytes) {
  if (h->xs_bytes >= bytes) return HM_OK;
  if (h->d_xs) cudaFree(h->d_xs);
  h->d_xs = nullptr;
  h->xs_bytes = 0;
  HM_CUDA_TRY(cudaMalloc(&h->d_xs, bytes));
  h->xs_bytes = bytes;
  return HM_OK;
}

// The window lists split by leaf kind: the dense leaves alone (the passes that
// treat them separately: tensor-core calls, BF16 single-column products) and
// the low-rank leaves alone.
int split_p2(MvPlan& P) {
  if (P.d_wind || P.nwin == 0) return HM_OK;
  std::vector<P2Desc> v((size_t)P.np2);
  std::vector<MvWin> win((size_t)P.nwin);
  if (P.np2 > 0) HM_CUDA_TRY(cudaMemcpy(v.data(), P.d_p2, sizeof(P2Desc) * v.size(), cudaMemcpyDeviceToHost));
  HM_CUDA_TRY(cudaMemcpy(win.data(), P.d_win, sizeof(MvWin) * win.size(), cudaMemcpyDeviceToHost));
  std::vector<P2Desc> dd, rr;
  std::vector<MvWin> wd(win), wr(win);
  for (size_t w = 0; w < win.size(); ++w) {
    wd[w].begin = (uint32_t)dd.size();
    wr[w].begin = (uint32_t)rr.size();
    for (uint32_t i = win[w].begin; i < win[w].end; ++i) (v[i].type == P2_RK ? rr : dd).push_back(v[i]);
    wd[w].end = (uint32_t)dd.size();
    wr[w].end = (uint32_t)rr.size();
  }
  if (dd.empty()) dd.push_back(P2Desc{});        // keeps the pointers valid; no window refers to them
  if (rr.empty()) rr.push_back(P2Desc{});
  HM_CUDA_TRY(cudaMalloc(&P.d_p2r, sizeof(P2Desc) * rr.size()));
  HM_CUDA_TRY(h2d_sync(P.d_p2r, rr.data(), sizeof(P2Desc) * rr.size()));
  HM_CUDA_TRY(cudaMalloc(&P.d_winr, sizeof(MvWin) * wr.size()));
  HM_CUDA_TRY(h2d_sync(P.d_winr, wr.data(), sizeof(MvWin) * wr.size()));
  HM_CUDA_TRY(cudaMalloc(&P.d_p2d, sizeof(P2Desc) * dd.size()));
  HM_CUDA_TRY(h2d_sync(P.d_p2d, dd.data(), sizeof(P2Desc) * dd.size()));
  HM_CUDA_TRY(cudaMalloc(&P.d_wind, sizeof(MvWin) * wd.size()));   // last: marks the split as complete
  HM_CUDA_TRY(h2d_sync(P.d_wind, wd.data(), sizeof(MvWin) * wd.size()));
  return HM_OK;
}

// y = the dense leaves' part of H x (one column): a warp per 32 output rows
// walks its window's dense descriptors; the leaves covering its rows are read
// column by column (32 consecutive rows a load, eight columns in flight).
template <typename TD>
__global__ void __launch_bounds__(256) mv_dense1_kernel(const MvWin* __restrict__ win, const P2Desc* __restrict__ d,
                                                        const TD* __restrict__ dn, const double* __restrict__ x,
                                                        int64_t nslab, double* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw >= nslab) return;
  const int64_t grow = gw * 32;
  const MvWin W = win[grow / MV_WROWS];
  const int r0 = (int)(grow - W.row0), r = r0 + lane;
  double acc = 0.0;
  for (uint32_t i = W.begin; i < W.end; ++i) {
    const P2Desc D = d[i];
    if (D.row_off >= r0 + 32 || D.row_off + (int)D.m <= r0) continue;
    const int lr = r - D.row_off;
    const bool mine = lr >= 0 && lr < (int)D.m;
    const bool tr = D.type == P2_DENSE_T;
    const TD* col = dn + D.off + (mine ? (tr ? (int64_t)lr * D.ld : (int64_t)lr) : 0);
    const int64_t cs = tr ? 1 : (int64_t)D.ld;
    const double* xs = x + D.aux;
    uint32_t c = 0;
    for (; c + 8 <= D.cnt; c += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = mine ? (double)__ldcs(col + (int64_t)(c + u) * cs) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc = fma(v[u], __ldg(xs + c + u), acc);
    }
    for (; c < D.cnt; ++c) acc = fma(mine ? (double)__ldcs(col + (int64_t)c * cs) : 0.0, __ldg(xs + c), acc);
  }
  if (r < (int)W.nrows) y[W.row0 + r] = acc;
}

// BF16 factors: y += the low-rank leaves' part, each lane owning 8
// consecutive output rows (one 16-byte load of 8 BF16 values where the leaf
// starts on an 8-row boundary of the window, two 8-byte loads on a 4-row
// boundary, element loads elsewhere; padding rows hold zeros).  Twice the rows
// of the 4-row kernel per entry: BF16 halves the bytes of an entry, and the
// 4-row form ran out of issue slots before HBM.
template <int SPLIT> struct P2Shape8 {
  static constexpr int CROWS = MV_WROWS / SPLIT;   // rows of one CTA
  static constexpr int WARPS = CROWS / 256;        // 32 lanes x 8 rows a warp
  static constexpr int EMAX = 1024 / SPLIT;
};
template <int SPLIT>
__global__ void __launch_bounds__(P2Shape8<SPLIT>::WARPS * 32) mv_phase2_bf16_kernel(
    const MvWin* __restrict__ win, const P2Desc* __restrict__ d, const __nv_bfloat16* __restrict__ rk,
    const double* __restrict__ z, double* __restrict__ y) {
  constexpr int U = 8;
  constexpr int CROWS = P2Shape8<SPLIT>::CROWS, EMAX = P2Shape8<SPLIT>::EMAX;
  __shared__ P2Desc sd[P2_NB];
  __shared__ int spre[P2_NB + 1];
  __shared__ uint64_t e_off[EMAX];
  __shared__ int32_t e_ro[EMAX];
  __shared__ uint32_t e_m[EMAX];
  __shared__ double e_z[EMAX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MvWin W = win[blockIdx.x / SPLIT];
  const int h0 = (int)(blockIdx.x % SPLIT) * CROWS;
  const int base = h0 + 8 * (warp * 32 + lane);
  const uint16_t* rkb = reinterpret_cast<const uint16_t*>(rk);
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
  for (uint32_t b0 = W.begin; b0 < W.end; b0 += P2_NB) {
    const int nb = (int)min((uint32_t)P2_NB, W.end - b0);
    __syncthreads();
    if (warp == 0) {
      int cnt = 0;
      if (lane < nb) {
        sd[lane] = d[b0 + lane];
        const int r0 = sd[lane].row_off, r1 = r0 + (int)sd[lane].m;
        cnt = (r1 > h0 && r0 < h0 + CROWS) ? (int)sd[lane].cnt : 0;
      }
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      spre[lane + 1] = incl;
      if (lane == 0) spre[0] = 0;
    }
    __syncthreads();
    const int total = spre[nb];
    for (int e0 = 0; e0 < total; e0 += EMAX) {
      const int ne = min(EMAX, total - e0);
      if (e0 > 0) __syncthreads();
      for (int e = threadIdx.x; e < ne; e += blockDim.x) {
        const int ge = e0 + e;
        int lo = 0, hi = nb - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (spre[mid] <= ge) lo = mid; else hi = mid - 1;
        }
        const P2Desc& D = sd[lo];
        const int c = ge - spre[lo];
        e_off[e] = D.off + (uint64_t)c * D.ld;
        e_z[e] = z[D.aux + c];
        e_ro[e] = D.row_off;
        e_m[e] = D.m;
      }
      __syncthreads();
      for (int e = 0; e < ne; e += U) {
        uint4 raw[U];
        double zz[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          raw[u] = make_uint4(0u, 0u, 0u, 0u);
          zz[u] = 0.0;
          const int ee = e + u;
          if (ee < ne) {
            const int ro = e_ro[ee];
            const int mm = (int)e_m[ee];
            const uint64_t o = e_off[ee];
            const int lr = base - ro;
            zz[u] = e_z[ee];
            if ((ro & 7) == 0) {
              if (lr >= 0 && lr < mm) raw[u] = __ldcs(reinterpret_cast<const uint4*>(rk + o + lr));
            } else if ((ro & 3) == 0) {
              if (lr >= 0 && lr < mm) {
                const uint2 a = __ldcs(reinterpret_cast<const uint2*>(rk + o + lr));
                raw[u].x = a.x; raw[u].y = a.y;
              }
              if (lr + 4 >= 0 && lr + 4 < mm) {
                const uint2 b = __ldcs(reinterpret_cast<const uint2*>(rk + o + lr + 4));
                raw[u].z = b.x; raw[u].w = b.y;
              }
            } else {
              uint32_t wv[4] = {0u, 0u, 0u, 0u};
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const int r = lr + q;
                if (r >= 0 && r < mm) wv[q >> 1] |= (uint32_t)rkb[o + (uint64_t)r] << (16 * (q & 1));
              }
              raw[u] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
            }
          }
        }
        // FP32 products and partial sums over the entries in flight, folded
        // into the FP64 row sums once per group
        float part[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) part[q] = 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float zf = (float)zz[u];
          const uint32_t w4[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            part[2 * q] = fmaf(bf_lo(w4[q]), zf, part[2 * q]);
            part[2 * q + 1] = fmaf(bf_hi(w4[q]), zf, part[2 * q + 1]);
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] += (double)part[q];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (base + q < (int)W.nrows) y[W.row0 + base + q] += acc[q];
}

// resident CTAs of phase 1 on the device, asked once per device
template <typename T>
static int64_t p1_wave(int device) {
  static std::atomic<int> known[64];
  std::atomic<int>* slot = device >= 0 && device < 64 ? &known[device] : nullptr;
  if (slot && slot->load(std::memory_order_relaxed) > 0) return slot->load(std::memory_order_relaxed);
  int nsm = 148, per_sm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mv_phase1_kernel<T>, 256, 0) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  if (slot) slot->store(nsm * per_sm, std::memory_order_relaxed);
  return (int64_t)nsm * per_sm;
}

template <typename T>
static int matvec_t(hm_handle* h, const double* d_x, double* d_y, int trans, cudaStream_t st, cudaEvent_t* ev) {
  using TX = typename MvT<T>::X;
  constexpr int XA = 16 / (int)sizeof(TX);
  MvPlan& P = trans ? h->bwd : h->fwd;
  const int64_t stride = pad_to(h->n + 64, 64);
  const TX* xs = nullptr;
  if (ev) HM_CUDA_TRY(cudaEventRecord(ev[0], st));
  if constexpr (std::is_same<T, double>::value) {
    xs = d_x;
  } else {
    HM_TRY(ensure_xs(h, sizeof(TX) * stride * XA));
    int64_t tot = stride * XA;
    unsigned g = (unsigned)std::min<int64_t>((tot + 255) / 256, 148 * 16);
    xcopy_kernel<TX><<<g, 256, 0, st>>>(d_x, h->n, (TX*)h->d_xs, stride, XA);
    xs = (const TX*)h->d_xs;
  }
  if (ev) HM_CUDA_TRY(cudaEventRecord(ev[1], st));
  if (P.np1 > 0) {
    // one wave of resident CTAs: the warps stride over equal-sized leaves and
    // finish together (a grid of several partial waves leaves a tail)
    const int64_t wave = p1_wave<T>(h->device);
    int64_t blocks = std::min<int64_t>((P.np1 + 7) / 8, wave * std::max(1, h->tune.p1_waves));
    mv_phase1_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(P.d_p1, P.np1, (const T*)h->d_rk, xs, stride, h->d_z);
  }
  if (ev) HM_CUDA_TRY(cudaEventRecord(ev[2], st));
  // dense leaves are FP64 with FP64 factors and FP32 otherwise
  using TD = typename std::conditional<std::is_same<T, double>::value, double, float>::type;
  bool slabs = false;
  if (h->tune.p2_split == 1) HM_TRY(ensure_slabs(h, trans, st, &slabs));
  if (slabs) {
    mv_slab_kernel<T, TD><<<(unsigned)P.nslab, SL_WARPS * 32, 0, st>>>(
        P.d_slab, P.d_ent, (const T*)h->d_rk, (const TD*)h->d_dense, h->d_z, d_x, d_y);
  } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    // dense leaves (FP32) first, written into y; then the BF16 low-rank part added
    HM_TRY(split_p2(P));
    const int64_t nslab = (h->n + 31) / 32;
    mv_dense1_kernel<float><<<(unsigned)((nslab + 7) / 8), 256, 0, st>>>(P.d_wind, P.d_p2d,
                                                                         (const float*)h->d_dense, d_x, nslab, d_y);
    if (h->tune.p2_split == 2)
      mv_phase2_bf16_kernel<2><<<(unsigned)(P.nwin * 2), P2Shape8<2>::WARPS * 32, 0, st>>>(
          P.d_winr, P.d_p2r, (const __nv_bfloat16*)h->d_rk, h->d_z, d_y);
    else                                       // splits 4 and 8: one warp a quarter window
      mv_phase2_bf16_kernel<4><<<(unsigned)(P.nwin * 4), P2Shape8<4>::WARPS * 32, 0, st>>>(
          P.d_winr, P.d_p2r, (const __nv_bfloat16*)h->d_rk, h->d_z, d_y);
  } else {
    auto p2 = [&](auto split) {
      constexpr int S = decltype(split)::value;
      mv_phase2_kernel<T, TD, S><<<(unsigned)(P.nwin * S), P2Shape<S>::WARPS * 32, 0, st>>>(
          P.d_win, P.d_p2, (const T*)h->d_rk, (const TD*)h->d_dense, h->d_z, d_x, d_y);
    };
    switch (h->tune.p2_split) {
      case 2: p2(std::integral_constant<int, 2>{}); break;
      case 8: p2(std::integral_constant<int, 8>{}); break;
      default: p2(std::integral_constant<int, 4>{});
    }
  }
  if (ev) HM_CUDA_TRY(cudaEventRecord(ev[3], st));
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

int matvec_device(hm_handle* h, const double* d_x, double* d_y, int trans, cudaStream_t st, cudaEvent_t* ev) {
  switch (h->storage) {
    case HM_F64: return matvec_t<double>(h, d_x, d_y, trans, st, ev);
    case HM_F32: return matvec_t<float>(h, d_x, d_y, trans, st, ev);
    default: return matvec_t<__nv_bfloat16>(h, d_x, d_y, trans, st, ev);
  }
}

// ---------------------------------------------------------------------------
// residual r = b - H x with compensated (double-double) sums, for iterative
// refinement: every product is split exactly (TwoProduct by FMA) and every
// sum carries its rounding error (TwoSum), the dot product and sum algorithms
// of Ogita, Rump & Oishi (2005), "Accurate sum and dot product".  The result
// is as accurate as if H x were summed in twice the FP64 precision, so the
// refinement is not stopped by the rounding of H x near b.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void dd_add_prod(double& p, double& c, double a, double b) {
  const double h = a * b;
  const double r = fma(a, b, -h);          // a b = h + r exactly
  double q;
  two_sum(p, h, p, q);
  c += q + r;
}

// z = F1' x per low-rank leaf and rank, as hi + lo; one warp per leaf
template <typename T>
__global__ void __launch_bounds__(256) mvdd_phase1_kernel(const P1Desc* __restrict__ d, int64_t nd,
                                                          const T* __restrict__ pool, const double* __restrict__ x,
                                                          double* __restrict__ zh, double* __restrict__ zl) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = gw; b < nd; b += nw) {
    const P1Desc D = d[b];
    for (int r = 0; r < D.k; ++r) {
      const T* f = pool + D.off + (int64_t)r * D.stride;
      double p = 0.0, c = 0.0;
      for (uint32_t j = lane; j < D.len; j += 32) dd_add_prod(p, c, from_store<T>(f[j]), x[D.seg0 + j]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double p2 = __shfl_xor_sync(0xffffffffu, p, o), c2 = __shfl_xor_sync(0xffffffffu, c, o);
        double q;
        two_sum(p, p2, p, q);
        c += c2 + q;
      }
      if (lane == 0) {
        const double hi = p + c;
        zh[D.zoff + r] = hi;
        zl[D.zoff + r] = c - (hi - p);
      }
    }
  }
}

// r = b - (sum over the window's leaves) per output row.  A CTA owns 32 rows
// (lane = row) and its 8 warps split the window's descriptors, every eighth
// one each, so the dense near-field leaves, neighbours in the list, spread over
// the warps; the warps' double-double sums are added in shared memory in warp
// order.  The sums are chains of dependent FP64 operations: one thread a row
// walking every descriptor kept an SM at two warps and took 380 us at
// n = 20000.
constexpr int MVDD_WARPS = 8;
constexpr int MVDD_SPLIT = MV_WROWS / 32;
template <typename T, typename TD>
__global__ void __launch_bounds__(MVDD_WARPS * 32) mvdd_phase2_kernel(const MvWin* __restrict__ win,
                                                                const P2Desc* __restrict__ d, const T* __restrict__ rk,
                                                                const TD* __restrict__ dn, const double* __restrict__ zh,
                                                                const double* __restrict__ zl,
                                                                const double* __restrict__ x,
                                                                const double* __restrict__ bvec, double* __restrict__ rvec) {
  __shared__ double sp[MVDD_WARPS][32], sc[MVDD_WARPS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MvWin W = win[blockIdx.x / MVDD_SPLIT];
  const int r0 = (int)(blockIdx.x % MVDD_SPLIT) * 32;             // this CTA's rows [r0, r0 + 32)
  if (r0 >= (int)W.nrows) return;
  double p = 0.0, c = 0.0;
  for (uint32_t b0 = W.begin; b0 < W.end; b0 += 32 * MVDD_WARPS) {
    const uint32_t b = b0 + lane * MVDD_WARPS + warp;
    P2Desc D{};
    bool cov = false;
    if (b < W.end) {
      D = d[b];
      cov = D.row_off < r0 + 32 && D.row_off + (int)D.m > r0;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, cov); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const uint64_t off = __shfl_sync(0xffffffffu, (unsigned long long)D.off, src);
      const int lr = r0 + lane - __shfl_sync(0xffffffffu, D.row_off, src);
      const int m = (int)__shfl_sync(0xffffffffu, D.m, src);
      const uint32_t ld = __shfl_sync(0xffffffffu, D.ld, src), aux = __shfl_sync(0xffffffffu, D.aux, src);
      const uint32_t cnt = __shfl_sync(0xffffffffu, D.cnt, src);
      const uint32_t type = __shfl_sync(0xffffffffu, (uint32_t)D.type, src);
      const bool mine = lr >= 0 && lr < m;
      if (type == P2_RK) {
        const T* f = rk + off + (mine ? lr : 0);
        for (uint32_t q = 0; q < cnt; q += 4) {
          double v[4], h[4], l[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = q + u < cnt;
            v[u] = in && mine ? from_store<T>(f[(uint64_t)(q + u) * ld]) : 0.0;
            h[u] = in ? __ldg(zh + aux + q + u) : 0.0;
            l[u] = in ? __ldg(zl + aux + q + u) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (mine && q + u < cnt) {
              dd_add_prod(p, c, v[u], h[u]);
              c = fma(v[u], l[u], c);
            }
        }
      } else {
        // dense: column by column, or along the rows of the leaf (H'x)
        const bool tr = type == P2_DENSE_T;
        const TD* f = dn + off + (mine ? (tr ? (uint64_t)lr * ld : (uint64_t)lr) : 0);
        const uint64_t cs = tr ? 1 : ld;
        for (uint32_t q = 0; q < cnt; q += 8) {
          double v[8], h[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const bool in = q + u < cnt;
            v[u] = in && mine ? (double)f[(q + u) * cs] : 0.0;
            h[u] = in ? __ldg(x + aux + q + u) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (mine && q + u < cnt) dd_add_prod(p, c, v[u], h[u]);
        }
      }
    }
  }
  sp[warp][lane] = p;
  sc[warp][lane] = c;
  __syncthreads();
  if (warp == 0 && r0 + lane < (int)W.nrows) {
    double ps = sp[0][lane], cs = sc[0][lane];
#pragma unroll
    for (int w = 1; w < MVDD_WARPS; ++w) {
      double q;
      two_sum(ps, sp[w][lane], ps, q);
      cs += q + sc[w][lane];
    }
    const uint32_t i = W.row0 + (uint32_t)(r0 + lane);
    double t, q;
    two_sum(bvec[i], -ps, t, q);
    rvec[i] = t + (q - cs);
  }
}

template <typename T>
static int residual_t(hm_handle* h, const double* d_x, const double* d_b, double* d_r, int trans, cudaStream_t st) {
  using TD = typename std::conditional<std::is_same<T, double>::value, double, float>::type;
  const MvPlan& P = trans ? h->bwd : h->fwd;
  const size_t need = sizeof(double) * 2 * (size_t)std::max<int64_t>(h->zlen, 1);
  if (h->dd_bytes < need) {
    if (h->d_dd) cudaFree(h->d_dd);
    h->d_dd = nullptr;
    h->dd_bytes = 0;
    cudaError_t e = cudaMalloc(&h->d_dd, need);
    if (e != cudaSuccess) return fail(HM_ERR_OOM, std::string("residual buffers: ") + cudaGetErrorString(e));
    h->dd_bytes = need;
  }
  double* zh = (double*)h->d_dd;
  double* zl = zh + std::max<int64_t>(h->zlen, 1);
  if (P.np1 > 0) {
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
    const int64_t blocks = std::min<int64_t>((P.np1 + 7) / 8, (int64_t)nsm * 8);
    mvdd_phase1_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(P.d_p1, P.np1, (const T*)h->d_rk, d_x, zh, zl);
  }
  mvdd_phase2_kernel<T, TD><<<(unsigned)(P.nwin * MVDD_SPLIT), MVDD_WARPS * 32, 0, st>>>(
      P.d_win, P.d_p2, (const T*)h->d_rk, (const TD*)h->d_dense, zh, zl, d_x, d_b, d_r);
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

int residual_device(hm_handle* h, const double* d_x, const double* d_b, double* d_r, int trans, cudaStream_t st) {
  switch (h->storage) {
    case HM_F64: return residual_t<double>(h, d_x, d_b, d_r, trans, st);
    case HM_F32: return residual_t<float>(h, d_x, d_b, d_r, trans, st);
    default: return residual_t<__nv_bfloat16>(h, d_x, d_b, d_r, trans, st);
  }
}

// ---------------------------------------------------------------------------
// exact FP64 rows (K14): y_i = sum_j K(x_rows[i], x_j) x_j + shift * x_rows[i]
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512) exact_rows_kernel(KernelDesc kd, const double* __restrict__ geom, int64_t n,
                                                         const int64_t* __restrict__ rows,
                                                         const double* __restrict__ x, double* __restrict__ y) {
  __shared__ double red[32];
  const int64_t i = rows[blockIdx.x];
  double s = 0.0;
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x) s = fma(kernel_eval(kd, geom, n, i, j), x[j], s);
  s = block_sum(s, red);
  if (threadIdx.x == 0) y[blockIdx.x] = s + kd.shift * x[i];
}

int exact_rows_device(hm_handle* h, const int64_t* d_rows, int64_t nrows, const double* d_x, double* d_y,
                      cudaStream_t st) {
  if (nrows <= 0) return HM_OK;
  for (int64_t b0 = 0; b0 < nrows; b0 += (1ll << 30)) {
    unsigned nb = (unsigned)std::min<int64_t>(nrows - b0, 1ll << 30);
    exact_rows_kernel<<<nb, 512, 0, st>>>(h->kd, h->d_geom, h->n, d_rows + b0, d_x, d_y + b0);
  }
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

// ---------------------------------------------------------------------------
// densify (to_fmat, src/utils.jl:162-192), leaf factors, shift, scale, copy
// ---------------------------------------------------------------------------
struct LeafDev {
  int64_t row0, col0, off;
  int32_t m, n, k, type;
};

template <typename T, typename TD>
__global__ void to_dense_kernel(const LeafDev* __restrict__ L, const T* __restrict__ rk, const TD* __restrict__ dn,
                                int64_t n, double* __restrict__ out) {
  const LeafDev D = L[blockIdx.x];
  const int eb = (int)sizeof(T), deb = (int)sizeof(TD);
  const int64_t tot = (int64_t)D.m * D.n;
  for (int64_t e = threadIdx.x; e < tot; e += blockDim.x) {
    const int i = (int)(e % D.m), j = (int)(e / D.m);
    double v;
    if (D.type == T_DENSE) {
      v = (double)dn[D.off + i + (int64_t)j * col_pad_dev(D.m, deb)];
    } else {
      const int64_t npad = col_pad_dev(D.n, eb), mpad = col_pad_dev(D.m, eb);
      const T* B = rk + D.off;
      const T* A = B + npad * D.k;
      v = 0.0;
      for (int q = 0; q < D.k; ++q) v = fma(from_store<T>(A[i + q * mpad]), from_store<T>(B[j + q * npad]), v);
    }
    out[(D.row0 + i) + (D.col0 + j) * n] = v;
  }
}

int to_dense(const hm_handle* h, double* d_out) {
  std::vector<LeafDev> L(h->leaves.size());
  for (size_t i = 0; i < L.size(); ++i) {
    const Leaf& x = h->leaves[i];
    L[i] = LeafDev{x.row0, x.col0, x.off, x.m, x.n, x.k, x.type};
  }
  if (L.empty()) return HM_OK;
  LeafDev* dL = nullptr;
  HM_CUDA_TRY(cudaMalloc(&dL, sizeof(LeafDev) * L.size()));
  HM_CUDA_TRY(cudaMemcpyAsync(dL, L.data(), sizeof(LeafDev) * L.size(), cudaMemcpyHostToDevice, h->stream));
  const unsigned nb = (unsigned)L.size();
  switch (h->storage) {
    case HM_F64:
      to_dense_kernel<double, double><<<nb, 256, 0, h->stream>>>(dL, (const double*)h->d_rk, (const double*)h->d_dense, h->n, d_out);
      break;
    case HM_F32:
      to_dense_kernel<float, float><<<nb, 256, 0, h->stream>>>(dL, (const float*)h->d_rk, (const float*)h->d_dense, h->n, d_out);
      break;
    default:
      to_dense_kernel<__nv_bfloat16, float><<<nb, 256, 0, h->stream>>>(dL, (const __nv_bfloat16*)h->d_rk, (const float*)h->d_dense, h->n, d_out);
  }
  HM_CUDA_TRY(cudaGetLastError());
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  cudaFree(dL);
  return HM_OK;
}

static inline double bf16_bits_to_double(uint16_t b) {
  uint32_t w = (uint32_t)b << 16;
  float f;
  std::memcpy(&f, &w, 4);
  return (double)f;
}

int leaf_factors_f64(const hm_handle* h, int64_t leaf, double* A, double* B) {
  const Leaf& L = h->leaves[leaf];
  if (L.type != T_RK) return fail(HM_ERR_ARG, "leaf is not low-rank");
  const int eb = elem_bytes(h->storage);
  const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
  const int64_t tot = (npad + mpad) * L.k;
  std::vector<char> buf(tot * eb);
  if (tot) HM_CUDA_TRY(cudaMemcpy(buf.data(), (const char*)h->d_rk + L.off * eb, tot * eb, cudaMemcpyDeviceToHost));
  auto get = [&](int64_t e) -> double {
    if (eb == 8) return ((const double*)buf.data())[e];
    if (eb == 4) return (double)((const float*)buf.data())[e];
    return bf16_bits_to_double(((const uint16_t*)buf.data())[e]);
  };
  for (int q = 0; q < L.k; ++q) {
    for (int j = 0; j < L.n; ++j) B[j + (int64_t)q * L.n] = get(j + q * npad);
    for (int i = 0; i < L.m; ++i) A[i + (int64_t)q * L.m] = get(npad * L.k + i + q * mpad);
  }
  return HM_OK;
}

template <typename TD>
__global__ void shift_kernel(const int64_t* __restrict__ offs, const int32_t* __restrict__ ms, int nleaf,
                             const int32_t* __restrict__ lds, TD* dn, double lam) {
  const int b = blockIdx.x;
  for (int i = threadIdx.x; i < ms[b]; i += blockDim.x) {
    TD* p = dn + offs[b] + i + (int64_t)i * lds[b];
    *p = (TD)((double)*p + lam);
  }
}

int apply_shift(hm_handle* h, double lam) {
  std::vector<int64_t> offs;
  std::vector<int32_t> ms, lds;
  const int deb = dense_elem_bytes(h->storage);
  for (auto& L : h->leaves)
    if (L.type == T_DENSE && L.row0 == L.col0 && L.m == L.n) {
      offs.push_back(L.off);
      ms.push_back(L.m);
      lds.push_back((int32_t)col_pad(L.m, deb));
    }
  if (!offs.empty()) {
    int64_t* d_o = nullptr;
    int32_t *d_m = nullptr, *d_l = nullptr;
    HM_CUDA_TRY(cudaMalloc(&d_o, 8 * offs.size()));
    HM_CUDA_TRY(cudaMalloc(&d_m, 4 * ms.size()));
    HM_CUDA_TRY(cudaMalloc(&d_l, 4 * lds.size()));
    HM_CUDA_TRY(h2d_sync(d_o, offs.data(), 8 * offs.size()));
    HM_CUDA_TRY(h2d_sync(d_m, ms.data(), 4 * ms.size()));
    HM_CUDA_TRY(h2d_sync(d_l, lds.data(), 4 * lds.size()));
    if (h->storage == HM_F64)
      shift_kernel<double><<<(unsigned)offs.size(), 128, 0, h->stream>>>(d_o, d_m, (int)offs.size(), d_l, (double*)h->d_dense, lam);
    else
      shift_kernel<float><<<(unsigned)offs.size(), 128, 0, h->stream>>>(d_o, d_m, (int)offs.size(), d_l, (float*)h->d_dense, lam);
    HM_CUDA_TRY(cudaGetLastError());
    HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    cudaFree(d_o); cudaFree(d_m); cudaFree(d_l);
  }
  h->kd.shift += lam;
  return HM_OK;
}

template <typename T>
__global__ void scale_kernel(T* p, int64_t cnt, double u) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x)
    p[e] = to_store<T>(from_store<T>(p[e]) * u);
}

int apply_scale(hm_handle* h, double u) {
  const int eb = elem_bytes(h->storage), deb = dense_elem_bytes(h->storage);
  // dense pool: every element (padding is zero and stays zero)
  if (h->dense_bytes) {
    if (h->storage == HM_F64) scale_kernel<double><<<592, 256, 0, h->stream>>>((double*)h->d_dense, h->dense_bytes / deb, u);
    else scale_kernel<float><<<592, 256, 0, h->stream>>>((float*)h->d_dense, h->dense_bytes / deb, u);
  }
  // low-rank leaves: the A factor only, as u*H scales H.A (src/harithm.jl:487)
  for (auto& L : h->leaves) {
    if (L.type != T_RK || L.k == 0) continue;
    const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
    const int64_t o = L.off + npad * L.k, cnt = mpad * L.k;
    unsigned g = (unsigned)std::min<int64_t>((cnt + 255) / 256, 64);
    if (h->storage == HM_F64) scale_kernel<double><<<g, 256, 0, h->stream>>>((double*)h->d_rk + o, cnt, u);
    else if (h->storage == HM_F32) scale_kernel<float><<<g, 256, 0, h->stream>>>((float*)h->d_rk + o, cnt, u);
    else scale_kernel<__nv_bfloat16><<<g, 256, 0, h->stream>>>((__nv_bfloat16*)h->d_rk + o, cnt, u);
  }
  HM_CUDA_TRY(cudaGetLastError());
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  h->kd.shift *= u;
  return HM_OK;
}

static int dup(void** dst, const void* src, size_t bytes) {
  *dst = nullptr;
  if (!bytes || !src) return HM_OK;
  cudaError_t e = cudaMalloc(dst, bytes);
  if (e != cudaSuccess) return fail(HM_ERR_OOM, std::string("copy: ") + cudaGetErrorString(e));
  HM_CUDA_TRY(cudaMemcpy(*dst, src, bytes, cudaMemcpyDeviceToDevice));
  return HM_OK;
}

int copy_handle(const hm_handle* h, hm_handle** out) {
  hm_handle* c = new hm_handle();
  c->prm = h->prm; c->n = h->n; c->dim = h->dim; c->device = h->device; c->kd = h->kd;
  c->cl_s = h->cl_s; c->cl_e = h->cl_e; c->cl_left = h->cl_left; c->cl_right = h->cl_right;
  c->cl_depth = h->cl_depth; c->nodes = h->nodes; c->leaves = h->leaves; c->depth = h->depth;
  c->storage = h->storage; c->kmax = h->kmax; c->rk_bytes = h->rk_bytes; c->dense_bytes = h->dense_bytes;
  c->zlen = h->zlen;
  c->tune = h->tune;                           // the same launch shapes: the same sums in the same order
  // h's pending work lands before the copies read it (they run on the legacy
  // stream, which the handles' non-blocking streams do not order with)
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) { delete c; return fail(HM_ERR_CUDA, cudaGetErrorString(e)); }
  e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) { delete c; return fail(HM_ERR_CUDA, cudaGetErrorString(e)); }
  int s = HM_OK;
  auto chk = [&](int st) { if (s == HM_OK) s = st; };
  chk(dup((void**)&c->d_geom, h->d_geom, sizeof(double) * h->n * h->dim));
  chk(dup(&c->d_rk, h->d_rk, h->rk_bytes));
  chk(dup(&c->d_dense, h->d_dense, h->dense_bytes));
  chk(dup((void**)&c->d_z, h->d_z, sizeof(double) * h->zlen));
  chk(dup((void**)&c->d_piv, h->d_piv, sizeof(int32_t) * h->piv_count));
  c->piv_count = h->d_piv ? h->piv_count : 0;
  for (int t = 0; t < 2 && s == HM_OK; ++t) {
    const MvPlan& a = t ? h->bwd : h->fwd;
    MvPlan& b = t ? c->bwd : c->fwd;
    b.np1 = a.np1; b.np2 = a.np2; b.nwin = a.nwin;
    chk(dup(&b.d_desc, a.d_desc, a.desc_bytes));
    if (s == HM_OK && b.d_desc) {
      b.desc_bytes = a.desc_bytes;
      b.d_p1 = (P1Desc*)b.d_desc;
      b.d_p2 = (P2Desc*)((char*)b.d_desc + sizeof(P1Desc) * a.np1);
      b.d_win = (MvWin*)((char*)b.d_desc + sizeof(P1Desc) * a.np1 + sizeof(P2Desc) * a.np2);
    }
  }
  if (s == HM_OK && h->lu) s = lu_copy(h, c);
  c->factorized = h->factorized;
  // and the copies land before c's kernels read them
  if (s == HM_OK && cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) s = fail(HM_ERR_CUDA, "copy");
  if (s != HM_OK) {
    free_handle_data(c);
    cudaStreamDestroy(c->stream);
    delete c;
    return s;
  }
  *out = c;
  return HM_OK;
}

}  // namespace hm
