// H-LU and triangular H-solve on the device (src/hlu.jl:227-562, with the
// H-arithmetic of src/harithm.jl:4-420 that the Schur updates use).
//
// The host walks the same recursion as the reference -- lu!, permute_hmat!,
// hmat_trisolve!, mat_full_solve, hmat_sub_mul! = hmul + hmat_add!, and the
// recompressions of rkmat_add!, rkmat_hmat_add and compress -- and issues one
// stream-ordered kernel per primitive.  Nothing is read back during the
// factorisation: ranks live on the device, every low-rank buffer has a fixed
// capacity `cap` and keeps its columns beyond the current rank at zero, so
// every product can run with static shapes.  Temporaries are stream-ordered
// allocations (cudaMallocAsync / cudaFreeAsync).  Pivoting is partial and
// stays inside each diagonal leaf, exactly as in the reference; the global
// permutation is one device array P with H[P,:] = L U.
#include "hm_internal.h"
#include "hm_lowrank.cuh"
#include "hm_core.cuh"
#include "hm_lu_tile.cuh"
#include "hm_lu_pair.cuh"


#include <algorithm>
#include <map>
#include <memory>
#include <stdexcept>

namespace hm {

// ---------------------------------------------------------------------------
// strided views: element (i,j) at p[i*rs + j*cs]
// ---------------------------------------------------------------------------
struct View {
  double* p;
  int64_t rs, cs;
  int rows, cols;
};
static inline View vsub(View v, int r0, int c0, int nr, int nc) {
  return View{v.p + (int64_t)r0 * v.rs + (int64_t)c0 * v.cs, v.rs, v.cs, nr, nc};
}
static inline View vtr(View v) { return View{v.p, v.cs, v.rs, v.cols, v.rows}; }
static inline View vrev(View v) {
  return View{v.p + (int64_t)(v.rows - 1) * v.rs + (int64_t)(v.cols - 1) * v.cs, -v.rs, -v.cs, v.rows, v.cols};
}

struct LuError : std::runtime_error {
  int code;
  LuError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define HM_LU_CUDA(expr)                                                                    \
  do {                                                                                      \
    cudaError_t _e = (expr);                                                                \
    if (_e != cudaSuccess) throw LuError(HM_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)
#define LU_LAUNCH_CHECK()                                                                   \
  do {                                                                                      \
    cudaError_t _e = cudaGetLastError();                                                    \
    if (_e != cudaSuccess) throw LuError(HM_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(_e)); \
  } while (0)

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
// C = alpha * A * B + beta * C   (A: m x k, B: k x n), FP64, 32x32 tiles
__device__ __forceinline__ void gemm_tile(const View& A, const View& B, const View& C, double alpha, double beta,
                                          int i0, int j0) {
  __shared__ double As[32][33];
  __shared__ double Bs[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int m = C.rows, n = C.cols, kk = A.cols;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k0 = 0; k0 < kk; k0 += 32) {
    for (int e = threadIdx.x; e < 1024; e += 256) {
      const int r = e & 31, c = e >> 5;
      As[r][c] = (i0 + r < m && k0 + c < kk) ? A.p[(int64_t)(i0 + r) * A.rs + (int64_t)(k0 + c) * A.cs] : 0.0;
      Bs[r][c] = (k0 + r < kk && j0 + c < n) ? B.p[(int64_t)(k0 + r) * B.rs + (int64_t)(j0 + c) * B.cs] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q) {
      const double a = As[tx][q];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = fma(a, Bs[q][ty + 8 * u], acc[u]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = i0 + tx, j = j0 + ty + 8 * u;
    if (i < m && j < n) {
      double* c = C.p + (int64_t)i * C.rs + (int64_t)j * C.cs;
      *c = (beta == 0.0) ? alpha * acc[u] : fma(alpha, acc[u], beta * *c);
    }
  }
}

__global__ void __launch_bounds__(256) lu_gemm_kernel(View A, View B, View C, double alpha, double beta) {
  gemm_tile(A, B, C, alpha, beta, blockIdx.y * 32, blockIdx.x * 32);
}

// a batch of independent products, one job per blockIdx.z
struct GemmJob {
  View A, B, C;
  double alpha, beta;
};
__global__ void __launch_bounds__(256) lu_gemm_batch_kernel(const GemmJob* __restrict__ jobs) {
  const GemmJob& J = jobs[blockIdx.z];
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
  if (i0 >= J.C.rows || j0 >= J.C.cols) return;
  gemm_tile(J.A, J.B, J.C, J.alpha, J.beta, i0, j0);
}

// Large products (the tile schedule's B_ik' A_kj cores and Q_i = A_ik W): C
// tiles of 128 x 128 per CTA, K in steps of 16 through shared memory, 8 x 8
// outputs per thread (rows tx + 16 u, columns 8 ty + v, so that a warp's
// stores of column-major C are 128-byte runs).  Tiles are read along whichever
// stride of the view is 1, so transposed views stay coalesced.
constexpr int GB_T = 128, GB_K = 16, GB_LD = GB_T + 4;
__device__ __forceinline__ void gemm_big_tile(const View& A, const View& B, const View& C, double alpha,
                                              double beta, int i0, int j0) {
  __shared__ __align__(16) double As[GB_K][GB_LD];
  __shared__ __align__(16) double Bs[GB_K][GB_LD];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m = C.rows, n = C.cols, K = A.cols;
  double acc[8][8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[u][v] = 0.0;
  // the next K step's tiles are loaded into registers while this one is
  // multiplied, so the global loads overlap the FMAs
  double ra[8], rb[8];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = tid + 256 * q;
      int i, kk;
      if (A.rs == 1) { i = e & 127; kk = e >> 7; } else { kk = e & 15; i = e >> 4; }
      ra[q] = (i0 + i < m && k0 + kk < K) ? A.p[(int64_t)(i0 + i) * A.rs + (int64_t)(k0 + kk) * A.cs] : 0.0;
      int j;
      if (B.rs == 1) { kk = e & 15; j = e >> 4; } else { j = e & 127; kk = e >> 7; }
      rb[q] = (k0 + kk < K && j0 + j < n) ? B.p[(int64_t)(k0 + kk) * B.rs + (int64_t)(j0 + j) * B.cs] : 0.0;
    }
  };
  auto stash = [&]() {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = tid + 256 * q;
      int i, kk;
      if (A.rs == 1) { i = e & 127; kk = e >> 7; } else { kk = e & 15; i = e >> 4; }
      As[kk][i] = ra[q];
      int j;
      if (B.rs == 1) { kk = e & 15; j = e >> 4; } else { j = e & 127; kk = e >> 7; }
      Bs[kk][j] = rb[q];
    }
  };
  load(0);
  for (int k0 = 0; k0 < K; k0 += GB_K) {
    stash();
    __syncthreads();
    if (k0 + GB_K < K) load(k0 + GB_K);
#pragma unroll 4
    for (int kk = 0; kk < GB_K; ++kk) {
      double a[8], b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) a[u] = As[kk][tx + 16 * u];
#pragma unroll
      for (int v = 0; v < 8; v += 2) {
        const double2 t = *reinterpret_cast<const double2*>(&Bs[kk][8 * ty + v]);
        b[v] = t.x;
        b[v + 1] = t.y;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int j = j0 + 8 * ty + v;
    if (j >= n) continue;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + tx + 16 * u;
      if (i < m) {
        double* c = C.p + (int64_t)i * C.rs + (int64_t)j * C.cs;
        *c = (beta == 0.0) ? alpha * acc[u][v] : fma(alpha, acc[u][v], beta * *c);
      }
    }
  }
}
__global__ void __launch_bounds__(256) lu_gemm_big_kernel(View A, View B, View C, double alpha, double beta) {
  gemm_big_tile(A, B, C, alpha, beta, blockIdx.y * GB_T, blockIdx.x * GB_T);
}
// Y = alpha * X + beta * Y (beta == 0: Y is not read)
__global__ void lu_axpby_kernel(View Y, View X, double alpha, double beta) {
  const int64_t tot = (int64_t)Y.rows * Y.cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % Y.rows), j = (int)(e / Y.rows);
    double* y = Y.p + (int64_t)i * Y.rs + (int64_t)j * Y.cs;
    const double x = X.p ? X.p[(int64_t)i * X.rs + (int64_t)j * X.cs] : 0.0;
    *y = (beta == 0.0) ? alpha * x : fma(alpha, x, beta * *y);
  }
}

// X <- L^{-1} X, L lower triangular (strided: upper/transposed/reversed
// triangles are views of this one) of at most MM rows (diagonal leaves): one warp
// per 32 columns of X, each column held in registers, loops fully unrolled.
template <int MM>
__global__ void __launch_bounds__(32) lu_trsm_small_kernel(View L, View X, int unit) {
  __shared__ double Ls[MM * MM];
  const int m = L.rows;
  for (int e = threadIdx.x; e < m * m; e += 32) {
    const int i = e % m, j = e / m;
    Ls[i + j * MM] = (j <= i) ? L.p[(int64_t)i * L.rs + (int64_t)j * L.cs] : 0.0;
  }
  __syncwarp();
  const int j = blockIdx.x * 32 + threadIdx.x;
  if (j >= X.cols) return;
  double* xp = X.p + (int64_t)j * X.cs;
  double x[MM];
#pragma unroll
  for (int i = 0; i < MM; ++i) x[i] = (i < m) ? xp[(int64_t)i * X.rs] : 0.0;
#pragma unroll
  for (int i = 0; i < MM; ++i) {
    if (i < m) {
      double s = x[i];
#pragma unroll
      for (int l = 0; l < i; ++l) s = fma(-Ls[i + l * MM], x[l], s);
      if (!unit) s = s / Ls[i + i * MM];
      x[i] = s;
    }
  }
#pragma unroll
  for (int i = 0; i < MM; ++i)
    if (i < m) xp[(int64_t)i * X.rs] = x[i];
}

// getrf of a leaf of at most 64 rows by one warp (same pivoting and
// arithmetic as lu_getrf_kernel; padded shared tile, warp barriers only)
__global__ void __launch_bounds__(32) lu_getrf_small_kernel(View C, int64_t* __restrict__ P, int64_t goff,
                                                            int* __restrict__ flags) {
  constexpr int LD = 65;
  __shared__ double S[64 * LD];
  __shared__ int perm[64];
  const int m = C.rows, lane = threadIdx.x;
  for (int e = lane; e < m * m; e += 32) {
    const int i = e % m, j = e / m;
    S[i + j * LD] = C.p[(int64_t)i * C.rs + (int64_t)j * C.cs];
  }
  for (int i = lane; i < m; i += 32) perm[i] = i;
  __syncwarp();
  for (int j = 0; j < m; ++j) {
    double best = -1.0, bv = 0.0;
    int64_t bi = INT64_MAX;
    for (int i = j + lane; i < m; i += 32) {
      const double a = fabs(S[i + j * LD]);
      if (a > best) { best = a; bi = i; bv = S[i + j * LD]; }
    }
    warp_argmax(best, bi, bv);
    if (lane == 0 && !(bv != 0.0)) atomicOr(flags, bi == INT64_MAX ? 6 : 4);
    // every candidate NaN: no maximum was found; keep the row (flagged above)
    const int p = bi == INT64_MAX ? j : (int)bi;
    if (p != j) {
      for (int c = lane; c < m; c += 32) {
        const double t = S[j + c * LD];
        S[j + c * LD] = S[p + c * LD];
        S[p + c * LD] = t;
      }
      if (lane == 0) { const int t = perm[j]; perm[j] = perm[p]; perm[p] = t; }
    }
    __syncwarp();
    const double piv = S[j + j * LD];
    if (piv != 0.0)
      for (int i = j + 1 + lane; i < m; i += 32) S[i + j * LD] /= piv;
    __syncwarp();
    for (int c = j + 1 + lane; c < m; c += 32) {
      const double ujc = S[j + c * LD];
      for (int i = j + 1; i < m; ++i) S[i + c * LD] = fma(-S[i + j * LD], ujc, S[i + c * LD]);
    }
    __syncwarp();
  }
  for (int e = lane; e < m * m; e += 32) {
    const int i = e % m, j = e / m;
    C.p[(int64_t)i * C.rs + (int64_t)j * C.cs] = S[i + j * LD];
  }
  for (int i = lane; i < m; i += 32) P[goff + i] = goff + perm[i];
}

// getrf with partial pivoting of an m x m dense leaf (LAPACK semantics: first
// maximum as pivot, full-row swaps); P[goff+i] = goff + p[i] with C[p] = L U.
__global__ void __launch_bounds__(256) lu_getrf_kernel(View C, int64_t* __restrict__ P, int64_t goff,
                                                       int* __restrict__ flags) {
  extern __shared__ double S[];
  const int m = C.rows;
  int* perm = reinterpret_cast<int*>(S + (int64_t)m * m);
  __shared__ int s_piv;
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
    const int i = e % m, j = e / m;
    S[e] = C.p[(int64_t)i * C.rs + (int64_t)j * C.cs];
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) perm[i] = i;
  __syncthreads();
  for (int j = 0; j < m; ++j) {
    if (threadIdx.x < 32) {
      double best = -1.0, bv = 0.0;
      int64_t bi = INT64_MAX;
      for (int i = j + threadIdx.x; i < m; i += 32) {
        const double a = fabs(S[i + j * m]);
        if (a > best) { best = a; bi = i; bv = S[i + j * m]; }
      }
      warp_argmax(best, bi, bv);
      if (threadIdx.x == 0) {
        // every candidate NaN: no maximum was found; keep the row
        s_piv = bi == INT64_MAX ? j : (int)bi;
        if (!(bv != 0.0)) atomicOr(flags, bi == INT64_MAX ? 6 : 4);   // exactly zero (or NaN) pivot
      }
    }
    __syncthreads();
    const int p = s_piv;
    if (p != j) {
      for (int c = threadIdx.x; c < m; c += blockDim.x) {
        const double t = S[j + c * m];
        S[j + c * m] = S[p + c * m];
        S[p + c * m] = t;
      }
      if (threadIdx.x == 0) { const int t = perm[j]; perm[j] = perm[p]; perm[p] = t; }
    }
    __syncthreads();
    const double piv = S[j + j * m];
    if (piv != 0.0) {
      for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) S[i + j * m] /= piv;
    }
    __syncthreads();
    const int rem = m - j - 1;
    for (int e = threadIdx.x; e < rem * rem; e += blockDim.x) {
      const int i = j + 1 + e % rem, c = j + 1 + e / rem;
      S[i + c * m] = fma(-S[i + j * m], S[j + c * m], S[i + c * m]);
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
    const int i = e % m, j = e / m;
    C.p[(int64_t)i * C.rs + (int64_t)j * C.cs] = S[e];
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) P[goff + i] = goff + perm[i];
}

// X <- X[p, :] with p[i] = P[goff+i] - goff, columns in chunks through smem
__global__ void lu_laswp_kernel(View X, const int64_t* __restrict__ P, int64_t goff, int chunk) {
  extern __shared__ double T[];
  const int m = X.rows;
  const int c0 = blockIdx.x * chunk;
  const int nc = min(chunk, X.cols - c0);
  for (int e = threadIdx.x; e < m * nc; e += blockDim.x) {
    const int i = e % m, c = e / m;
    const int64_t src = P[goff + i] - goff;
    T[e] = X.p[src * X.rs + (int64_t)(c0 + c) * X.cs];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < m * nc; e += blockDim.x) {
    const int i = e % m, c = e / m;
    X.p[(int64_t)i * X.rs + (int64_t)(c0 + c) * X.cs] = T[e];
  }
}

// y[i, c] = b[P[i], c]
__global__ void lu_gather_rows_kernel(View Y, View Bv, const int64_t* __restrict__ P) {
  const int64_t tot = (int64_t)Y.rows * Y.cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % Y.rows), c = (int)(e / Y.rows);
    Y.p[(int64_t)i * Y.rs + (int64_t)c * Y.cs] = Bv.p[P[i] * Bv.rs + (int64_t)c * Bv.cs];
  }
}

// pieces of a low-rank sum, gathered into contiguous [s_i A_i] / [B_i] with
// their first k_i columns, rows placed at offsets ro_i / co_i (zeros
// elsewhere) -- the concatenations of rkmat_add! and rkmat_hmat_add
struct Piece {
  const double* A; int64_t lda;
  const double* B; int64_t ldb;
  const int32_t* k;
  int m, n, ro, co;
  double s;
};
constexpr int MAX_PIECES = 4;
struct GatherArgs {
  Piece pc[MAX_PIECES];
  int np;
  double* SA; double* SB;     // M x rmax, N x rmax
  int M, N, rmax;
  int32_t* r_out;
  int* flags;
};
__device__ void gather_pieces(const GatherArgs& g);
__global__ void __launch_bounds__(256) lu_gather_pieces_kernel(GatherArgs g) { gather_pieces(g); }
__device__ void gather_pieces(const GatherArgs& g) {
  __shared__ int pre[MAX_PIECES + 1];
  if (threadIdx.x == 0) {
    int t = 0;
    for (int q = 0; q < g.np; ++q) { pre[q] = t; t += *g.pc[q].k; }
    pre[g.np] = t;
    if (t > g.rmax) atomicOr(g.flags, 1);
    *g.r_out = t;
  }
  __syncthreads();
  const int r = min(pre[g.np], g.rmax);
  for (int64_t e = threadIdx.x; e < (int64_t)g.M * r; e += blockDim.x) {
    const int i = (int)(e % g.M), c = (int)(e / g.M);
    int q = 0;
    while (q + 1 < g.np && pre[q + 1] <= c) ++q;
    const Piece& P = g.pc[q];
    const int cc = c - pre[q];
    const int ii = i - P.ro;
    g.SA[e] = (ii >= 0 && ii < P.m) ? P.s * P.A[ii + (int64_t)cc * P.lda] : 0.0;
  }
  for (int64_t e = threadIdx.x; e < (int64_t)g.N * r; e += blockDim.x) {
    const int j = (int)(e % g.N), c = (int)(e / g.N);
    int q = 0;
    while (q + 1 < g.np && pre[q + 1] <= c) ++q;
    const Piece& P = g.pc[q];
    const int cc = c - pre[q];
    const int jj = j - P.co;
    g.SB[e] = (jj >= 0 && jj < P.n) ? P.B[jj + (int64_t)cc * P.ldb] : 0.0;
  }
}

__global__ void lu_copy_int_kernel(int32_t* dst, const int32_t* src) { *dst = *src; }

__global__ void lu_set_int_kernel(int32_t* dst, int v) { *dst = v; }

template <typename T>
__global__ void lu_load_kernel(const T* __restrict__ src, int64_t ld_src, int rows, int cols, double* __restrict__ dst,
                               int64_t ld_dst, int dst_cols) {
  const int64_t tot = (int64_t)rows * dst_cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % rows), c = (int)(e / rows);
    dst[i + (int64_t)c * ld_dst] = c < cols ? from_store<T>(src[i + (int64_t)c * ld_src]) : 0.0;
  }
}

// ---------------------------------------------------------------------------
// host-side block tree of the factorisation and of the temporaries
// ---------------------------------------------------------------------------
struct Blk;
using BP = std::shared_ptr<Blk>;

struct Ctx {
  cudaStream_t st;
  int cap;
  int64_t* P;          // device permutation
  int* flags;          // device error bits: 1 rank overflow, 2 non-finite, 4 singular
  double eps_trunc;
  const hm_handle* h;
  struct Arena* ar = nullptr;      // when set, temporaries come from this fixed buffer
};

// A fixed device buffer handed out front to back; nothing is returned before
// the sequence that uses it ends.  A captured solve takes its temporaries from
// one, so the graph holds no allocation nodes.
struct Arena {
  char* base = nullptr;
  size_t size = 0, used = 0;
};
static inline size_t arena_round(size_t b) { return (std::max<size_t>(b, 8) + 255) & ~(size_t)255; }

struct Blk {
  int8_t type = T_H;
  int m = 0, n = 0;
  int32_t s = -1, t = -1;             // clusters (for the isleaf tests of hmul)
  int64_t row0 = 0;                   // global first row (persistent blocks)
  double* C = nullptr;                // dense, column-major, ld = ldc
  int64_t ldc = 0;
  double* A = nullptr;                // low-rank: A (m x cap), B (n x cap)
  double* B = nullptr;
  int64_t lda = 0, ldb = 0;
  int32_t* k = nullptr;
  int cap = 0;
  BP ch[4];
  std::vector<void*> own;
  char* part = nullptr;               // the rest of a reserved allocation (dmalloc takes from it first)
  size_t left = 0;
  cudaStream_t st = nullptr;
  ~Blk() {
    for (void* p : own) cudaFreeAsync(p, st);
  }
  View Cv() const { return View{C, 1, ldc, m, n}; }
  View Av() const { return View{A, 1, lda, m, cap}; }
  View Bv() const { return View{B, 1, ldb, n, cap}; }
};

struct JobTape;
static thread_local JobTape* g_tape = nullptr;
static void tape_note_temporary(size_t bytes);

static void* dmalloc(Ctx& c, Blk& b, size_t bytes) {
  if (c.ar) {
    const size_t r = arena_round(bytes);
    if (c.ar->used + r > c.ar->size) throw LuError(HM_ERR_CUDA, "solve arena exhausted");
    void* q = c.ar->base + c.ar->used;
    c.ar->used += r;
    return q;
  }
  tape_note_temporary(bytes);
  void* p = nullptr;
  const size_t r = arena_round(bytes);
  if (r <= b.left) {
    p = b.part;
    b.part += r;
    b.left -= r;
    return p;
  }
  cudaError_t e = cudaMallocAsync(&p, std::max<size_t>(bytes, 8), c.st);
  if (e != cudaSuccess) throw LuError(HM_ERR_OOM, std::string("H-LU temporary: ") + cudaGetErrorString(e));
  b.own.push_back(p);
  return p;
}

// One allocation for the next dmalloc calls on b, `bytes` of them in whole
// arena_round units.  The factorisations of a batch allocate at the same time
// and wait for one another in the allocator, up to half a millisecond a call:
// 16 problems of 1024 to 8192 points, factorised and solved, 95.7 ms with an
// allocation per panel and inverse, 78.4 ms so.
static void reserve(Ctx& c, Blk& b, size_t bytes) {
  if (c.ar || bytes == 0) return;
  b.left = 0;
  b.part = (char*)dmalloc(c, b, bytes);
  b.left = bytes;
}

static BP new_dense(Ctx& c, int m, int n, int32_t s, int32_t t) {
  BP b = std::make_shared<Blk>();
  b->st = c.st;
  b->type = T_DENSE; b->m = m; b->n = n; b->s = s; b->t = t;
  b->C = (double*)dmalloc(c, *b, sizeof(double) * (size_t)m * n);
  b->ldc = std::max(m, 1);
  return b;
}

static BP new_rk(Ctx& c, int m, int n, int32_t s, int32_t t, bool alloc_a = true, bool alloc_b = true) {
  BP b = std::make_shared<Blk>();
  b->st = c.st;
  b->type = T_RK; b->m = m; b->n = n; b->s = s; b->t = t; b->cap = c.cap;
  if (alloc_a) { b->A = (double*)dmalloc(c, *b, sizeof(double) * (size_t)m * c.cap); b->lda = std::max(m, 1); }
  if (alloc_b) { b->B = (double*)dmalloc(c, *b, sizeof(double) * (size_t)n * c.cap); b->ldb = std::max(n, 1); }
  b->k = (int32_t*)dmalloc(c, *b, sizeof(int32_t));
  return b;
}

static bool is_leaf_cluster(const Ctx& c, int32_t cl) { return cl >= 0 && c.h->cl_left[cl] < 0; }

// ---- primitive launches --------------------------------------------------

static void gemm(Ctx& c, View C, View A, View B, double alpha, double beta) {
  if (C.rows == 0 || C.cols == 0) return;
  // 128 x 128 tiles once they fill the GPU; medium products keep the 32 x 32
  // tiles (more CTAs)
  const int64_t big_tiles = (int64_t)((C.rows + GB_T - 1) / GB_T) * ((C.cols + GB_T - 1) / GB_T);
  if (A.cols > 0 && (double)C.rows * C.cols * A.cols >= 4.0e6 && big_tiles >= 148) {
    dim3 g((C.cols + GB_T - 1) / GB_T, (C.rows + GB_T - 1) / GB_T);
    lu_gemm_big_kernel<<<g, 256, 0, c.st>>>(A, B, C, alpha, beta);
    LU_LAUNCH_CHECK();
    return;
  }
  if (A.cols == 0) {
    if (beta != 1.0) {
      lu_axpby_kernel<<<64, 256, 0, c.st>>>(C, View{nullptr, 0, 0, C.rows, C.cols}, 0.0, beta);
      LU_LAUNCH_CHECK();
    }
    return;
  }
  dim3 g((C.cols + 31) / 32, (C.rows + 31) / 32);
  lu_gemm_kernel<<<g, 256, 0, c.st>>>(A, B, C, alpha, beta);
  LU_LAUNCH_CHECK();
}

static void axpby(Ctx& c, View Y, View X, double alpha, double beta) {
  const int64_t tot = (int64_t)Y.rows * Y.cols;
  if (tot == 0) return;
  unsigned g = (unsigned)std::min<int64_t>((tot + 255) / 256, 1024);
  lu_axpby_kernel<<<g, 256, 0, c.st>>>(Y, X, alpha, beta);
  LU_LAUNCH_CHECK();
}

// X <- L^-1 X for triangles of 65 to TRSM_ROWS rows, 32 columns a CTA, staged in
// shared memory.  Larger ones are halved, with a product by all SMs between the
// halves (trsm_lower).  One thread a column with the triangle read from L2 was a
// chain of rows^2 / 2 dependent steps: 100 right-hand sides at n = 8192, 32 tiles
// of 256 rows, 165 ms so, 11 now; 8 tiles of 1024 rows 730 and 11 ms; the LU of the
// latter, whose panels take this way too, 544 and 33 ms.  Pieces of up to 512 rows:
// 12 ms and 37 ms.  The recursion's leaves of 94 rows (n = 3000, one column): 7.8
// and 3.4 ms.
constexpr int TRSM_ROWS = 256;
__global__ void __launch_bounds__(256) lu_trsm_block_kernel(View L, View X, int unit) {
  extern __shared__ double sm[];
  const int S = L.rows, ldx = tp_ldx(S), c0 = (int)blockIdx.x * TP_COLS, nc = min(TP_COLS, X.cols - c0);
  double* xg = X.p + (int64_t)c0 * X.cs;
  double* tri = sm + TP_COLS * ldx;                      // 32 x 33, then the 32 reciprocals
  for (int e = threadIdx.x; e < TP_COLS * S; e += blockDim.x) {
    const int cc = e / S, i = e % S;
    sm[cc * ldx + i] = cc < nc ? xg[(int64_t)cc * X.cs + (int64_t)i * X.rs] : 0.0;
  }
  __syncthreads();
  tile_trsm(L.p, L.rs, L.cs, S, unit != 0, sm, ldx, nc, 0, tri, tri + 32 * 33);
  for (int e = threadIdx.x; e < nc * S; e += blockDim.x) {
    const int cc = e / S, i = e % S;
    xg[(int64_t)cc * X.cs + (int64_t)i * X.rs] = sm[cc * ldx + i];
  }
}

static void trsm_lower(Ctx& c, View L, View X, bool unit) {
  if (X.cols == 0 || L.rows == 0) return;
  if (L.rows <= 32) {
    lu_trsm_small_kernel<32><<<(X.cols + 31) / 32, 32, 0, c.st>>>(L, X, unit ? 1 : 0);
    LU_LAUNCH_CHECK();
    return;
  }
  if (L.rows <= 64) {
    lu_trsm_small_kernel<64><<<(X.cols + 31) / 32, 32, 0, c.st>>>(L, X, unit ? 1 : 0);
    LU_LAUNCH_CHECK();
    return;
  }
  // dense diagonal tiles (solves of many columns, panels of large tiles) and the
  // largest leaves: halves of at most TRSM_ROWS rows with a product between them
  if (L.rows > TRSM_ROWS) {
    const int m = (L.rows / 2 + 31) / 32 * 32, r = L.rows - m;
    const View X1 = vsub(X, 0, 0, m, X.cols), X2 = vsub(X, m, 0, r, X.cols);
    trsm_lower(c, vsub(L, 0, 0, m, m), X1, unit);
    gemm(c, X2, vsub(L, m, 0, r, m), X1, -1.0, 1.0);
    trsm_lower(c, vsub(L, m, m, r, r), X2, unit);
    return;
  }
  if (smem_attr((const void*)lu_trsm_block_kernel, (int)tp_smem(TRSM_ROWS)) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "trsm smem attribute");
  lu_trsm_block_kernel<<<(X.cols + TP_COLS - 1) / TP_COLS, 256, tp_smem(L.rows), c.st>>>(L, X, unit ? 1 : 0);
  LU_LAUNCH_CHECK();
}

// rows of a diagonal leaf at most, of the recursion (the leaf and its pivots in
// 200 KB) and of the tiles (lu_diag_kernel<160>)
constexpr int LU_LEAF_MAX = 159;
static_assert(sizeof(double) * LU_LEAF_MAX * LU_LEAF_MAX + sizeof(int) * LU_LEAF_MAX <= 200 * 1024, "leaf in shared memory");
[[noreturn]] static void leaf_too_large() {
  throw LuError(HM_ERR_UNSUPPORTED, "diagonal leaf above " + std::to_string(LU_LEAF_MAX) + " rows (MinBlock too large)");
}

static void getrf(Ctx& c, View C, int64_t goff) {
  const int m = C.rows;
  if (m != C.cols) throw LuError(HM_ERR_UNSUPPORTED, "non-square diagonal leaf");
  if (m <= 64) {
    lu_getrf_small_kernel<<<1, 32, 0, c.st>>>(C, c.P, goff, c.flags);
    LU_LAUNCH_CHECK();
    return;
  }
  if (m > LU_LEAF_MAX) leaf_too_large();
  const size_t smem = sizeof(double) * (size_t)m * m + sizeof(int) * m;
  if (smem_attr((const void*)lu_getrf_kernel, 200 * 1024) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "getrf smem attribute");
  lu_getrf_kernel<<<1, 256, smem, c.st>>>(C, c.P, goff, c.flags);
  LU_LAUNCH_CHECK();
}

static void laswp(Ctx& c, View X, int64_t goff) {
  if (X.rows == 0 || X.cols == 0) return;
  int chunk = (int)std::max<int64_t>(1, std::min<int64_t>(X.cols, (48 * 1024 / 8) / X.rows));
  const size_t smem = sizeof(double) * (size_t)X.rows * chunk;
  lu_laswp_kernel<<<(X.cols + chunk - 1) / chunk, 256, smem, c.st>>>(X, c.P, goff, chunk);
  LU_LAUNCH_CHECK();
}

static void copy_int(Ctx& c, int32_t* dst, const int32_t* src) {
  lu_copy_int_kernel<<<1, 1, 0, c.st>>>(dst, src);
  LU_LAUNCH_CHECK();
}

// ---- recompression --------------------------------------------------------
// target (low-rank) = truncated sum of pieces: QR of both concatenations and
// compress() of the core (src/harithm.jl:374-396, 49-56, src/hlu.jl:159-190)
static void recompress(Ctx& c, Blk& target, const std::vector<Piece>& pcs) {
  if (pcs.size() > (size_t)MAX_PIECES) throw LuError(HM_ERR_UNSUPPORTED, "too many pieces");
  Blk tmp;
  tmp.st = c.st;
  const int M = target.m, N = target.n;
  double* SA = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)M * RCORE_MAX);
  double* SB = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)N * RCORE_MAX);
  int32_t* r = (int32_t*)dmalloc(c, tmp, sizeof(int32_t));
  GatherArgs g{};
  for (size_t q = 0; q < pcs.size(); ++q) g.pc[q] = pcs[q];
  g.np = (int)pcs.size();
  g.SA = SA; g.SB = SB; g.M = M; g.N = N; g.rmax = RCORE_MAX; g.r_out = r; g.flags = c.flags;
  lu_gather_pieces_kernel<<<1, 256, 0, c.st>>>(g);
  LU_LAUNCH_CHECK();
  CoreJob J{};
  J.A = SA; J.B = SB; J.outA = target.A; J.outB = target.B;
  J.m = M; J.n = N; J.r = 0; J.lda = std::max(M, 1); J.ldb = std::max(N, 1);
  J.ldoa = (int32_t)target.lda; J.ldob = (int32_t)target.ldb; J.kcap = target.cap;
  J.zero_test = 1; J.rank = target.k; J.r_dev = r; J.pre_status = nullptr; J.zero_fill = 1;
  int s = launch_core_one(J, c.eps_trunc, c.flags, c.st);
  if (s != HM_OK) throw LuError(s, "recompression launch");
}

// target (low-rank) = compress(D) for a dense D (src/hlu.jl:159-190): fully
// pivoted ACA far below eps_trunc * s_1, then the exact SVD of its core
static void compress_dense_into(Ctx& c, Blk& target, View D) {
  Blk tmp;
  tmp.st = c.st;
  const int m = D.rows, n = D.cols;
  double* R = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)m * n);
  double* U = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)m * RCORE_MAX);
  double* V = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)n * RCORE_MAX);
  int32_t* rk = (int32_t*)dmalloc(c, tmp, sizeof(int32_t) * 2);
  axpby(c, View{R, 1, std::max(m, 1), m, n}, D, 1.0, 0.0);
  AcaFpJob J{};
  J.R = R; J.U = U; J.V = V; J.m = m; J.n = n; J.cap = RCORE_MAX; J.min_rank = 1; J.eps = 0.0;
  J.rank = rk; J.status = rk + 1; J.rel_mode = 1; J.eps_trunc = c.eps_trunc;
  int s = launch_aca_fp_one(J, c.st);
  if (s != HM_OK) throw LuError(s, "compress launch");
  CoreJob K{};
  K.A = U; K.B = V; K.outA = target.A; K.outB = target.B; K.m = m; K.n = n; K.r = 0;
  K.lda = std::max(m, 1); K.ldb = std::max(n, 1); K.ldoa = (int32_t)target.lda; K.ldob = (int32_t)target.ldb;
  K.kcap = target.cap; K.zero_test = 0; K.rank = target.k; K.r_dev = rk; K.pre_status = rk + 1; K.zero_fill = 1;
  s = launch_core_one(K, c.eps_trunc, c.flags, c.st);
  if (s != HM_OK) throw LuError(s, "compress core launch");
}

// ---- H-matrix products with dense blocks ----------------------------------
// Y += s H X   (hmat_matvec! with a matrix, src/harithm.jl:340-354)
static void hmm(Ctx& c, View Y, double s, const Blk& H, View X) {
  if (H.type == T_DENSE) {
    gemm(c, Y, H.Cv(), X, s, 1.0);
  } else if (H.type == T_RK) {
    Blk tmp;
    tmp.st = c.st;
    double* T = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)H.cap * X.cols);
    View Tv{T, 1, H.cap, H.cap, X.cols};
    gemm(c, Tv, vtr(H.Bv()), X, 1.0, 0.0);
    gemm(c, Y, H.Av(), Tv, s, 1.0);
  } else {
    const int m = H.ch[0]->m, n = H.ch[0]->n;
    hmm(c, vsub(Y, 0, 0, m, Y.cols), s, *H.ch[0], vsub(X, 0, 0, n, X.cols));
    hmm(c, vsub(Y, 0, 0, m, Y.cols), s, *H.ch[1], vsub(X, n, 0, H.n - n, X.cols));
    hmm(c, vsub(Y, m, 0, H.m - m, Y.cols), s, *H.ch[2], vsub(X, 0, 0, n, X.cols));
    hmm(c, vsub(Y, m, 0, H.m - m, Y.cols), s, *H.ch[3], vsub(X, n, 0, H.n - n, X.cols));
  }
}

// Y += s H' X   (transpose_hmat_mat_mul, src/harithm.jl:243-260)
static void hmm_t(Ctx& c, View Y, double s, const Blk& H, View X) {
  if (H.type == T_DENSE) {
    gemm(c, Y, vtr(H.Cv()), X, s, 1.0);
  } else if (H.type == T_RK) {
    Blk tmp;
    tmp.st = c.st;
    double* T = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)H.cap * X.cols);
    View Tv{T, 1, H.cap, H.cap, X.cols};
    gemm(c, Tv, vtr(H.Av()), X, 1.0, 0.0);
    gemm(c, Y, H.Bv(), Tv, s, 1.0);
  } else {
    const int m = H.ch[0]->m, n = H.ch[0]->n;
    hmm_t(c, vsub(Y, 0, 0, n, Y.cols), s, *H.ch[0], vsub(X, 0, 0, m, X.cols));
    hmm_t(c, vsub(Y, 0, 0, n, Y.cols), s, *H.ch[2], vsub(X, m, 0, H.m - m, X.cols));
    hmm_t(c, vsub(Y, n, 0, H.n - n, Y.cols), s, *H.ch[1], vsub(X, 0, 0, m, X.cols));
    hmm_t(c, vsub(Y, n, 0, H.n - n, Y.cols), s, *H.ch[3], vsub(X, m, 0, H.m - m, X.cols));
  }
}

// Y += s X H   (v*H of src/harithm.jl:331-371 for a matrix v)
static void xh(Ctx& c, View Y, double s, View X, const Blk& H) {
  hmm_t(c, vtr(Y), s, H, vtr(X));
}

// dense copy of H (to_fmat, src/utils.jl:162-192)
static void densify_into(Ctx& c, View D, const Blk& H) {
  if (H.type == T_DENSE) {
    axpby(c, D, H.Cv(), 1.0, 0.0);
  } else if (H.type == T_RK) {
    gemm(c, D, H.Av(), vtr(H.Bv()), 1.0, 0.0);
  } else {
    const int m = H.ch[0]->m, n = H.ch[0]->n;
    densify_into(c, vsub(D, 0, 0, m, n), *H.ch[0]);
    densify_into(c, vsub(D, 0, n, m, H.n - n), *H.ch[1]);
    densify_into(c, vsub(D, m, 0, H.m - m, n), *H.ch[2]);
    densify_into(c, vsub(D, m, n, H.m - m, H.n - n), *H.ch[3]);
  }
}

static BP dense_of(Ctx& c, const Blk& H) {
  BP d = new_dense(c, H.m, H.n, H.s, H.t);
  densify_into(c, d->Cv(), H);
  return d;
}

static BP copy_blk(Ctx& c, const Blk& a) {
  if (a.type == T_DENSE) {
    BP d = new_dense(c, a.m, a.n, a.s, a.t);
    d->row0 = a.row0;
    axpby(c, d->Cv(), a.Cv(), 1.0, 0.0);
    return d;
  }
  if (a.type == T_RK) {
    BP r = new_rk(c, a.m, a.n, a.s, a.t);
    r->row0 = a.row0;
    axpby(c, r->Av(), a.Av(), 1.0, 0.0);
    axpby(c, r->Bv(), a.Bv(), 1.0, 0.0);
    copy_int(c, r->k, a.k);
    return r;
  }
  BP h = std::make_shared<Blk>();
  h->st = c.st;
  h->type = T_H; h->m = a.m; h->n = a.n; h->s = a.s; h->t = a.t; h->row0 = a.row0;
  for (int q = 0; q < 4; ++q) h->ch[q] = copy_blk(c, *a.ch[q]);
  return h;
}

// ---- H-add (src/harithm.jl:4-151, 374-420) ---------------------------------
static void hmat_full_add(Ctx& c, Blk& a, View D, double s);
static void hmat_add(Ctx& c, Blk& a, const Blk& b, double s);

static void hmat_full_add(Ctx& c, Blk& a, View D, double s) {
  if (a.type == T_DENSE) {
    axpby(c, a.Cv(), D, s, 1.0);
  } else if (a.type == T_RK) {
    // C = A B' + s b; a.A, a.B = compress(C)   (src/harithm.jl:12-15)
    Blk tmp;
    tmp.st = c.st;
    double* T = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)a.m * a.n);
    View Tv{T, 1, std::max(a.m, 1), a.m, a.n};
    axpby(c, Tv, D, s, 0.0);
    gemm(c, Tv, a.Av(), vtr(a.Bv()), 1.0, 1.0);
    compress_dense_into(c, a, Tv);
  } else {
    const int m = a.ch[0]->m, n = a.ch[0]->n;
    hmat_full_add(c, *a.ch[0], vsub(D, 0, 0, m, n), s);
    hmat_full_add(c, *a.ch[1], vsub(D, 0, n, m, a.n - n), s);
    hmat_full_add(c, *a.ch[2], vsub(D, m, 0, a.m - m, n), s);
    hmat_full_add(c, *a.ch[3], vsub(D, m, n, a.m - m, a.n - n), s);
  }
}

// A B' + s H as a new low-rank block (src/harithm.jl:58-91)
static BP rkmat_hmat_add(Ctx& c, View A, View B, const int32_t* k, double s, const Blk& H) {
  BP out = new_rk(c, A.rows, B.rows, H.s, H.t);
  if (H.type == T_DENSE) {
    Blk tmp;
    tmp.st = c.st;
    double* T = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)H.m * H.n);
    View Tv{T, 1, std::max(H.m, 1), H.m, H.n};
    axpby(c, Tv, H.Cv(), s, 0.0);
    gemm(c, Tv, A, vtr(B), 1.0, 1.0);
    compress_dense_into(c, *out, Tv);
  } else if (H.type == T_RK) {
    std::vector<Piece> pcs = {
        Piece{A.p, A.cs, B.p, B.cs, k, A.rows, B.rows, 0, 0, 1.0},
        Piece{H.A, H.lda, H.B, H.ldb, H.k, H.m, H.n, 0, 0, s}};
    recompress(c, *out, pcs);
  } else {
    const int m = H.ch[0]->m, n = H.ch[0]->n;
    BP r11 = rkmat_hmat_add(c, vsub(A, 0, 0, m, A.cols), vsub(B, 0, 0, n, B.cols), k, s, *H.ch[0]);
    BP r12 = rkmat_hmat_add(c, vsub(A, 0, 0, m, A.cols), vsub(B, n, 0, H.n - n, B.cols), k, s, *H.ch[1]);
    BP r21 = rkmat_hmat_add(c, vsub(A, m, 0, H.m - m, A.cols), vsub(B, 0, 0, n, B.cols), k, s, *H.ch[2]);
    BP r22 = rkmat_hmat_add(c, vsub(A, m, 0, H.m - m, A.cols), vsub(B, n, 0, H.n - n, B.cols), k, s, *H.ch[3]);
    // A0 = [A11 A12 0 0; 0 0 A21 A22], B0 = [B11 0 B21 0; 0 B12 0 B22]  (src/harithm.jl:82-86)
    std::vector<Piece> pcs = {
        Piece{r11->A, r11->lda, r11->B, r11->ldb, r11->k, m, n, 0, 0, 1.0},
        Piece{r12->A, r12->lda, r12->B, r12->ldb, r12->k, m, H.n - n, 0, n, 1.0},
        Piece{r21->A, r21->lda, r21->B, r21->ldb, r21->k, H.m - m, n, m, 0, 1.0},
        Piece{r22->A, r22->lda, r22->B, r22->ldb, r22->k, H.m - m, H.n - n, m, n, 1.0}};
    recompress(c, *out, pcs);
  }
  return out;
}

static void hmat_add(Ctx& c, Blk& a, const Blk& b, double s) {
  if (b.type == T_DENSE) {
    hmat_full_add(c, a, b.Cv(), s);
  } else if (a.type == T_DENSE && b.type == T_RK) {
    gemm(c, a.Cv(), b.Av(), vtr(b.Bv()), s, 1.0);
  } else if (a.type == T_DENSE && b.type == T_H) {
    // a.C += s * (a.C + dense(b))  as written in src/harithm.jl:112; not
    // reached from lu! (a dense target has a leaf cluster, so b is never H)
    BP d = dense_of(c, b);
    axpby(c, d->Cv(), a.Cv(), 1.0, 1.0);
    axpby(c, a.Cv(), d->Cv(), s, 1.0);
  } else if (a.type == T_RK && b.type == T_RK) {
    std::vector<Piece> pcs = {
        Piece{a.A, a.lda, a.B, a.ldb, a.k, a.m, a.n, 0, 0, 1.0},
        Piece{b.A, b.lda, b.B, b.ldb, b.k, b.m, b.n, 0, 0, s}};
    recompress(c, a, pcs);
  } else if (a.type == T_RK && b.type == T_H) {
    BP r = rkmat_hmat_add(c, a.Av(), a.Bv(), a.k, s, b);
    axpby(c, a.Av(), r->Av(), 1.0, 0.0);
    axpby(c, a.Bv(), r->Bv(), 1.0, 0.0);
    copy_int(c, a.k, r->k);
  } else if (a.type == T_H && b.type == T_RK) {
    const int m = a.ch[0]->m, n = a.ch[0]->n;
    auto part = [&](int r0, int mr, int c0, int nc) {
      Blk v;
      v.st = c.st;
      v.type = T_RK; v.m = mr; v.n = nc; v.cap = b.cap; v.k = b.k;
      v.A = b.A + r0; v.lda = b.lda; v.B = b.B + c0; v.ldb = b.ldb;
      return v;
    };
    Blk c11 = part(0, m, 0, n), c21 = part(m, a.m - m, 0, n);
    Blk c12 = part(0, m, n, a.n - n), c22 = part(m, a.m - m, n, a.n - n);
    hmat_add(c, *a.ch[0], c11, s);
    hmat_add(c, *a.ch[2], c21, s);
    hmat_add(c, *a.ch[1], c12, s);
    hmat_add(c, *a.ch[3], c22, s);
  } else if (a.type == T_H && b.type == T_H) {
    for (int q = 0; q < 4; ++q) hmat_add(c, *a.ch[q], *b.ch[q], s);
  }
}

static BP hadd(Ctx& c, const Blk& a, const Blk& b) {
  BP r = copy_blk(c, a);
  hmat_add(c, *r, b, 1.0);
  return r;
}

// ---- H x H (src/harithm.jl:162-314) -----------------------------------------
static BP hmul(Ctx& c, const Blk& a, const Blk& b) {
  BP M;
  if (a.type == T_DENSE) {
    if (b.type == T_H && !is_leaf_cluster(c, a.s) && !is_leaf_cluster(c, a.t))
      throw LuError(HM_ERR_UNSUPPORTED, "full_mat_mul branch that has no method in the reference");
    if (b.type == T_H) {
      BP db = dense_of(c, b);
      M = new_dense(c, a.m, b.n, a.s, b.t);
      gemm(c, M->Cv(), a.Cv(), db->Cv(), 1.0, 0.0);
    } else if (b.type == T_DENSE) {
      M = new_dense(c, a.m, b.n, a.s, b.t);
      gemm(c, M->Cv(), a.Cv(), b.Cv(), 1.0, 0.0);
    } else {
      M = new_rk(c, a.m, b.n, a.s, b.t, true, false);
      M->B = b.B; M->ldb = b.ldb;
      gemm(c, M->Av(), a.Cv(), b.Av(), 1.0, 0.0);
      copy_int(c, M->k, b.k);
    }
  } else if (b.type == T_DENSE) {
    if (a.type == T_H && !is_leaf_cluster(c, b.s) && !is_leaf_cluster(c, b.t))
      throw LuError(HM_ERR_UNSUPPORTED, "mat_full_mul branch that has no method in the reference");
    if (a.type == T_H) {
      M = new_dense(c, a.m, b.n, a.s, b.t);
      axpby(c, M->Cv(), View{nullptr, 0, 0, a.m, b.n}, 0.0, 0.0);
      hmm(c, M->Cv(), 1.0, a, b.Cv());
    } else {
      M = new_rk(c, a.m, b.n, a.s, b.t, false, true);
      M->A = a.A; M->lda = a.lda;
      gemm(c, M->Bv(), vtr(b.Cv()), a.Bv(), 1.0, 0.0);
      copy_int(c, M->k, a.k);
    }
  } else if (a.type == T_RK && b.type == T_RK) {
    M = new_rk(c, a.m, b.n, a.s, b.t, false, true);
    M->A = a.A; M->lda = a.lda;
    Blk tmp;
    tmp.st = c.st;
    double* W = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)b.cap * a.cap);
    View Wv{W, 1, b.cap, b.cap, a.cap};
    gemm(c, Wv, vtr(b.Av()), a.Bv(), 1.0, 0.0);
    gemm(c, M->Bv(), b.Bv(), Wv, 1.0, 0.0);
    copy_int(c, M->k, a.k);
  } else if (a.type == T_RK && b.type == T_H) {
    M = new_rk(c, a.m, b.n, a.s, b.t, false, true);
    M->A = a.A; M->lda = a.lda;
    axpby(c, M->Bv(), View{nullptr, 0, 0, b.n, M->cap}, 0.0, 0.0);
    hmm_t(c, M->Bv(), 1.0, b, a.Bv());
    copy_int(c, M->k, a.k);
  } else if (a.type == T_H && b.type == T_RK) {
    M = new_rk(c, a.m, b.n, a.s, b.t, true, false);
    M->B = b.B; M->ldb = b.ldb;
    axpby(c, M->Av(), View{nullptr, 0, 0, a.m, M->cap}, 0.0, 0.0);
    hmm(c, M->Av(), 1.0, a, b.Av());
    copy_int(c, M->k, b.k);
  } else {
    M = std::make_shared<Blk>();
    M->st = c.st;
    M->type = T_H; M->m = a.m; M->n = b.n; M->s = a.s; M->t = b.t;
    for (int i = 0; i < 2; ++i)
      for (int j = 0; j < 2; ++j) {
        BP H1 = hmul(c, *a.ch[2 * i + 0], *b.ch[0 + j]);
        BP H2 = hmul(c, *a.ch[2 * i + 1], *b.ch[2 + j]);
        M->ch[2 * i + j] = hadd(c, *H1, *H2);
      }
  }
  M->s = a.s;
  M->t = b.t;
  return M;
}

static void sub_mul(Ctx& c, Blk& cc, const Blk& a, const Blk& b) {
  BP M = hmul(c, a, b);
  hmat_add(c, cc, *M, -1.0);
}

// ---- triangular solves (src/hlu.jl:236-442) ----------------------------------
static void mfs(Ctx& c, const Blk& a, View X, bool unit, bool lower) {
  if (a.type == T_RK) throw LuError(HM_ERR_UNSUPPORTED, "A should not be a low-rank matrix");
  if (lower) {
    if (a.type == T_DENSE) {
      trsm_lower(c, a.Cv(), X, unit);
    } else {
      const int n = a.ch[0]->m;
      View X1 = vsub(X, 0, 0, n, X.cols), X2 = vsub(X, n, 0, X.rows - n, X.cols);
      mfs(c, *a.ch[0], X1, unit, true);
      hmm(c, X2, -1.0, *a.ch[2], X1);
      mfs(c, *a.ch[3], X2, unit, true);
    }
  } else {
    if (a.type == T_DENSE) {
      // X <- X U^{-1}  ==  X' <- U'^{-1} X'
      trsm_lower(c, vtr(a.Cv()), vtr(X), unit);
    } else {
      const int n = a.ch[0]->m;
      View X1 = vsub(X, 0, 0, X.rows, n), X2 = vsub(X, 0, n, X.rows, X.cols - n);
      mfs(c, *a.ch[0], X1, unit, false);
      xh(c, X2, -1.0, X1, *a.ch[1]);
      mfs(c, *a.ch[3], X2, unit, false);
    }
  }
}

static void trisolve(Ctx& c, const Blk& a, Blk& b, bool lower, bool unit) {
  if (a.type == T_RK) throw LuError(HM_ERR_UNSUPPORTED, "A should not be a low-rank matrix");
  if (lower) {
    if (a.type == T_DENSE && b.type == T_DENSE) trsm_lower(c, a.Cv(), b.Cv(), unit);
    else if (a.type == T_DENSE && b.type == T_RK) trsm_lower(c, a.Cv(), b.Av(), unit);
    else if (a.type == T_DENSE && b.type == T_H) throw LuError(HM_ERR_UNSUPPORTED, "This is never used");
    else if (a.type == T_H && b.type == T_H) {
      trisolve(c, *a.ch[0], *b.ch[0], lower, unit);
      trisolve(c, *a.ch[0], *b.ch[1], lower, unit);
      sub_mul(c, *b.ch[2], *a.ch[2], *b.ch[0]);
      sub_mul(c, *b.ch[3], *a.ch[2], *b.ch[1]);
      trisolve(c, *a.ch[3], *b.ch[2], lower, unit);
      trisolve(c, *a.ch[3], *b.ch[3], lower, unit);
    } else if (a.type == T_H && b.type == T_DENSE) mfs(c, a, b.Cv(), unit, true);
    else if (a.type == T_H && b.type == T_RK) mfs(c, a, b.Av(), unit, true);
  } else {
    if (a.type == T_DENSE && b.type == T_DENSE) trsm_lower(c, vtr(a.Cv()), vtr(b.Cv()), unit);
    else if (a.type == T_DENSE && b.type == T_RK) trsm_lower(c, vtr(a.Cv()), b.Bv(), unit);
    else if (a.type == T_H && b.type == T_DENSE) mfs(c, a, b.Cv(), unit, false);
    else if (a.type == T_H && b.type == T_RK) mfs(c, a, vtr(b.Bv()), unit, false);
    else if (a.type == T_H && b.type == T_H) {
      trisolve(c, *a.ch[0], *b.ch[0], lower, unit);
      trisolve(c, *a.ch[0], *b.ch[2], lower, unit);
      sub_mul(c, *b.ch[1], *b.ch[0], *a.ch[1]);
      sub_mul(c, *b.ch[3], *b.ch[2], *a.ch[1]);
      trisolve(c, *a.ch[3], *b.ch[1], lower, unit);
      trisolve(c, *a.ch[3], *b.ch[3], lower, unit);
    } else throw LuError(HM_ERR_UNSUPPORTED, "Invalid");
  }
}

// ---- LU (src/hlu.jl:446-515) --------------------------------------------------
static void permute(Ctx& c, Blk& H) {
  if (H.type == T_DENSE) laswp(c, H.Cv(), H.row0);
  else if (H.type == T_RK) laswp(c, H.Av(), H.row0);
  else
    for (int q = 0; q < 4; ++q) permute(c, *H.ch[q]);
}

static void lu_rec(Ctx& c, Blk& H) {
  if (H.type == T_RK) throw LuError(HM_ERR_UNSUPPORTED, "H should not be a low-rank matrix");
  if (H.type == T_DENSE) {
    getrf(c, H.Cv(), H.row0);
    return;
  }
  lu_rec(c, *H.ch[0]);
  permute(c, *H.ch[1]);
  trisolve(c, *H.ch[0], *H.ch[1], true, true);
  trisolve(c, *H.ch[0], *H.ch[2], false, false);
  sub_mul(c, *H.ch[3], *H.ch[2], *H.ch[1]);
  lu_rec(c, *H.ch[3]);
  permute(c, *H.ch[2]);
}

// ---- solve (src/hlu.jl:524-562) -----------------------------------------------
static void solve_rec(Ctx& c, const Blk& a, View y, bool lower) {
  if (a.type == T_RK) throw LuError(HM_ERR_UNSUPPORTED, "a cannot be a low-rank matrix");
  const int m = a.type == T_H ? a.ch[0]->m : a.m;
  if (lower) {
    if (a.type == T_DENSE) {
      trsm_lower(c, a.Cv(), y, true);
    } else {
      solve_rec(c, *a.ch[0], vsub(y, 0, 0, m, y.cols), true);
      hmm(c, vsub(y, m, 0, y.rows - m, y.cols), -1.0, *a.ch[2], vsub(y, 0, 0, m, y.cols));
      solve_rec(c, *a.ch[3], vsub(y, m, 0, y.rows - m, y.cols), true);
    }
  } else {
    if (a.type == T_DENSE) {
      trsm_lower(c, vrev(a.Cv()), vrev(y), false);       // U^{-1} y as a reversed lower solve
    } else {
      solve_rec(c, *a.ch[3], vsub(y, m, 0, y.rows - m, y.cols), false);
      hmm(c, vsub(y, 0, 0, m, y.cols), -1.0, *a.ch[1], vsub(y, m, 0, y.rows - m, y.cols));
      solve_rec(c, *a.ch[0], vsub(y, 0, 0, m, y.cols), false);
    }
  }
}

// transposed solve H' x = b with H[P,:] = L U: U' z = b (lower, non-unit),
// L' w = z (upper, unit), x[P] = w.  No counterpart in the reference (the
// adjoint of H\y); the same leaf kernels run on transposed/reversed views.
static void solve_t_rec(Ctx& c, const Blk& a, View y, bool upper_t) {
  if (a.type == T_RK) throw LuError(HM_ERR_UNSUPPORTED, "a cannot be a low-rank matrix");
  const int m = a.type == T_H ? a.ch[0]->m : a.m;
  if (upper_t) {                       // U' is lower triangular
    if (a.type == T_DENSE) {
      trsm_lower(c, vtr(a.Cv()), y, false);
    } else {
      solve_t_rec(c, *a.ch[0], vsub(y, 0, 0, m, y.cols), true);
      hmm_t(c, vsub(y, m, 0, y.rows - m, y.cols), -1.0, *a.ch[1], vsub(y, 0, 0, m, y.cols));
      solve_t_rec(c, *a.ch[3], vsub(y, m, 0, y.rows - m, y.cols), true);
    }
  } else {                             // L' is unit upper triangular
    if (a.type == T_DENSE) {
      trsm_lower(c, vrev(vtr(a.Cv())), vrev(y), true);
    } else {
      solve_t_rec(c, *a.ch[3], vsub(y, m, 0, y.rows - m, y.cols), false);
      hmm_t(c, vsub(y, 0, 0, m, y.cols), -1.0, *a.ch[2], vsub(y, m, 0, y.rows - m, y.cols));
      solve_t_rec(c, *a.ch[0], vsub(y, 0, 0, m, y.cols), false);
    }
  }
}

// x[P[i], c] = w[i, c]
__global__ void lu_scatter_rows_kernel(View Xv, View W, const int64_t* __restrict__ P) {
  const int64_t tot = (int64_t)W.rows * W.cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % W.rows), c = (int)(e / W.rows);
    Xv.p[P[i] * Xv.rs + (int64_t)c * Xv.cs] = W.p[(int64_t)i * W.rs + (int64_t)c * W.cs];
  }
}

// ---------------------------------------------------------------------------
// batched helpers
// ---------------------------------------------------------------------------
// Job arrays of a sequence that is later captured into a CUDA graph: the first
// (recording) run keeps every uploaded array alive in order; the capture run
// takes the same arrays back instead of uploading (a host-to-device copy of
// pageable memory cannot be captured).  The job contents are identical since
// the capture replays the recorded sequence on the same buffers.
struct JobTape {
  bool record = false, replay = false;
  std::vector<void*> bufs;
  std::vector<size_t> bytes;
  size_t pos = 0;
  size_t temp_bytes = 0;   // arena size that holds every temporary of the recorded run
  ~JobTape() {             // the owner has synchronised the device
    for (void* p : bufs) cudaFreeAsync(p, cudaStreamLegacy);
  }
};
static void tape_note_temporary(size_t bytes) {
  if (g_tape && g_tape->record) g_tape->temp_bytes += arena_round(bytes);
}

template <typename J>
static J* upload_jobs(Ctx& c, Blk& owner, const std::vector<J>& v) {
  if (g_tape && g_tape->replay) {
    if (g_tape->pos >= g_tape->bufs.size() || g_tape->bytes[g_tape->pos] != sizeof(J) * v.size())
      throw LuError(HM_ERR_CUDA, "job tape does not match the recorded sequence");
    return (J*)g_tape->bufs[g_tape->pos++];
  }
  J* d = nullptr;
  if (g_tape && g_tape->record) {
    if (cudaMallocAsync(&d, sizeof(J) * v.size(), c.st) != cudaSuccess) throw LuError(HM_ERR_OOM, "job tape");
    g_tape->bufs.push_back(d);
    g_tape->bytes.push_back(sizeof(J) * v.size());
  } else {
    d = (J*)dmalloc(c, owner, sizeof(J) * v.size());
  }
  if (cudaMemcpyAsync(d, v.data(), sizeof(J) * v.size(), cudaMemcpyHostToDevice, c.st) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "job upload");
  return d;
}

// copies of stored leaves into the FP64 working buffers of the factorisation,
// collected and launched as one kernel (one CTA per block)
struct LoadJob {
  const void* src;
  int64_t ld_src;
  int rows, cols;          // valid source columns; columns [cols, dst_cols) become zero
  int type;                // HM_F64 / HM_F32 / HM_BF16 element type of src
  double* dst;
  int64_t ld_dst;
  int dst_cols;
  int32_t* kdst;           // if set: *kdst = kval
  int kval;
};
__global__ void lu_load_batch_kernel(const LoadJob* __restrict__ jobs) {
  const LoadJob J = jobs[blockIdx.x];
  const int64_t tot = (int64_t)J.rows * J.dst_cols;
  for (int64_t e = threadIdx.x; e < tot; e += blockDim.x) {
    const int i = (int)(e % J.rows), c = (int)(e / J.rows);
    double v = 0.0;
    if (c < J.cols) {
      const int64_t s = i + (int64_t)c * J.ld_src;
      if (J.type == HM_F64) v = ((const double*)J.src)[s];
      else if (J.type == HM_F32) v = (double)((const float*)J.src)[s];
      else v = (double)__bfloat162float(((const __nv_bfloat16*)J.src)[s]);
    }
    J.dst[i + (int64_t)c * J.ld_dst] = v;
  }
  if (threadIdx.x == 0 && J.kdst) *J.kdst = J.kval;
}

struct Loader {
  std::vector<LoadJob> jobs;
  void flush(Ctx& c) {
    for (size_t b = 0; b < jobs.size(); b += 65535) {
      const size_t nb = std::min<size_t>(65535, jobs.size() - b);
      Blk tmp;
      tmp.st = c.st;
      std::vector<LoadJob> part(jobs.begin() + b, jobs.begin() + b + nb);
      LoadJob* d = upload_jobs(c, tmp, part);
      lu_load_batch_kernel<<<(unsigned)nb, 256, 0, c.st>>>(d);
      LU_LAUNCH_CHECK();
    }
    jobs.clear();
  }
};

static BP build_tree(Ctx& c, const hm_handle* h, int32_t node, Loader& ld);
static BP build_from_handle(Ctx& c, const hm_handle* h, int32_t node);

// independent products in one launch
static void gemm_batch(Ctx& c, const std::vector<GemmJob>& jobs) {
  if (jobs.empty()) return;
  int gx = 1, gy = 1;
  for (auto& j : jobs) {
    gx = std::max(gx, (j.C.cols + 31) / 32);
    gy = std::max(gy, (j.C.rows + 31) / 32);
  }
  for (size_t b = 0; b < jobs.size(); b += 65535) {
    const size_t nb = std::min<size_t>(65535, jobs.size() - b);
    Blk tmp;
    tmp.st = c.st;
    std::vector<GemmJob> part(jobs.begin() + b, jobs.begin() + b + nb);
    lu_gemm_batch_kernel<<<dim3(gx, gy, (unsigned)nb), 256, 0, c.st>>>(upload_jobs(c, tmp, part));
    LU_LAUNCH_CHECK();
  }
}

// truncation tolerance from which the tile recompressions run in FP32
constexpr double MIXED_CORE_EPS = 1e-6;

// ---------------------------------------------------------------------------
// tile LU.  When every leaf outside the diagonal tiles (row group x column
// group blocks) is one low-rank block covering its whole tile -- the
// partition of the aca2 route with the identity adjacency -- the recursion of
// lu! is carried out tile by tile (right-looking), which performs the same
// operations with leaf-local pivoting but batches them.  The diagonal tiles
// are held dense: their low-rank blocks (a few per cent of the matrix) are
// expanded at load, so a step's update of a tile is one rank-k product instead
// of a recompression per block, and its LU one kernel instead of a recursion of
// about a hundred launches (8 leaves of 32 rows: 3.2 ms, now 0.1 ms); the
// result is the same LU without the truncations inside the tile.  Per step k
// the diagonal tile is factorised, the whole row panel (A factors of tiles
// (k, j>k)) and column panel (B factors of tiles (i>k, k)) are solved as one
// wide triangular solve each, and every pair of trailing tiles is updated and
// recompressed by one CTA that forms its core B_ik' A_kj itself.  Updates are
// truncated per step (the recursion sums some products before truncating); both
// stay within eps_trunc of the exact Schur complement.
// ---------------------------------------------------------------------------
struct TileLU {
  int T = 0;
  std::vector<int64_t> start, size;      // tile ranges
  std::vector<BP> diag;                  // diagonal tiles, dense
  std::vector<double*> Ap, Bp;           // row panels (m_i x T*cap), column panels (n_j x T*cap)
  int32_t* kmat = nullptr;               // ranks of the off-diagonal tiles, T x T
  BP hold;                               // owns the panel memory
  double* Ai(int i, int j, int cap) const { return Ap[i] + (int64_t)j * cap * size[i]; }
  double* Bj(int i, int j, int cap) const { return Bp[j] + (int64_t)i * cap * size[j]; }
  // for the sweep solve (built on the first solve): the inverses of the
  // diagonal tiles' unit-lower L and upper U, each stored column-major and
  // row-major, and device tables of the panels
  BP sweep_hold;
  const double** d_Ap = nullptr;
  const double** d_Bp = nullptr;
  const double** d_inv[4] = {nullptr, nullptr, nullptr, nullptr};   // see sweep_finish
  int64_t* d_start = nullptr;
  int32_t* d_size = nullptr;
};

// tile structure of the handle, or false when the partition has no such level
// A tiling of [0, n) by clusters gcl (sorted by start) can run the tile
// schedule when every leaf off the tile diagonal is a low-rank leaf whose rows
// and columns are unions of whole tiles (a leaf spanning several tiles is
// loaded as its tile parts, which keep its rank) and every diagonal tile is a
// node of the block tree (leaves inside it stay in its recursive tree).
static bool tile_check(const hm_handle* h, const std::vector<int32_t>& gcl, std::vector<int32_t>& diag_node) {
  const int T = (int)gcl.size();
  if (T < 2) return false;
  if (h->cl_s[gcl[0]] != 0 || h->cl_e[gcl[T - 1]] != h->n) return false;
  for (int i = 1; i < T; ++i)
    if (h->cl_s[gcl[i]] != h->cl_e[gcl[i - 1]]) return false;
  std::vector<int64_t> st(T);
  for (int i = 0; i < T; ++i) st[i] = h->cl_s[gcl[i]];
  auto tile_of = [&](int64_t r) { return (int)(std::upper_bound(st.begin(), st.end(), r) - st.begin()) - 1; };
  auto aligned = [&](int64_t a, int64_t len, int t0, int t1) { return a == st[t0] && a + len == h->cl_e[gcl[t1]]; };
  for (auto& L : h->leaves) {
    const int i0 = tile_of(L.row0), i1 = tile_of(L.row0 + L.m - 1);
    const int j0 = tile_of(L.col0), j1 = tile_of(L.col0 + L.n - 1);
    if (i0 == i1 && j0 == j1 && i0 == j0) continue;            // inside a diagonal tile
    const bool overlap = !(i1 < j0 || j1 < i0);                 // would cover part of a diagonal tile
    if (overlap || L.type != T_RK || !aligned(L.row0, L.m, i0, i1) || !aligned(L.col0, L.n, j0, j1))
      return false;
  }
  const int64_t ncl = (int64_t)h->cl_s.size();
  diag_node.assign(T, -1);
  std::vector<int32_t> tile_of_cluster(ncl, -1);
  for (int i = 0; i < T; ++i) tile_of_cluster[gcl[i]] = i;
  for (int32_t id = 0; id < (int32_t)h->nodes.size(); ++id) {
    const Node& nd = h->nodes[id];
    if (nd.s == nd.t && tile_of_cluster[nd.s] >= 0) diag_node[tile_of_cluster[nd.s]] = id;
  }
  for (int i = 0; i < T; ++i)
    if (diag_node[i] < 0) return false;
  return true;
}

// The tile level.  First candidate: the highest clusters that are the row
// cluster of some leaf (for a balanced partition, the clusters of the first
// admissible level; for a KMeans tree the tiles may sit at several depths).
// Otherwise the shallowest depth whose clusters form a valid tiling (a median
// bisection of an n that is not a power of two mixes cluster sizes on both
// sides of MaxBlock on one level, so the admissible blocks start one level
// lower on part of it).  Tiles of at most TILE_MAX rows where there is a tiling
// of such, the leaves above that taken in parts: a diagonal tile is dense, and
// its LU, S^3 on the eight SMs of a cluster, is the longer the larger it is.
// H-LU, n = 16384 (bbfmm), tiles of 4096 rows 410 ms, cut into tiles of 2048 150;
// as block trees 302 and 238 ms.
constexpr int64_t TILE_MAX = 2048;

static bool tile_structure(const hm_handle* h, std::vector<int32_t>& gcl, std::vector<int32_t>& diag_node) {
  const int64_t ncl = (int64_t)h->cl_s.size();
  auto by_start = [&](int32_t a, int32_t b) { return h->cl_s[a] < h->cl_s[b]; };
  auto rows = [&](int64_t c) { return h->cl_e[c] - h->cl_s[c]; };
  auto largest = [&] {
    int64_t m = 0;
    for (int32_t c : gcl) m = std::max(m, rows(c));
    return m;
  };
  std::vector<char> is_row(ncl, 0);
  for (auto& L : h->leaves) is_row[L.s] = 1;
  // the highest clusters of at most `most` rows that are a leaf's row cluster or lie below one
  auto highest = [&](int64_t most) {
    std::vector<char> covered(ncl, 0), below(ncl, 0);
    gcl.clear();
    for (int64_t c = 0; c < ncl; ++c) {
      const bool row = is_row[c] || below[c];
      const bool take = !covered[c] && row && (rows(c) <= most || h->cl_left[c] < 0);
      if (take) gcl.push_back((int32_t)c);
      if (h->cl_left[c] >= 0)
        for (int64_t ch : {h->cl_left[c], h->cl_right[c]}) {
          covered[ch] = covered[c] || take;
          below[ch] = row;
        }
    }
    std::sort(gcl.begin(), gcl.end(), by_start);
    return tile_check(h, gcl, diag_node);
  };
  if (highest(TILE_MAX)) return true;
  std::vector<int32_t> first, first_node;       // a tiling with a larger tile
  if (highest(INT64_MAX)) {
    first = gcl;
    first_node = diag_node;
  }
  int maxd = 0;
  for (int64_t c = 0; c < ncl; ++c) maxd = std::max(maxd, (int)h->cl_depth[c]);
  for (int d = 1; d <= maxd; ++d) {
    gcl.clear();
    int64_t cover = 0;
    for (int64_t c = 0; c < ncl; ++c)
      if (h->cl_depth[c] == d) {
        gcl.push_back((int32_t)c);
        cover += rows(c);
      }
    if (cover != h->n) break;                   // a cluster leaf above depth d: no deeper level covers
    std::sort(gcl.begin(), gcl.end(), by_start);
    if (!tile_check(h, gcl, diag_node)) continue;
    if (largest() <= TILE_MAX) return true;
    if (first.empty()) {
      first = gcl;
      first_node = diag_node;
    }
  }
  gcl.swap(first);
  diag_node.swap(first_node);
  return !gcl.empty();
}

// The recompressions of step k's pairs (tile_pair's mode), every launch sized
// without knowing a rank: first all pairs by the register kernel, whose pairs
// of larger rank go on a list for the next kernel, to the last one, which
// takes any rank the capacity allows.  ws: the lists and their counts.
struct PairLists {
  int32_t* list[3];          // [T (T - 1)] each
  int* count;                // [8]
  void* scratch;             // of the last kernel: blocks x 2 smax rl
  int smax, blocks;
};
template <typename TS>
static void recompress_pairs_t(Ctx& c, const TileLU& TL, const PairLists& W, int k, int mode) {
  const int T = TL.T;
  const int64_t njobs = tile_pair_count(T, k, mode);
  if (njobs <= 0) return;
  if (njobs > INT32_MAX) throw LuError(HM_ERR_UNSUPPORTED, "too many tile pairs");
  HM_LU_CUDA(cudaMemsetAsync(W.count, 0, 8 * sizeof(int), c.st));
  PairArgs a{};
  a.Ap = (double* const*)TL.d_Ap; a.Bp = (double* const*)TL.d_Bp; a.size = TL.d_size; a.kmat = TL.kmat;
  a.T = T; a.cap = c.cap; a.k = k; a.mode = mode; a.eps = c.eps_trunc; a.flags = c.flags;
  a.out = W.list[0]; a.nout = W.count;
  auto next = [&](int i) {             // the list just written becomes the input
    a.in = W.list[i]; a.nin = W.count + i;
    a.out = i < 2 ? W.list[i + 1] : nullptr; a.nout = i < 2 ? W.count + i + 1 : nullptr;
  };
  // what the later kernels take: up to 24 columns of 256 rows, or what else fits
  // twice on an SM, staged in shared memory; the rest in scratch.  Each follows
  // where some pair is left to it: the register kernels hold 12 columns, but only
  // of tiles of up to 512 rows.
  const int rl =
      (int)std::min<size_t>(24, (104 * 1024 - sizeof(double) * c.cap * c.cap) / (sizeof(TS) * (2 * W.smax + 3 * 25)));
  const int rmax = std::min(2 * c.cap, RCORE_MAX);
  const int taken = W.smax <= 512 ? 12 : 0;
  const bool staged = rl > taken && rmax > taken, scratch = rmax > std::max(rl, taken);
  auto smem = [&](int q, bool st) {
    return sizeof(TS) * ((size_t)3 * q * (q + 1) + (st ? (size_t)2 * W.smax * q : 0)) +
           (st ? sizeof(double) * c.cap * c.cap : 0);
  };
  const unsigned pers = (unsigned)std::min<int64_t>(njobs, 148 * 4);
  // the second register kernel; with nothing behind it a pair it cannot take is an error
  auto second = [&] {
    next(0);
    if (!staged && !scratch) a.out = nullptr;
  };
  if (W.smax <= 256) {
    lu_pair_kernel<TS, 1, 8><<<(unsigned)njobs, 64, 0, c.st>>>(a);
    LU_LAUNCH_CHECK();
    second();
    lu_pair_kernel<TS, 1, 12><<<pers, 64, 0, c.st>>>(a);
  } else {
    lu_pair_kernel<TS, 2, 8><<<(unsigned)njobs, 128, 0, c.st>>>(a);
    LU_LAUNCH_CHECK();
    second();
    lu_pair_kernel<TS, 2, 12><<<pers, 128, 0, c.st>>>(a);
  }
  LU_LAUNCH_CHECK();
  if (smem_attr((const void*)lu_tile_core_kernel<TS>, (int)sizeof(double) * 3 * RCORE_MAX * (RCORE_MAX + 1)) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "tile core smem");
  if (staged) {
    next(1);
    if (!scratch) a.out = nullptr;
    lu_tile_core_kernel<TS><<<std::min<unsigned>(pers, 148 * 2), TC_THREADS, smem(rl, true), c.st>>>(a, rl, W.smax, (TS*)nullptr);
    LU_LAUNCH_CHECK();
  }
  if (scratch) {
    next(staged ? 2 : 1);
    a.out = nullptr;
    // as many CTAs as are resident (at most 3 by their registers)
    const unsigned res = 148 * (unsigned)std::max<size_t>(1, std::min<size_t>(3, (size_t)227 * 1024 / (smem(rmax, false) + 4096)));
    lu_tile_core_kernel<TS><<<std::min({pers, res, (unsigned)W.blocks}), TC_THREADS, smem(rmax, false), c.st>>>(
        a, rmax, W.smax, (TS*)W.scratch);
    LU_LAUNCH_CHECK();
  }
}
static void recompress_pairs(Ctx& c, const TileLU& TL, const PairLists& W, int k, int mode) {
  // FP32 when the truncation tolerance is loose (>= 1e-6, the mixed-precision scheme)
  if (c.eps_trunc >= MIXED_CORE_EPS) recompress_pairs_t<float>(c, TL, W, k, mode);
  else recompress_pairs_t<double>(c, TL, W, k, mode);
}

static void tile_factor(Ctx& c, const hm_handle* h, TileLU& TL, const std::vector<int32_t>& gcl,
                        const std::vector<int32_t>& dnode, cudaStream_t look) {
  const int T = (int)gcl.size(), cap = c.cap;
  TL.T = T;
  TL.start.resize(T);
  TL.size.resize(T);
  for (int i = 0; i < T; ++i) {
    TL.start[i] = h->cl_s[gcl[i]];
    TL.size[i] = h->cl_e[gcl[i]] - h->cl_s[gcl[i]];
  }
  TL.hold = std::make_shared<Blk>();
  TL.hold->st = c.st;
  TL.Ap.resize(T);
  TL.Bp.resize(T);
  {
    size_t tot = arena_round(sizeof(int32_t) * T * T) + 2 * arena_round(sizeof(void*) * T) +
                 arena_round(sizeof(int64_t) * T) + arena_round(sizeof(int32_t) * T);
    for (int i = 0; i < T; ++i)
      tot += 2 * arena_round(sizeof(double) * TL.size[i] * T * cap) + arena_round(sizeof(double) * TL.size[i] * TL.size[i]);
    reserve(c, *TL.hold, tot);
  }
  for (int i = 0; i < T; ++i) {
    TL.Ap[i] = (double*)dmalloc(c, *TL.hold, sizeof(double) * TL.size[i] * T * cap);
    TL.Bp[i] = (double*)dmalloc(c, *TL.hold, sizeof(double) * TL.size[i] * T * cap);
  }
  TL.kmat = (int32_t*)dmalloc(c, *TL.hold, sizeof(int32_t) * T * T);
  {
    std::vector<const double*> ap(TL.Ap.begin(), TL.Ap.end()), bp(TL.Bp.begin(), TL.Bp.end());
    std::vector<int32_t> sz(TL.size.begin(), TL.size.end());
    TL.d_Ap = (const double**)dmalloc(c, *TL.hold, sizeof(void*) * T);
    TL.d_Bp = (const double**)dmalloc(c, *TL.hold, sizeof(void*) * T);
    TL.d_start = (int64_t*)dmalloc(c, *TL.hold, sizeof(int64_t) * T);
    TL.d_size = (int32_t*)dmalloc(c, *TL.hold, sizeof(int32_t) * T);
    if (cudaMemcpyAsync(TL.d_Ap, ap.data(), sizeof(void*) * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess ||
        cudaMemcpyAsync(TL.d_Bp, bp.data(), sizeof(void*) * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess ||
        cudaMemcpyAsync(TL.d_start, TL.start.data(), sizeof(int64_t) * T, cudaMemcpyHostToDevice, c.st) !=
            cudaSuccess ||
        cudaMemcpyAsync(TL.d_size, sz.data(), sizeof(int32_t) * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess ||
        cudaStreamSynchronize(c.st) != cudaSuccess)
      throw LuError(HM_ERR_CUDA, "tile tables");
  }
  if (cudaMemsetAsync(TL.kmat, 0, sizeof(int32_t) * T * T, c.st) != cudaSuccess) throw LuError(HM_ERR_CUDA, "memset");
  // load the off-diagonal tiles into the panels and the diagonal tiles as trees
  const int eb = elem_bytes(h->storage);
  std::vector<int32_t> kh(T * T, 0);
  auto tile_of = [&](int64_t r) {
    return (int)(std::upper_bound(TL.start.begin(), TL.start.end(), r) - TL.start.begin()) - 1;
  };
  Loader ld;
  const char* base = (const char*)h->d_rk;
  for (auto& L : h->leaves) {
    const int i0 = tile_of(L.row0), i1 = tile_of(L.row0 + L.m - 1);
    const int j0 = tile_of(L.col0), j1 = tile_of(L.col0 + L.n - 1);
    if (i0 == i1 && j0 == j1 && i0 == j0) continue;            // part of a diagonal tile's tree
    if (L.k > cap) throw LuError(HM_ERR_RANK, "leaf rank above the H-LU rank capacity");
    const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
    // a leaf spanning several tiles: tile (i, j) holds rows of A and of B
    for (int i = i0; i <= i1; ++i)
      for (int j = j0; j <= j1; ++j) {
        kh[i * T + j] = L.k;
        const int64_t ro = TL.start[i] - L.row0, co = TL.start[j] - L.col0;
        ld.jobs.push_back(LoadJob{base + (L.off + co) * eb, npad, (int)TL.size[j], L.k, h->storage,
                                  TL.Bj(i, j, cap), TL.size[j], cap, nullptr, 0});
        ld.jobs.push_back(LoadJob{base + (L.off + npad * L.k + ro) * eb, mpad, (int)TL.size[i], L.k, h->storage,
                                  TL.Ai(i, j, cap), TL.size[i], cap, nullptr, 0});
      }
  }
  if (cudaMemcpyAsync(TL.kmat, kh.data(), sizeof(int32_t) * T * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "rank upload");
  cudaStreamSynchronize(c.st);       // kh leaves scope before the async copy otherwise
  ld.flush(c);
  // the diagonal tiles: every leaf expanded into the dense tile, and the row
  // ranges of the diagonal leaves (the pivots stay inside them)
  TL.diag.resize(T);
  std::vector<int32_t> leaf;                       // tile by tile: leaf starts, then the size
  std::vector<int> leaf0(T), nleaf(T);
  int mmax = 1, smax = 1;
  {
    const int deb = dense_elem_bytes(h->storage), dt = h->storage == HM_F64 ? HM_F64 : HM_F32;
    std::vector<DiagLoad> jobs;
    std::vector<std::pair<int64_t, int>> cuts;     // (first row, rows) of a tile's diagonal leaves
    for (int i = 0; i < T; ++i) {
      const int S = (int)TL.size[i];
      smax = std::max(smax, S);
      TL.diag[i] = std::make_shared<Blk>();             // its array is TL.hold's
      TL.diag[i]->st = c.st;
      TL.diag[i]->type = T_DENSE;
      TL.diag[i]->m = TL.diag[i]->n = S;
      TL.diag[i]->s = TL.diag[i]->t = gcl[i];
      TL.diag[i]->C = (double*)dmalloc(c, *TL.hold, sizeof(double) * (size_t)S * S);
      TL.diag[i]->ldc = std::max(S, 1);
      TL.diag[i]->row0 = TL.start[i];
      cuts.clear();
      std::vector<int32_t> todo(1, dnode[i]);
      while (!todo.empty()) {
        const Node& nd = h->nodes[todo.back()];
        todo.pop_back();
        if (nd.type == T_H) {
          for (int q = 0; q < 4; ++q) todo.push_back(nd.child[q]);
          continue;
        }
        const Leaf& L = h->leaves[nd.leaf];
        DiagLoad J{};
        J.m = L.m; J.n = L.n; J.k = L.k; J.dense = nd.type == T_DENSE; J.ctype = dt; J.rtype = h->storage;
        J.dst = TL.diag[i]->C + (L.row0 - TL.start[i]) + (L.col0 - TL.start[i]) * (int64_t)S;
        J.ldd = S;
        if (J.dense) {
          J.C = (const char*)h->d_dense + L.off * deb;
          J.ldc = col_pad(L.m, deb);
        } else {
          const int64_t npad = col_pad(L.n, eb), mpad = col_pad(L.m, eb);
          J.B = base + L.off * eb;
          J.ldb = npad;
          J.A = base + (L.off + npad * L.k) * eb;
          J.lda = mpad;
        }
        jobs.push_back(J);
        if (nd.s == nd.t) {
          if (!J.dense || L.m != L.n) throw LuError(HM_ERR_UNSUPPORTED, "H should not be a low-rank matrix");
          cuts.push_back({L.row0 - TL.start[i], L.m});
          mmax = std::max(mmax, L.m);
        }
      }
      std::sort(cuts.begin(), cuts.end());
      leaf0[i] = (int)leaf.size();
      nleaf[i] = (int)cuts.size();
      int64_t next = 0;
      for (auto& q : cuts) {
        if (q.first != next) throw LuError(HM_ERR_UNSUPPORTED, "diagonal leaves do not cover their tile");
        leaf.push_back((int32_t)q.first);
        next += q.second;
      }
      if (next != S) throw LuError(HM_ERR_UNSUPPORTED, "diagonal leaves do not cover their tile");
      leaf.push_back(S);
    }
    if (mmax > LU_LEAF_MAX) leaf_too_large();
    for (size_t b = 0; b < jobs.size(); b += (size_t)1 << 30) {
      const size_t nb = std::min<size_t>((size_t)1 << 30, jobs.size() - b);
      Blk tmp;
      tmp.st = c.st;
      std::vector<DiagLoad> part(jobs.begin() + b, jobs.begin() + b + nb);
      lu_diag_load_kernel<<<dim3((unsigned)nb, 4), 256, 0, c.st>>>(upload_jobs(c, tmp, part));
      LU_LAUNCH_CHECK();
    }
  }
  int32_t* d_leaf = (int32_t*)dmalloc(c, *TL.hold, sizeof(int32_t) * leaf.size());
  double** d_D = (double**)dmalloc(c, *TL.hold, sizeof(void*) * T);
  {
    std::vector<double*> D(T);
    for (int i = 0; i < T; ++i) D[i] = TL.diag[i]->C;
    if (cudaMemcpyAsync(d_leaf, leaf.data(), sizeof(int32_t) * leaf.size(), cudaMemcpyHostToDevice, c.st) != cudaSuccess ||
        cudaMemcpyAsync(d_D, D.data(), sizeof(void*) * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess ||
        cudaStreamSynchronize(c.st) != cudaSuccess)
      throw LuError(HM_ERR_CUDA, "diagonal tile tables");
  }
  // the LU kernel by the largest leaf
  const void* diag_fn = mmax <= 32 ? (const void*)lu_diag_kernel<32> : mmax <= 64 ? (const void*)lu_diag_kernel<64>
                                                                                : (const void*)lu_diag_kernel<160>;
  const int M = mmax <= 32 ? 32 : mmax <= 64 ? 64 : 160;
  const size_t diag_smem = M == 32 ? diag_lu_smem<32>() : M == 64 ? diag_lu_smem<64>() : diag_lu_smem<160>();
  const bool panel_sm = tp_smem(smax) <= 220 * 1024;     // a panel's columns fit in shared memory
  if (smem_attr(diag_fn, (int)diag_smem) != cudaSuccess ||
      (panel_sm && smem_attr((const void*)lu_panel_kernel, 220 * 1024) != cudaSuccess))
    throw LuError(HM_ERR_CUDA, "tile kernels smem");

  // Step k: the diagonal tile's LU and the panels (x: the stream they run on),
  // then the trailing update.  With a look-ahead stream, the LU and panels of
  // tile k+1 run there as soon as step k has updated tile row and column k+1,
  // overlapping the rest of step k's update on the main stream.
  auto panels = [&](Ctx& x, int k) {
    const int mk = (int)TL.size[k];
    const int R = (T - k - 1) * cap;
    DiagLu dl{TL.diag[k]->C, mk, nleaf[k], d_leaf + leaf0[k], x.P, TL.start[k], x.flags};
    if (M == 32) lu_diag_kernel<32><<<DL_CTAS, 32 * DL_WARPS, diag_smem, x.st>>>(dl);
    else if (M == 64) lu_diag_kernel<64><<<DL_CTAS, 32 * DL_WARPS, diag_smem, x.st>>>(dl);
    else lu_diag_kernel<160><<<DL_CTAS, 32 * DL_WARPS, diag_smem, x.st>>>(dl);
    LU_LAUNCH_CHECK();
    if (k > 0) laswp(x, View{TL.Ap[k], 1, mk, mk, k * cap}, TL.start[k]);
    if (R == 0) return;
    View Ua{TL.Ai(k, k + 1, cap), 1, mk, mk, R};          // A factors of tiles (k, j>k)
    View Lb{TL.Bj(k + 1, k, cap), 1, mk, mk, R};          // B factors of tiles (i>k, k)
    if (panel_sm) {                                       // L_kk^{-1} P_k A_kj and B_ik' U_kk^{-1}
      PanelArgs pa{TL.diag[k]->C, mk, T, k, cap, x.P, TL.start[k], TL.Ap[k], TL.Bp[k], TL.kmat};
      lu_panel_kernel<<<dim3((T - k - 1 + TP_TILES - 1) / TP_TILES, 2), 256, tp_smem(mk), x.st>>>(pa);
      LU_LAUNCH_CHECK();
    } else {
      laswp(x, Ua, TL.start[k]);
      mfs(x, *TL.diag[k], Ua, true, true);
      mfs(x, *TL.diag[k], vtr(Lb), false, false);
    }
  };
  // updates of the trailing diagonal tiles i in [i0, i1)
  auto diag_updates = [&](int k, int i0, int i1) {
    if (i1 <= i0) return;
    DiagUpdate du{TL.d_Ap, TL.d_Bp, d_D, TL.d_size, TL.kmat, T, cap, k, i0};
    lu_diag_update_kernel<<<dim3((smax + 31) / 32, i1 - i0), 256, sizeof(double) * (cap * cap + 32 * cap), c.st>>>(du);
    LU_LAUNCH_CHECK();
  };
  Ctx cl = c;
  cl.st = look;
  cudaEvent_t ev_up = nullptr, ev_dn = nullptr;
  if (look && (cudaEventCreateWithFlags(&ev_up, cudaEventDisableTiming) != cudaSuccess ||
               cudaEventCreateWithFlags(&ev_dn, cudaEventDisableTiming) != cudaSuccess))
    throw LuError(HM_ERR_CUDA, "look-ahead events");
  struct EvGuard {
    cudaEvent_t a, b;
    cudaStream_t s;
    ~EvGuard() {
      if (s) cudaStreamSynchronize(s);
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
    }
  } evg{ev_up, ev_dn, look};
  // lists of the pairs each recompression kernel leaves to the next, and the
  // last one's scratch
  Blk wsb;
  wsb.st = c.st;
  PairLists ws{};
  ws.smax = smax;
  const size_t per = sizeof(double) * ((size_t)2 * smax * std::min(2 * cap, RCORE_MAX) + cap * cap);
  ws.blocks = (int)std::max<size_t>(16, std::min<size_t>(148 * 3, ((size_t)256 << 20) / per));
  reserve(c, wsb, std::size(ws.list) * arena_round(sizeof(int32_t) * (size_t)T * T) + arena_round(8 * sizeof(int)) +
                      arena_round(per * ws.blocks));
  for (auto& l : ws.list) l = (int32_t*)dmalloc(c, wsb, sizeof(int32_t) * (size_t)T * T);
  ws.count = (int*)dmalloc(c, wsb, 8 * sizeof(int));
  ws.scratch = dmalloc(c, wsb, per * ws.blocks);
  panels(c, 0);
  for (int k = 0; k + 1 < T; ++k) {
    if (look) {
      diag_updates(k, k + 1, k + 2);
      recompress_pairs(c, TL, ws, k, 1);                  // tile row and column k+1
      if (cudaEventRecord(ev_up, c.st) != cudaSuccess || cudaStreamWaitEvent(look, ev_up, 0) != cudaSuccess)
        throw LuError(HM_ERR_CUDA, "look-ahead wait");
      panels(cl, k + 1);
      if (cudaEventRecord(ev_dn, look) != cudaSuccess) throw LuError(HM_ERR_CUDA, "look-ahead record");
      recompress_pairs(c, TL, ws, k, 2);                  // the rest
      diag_updates(k, k + 2, T);
      if (cudaStreamWaitEvent(c.st, ev_dn, 0) != cudaSuccess) throw LuError(HM_ERR_CUDA, "look-ahead join");
    } else {
      diag_updates(k, k + 1, T);
      recompress_pairs(c, TL, ws, k, 0);
      panels(c, k + 1);
    }
  }
}

// ---- sweep solve ---------------------------------------------------------
// The triangular solves over the tile level as one kernel per tile: step k of
// a sweep finishes tile k (the update from the tile finished at step k-1, then
// the diagonal tile's triangular solve) in a few finisher CTAs, while the
// other CTAs apply the same finished tile's update to every later tile: 2T
// launches a solve.  The diagonal solves multiply by the inverses of the
// diagonal tiles' L and U factors (computed once from the factored tiles), so
// a step has no row-by-row dependency chain.
constexpr int SW_THREADS = 256;

struct SweepTab {
  const double* const* Ap;
  const double* const* Bp;
  // per tile, the inverse factor sweep_finish applies for which = 0, 1, 2, 3
  const double* const* Inv0;
  const double* const* Inv1;
  const double* const* Inv2;
  const double* const* Inv3;
  const int64_t* start;
  const int32_t* size;
  const int32_t* kmat;
  int T, cap;
};

// The low-rank factors of tile (i, s) as used by a sweep step: y_i -= P (Q' y_s)
// with, non-transposed, P = A_is and Q = B_is (tile (i,s) = A B') and,
// transposed, P = B_si and Q = A_si (tile (s,i)' = B A'); r is the rank.
__device__ __forceinline__ void sweep_factors(const SweepTab& t, int i, int s, bool trans, const double*& P,
                                              const double*& Q, int& r) {  // inlined: no addresses taken
  const int Si = t.size[i], Ss = t.size[s];
  if (!trans) {
    P = t.Ap[i] + (int64_t)s * t.cap * Si;
    Q = t.Bp[s] + (int64_t)i * t.cap * Ss;
    r = t.kmat[i * t.T + s];
  } else {
    P = t.Bp[i] + (int64_t)s * t.cap * Si;
    Q = t.Ap[s] + (int64_t)i * t.cap * Ss;
    r = t.kmat[s * t.T + i];
  }
}

// zsh[q + c r] = (Q' y_s)[q, c], y_s = the finished tile s in F.  Plain loads
// of y_s: the step that writes it may still run when this one starts (dependent
// launches), and the non-coherent load asks for data nobody writes meanwhile.
__device__ void sweep_z(const SweepTab& t, const double* F, int64_t ldy, int nc, int s, const double* Q, int r,
                        double* zsh) {
  const int Ss = t.size[s];
  const double* ys = F + t.start[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int qc = warp; qc < r * nc; qc += SW_THREADS / 32) {
    const int q = qc % r, cc = qc / r;
    double acc = 0.0;
#pragma unroll 8
    for (int row = lane; row < Ss; row += 32)
      acc = fma(__ldg(Q + row + (int64_t)q * Ss), ys[row + cc * ldy], acc);
    acc = warp_sum(acc);
    if (lane == 0) zsh[q + cc * r] = acc;
  }
  __syncthreads();
}

// Each step's launch may start while the previous one runs (programmatic
// dependent launch): what does not depend on it -- the inverse's rows, the
// factor columns of the first dot products -- is loaded before the wait, so a
// step costs one round of dependent loads instead of a launch and four.
__device__ __forceinline__ void sweep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void sweep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// this warp's first factor column of Q (rows lane + 32 j), and its dot product
// with y_s; later columns and rows past SW_QREG loads go the plain way
constexpr int SW_QREG = 12;
__device__ __forceinline__ void sweep_q_prefetch(const double* Q, int r, int Ss, int warp, int lane, double (&qreg)[SW_QREG]) {
#pragma unroll
  for (int j = 0; j < SW_QREG; ++j) {
    const int row = lane + 32 * j;
    qreg[j] = warp < r && row < Ss ? __ldg(Q + row + (int64_t)warp * Ss) : 0.0;
  }
}
// one column of z = Q' y_s into zsh (no barrier); yreg: y_s at this lane's rows
__device__ __forceinline__ void sweep_z1(const double* Q, const double* ys, int r, int Ss, int warp, int lane,
                                         const double (&qreg)[SW_QREG], const double (&yreg)[SW_QREG], double* zsh) {
  for (int q = warp; q < r; q += SW_THREADS / 32) {
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < SW_QREG; ++j) {
      const int row = lane + 32 * j;
      const double v = q == warp ? qreg[j] : (row < Ss ? __ldg(Q + row + (int64_t)q * Ss) : 0.0);
      acc = fma(v, yreg[j], acc);
    }
    for (int row = lane + 32 * SW_QREG; row < Ss; row += 32) acc = fma(__ldg(Q + row + (int64_t)q * Ss), ys[row], acc);
    acc = warp_sum(acc);
    if (lane == 0) zsh[q] = acc;
  }
}

// A_i -= P (Q' y_s): the finished tile s applied to the pending tile i
__device__ void sweep_update(const SweepTab& t, double* A, const double* F, int64_t ldy, int nc, int i, int s,
                             bool trans, double* zsh) {
  const double* P;
  const double* Q;
  int r;
  sweep_factors(t, i, s, trans, P, Q, r);
  const int Si = t.size[i], Ss = t.size[s], warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double qreg[SW_QREG];
  sweep_q_prefetch(Q, r, Ss, warp, lane, qreg);
  sweep_wait();
  if (r <= 0) return;
  double* yi = A + t.start[i];
  const double* ys = F + t.start[s];
  if (nc == 1) {
    double yreg[SW_QREG], preg[8];
#pragma unroll
    for (int j = 0; j < SW_QREG; ++j) yreg[j] = lane + 32 * j < Ss ? ys[lane + 32 * j] : 0.0;
    const int row = threadIdx.x;                          // this thread's first row
    const double y0 = row < Si ? yi[row] : 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) preg[q] = q < r && row < Si ? __ldg(P + row + (int64_t)q * Si) : 0.0;
    sweep_z1(Q, ys, r, Ss, warp, lane, qreg, yreg, zsh);
    __syncthreads();
    if (row < Si) {
      double acc = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < r) acc = fma(preg[q], zsh[q], acc);
      for (int q = 8; q < r; ++q) acc = fma(__ldg(P + row + (int64_t)q * Si), zsh[q], acc);
      yi[row] = y0 - acc;
    }
    for (int e = row + SW_THREADS; e < Si; e += SW_THREADS) {
      double acc = 0.0;
      for (int q = 0; q < r; ++q) acc = fma(__ldg(P + e + (int64_t)q * Si), zsh[q], acc);
      yi[e] -= acc;
    }
    return;
  }
  sweep_z(t, F, ldy, nc, s, Q, r, zsh);
  for (int e = threadIdx.x; e < Si * nc; e += SW_THREADS) {
    const int row = e % Si, cc = e / Si;
    double acc = 0.0;
#pragma unroll 8
    for (int q = 0; q < r; ++q) acc = fma(__ldg(P + row + (int64_t)q * Si), zsh[q + cc * r], acc);
    yi[row + cc * ldy] -= acc;
  }
}

// Finisher f of tile k: SW_ROWS rows from f SW_ROWS on of M (A_k - P (Q' y_s))
// written to F, where M = Inv[which][k] (M[q*S + r] = M(r, q); which 0 and 2
// lower, 1 and 3 upper).  A half warp per segment of the columns q the rows
// need, a lane per row: each thread loads its part of M into registers before
// the wait, then the update of tile k from the finished tile s (if any) is
// recomputed for the rows q needed, and the 16 segment sums of a row are added
// in shared memory.
constexpr int SW_MREG = 24;
constexpr int SW_ROWS = 16;
constexpr int SW_SEGS = SW_THREADS / SW_ROWS;
__device__ void sweep_finish(const SweepTab& t, const double* A, double* F, int64_t ldy, int nc, int k, int s,
                             bool has_src, bool trans, int which, int f, int chunk, double* sh) {
  const int S = t.size[k];
  const int r0 = f * SW_ROWS, r1 = min(S, r0 + SW_ROWS), nr = r1 - r0;
  const bool lower = which == 0 || which == 2;
  const int qa = lower ? 0 : r0, qb = lower ? r1 : S, span = qb - qa;
  const int segl = (span + SW_SEGS - 1) / SW_SEGS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = lane % SW_ROWS, seg = threadIdx.x / SW_ROWS;
  const bool row_ok = rl < nr;
  const int qs = qa + seg * segl;                     // this thread's columns [qs, qs + segl)
  const double* const* inv = which == 0 ? t.Inv0 : which == 1 ? t.Inv1 : which == 2 ? t.Inv2 : t.Inv3;
  const double* M = inv[k] + r0 + rl;                 // M(r0 + rl, q) = M[q*S]
  double mreg[SW_MREG];
#pragma unroll
  for (int j = 0; j < SW_MREG; ++j)
    mreg[j] = (row_ok && j < segl && qs + j < qb) ? __ldg(M + (int64_t)(qs + j) * S) : 0.0;
  double* ysh = sh;                                   // span x chunk
  double* part = ysh + (size_t)S * chunk;             // SW_SEGS x SW_ROWS x chunk
  double* zsh = part + (size_t)SW_THREADS * chunk;    // cap x nc
  const double* P = nullptr;
  const double* Q = nullptr;
  int r = 0;
  if (has_src) sweep_factors(t, k, s, trans, P, Q, r);
  const int Ss = has_src ? t.size[s] : 0;
  const double* ys = F + (has_src ? t.start[s] : 0);
  const double* yk = A + t.start[k];
  double* out = F + t.start[k];
  double qreg[SW_QREG];
  sweep_q_prefetch(Q, r, Ss, warp, lane, qreg);
  sweep_wait();
  if (nr <= 0) return;
  auto times_m = [&](const double* yv) {              // this thread's part of its row of M yv
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < SW_MREG; ++j)
      if (j < segl && qs + j < qb) acc = fma(mreg[j], yv[qs + j], acc);
    if (row_ok)                                       // segments longer than the registers hold
#pragma unroll 8
      for (int q = qs + SW_MREG; q < min(qs + segl, qb); ++q) acc = fma(__ldg(M + (int64_t)q * S), yv[q], acc);
    return acc;
  };
  if (nc == 1) {
    double yreg[SW_QREG], preg[8];
#pragma unroll
    for (int j = 0; j < SW_QREG; ++j) yreg[j] = r > 0 && lane + 32 * j < Ss ? ys[lane + 32 * j] : 0.0;
    const int q0 = threadIdx.x;
    const double y0 = q0 < span ? yk[qa + q0] : 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) preg[j] = j < r && q0 < span ? __ldg(P + qa + q0 + (int64_t)j * S) : 0.0;
    if (r > 0) sweep_z1(Q, ys, r, Ss, warp, lane, qreg, yreg, zsh);
    __syncthreads();
    if (q0 < span) {
      double v = y0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < r) v = fma(-preg[j], zsh[j], v);
      for (int j = 8; j < r; ++j) v = fma(-__ldg(P + qa + q0 + (int64_t)j * S), zsh[j], v);
      ysh[q0] = v;
    }
    for (int q = q0 + SW_THREADS; q < span; q += SW_THREADS) {
      double v = yk[qa + q];
      for (int j = 0; j < r; ++j) v = fma(-__ldg(P + qa + q + (int64_t)j * S), zsh[j], v);
      ysh[q] = v;
    }
    __syncthreads();
    part[threadIdx.x] = times_m(ysh - qa);
    __syncthreads();
    if (threadIdx.x < nr) {
      double acc = 0.0;
#pragma unroll
      for (int w = 0; w < SW_SEGS; ++w) acc += part[w * SW_ROWS + threadIdx.x];
      out[r0 + threadIdx.x] = acc;
    }
    return;
  }
  if (r > 0) sweep_z(t, F, ldy, nc, s, Q, r, zsh);
  for (int c0 = 0; c0 < nc; c0 += chunk) {
    const int ncc = min(chunk, nc - c0);
    __syncthreads();                                  // ysh and part free
    for (int e = threadIdx.x; e < span * ncc; e += SW_THREADS) {
      const int q = e % span, cc = e / span;
      double v = yk[qa + q + (int64_t)(c0 + cc) * ldy];
#pragma unroll 8
      for (int j = 0; j < r; ++j) v = fma(-__ldg(P + qa + q + (int64_t)j * S), zsh[j + (c0 + cc) * r], v);
      ysh[q + cc * span] = v;
    }
    __syncthreads();
    for (int cc = 0; cc < ncc; ++cc) part[cc * SW_THREADS + threadIdx.x] = times_m(ysh + cc * span - qa);
    __syncthreads();
    for (int e = threadIdx.x; e < nr * ncc; e += SW_THREADS) {
      const int ii = e % nr, cc = e / nr;
      double acc = 0.0;
#pragma unroll
      for (int w = 0; w < SW_SEGS; ++w) acc += part[cc * SW_THREADS + w * SW_ROWS + ii];
      out[r0 + ii + (int64_t)(c0 + cc) * ldy] = acc;
    }
  }
}

// Step k of a sweep (dir +1 forward, -1 backward; which: 0 L, 1 U, 2 U', 3 L').
// A holds the pending right-hand sides, F receives the finished tiles; the
// finished tile s = k - dir is applied to tile k by the nf finisher CTAs and
// to every later tile of the sweep by one CTA each.  Bound: the latency of the
// chain of steps (grid completion, y_s, two barriers, 24 FMAs a thread).  64
// tiles of 312 rows, one column: 13.4 us a step with plain launches and a warp
// per row of M, 4.9 us so; a solve at n = 65536 (256 tiles) 1.7 ms, was 6.7.
__global__ void __launch_bounds__(SW_THREADS, 2) lu_sweep_kernel(SweepTab t, double* A, double* F, int64_t ldy,
                                                              int nc, int k, int dir, int which, int nf, int chunk) {
  extern __shared__ double sh[];
  sweep_release();
  const bool trans = which >= 2;
  const int s = k - dir;
  const bool has_src = s >= 0 && s < t.T;
  if ((int)blockIdx.x < nf) sweep_finish(t, A, F, ldy, nc, k, s, has_src, trans, which, blockIdx.x, chunk, sh);
  else if (has_src) sweep_update(t, A, F, ldy, nc, k + dir * ((int)blockIdx.x - nf + 1), s, trans, sh);
  else sweep_wait();
}

// The same inverses for tiles whose columns do not fit in shared memory, of the
// unit-lower L (upper = 0) or the upper U (upper = 1) of the
// packed S x S tiles D (column-major), one thread per column of the inverse,
// written row-major to W (W[i*S + j] = inverse(i, j)) and column-major to Wc.
// All threads of a tile run the same substitution, so the reads of D are
// broadcasts and the reads and writes of W are coalesced.
__global__ void lu_tri_inverse_kernel(const double* const* __restrict__ D, double* const* __restrict__ W,
                                      double* const* __restrict__ Wc, const int32_t* __restrict__ size, int upper) {
  const int tile = blockIdx.y;
  const int S = size[tile];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x * blockDim.x >= S) return;
  const double* d = D[tile];
  double* w = W[tile];
  double* wc = Wc[tile];
  const bool act = j < S;
  if (!upper) {
    for (int i = 0; i < S; ++i) {
      double s = (i == j) ? 1.0 : 0.0;
      for (int l = 0; l < i; ++l) s = fma(-d[i + (int64_t)l * S], act ? w[(int64_t)l * S + j] : 0.0, s);
      if (act) {
        const double v = (i < j) ? 0.0 : s;
        w[(int64_t)i * S + j] = v;
        wc[i + (int64_t)j * S] = v;
      }
    }
  } else {
    for (int i = S - 1; i >= 0; --i) {
      double s = (i == j) ? 1.0 : 0.0;
      for (int l = i + 1; l < S; ++l) s = fma(-d[i + (int64_t)l * S], act ? w[(int64_t)l * S + j] : 0.0, s);
      if (act) {
        const double v = (i > j) ? 0.0 : s / d[i + (int64_t)i * S];
        w[(int64_t)i * S + j] = v;
        wc[i + (int64_t)j * S] = v;
      }
    }
  }
}

// inverse factors and device tables, once per factorisation
static void ensure_sweep(Ctx& c, TileLU& TL) {
  if (TL.d_inv[0]) return;
  const int T = TL.T;
  auto hold = std::make_shared<Blk>();
  hold->st = c.st;
  Blk tmp;
  tmp.st = c.st;
  int smax = 0;
  std::vector<double*> D(T);
  std::vector<const double*> inv[4];         // Lc, Uc, Ur, Lr: the matrices of which = 0..3
  {
    size_t tot = 4 * arena_round(sizeof(void*) * T);
    for (int k = 0; k < T; ++k) tot += 4 * arena_round(sizeof(double) * (size_t)TL.size[k] * TL.size[k]);
    reserve(c, *hold, tot);
  }
  for (int k = 0; k < T; ++k) {
    const int S = (int)TL.size[k];
    smax = std::max(smax, S);
    D[k] = TL.diag[k]->C;
    for (int w = 0; w < 4; ++w) inv[w].push_back((double*)dmalloc(c, *hold, sizeof(double) * (size_t)S * S));
  }
  std::vector<int32_t> sz(T);
  for (int k = 0; k < T; ++k) sz[k] = (int32_t)TL.size[k];
  std::vector<const double*> Ap(TL.Ap.begin(), TL.Ap.end()), Bp(TL.Bp.begin(), TL.Bp.end());
  auto up = [&](const void* src, size_t bytes) {
    void* d = dmalloc(c, *hold, bytes);
    if (cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, c.st) != cudaSuccess)
      throw LuError(HM_ERR_CUDA, "sweep tables");
    return d;
  };
  double** dD = (double**)dmalloc(c, tmp, sizeof(void*) * T);
  if (cudaMemcpyAsync(dD, D.data(), sizeof(void*) * T, cudaMemcpyHostToDevice, c.st) != cudaSuccess)
    throw LuError(HM_ERR_CUDA, "sweep tables");
  if (!TL.d_Ap) {                            // a copied factorisation has no tables yet
    TL.d_Ap = (const double**)up(Ap.data(), sizeof(void*) * T);
    TL.d_Bp = (const double**)up(Bp.data(), sizeof(void*) * T);
    TL.d_start = (int64_t*)up(TL.start.data(), sizeof(int64_t) * T);
    TL.d_size = (int32_t*)up(sz.data(), sizeof(int32_t) * T);
  }
  for (int w = 0; w < 4; ++w) TL.d_inv[w] = (const double**)up(inv[w].data(), sizeof(void*) * T);
  // L^-1: row-major (which 3) and column-major (which 0); U^-1: row-major (2), column-major (1)
  if (tp_smem(smax) <= 220 * 1024) {
    if (smem_attr((const void*)lu_inverse_kernel, 220 * 1024) != cudaSuccess) throw LuError(HM_ERR_CUDA, "inverse smem");
    InverseArgs ia{dD, {(double* const*)TL.d_inv[0], (double* const*)TL.d_inv[1]},
                   {(double* const*)TL.d_inv[3], (double* const*)TL.d_inv[2]}, TL.d_size};
    for (int t = 0; t < T; t += 65535) {       // grid.y
      InverseArgs b = ia;
      for (int w = 0; w < 2; ++w) { b.C[w] += t; b.R[w] += t; }
      b.D += t;
      b.size += t;
      lu_inverse_kernel<<<dim3((smax + TP_COLS - 1) / TP_COLS, std::min(65535, T - t), 2), 256, tp_smem(smax), c.st>>>(b);
      LU_LAUNCH_CHECK();
    }
  } else {
    const dim3 g((smax + 127) / 128, T);
    lu_tri_inverse_kernel<<<g, 128, 0, c.st>>>(dD, (double* const*)TL.d_inv[3], (double* const*)TL.d_inv[0],
                                               TL.d_size, 0);
    LU_LAUNCH_CHECK();
    lu_tri_inverse_kernel<<<g, 128, 0, c.st>>>(dD, (double* const*)TL.d_inv[2], (double* const*)TL.d_inv[1],
                                               TL.d_size, 1);
    LU_LAUNCH_CHECK();
  }
  if (cudaStreamSynchronize(c.st) != cudaSuccess) throw LuError(HM_ERR_CUDA, "sweep set-up");
  TL.sweep_hold = hold;
}

static void tile_solve(Ctx& c, const TileLU& TL, View X, bool trans, double* Zext);

// the two sweeps of a\y (trans 0) or a'\y (trans 1) on X in place (X already
// permuted for a\y; permuted afterwards by the caller for a'\y).  The
// forward sweep finishes tiles into a second array W, the backward sweep
// takes W as its right-hand sides and finishes into X.
static void tile_sweeps(Ctx& c, const TileLU& TL, View X, bool trans) {
  const int T = TL.T, nc = X.cols;
  int smax = 1;
  for (int k = 0; k < T; ++k) smax = std::max<int>(smax, (int)TL.size[k]);
  const int chunk = std::min(nc, 8);                               // columns staged per pass
  const size_t smem = sizeof(double) * ((size_t)smax * chunk + (size_t)SW_THREADS * chunk + (size_t)c.cap * nc);
  if (smem > 200 * 1024 || X.rs != 1) {
    tile_solve(c, TL, X, trans, nullptr);
    return;
  }
  if (smem_attr((const void*)lu_sweep_kernel, 200 * 1024) != cudaSuccess) throw LuError(HM_ERR_CUDA, "sweep smem");
  Blk tmp;
  tmp.st = c.st;
  double* W = (double*)dmalloc(c, tmp, sizeof(double) * (size_t)X.cs * nc);
  SweepTab t{TL.d_Ap, TL.d_Bp, TL.d_inv[0], TL.d_inv[1], TL.d_inv[2], TL.d_inv[3], TL.d_start, TL.d_size,
             TL.kmat, T, c.cap};
  // the first launch is a plain one: what it loads early is then complete
  auto step = [&](double* A, double* F, int k, int dir, int which, bool overlap) {
    const int nf = ((int)TL.size[k] + SW_ROWS - 1) / SW_ROWS;
    const int nu = dir > 0 ? (k > 0 ? T - 1 - k : 0) : (k < T - 1 ? k : 0);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(nf + nu));
    cfg.blockDim = dim3(SW_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    HM_LU_CUDA(cudaLaunchKernelEx(&cfg, lu_sweep_kernel, t, A, F, X.cs, nc, k, dir, which, nf, chunk));
  };
  for (int k = 0; k < T; ++k) step(X.p, W, k, 1, trans ? 2 : 0, k > 0);
  for (int k = T - 1; k >= 0; --k) step(W, X.p, k, -1, trans ? 3 : 1, true);
}

// y = P b, forward (unit L), backward (U) tile by tile; trans: U' then L'
// (the launch-per-operation form, used beyond SWEEP_MAX_COLS right-hand sides)
static void tile_solve(Ctx& c, const TileLU& TL, View X, bool trans, double* Zext) {
  const int T = TL.T, cap = c.cap, nc = X.cols;
  auto yv = [&](int i) { return vsub(X, (int)TL.start[i], 0, (int)TL.size[i], nc); };
  Blk tmp;
  tmp.st = c.st;
  double* Z = Zext ? Zext : (double*)dmalloc(c, tmp, sizeof(double) * (size_t)T * cap * nc);
  if (!trans) {
    for (int k = 0; k < T; ++k) {                       // L y = b
      solve_rec(c, *TL.diag[k], yv(k), true);
      const int R = (T - k - 1) * cap;
      if (R == 0) break;
      View Zv{Z, 1, R, R, nc};
      gemm(c, Zv, vtr(View{TL.Bj(k + 1, k, cap), 1, TL.size[k], (int)TL.size[k], R}), yv(k), 1.0, 0.0);
      std::vector<GemmJob> g;
      for (int i = k + 1; i < T; ++i)
        g.push_back(GemmJob{View{TL.Ai(i, k, cap), 1, TL.size[i], (int)TL.size[i], cap},
                            vsub(Zv, (i - k - 1) * cap, 0, cap, nc), yv(i), -1.0, 1.0});
      gemm_batch(c, g);
    }
    for (int k = T - 1; k >= 0; --k) {                  // U x = y
      const int R = (T - k - 1) * cap;
      if (R > 0) {
        View Zv{Z, 1, R, R, nc};
        std::vector<GemmJob> g;
        for (int j = k + 1; j < T; ++j)
          g.push_back(GemmJob{vtr(View{TL.Bj(k, j, cap), 1, TL.size[j], (int)TL.size[j], cap}), yv(j),
                              vsub(Zv, (j - k - 1) * cap, 0, cap, nc), 1.0, 0.0});
        gemm_batch(c, g);
        gemm(c, yv(k), View{TL.Ai(k, k + 1, cap), 1, TL.size[k], (int)TL.size[k], R}, Zv, -1.0, 1.0);
      }
      solve_rec(c, *TL.diag[k], yv(k), false);
    }
  } else {
    for (int k = 0; k < T; ++k) {                       // U' z = b
      solve_t_rec(c, *TL.diag[k], yv(k), true);
      const int R = (T - k - 1) * cap;
      if (R == 0) break;
      View Zv{Z, 1, R, R, nc};
      gemm(c, Zv, vtr(View{TL.Ai(k, k + 1, cap), 1, TL.size[k], (int)TL.size[k], R}), yv(k), 1.0, 0.0);
      std::vector<GemmJob> g;
      for (int j = k + 1; j < T; ++j)
        g.push_back(GemmJob{View{TL.Bj(k, j, cap), 1, TL.size[j], (int)TL.size[j], cap},
                            vsub(Zv, (j - k - 1) * cap, 0, cap, nc), yv(j), -1.0, 1.0});
      gemm_batch(c, g);
    }
    for (int k = T - 1; k >= 0; --k) {                  // L' w = z
      const int R = (T - k - 1) * cap;
      if (R > 0) {
        View Zv{Z, 1, R, R, nc};
        std::vector<GemmJob> g;
        for (int i = k + 1; i < T; ++i)
          g.push_back(GemmJob{vtr(View{TL.Ai(i, k, cap), 1, TL.size[i], (int)TL.size[i], cap}), yv(i),
                              vsub(Zv, (i - k - 1) * cap, 0, cap, nc), 1.0, 0.0});
        gemm_batch(c, g);
        gemm(c, yv(k), View{TL.Bj(k + 1, k, cap), 1, TL.size[k], (int)TL.size[k], R}, Zv, -1.0, 1.0);
      }
      solve_t_rec(c, *TL.diag[k], yv(k), false);
    }
  }
}

static void tile_densify(Ctx& c, const TileLU& TL, View D) {
  const int T = TL.T, cap = c.cap;
  std::vector<GemmJob> g;
  for (int i = 0; i < T; ++i)
    for (int j = 0; j < T; ++j) {
      View blk = vsub(D, (int)TL.start[i], (int)TL.start[j], (int)TL.size[i], (int)TL.size[j]);
      if (i == j) densify_into(c, blk, *TL.diag[i]);
      else
        g.push_back(GemmJob{View{TL.Ai(i, j, cap), 1, TL.size[i], (int)TL.size[i], cap},
                            vtr(View{TL.Bj(i, j, cap), 1, TL.size[j], (int)TL.size[j], cap}), blk, 1.0, 0.0});
    }
  gemm_batch(c, g);
}

// ---------------------------------------------------------------------------
// state, entry points
// ---------------------------------------------------------------------------
// One captured solve: the launch sequence of a\y (or a'\y) for a fixed number
// of right-hand sides, recorded into a CUDA graph that works on the plan's own
// input/output buffers.  A call copies b in, launches the graph, copies x out.
struct SolvePlan {
  int64_t ncols = 0;
  int trans = 0;
  double* xin = nullptr;   // n x ncols, right-hand sides (the transposed solve works in place here)
  double* xout = nullptr;  // n x ncols, solution
  double* Z = nullptr;     // tile-solve product scratch
  Arena arena;             // temporaries of the captured sequence
  JobTape tape;
  cudaGraphExec_t exec = nullptr;
  bool no_graph = false;   // capture failed: the plan runs its sequence directly
  ~SolvePlan() {           // the owner has synchronised the device
    if (exec) cudaGraphExecDestroy(exec);
    for (void* p : {(void*)xin, (void*)xout, (void*)Z, (void*)arena.base})
      if (p) cudaFreeAsync(p, cudaStreamLegacy);
  }
};

struct LuState {
  BP root;                       // recursive format
  std::unique_ptr<TileLU> tile;  // tile format
  int64_t* P = nullptr;
  int* flags = nullptr;
  int cap = 0;
  cudaStream_t st = nullptr;
  // look-ahead stream of the tile schedule (blocks made there keep it as
  // their stream, so it lives as long as the factors)
  cudaStream_t look = nullptr;
  std::vector<std::unique_ptr<SolvePlan>> plans;
  ~LuState() {
    if (!plans.empty()) cudaDeviceSynchronize();
    plans.clear();
    if (look) cudaStreamSynchronize(look);
    root.reset();
    tile.reset();
    if (P) cudaFreeAsync(P, st);
    if (flags) cudaFreeAsync(flags, st);
    if (st) cudaStreamSynchronize(st);
    if (look) {
      cudaStreamSynchronize(look);
      cudaStreamDestroy(look);
    }
  }
  // a second stream (nullptr if it cannot be made: the schedule then runs on
  // one stream)
  void make_look() {
    if (look) return;
    // high priority: its small kernels are scheduled between the blocks of the
    // main stream's large recompression launches instead of after them
    int least = 0, greatest = 0;
    cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (cudaStreamCreateWithPriority(&look, cudaStreamNonBlocking, greatest) != cudaSuccess) {
      cudaGetLastError();
      look = nullptr;
    }
  }
};

static BP build_tree(Ctx& c, const hm_handle* h, int32_t node, Loader& ld) {
  const Node& nd = h->nodes[node];
  const int m = (int)(h->cl_e[nd.s] - h->cl_s[nd.s]), n = (int)(h->cl_e[nd.t] - h->cl_s[nd.t]);
  if (nd.type == T_H) {
    BP b = std::make_shared<Blk>();
    b->st = c.st;
    b->type = T_H; b->m = m; b->n = n; b->s = nd.s; b->t = nd.t; b->row0 = h->cl_s[nd.s];
    for (int q = 0; q < 4; ++q) b->ch[q] = build_tree(c, h, nd.child[q], ld);
    return b;
  }
  const Leaf& L = h->leaves[nd.leaf];
  const int eb = elem_bytes(h->storage), deb = dense_elem_bytes(h->storage);
  if (nd.type == T_DENSE) {
    BP d = new_dense(c, m, n, nd.s, nd.t);
    d->row0 = L.row0;
    const int dt = h->storage == HM_F64 ? HM_F64 : HM_F32;
    ld.jobs.push_back(LoadJob{(const char*)h->d_dense + L.off * deb, col_pad(m, deb), m, n, dt, d->C, d->ldc, n,
                              nullptr, 0});
    return d;
  }
  if (L.k > c.cap) throw LuError(HM_ERR_RANK, "leaf rank above the H-LU rank capacity");
  BP r = new_rk(c, m, n, nd.s, nd.t);
  r->row0 = L.row0;
  const int64_t npad = col_pad(n, eb), mpad = col_pad(m, eb);
  const char* base = (const char*)h->d_rk;
  ld.jobs.push_back(LoadJob{base + L.off * eb, npad, n, L.k, h->storage, r->B, r->ldb, c.cap, nullptr, 0});
  ld.jobs.push_back(LoadJob{base + (L.off + npad * L.k) * eb, mpad, m, L.k, h->storage, r->A, r->lda, c.cap,
                            r->k, L.k});
  return r;
}

static BP build_from_handle(Ctx& c, const hm_handle* h, int32_t node) {
  Loader ld;
  BP b = build_tree(c, h, node, ld);
  ld.flush(c);
  return b;
}

static int finish(Ctx& c, const char* what) {
  int flags = 0;
  HM_CUDA_TRY(cudaMemcpyAsync(&flags, c.flags, sizeof(int), cudaMemcpyDeviceToHost, c.st));
  HM_CUDA_TRY(cudaStreamSynchronize(c.st));
  if (flags & 4) return fail(HM_ERR_SINGULAR, std::string(what) + ": exactly zero pivot in a diagonal leaf");
  if (flags & 2) return fail(HM_ERR_NONFINITE, std::string(what) + ": non-finite values");
  if (flags & 1) return fail(HM_ERR_RANK, std::string(what) + ": a rank exceeded the capacity " + std::to_string(c.cap));
  return HM_OK;
}

int lu_factor(hm_handle* h) {
  // the factorisation allocates and frees many stream-ordered temporaries:
  // keep freed memory in the device's pool instead of returning it to the
  // driver at every synchronisation
  {
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, h->device) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  LuState* S = new LuState();
  S->st = h->stream;
  // capacity of low-rank blocks: twice the largest leaf rank (updated blocks
  // are truncated back after every addition), at least 12; HM_ERR_RANK if a
  // truncated rank ever exceeds it (raise rank_cap then)
  S->cap = h->prm.rank_cap > 0 ? h->prm.rank_cap : std::max(12, 2 * std::max(h->kmax, 1));
  S->cap = std::min(S->cap, RCORE_MAX / 2);
  HM_CUDA_TRY(cudaMallocAsync((void**)&S->P, sizeof(int64_t) * h->n, h->stream));
  HM_CUDA_TRY(cudaMallocAsync((void**)&S->flags, sizeof(int), h->stream));
  HM_CUDA_TRY(cudaMemsetAsync(S->flags, 0, sizeof(int), h->stream));
  const double eps_lu = h->prm.eps_trunc_lu > 0.0 ? h->prm.eps_trunc_lu : h->prm.eps_trunc;
  Ctx c{h->stream, S->cap, S->P, S->flags, eps_lu, h};
  const int mode = h->prm.lu_mode;     // 0 auto, 1 recursion, 2 tiles
  try {
    if (h->kmax > S->cap) throw LuError(HM_ERR_RANK, "a leaf rank exceeds the H-LU rank capacity");
    std::vector<int32_t> gcl, dnode;
    const bool tiled = mode != 1 && tile_structure(h, gcl, dnode);
    if (mode == 2 && !tiled) throw LuError(HM_ERR_UNSUPPORTED, "the partition has no tile level");
    if (tiled) {
      S->tile.reset(new TileLU());
      S->make_look();
      tile_factor(c, h, *S->tile, gcl, dnode, S->look);
    } else {
      S->root = build_from_handle(c, h, 0);
      lu_rec(c, *S->root);
    }
  } catch (const LuError& e) {
    cudaStreamSynchronize(h->stream);
    delete S;
    return fail(e.code, std::string("lu!: ") + e.what());
  }
  int s = finish(c, "lu!");
  if (s != HM_OK) {
    delete S;
    return s;
  }
  h->lu = S;
  h->factorized = true;
  return HM_OK;
}

// right-hand sides per sweep solve (the update's z values sit in shared memory)
static constexpr int SWEEP_MAX_COLS = 64;

// The launch sequence of a\y (trans = 0) or a'\y (trans = 1) from d_b into d_x.
// W, when given, is the working copy of b for the transposed solve; it may be
// d_b itself (the solve then overwrites b).
static void issue_solve(Ctx& c, LuState* S, const hm_handle* h, const double* d_b, double* d_x, int nc,
                        int trans, double* Z, double* W) {
  View B{const_cast<double*>(d_b), 1, h->n, (int)h->n, nc};
  View X{d_x, 1, h->n, (int)h->n, nc};
  const int64_t tot = h->n * nc;
  const unsigned g = (unsigned)std::min<int64_t>((tot + 255) / 256, 4096);
  if (!trans) {
    // a\y (src/hlu.jl:553-562): permute!(w, P), unit-L forward, U backward
    lu_gather_rows_kernel<<<g, 256, 0, c.st>>>(X, B, S->P);
    LU_LAUNCH_CHECK();
    if (S->tile && S->tile->d_inv[0] && nc <= SWEEP_MAX_COLS) {
      tile_sweeps(c, *S->tile, X, false);
    } else if (S->tile) {
      tile_solve(c, *S->tile, X, false, Z);
    } else {
      solve_rec(c, *S->root, X, true);
      solve_rec(c, *S->root, X, false);
    }
  } else {
    Blk tmp;
    tmp.st = c.st;
    double* w = W ? W : (double*)dmalloc(c, tmp, sizeof(double) * (size_t)tot);
    View Wv{w, 1, h->n, (int)h->n, nc};
    if (w != d_b) axpby(c, Wv, B, 1.0, 0.0);
    if (S->tile && S->tile->d_inv[0] && nc <= SWEEP_MAX_COLS) {
      tile_sweeps(c, *S->tile, Wv, true);
    } else if (S->tile) {
      tile_solve(c, *S->tile, Wv, true, Z);
    } else {
      solve_t_rec(c, *S->root, Wv, true);
      solve_t_rec(c, *S->root, Wv, false);
    }
    lu_scatter_rows_kernel<<<g, 256, 0, c.st>>>(X, Wv, S->P);
    LU_LAUNCH_CHECK();
  }
}

// Solves with at most this many right-hand sides are captured into a graph.
static constexpr int64_t SOLVE_GRAPH_MAX_COLS = 64;
static constexpr size_t SOLVE_MAX_PLANS = 8;

static SolvePlan* new_plan(LuState* S, const hm_handle* h, int64_t nc, int trans, cudaStream_t st) {
  auto pl = std::make_unique<SolvePlan>();
  pl->ncols = nc;
  pl->trans = trans;
  const size_t xb = sizeof(double) * (size_t)h->n * nc;
  const size_t zb = S->tile ? sizeof(double) * (size_t)S->tile->T * S->cap * nc : 8;
  if (cudaMallocAsync(&pl->xin, xb, st) != cudaSuccess || cudaMallocAsync(&pl->xout, xb, st) != cudaSuccess ||
      cudaMallocAsync(&pl->Z, zb, st) != cudaSuccess) {
    cudaGetLastError();
    throw LuError(HM_ERR_OOM, "solve plan buffers");
  }
  if (S->plans.size() >= SOLVE_MAX_PLANS) {
    cudaDeviceSynchronize();
    S->plans.erase(S->plans.begin());
  }
  S->plans.push_back(std::move(pl));
  return S->plans.back().get();
}

// Records the plan's sequence into a graph on a private stream.  Nothing runs
// during capture; a failure leaves the plan without a graph.
static void capture_plan(LuState* S, hm_handle* h, SolvePlan* pl, cudaStream_t caller) {
  cudaStream_t cs = nullptr;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    pl->no_graph = true;
    return;
  }
  if (pl->tape.temp_bytes > 0 &&
      cudaMallocAsync((void**)&pl->arena.base, pl->tape.temp_bytes, caller) != cudaSuccess) {
    cudaGetLastError();
    cudaStreamDestroy(cs);
    pl->no_graph = true;
    return;
  }
  pl->arena.size = pl->tape.temp_bytes;
  pl->arena.used = 0;
  Ctx c{cs, S->cap, S->P, S->flags, h->prm.eps_trunc, h, &pl->arena};
  pl->tape.record = false;
  pl->tape.replay = true;
  pl->tape.pos = 0;
  bool ok = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
  if (ok) {
    g_tape = &pl->tape;
    try {
      issue_solve(c, S, h, pl->xin, pl->xout, (int)pl->ncols, pl->trans, pl->Z, pl->xin);
    } catch (const LuError&) {
      ok = false;
    }
    g_tape = nullptr;
    cudaGraph_t graph = nullptr;
    if (cudaStreamEndCapture(cs, &graph) != cudaSuccess) ok = false;
    if (ok && pl->tape.pos != pl->tape.bufs.size()) ok = false;
    if (ok && cudaGraphInstantiate(&pl->exec, graph, 0) != cudaSuccess) {
      pl->exec = nullptr;
      ok = false;
    }
    if (graph) cudaGraphDestroy(graph);
  }
  cudaGetLastError();                  // capture errors are not sticky; clear them
  pl->tape.replay = false;
  pl->no_graph = !ok;
  cudaStreamDestroy(cs);
  // the plan's buffers were allocated in the caller's stream order; later
  // calls may come on other streams
  cudaStreamSynchronize(caller);
}

int lu_solve_device(hm_handle* h, const double* d_b, double* d_x, int64_t ncols, int trans, cudaStream_t st) {
  LuState* S = h->lu;
  if (!S) return fail(HM_ERR_STATE, "a has not been factorized");
  if (ncols <= 0) return HM_OK;
  Ctx c{st, S->cap, S->P, S->flags, h->prm.eps_trunc, h};
  try {
    if (S->tile) ensure_sweep(c, *S->tile);
    if (ncols > SOLVE_GRAPH_MAX_COLS) {
      issue_solve(c, S, h, d_b, d_x, (int)ncols, trans, nullptr, nullptr);
    } else {
      SolvePlan* pl = nullptr;
      for (auto& q : S->plans)
        if (q->ncols == ncols && q->trans == trans) pl = q.get();
      const size_t xb = sizeof(double) * (size_t)h->n * ncols;
      if (pl && pl->exec) {
        HM_LU_CUDA(cudaMemcpyAsync(pl->xin, d_b, xb, cudaMemcpyDeviceToDevice, st));
        HM_LU_CUDA(cudaGraphLaunch(pl->exec, st));
        HM_LU_CUDA(cudaMemcpyAsync(d_x, pl->xout, xb, cudaMemcpyDeviceToDevice, st));
      } else if (pl) {                 // capture failed earlier: direct run on the plan's buffers
        HM_LU_CUDA(cudaMemcpyAsync(pl->xin, d_b, xb, cudaMemcpyDeviceToDevice, st));
        issue_solve(c, S, h, pl->xin, pl->xout, (int)ncols, trans, pl->Z, pl->xin);
        HM_LU_CUDA(cudaMemcpyAsync(d_x, pl->xout, xb, cudaMemcpyDeviceToDevice, st));
      } else {                         // first solve of this shape: run it recording, then capture
        pl = new_plan(S, h, ncols, trans, st);
        HM_LU_CUDA(cudaMemcpyAsync(pl->xin, d_b, xb, cudaMemcpyDeviceToDevice, st));
        pl->tape.record = true;
        g_tape = &pl->tape;
        try {
          issue_solve(c, S, h, pl->xin, pl->xout, (int)ncols, trans, pl->Z, pl->xin);
        } catch (...) {
          g_tape = nullptr;
          pl->tape.record = false;
          throw;
        }
        g_tape = nullptr;
        pl->tape.record = false;
        HM_LU_CUDA(cudaMemcpyAsync(d_x, pl->xout, xb, cudaMemcpyDeviceToDevice, st));
        capture_plan(S, h, pl, st);
      }
    }
  } catch (const LuError& e) {
    return fail(e.code, std::string("H\\y: ") + e.what());
  }
  HM_CUDA_TRY(cudaGetLastError());
  return HM_OK;
}

__global__ void lu_colnorm2_kernel(View X, double* __restrict__ out) {
  __shared__ double red[32];
  const int c = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < X.rows; i += blockDim.x) {
    const double v = X.p[(int64_t)i * X.rs + (int64_t)c * X.cs];
    s = fma(v, v, s);
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[c] = s;
}

// Iterative refinement: x = (LU)^{-1} b, then r = b - H x with the FP64
// H-matvec of the unfactorised matrix (the matvec pools stay intact after
// lu!), x += (LU)^{-1} r, until max_c |r_c|/|b_c| <= tol or max_iter steps.
int lu_solve_refined(hm_handle* h, const double* d_b, double* d_x, int64_t ncols, int trans, double tol,
                     int max_iter, cudaStream_t st, int* iters, double* relres) {
  if (!h->lu) return fail(HM_ERR_STATE, "a has not been factorized");
  const int64_t n = h->n, tot = n * ncols;
  double *r = nullptr, *d = nullptr, *nrm = nullptr;
  HM_CUDA_TRY(cudaMallocAsync(&r, sizeof(double) * tot, st));
  HM_CUDA_TRY(cudaMallocAsync(&d, sizeof(double) * tot, st));
  HM_CUDA_TRY(cudaMallocAsync(&nrm, sizeof(double) * 2 * ncols, st));
  std::vector<double> hb(ncols), hr(ncols);
  int status = HM_OK, it = 0;
  double worst = 0.0;
  View Bv{const_cast<double*>(d_b), 1, n, (int)n, (int)ncols};
  View Rv{r, 1, n, (int)n, (int)ncols};
  Ctx c{st, h->lu->cap, h->lu->P, h->lu->flags, h->prm.eps_trunc, h};
  auto norms = [&](View V, double* dst, std::vector<double>& host) -> int {
    lu_colnorm2_kernel<<<(unsigned)ncols, 256, 0, st>>>(V, dst);
    HM_CUDA_TRY(cudaGetLastError());
    HM_CUDA_TRY(cudaMemcpyAsync(host.data(), dst, sizeof(double) * ncols, cudaMemcpyDeviceToHost, st));
    HM_CUDA_TRY(cudaStreamSynchronize(st));
    return HM_OK;
  };
  status = norms(Bv, nrm, hb);
  if (status == HM_OK) status = lu_solve_device(h, d_b, d_x, ncols, trans, st);
  for (; status == HM_OK; ++it) {
    // r = b - H x, summed in twice the FP64 precision
    for (int64_t q = 0; q < ncols && status == HM_OK; ++q)
      status = residual_device(h, d_x + q * n, d_b + q * n, r + q * n, trans, st);
    if (status != HM_OK) break;
    status = norms(Rv, nrm + ncols, hr);
    if (status != HM_OK) break;
    worst = 0.0;
    bool finite = true;
    for (int64_t q = 0; q < ncols; ++q) {
      const double v = hb[q] > 0 ? std::sqrt(hr[q] / hb[q]) : std::sqrt(hr[q]);
      if (!std::isfinite(v) || !std::isfinite(hb[q])) finite = false;   // std::max would drop a NaN
      worst = std::max(worst, v);
    }
    if (!finite) { status = fail(HM_ERR_NONFINITE, "refinement: non-finite residual"); break; }
    if (worst <= tol || it >= max_iter) break;
    status = lu_solve_device(h, r, d, ncols, trans, st);
    if (status != HM_OK) break;
    try {
      axpby(c, View{d_x, 1, n, (int)n, (int)ncols}, View{d, 1, n, (int)n, (int)ncols}, 1.0, 1.0);
    } catch (const LuError& e) {
      status = fail(e.code, e.what());
      break;
    }
  }
  cudaFreeAsync(r, st);
  cudaFreeAsync(d, st);
  cudaFreeAsync(nrm, st);
  cudaStreamSynchronize(st);
  if (iters) *iters = it;
  if (relres) *relres = worst;
  return status;
}

void lu_describe(const hm_handle* h, int64_t* tiles, int64_t* cap) {
  *tiles = h->lu && h->lu->tile ? h->lu->tile->T : 0;
  *cap = h->lu ? h->lu->cap : 0;
}

int lu_perm(const hm_handle* h, int64_t* P) {
  if (!h->lu) return fail(HM_ERR_STATE, "a has not been factorized");
  HM_CUDA_TRY(cudaMemcpyAsync(P, h->lu->P, sizeof(int64_t) * h->n, cudaMemcpyDeviceToHost, h->stream));
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  return HM_OK;
}

int lu_to_dense(const hm_handle* h, double* d_out) {
  if (!h->lu) return fail(HM_ERR_STATE, "a has not been factorized");
  Ctx c{h->stream, h->lu->cap, h->lu->P, h->lu->flags, h->prm.eps_trunc, h};
  try {
    View D{d_out, 1, h->n, (int)h->n, (int)h->n};
    if (h->lu->tile) tile_densify(c, *h->lu->tile, D);
    else densify_into(c, D, *h->lu->root);
  } catch (const LuError& e) {
    return fail(e.code, e.what());
  }
  HM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  return HM_OK;
}

void lu_free(hm_handle* h) {
  delete h->lu;
  h->lu = nullptr;
}

int lu_copy(const hm_handle* src, hm_handle* dst) {
  if (!src->lu) return HM_OK;
  LuState* S = new LuState();
  S->st = dst->stream;
  S->cap = src->lu->cap;
  HM_CUDA_TRY(cudaStreamSynchronize(src->stream));
  HM_CUDA_TRY(cudaMallocAsync((void**)&S->P, sizeof(int64_t) * src->n, dst->stream));
  HM_CUDA_TRY(cudaMallocAsync((void**)&S->flags, sizeof(int), dst->stream));
  HM_CUDA_TRY(cudaMemcpyAsync(S->P, src->lu->P, sizeof(int64_t) * src->n, cudaMemcpyDeviceToDevice, dst->stream));
  HM_CUDA_TRY(cudaMemsetAsync(S->flags, 0, sizeof(int), dst->stream));
  Ctx c{dst->stream, S->cap, S->P, S->flags, src->prm.eps_trunc, src};
  try {
    if (src->lu->tile) {
      const TileLU& A = *src->lu->tile;
      TileLU* B = new TileLU();
      S->tile.reset(B);
      B->T = A.T;
      B->start = A.start;
      B->size = A.size;
      B->hold = std::make_shared<Blk>();
      B->hold->st = c.st;
      B->Ap.resize(A.T);
      B->Bp.resize(A.T);
      for (int i = 0; i < A.T; ++i) {
        const size_t bytes = sizeof(double) * A.size[i] * A.T * S->cap;
        B->Ap[i] = (double*)dmalloc(c, *B->hold, bytes);
        B->Bp[i] = (double*)dmalloc(c, *B->hold, bytes);
        if (cudaMemcpyAsync(B->Ap[i], A.Ap[i], bytes, cudaMemcpyDeviceToDevice, c.st) != cudaSuccess ||
            cudaMemcpyAsync(B->Bp[i], A.Bp[i], bytes, cudaMemcpyDeviceToDevice, c.st) != cudaSuccess)
          throw LuError(HM_ERR_CUDA, "panel copy");
      }
      B->kmat = (int32_t*)dmalloc(c, *B->hold, sizeof(int32_t) * A.T * A.T);
      if (cudaMemcpyAsync(B->kmat, A.kmat, sizeof(int32_t) * A.T * A.T, cudaMemcpyDeviceToDevice, c.st) !=
          cudaSuccess)
        throw LuError(HM_ERR_CUDA, "rank copy");
      B->diag.resize(A.T);
      for (int i = 0; i < A.T; ++i) B->diag[i] = copy_blk(c, *A.diag[i]);
    } else {
      S->root = copy_blk(c, *src->lu->root);
    }
  } catch (const LuError& e) {
    delete S;
    return fail(e.code, e.what());
  }
  HM_CUDA_TRY(cudaStreamSynchronize(dst->stream));
  dst->lu = S;
  return HM_OK;
}

}  // namespace hm
