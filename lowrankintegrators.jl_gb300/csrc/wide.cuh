// wide.cuh - FP64 building blocks for one instance spread over thread-block
// clusters (engine_wide.cu, adjoint.cu): the rows of a tall panel are split
// over the CTAs of a cluster, reductions and small matrices go through
// distributed shared memory.
//
// GB300 runs FP64 at 1/64 of the FP32 rate (about 1.9 multiply-adds per clock
// and SM), so a warp's FP64 instruction occupies its unit for 16 clocks of
// the SM and shared-memory operand loads are free beside it: the products
// below give one output to a thread (or to a few lanes when outputs are
// fewer than threads) and keep no register tiles; what counts is that every
// SM of the cluster has all its FP64 units busy and that scalar work
// (square roots, divisions) is done by one warp only.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "engine_api.h"

namespace lri {
namespace wide {

namespace cg = cooperative_groups;

constexpr int WT = 256;          // threads per CTA
constexpr int WC_MAX = 16;       // CTAs per cluster (above 8: opt-in)
constexpr int WR_MAX = 64;       // widest panel

// Launch attributes of a cluster kernel: clusters above 8 CTAs and the largest
// dynamic shared memory (once per device, as set_smem_limit).
template <typename F>
inline cudaError_t cluster_attributes(F* kern, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = (dev < 64) ? (uint64_t(1) << dev) : 0;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmemMax);
  if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}
inline void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int blocks, int C, size_t smem,
                           cudaStream_t st) {
  cfg.gridDim = dim3(blocks, 1, 1);
  cfg.blockDim = dim3(WT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

// This CTA's part of a cluster.
struct Team {
  cg::cluster_group cl;
  int q, C;
  __device__ int rows_per(int N) const { return (N + C - 1) / C; }
  __device__ int lo(int N) const { return min(N, q * rows_per(N)); }
  __device__ int hi(int N) const { return min(N, (q + 1) * rows_per(N)); }
  template <typename P>
  __device__ P* at(P* p, int rank) const { return cl.map_shared_rank(p, rank); }
  // all threads of the cluster; orders shared, distributed and global accesses
  __device__ void sync() const {
    __threadfence();
    cl.sync();
  }
};

// out(o) for o in [0, nout): f(o, l, L) returns lane l's share (of L) of the
// sum, summed over the lanes; done(o, v) runs on one lane.  L is the largest
// power of two <= 32 with nout * L <= WT, so few outputs still fill the CTA.
template <class F, class D>
__device__ __forceinline__ void outputs(int nout, const F& f, const D& done) {
  int L = 1;
  while (L < 32 && nout * L * 2 <= WT) L *= 2;
  const int l = threadIdx.x & (L - 1);
  const int per = WT / L;
  for (int o0 = 0; o0 < nout; o0 += per) {  // uniform trip count: every lane reaches the shuffles
    const int o = o0 + threadIdx.x / L;
    double v = (o < nout) ? f(o, l, L) : 0.0;
    for (int s = L >> 1; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (o < nout && l == 0) done(o, v);
  }
}

// Adds every CTA's part[0 .. len) (shared memory, the same address in every
// CTA): done(e, sum) runs for each e on one CTA.  The terms are added in
// rank order.  Cluster-synchronises before (the parts are complete) and
// after (done's global writes are visible, part may be reused).
template <class D>
__device__ void reduce_parts(const Team& tm, double* part, int len, const D& done) {
  tm.sync();
  const int per = (len + tm.C - 1) / tm.C, e0 = tm.q * per, e1 = min(len, e0 + per);
  for (int e = e0 + threadIdx.x; e < e1; e += WT) {
    double s = 0.0;
    for (int k = 0; k < tm.C; ++k) s += tm.at(part, k)[e];
    done(e, s);
  }
  tm.sync();
}

// rows [lo, lo + rows) of a global panel (ld N) into a smem panel
static __device__ void load_rows(const double* X, int N, int lo, int rows, int r, double* p, int ld) {
  for (int e = threadIdx.x; e < rows * r; e += WT) {
    const int i = e % rows, k = e / rows;
    p[k * ld + 1 + i] = X[lo + i + (int64_t)k * N];
  }
}

// pushes this CTA's first and last rows into the neighbours' halo rows
// (panel at the same shared address in every CTA); the cluster must
// synchronise before they are read
static __device__ void push_halos(const Team& tm, int N, int rows, int r, double* p, int ld) {
  if (rows == 0) return;
  const int R0 = tm.rows_per(N);
  const bool up = tm.q > 0, dn = tm.q + 1 < tm.C && tm.lo(N) + rows < N;
  for (int e = threadIdx.x; e < 2 * r; e += WT) {
    const int k = e >> 1;
    if (!(e & 1) && up) tm.at(p, tm.q - 1)[k * ld + 1 + R0] = p[k * ld + 1];
    if ((e & 1) && dn) tm.at(p, tm.q + 1)[k * ld] = p[k * ld + rows];
  }
}

// the same with the halo rows from memory (zero outside [0, N))
static __device__ void load_rows_halo(const double* X, int N, int lo, int rows, int r, double* p, int ld) {
  for (int e = threadIdx.x; e < (rows + 2) * r; e += WT) {
    const int i = e % (rows + 2), k = e / (rows + 2), g = lo - 1 + i;
    p[k * ld + i] = (g >= 0 && g < N) ? X[g + (int64_t)k * N] : 0.0;
  }
}

// T w (or T^T w) at row i, column k of a smem panel, T = [sub | dia | sup]
struct Tri {
  const double* tri;
  int N, lo;
  __device__ double mul(const double* p, int ld, int i, int k) const {
    const int gi = lo + i;
    const double cd = tri[N + gi], cs = gi > 0 ? tri[gi] : 0.0, cp = gi + 1 < N ? tri[2 * N + gi] : 0.0;
    const double* w = p + k * ld + i;
    return fma(cs, w[0], fma(cp, w[2], cd * w[1]));
  }
  __device__ double mul_t(const double* p, int ld, int i, int k) const {
    const int gi = lo + i;
    const double cd = tri[N + gi], cs = gi > 0 ? tri[2 * N + gi - 1] : 0.0, cp = gi + 1 < N ? tri[gi + 1] : 0.0;
    const double* w = p + k * ld + i;
    return fma(cs, w[0], fma(cp, w[2], cd * w[1]));
  }
};

// Shared scratch of the distributed QR, carved from dynamic memory.
struct QrSmem {
  double* slot;  // 2 x C x r: partial dots of every CTA, alternating by column
  double* row;   // 2 x r: the pivot row
  double* part;  // (WT / 32) x r
  double* dots;  // r
  double* v1;    // r x (r + 1): pivot rows of V, v1[k LT + j], j < k
  double* tri;   // r x (r + 1): T of the compact WY form, T(i, k) at i LT + k
  double* coef;  // beta, tau, scal
  __host__ __device__ static constexpr size_t doubles(int C, int r) {
    return (size_t)r * (2 * C + 2 + WT / 32 + 1) + 2 * (size_t)r * (r + 1) + 4;
  }
  __device__ static QrSmem carve(double* p, int C, int r) {
    QrSmem s;
    s.slot = p;
    s.row = s.slot + 2 * C * r;
    s.part = s.row + 2 * r;
    s.dots = s.part + (WT / 32) * r;
    s.v1 = s.dots + r;
    s.tri = s.v1 + r * (r + 1);
    s.coef = s.tri + r * (r + 1);
    return s;
  }
};

// Householder QR (LAPACK signs) of an N x r panel whose rows [lo, lo + rows)
// are this CTA's a[k ld + i]; the explicit Q goes to qout (same layout) and,
// when R is given, the factor to R (global, ld ldr, zeros below).  One
// cluster barrier per column: a single pass forms x^T A for every column (the
// trailing ones, and the earlier reflectors for the compact WY form), its
// partials and the pivot row are pushed to every CTA, and every CTA derives
// the reflector from the same sums.  Q = [I; 0] - V (T V1^T), T from those
// products, replaces the backward accumulation: N r^2 / 2 multiply-adds and
// no further barrier.  a is overwritten.
static __device__ __noinline__ void qr(const Team& tm, int N, int lo, int rows, int r, double* a, int ld,
                                       double* qout, double* R, int ldr, const QrSmem& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int LT = r + 1;
  const int R0 = tm.rows_per(N);
  for (int e = tid; e < r * LT; e += WT) s.tri[e] = s.v1[e] = 0.0;
  __syncthreads();
  for (int k = 0; k < r; ++k) {
    double* slot = s.slot + (k & 1) * tm.C * r;
    double* row = s.row + (k & 1) * r;
    double* x = a + k * ld;
    const int i0 = max(0, k + 1 - lo);  // rows below the pivot
    // partial dots: lane = column, warp = row class
    for (int j = lane; j < r; j += 32) {
      double p = 0.0;
      for (int i = i0 + warp; i < rows; i += WT / 32) p = fma(x[i], a[j * ld + i], p);
      s.part[warp * r + j] = p;
    }
    if (tm.q == k / R0)
      for (int e = tid; e < r * tm.C; e += WT) tm.at(row, e / r)[e % r] = a[(e % r) * ld + (k - lo)];
    __syncthreads();
    if (tid < r) {
      double p = 0.0;
#pragma unroll
      for (int w = 0; w < WT / 32; ++w) p += s.part[w * r + tid];
      for (int c = 0; c < tm.C; ++c) tm.at(slot, c)[tm.q * r + tid] = p;
    }
    tm.cl.sync();
    // totals: four lanes per column
    for (int j0 = 0; j0 < r; j0 += WT / 4) {
      const int j = j0 + (tid >> 2);
      double p = 0.0;
      if (j < r)
        for (int c = tid & 3; c < tm.C; c += 4) p += slot[c * r + j];
      p += __shfl_xor_sync(0xffffffffu, p, 1);
      p += __shfl_xor_sync(0xffffffffu, p, 2);
      if (j < r && (tid & 3) == 0) s.dots[j] = p;
    }
    __syncthreads();
    if (warp == 0) {
      const double xn2 = s.dots[k], alpha = row[k];
      double beta = alpha, tau = 0.0, scal = 0.0;
      if (xn2 > 0.0) {
        beta = -copysign(sqrt(fma(alpha, alpha, xn2)), alpha);
        tau = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      if (lane == 0) {
        s.coef[0] = beta;
        s.coef[1] = tau;
        s.coef[2] = scal;
      }
    }
    __syncthreads();
    const double beta = s.coef[0], tau = s.coef[1], scal = s.coef[2];
    // w_j (trailing columns) and z_j = -tau V_j^T v_k (earlier reflectors)
    if (tid < r) {
      const int j = tid;
      const double rk = row[j];
      const double t = (j != k) ? tau * fma(scal, s.dots[j], rk) : 0.0;
      if (j < k) {
        s.v1[k * LT + j] = rk;
        s.tri[j * LT + k] = -t;
      }
      if (j == k) s.tri[k * LT + k] = tau;
      if (R && tm.q == 0) R[k + (int64_t)j * ldr] = (j > k) ? rk - t : ((j == k) ? beta : 0.0);
      s.dots[j] = t;
    }
    __syncthreads();
    // trailing update, the reflector stored in column k
    const int ib = max(0, k - lo), nr = rows - ib, nj = r - k - 1;
    if (tau != 0.0 && nr > 0) {
      for (int e = tid; e < nr * nj; e += WT) {
        const int i = ib + e % nr, j = k + 1 + e / nr;
        const double vi = (lo + i == k) ? 1.0 : x[i] * scal;
        a[j * ld + i] = fma(-vi, s.dots[j], a[j * ld + i]);
      }
      __syncthreads();
      for (int i = i0 + tid; i < rows; i += WT) x[i] *= scal;
    }
    __syncthreads();
  }
  // T: column k is T[:, 0:k] z_k (z_k sits in column k), diagonal tau; eight
  // lanes per row
  constexpr int TU = WR_MAX * 8 / WT;
  for (int k = 1; k < r; ++k) {
    double v[TU];
#pragma unroll
    for (int u = 0; u < TU; ++u) {
      const int i = (tid + u * WT) >> 3;
      double p = 0.0;
      if (i < k)
        for (int l = i + (tid & 7); l < k; l += 8) p = fma(s.tri[i * LT + l], s.tri[l * LT + k], p);
      p += __shfl_xor_sync(0xffffffffu, p, 1);
      p += __shfl_xor_sync(0xffffffffu, p, 2);
      p += __shfl_xor_sync(0xffffffffu, p, 4);
      v[u] = p;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < TU; ++u) {
      const int i = (tid + u * WT) >> 3;
      if (i < k && (tid & 7) == 0) s.tri[i * LT + k] = v[u];
    }
    __syncthreads();
  }
  // X = T V1^T (V1 unit lower triangular), X(i, j) at j LT + i for i <= j, over
  // the rows of v1 that it is formed from
  constexpr int XU = WR_MAX * WR_MAX / WT;
  double xv[XU];
#pragma unroll
  for (int u = 0; u < XU; ++u) {
    const int e = tid + u * WT, i = e % r, j = e / r;
    double p = 0.0;
    if (j < r && i <= j) {
      p = s.tri[i * LT + j];
      for (int l = i; l < j; ++l) p = fma(s.tri[i * LT + l], s.v1[j * LT + l], p);
    }
    xv[u] = p;
  }
  // explicit V: zeros above the unit diagonal
  for (int e = tid; e < rows * r; e += WT) {
    const int i = e % rows, k = e / rows;
    if (lo + i <= k) a[k * ld + i] = (lo + i == k) ? 1.0 : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < XU; ++u) {
    const int e = tid + u * WT, i = e % r, j = e / r;
    if (j < r && i <= j) s.v1[j * LT + i] = xv[u];
  }
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int i = e % rows, j = e / rows;
    double p = (lo + i == j) ? 1.0 : 0.0;
    for (int k = 0; k <= j; ++k) p = fma(-a[k * ld + i], s.v1[j * LT + k], p);
    qout[j * ld + i] = p;
  }
  __syncthreads();
}

}  // namespace wide
}  // namespace lri
