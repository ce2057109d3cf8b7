// wide.cuh - building blocks for one side of an instance on a thread-block
// cluster (engine_wide.cu, engine_sides.cu, adjoint.cu): the rows of a tall
// panel are split over the CTAs of a cluster (one CTA for small panels) and
// stay in shared memory; reductions and small matrices go through distributed
// shared memory.
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

#include "engine.cuh"
#include "engine_api.h"
#include "fast_div.h"

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
  __device__ P* at(P* p, int rank) const { return C > 1 ? cl.map_shared_rank(p, rank) : p; }
  __device__ void barrier() const {
    if (C > 1) cl.sync();
    else __syncthreads();
  }
  // all threads of the cluster; orders shared, distributed and global accesses
  __device__ void sync() const {
    if (C > 1) __threadfence();
    barrier();
  }
};

// Lanes per output for nout outputs on WT threads: the largest power of two <=
// 32 that still fits, else (more outputs than threads) the one of 1 .. 8 that
// leaves the fewest threads idle in the last round.
__device__ __forceinline__ int lanes_for(int nout) {
  int L = 1;
  if (nout <= WT) {
    while (L < 32 && nout * L * 2 <= WT) L *= 2;
    return L;
  }
  int best = (nout + WT - 1) / WT * 8;
  for (int t = 2; t <= 8; t *= 2) {
    const int cost = (nout * t + WT - 1) / WT * (8 / t);
    if (cost < best) {
      best = cost;
      L = t;
    }
  }
  return L;
}

// Lanes per output for nout FP64 sums of K terms: a warp's FP64 instruction
// occupies its scheduler's unit for 64 clocks, so the cost is the instructions
// per scheduler, ceil(warps / 4) (ceil(K / L) + log2 L); more lanes shorten the
// sums but add shuffle-and-add steps that whole warps execute.
__device__ __forceinline__ int lanes_f64(int nout, int K) {
  int best = 1 << 30, L = 1;
#pragma unroll
  for (int g = 0; g <= 5; ++g) {
    const int warps = ((nout << g) + 31) >> 5, cost = ((warps + 3) >> 2) * (((K + (1 << g) - 1) >> g) + g);
    if (cost < best) {
      best = cost;
      L = 1 << g;
    }
  }
  return L;
}

// out(o) for o in [0, nout): f(o, l, L) returns lane l's share (of L) of a sum
// of K terms, summed over the lanes; done(o, v) runs on one lane.  (L given:
// sums bound by something else than FP64 issue.)
template <class F, class D>
__device__ __forceinline__ void outputs(int nout, int K, const F& f, const D& done, int L = 0) {
  if (L == 0) L = lanes_f64(nout, K);
  const int l = threadIdx.x & (L - 1);
  const int per = WT / L;
  const int warp0 = (threadIdx.x & ~31) / L;  // the warp's first output of a round
  for (int o0 = 0; o0 + warp0 < nout; o0 += per) {  // warp-uniform: every lane reaches the shuffles
    const int o = o0 + threadIdx.x / L;
    double v = (o < nout) ? f(o, l, L) : 0.0;
    for (int s = L >> 1; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (o < nout && l == 0) done(o, v);
  }
}

// The products with a Gram matrix G = I + E: Y G = Y + Y E, with Y E on the FP32
// pipe while max |E| <= 2^-36.  That adds at most 2^-60 of a row's largest entry
// to each of its entries, where the rounding of G's own entries (sums over the
// rows of two bases, 2^-53 each) acts on them in the same way in the full
// product: errors against 64-bit results are the same in both forms
// (geometric means over 30 problems: FP64 ensembles 7.02e-16 and 7.05e-16 with
// the full product, gradients 1.78e-15 and 1.85e-15).  The FP32 range allows it
// for panels whose entries all stay below 2^100 and of which one reaches 2^-80
// (what falls under the range is then below 2^-64 of it); the others take
// the full product.  Both tests without an FP64 instruction, false for NaN.
__device__ __forceinline__ bool below_2_100(double x) { return (__double2hiint(x) & 0x7fffffff) < 0x46300000; }
__device__ __forceinline__ bool reaches_2_m80(double x) {
  return (unsigned)((__double2hiint(x) & 0x7fffffff) - ((1023 - 80) << 20)) < (unsigned)(0x7ff00000 - ((1023 - 80) << 20));
}
// whether the full product is needed: a value too large anywhere in the CTA, or
// none of size (all threads; a barrier)
__device__ __forceinline__ bool out_of_f32(int big, int reaches) {
  return __syncthreads_or(big) || !__syncthreads_or(reaches);
}

// Adds every CTA's part[0 .. len) (shared memory, the same address in every
// CTA): done(e, sum) runs for each e on one CTA.  The terms are added in
// rank order.  Cluster-synchronises before (the parts are complete) and
// after (done's global writes are visible, part may be reused).
template <typename A, class D>
__device__ void reduce_parts(const Team& tm, A* part, int len, const D& done) {
  tm.sync();
  const int per = (len + tm.C - 1) / tm.C, e0 = tm.q * per, e1 = min(len, e0 + per);
  for (int e = e0 + threadIdx.x; e < e1; e += WT) {
    A s = part[e];
    if (tm.C > 1) {
      s = tm.at(part, 0)[e];
      for (int k = 1; k < tm.C; ++k) s += tm.at(part, k)[e];
    }
    done(e, s);
  }
  tm.sync();
}

// rows [lo, lo + rows) of a global panel (ld N) into a smem panel
template <typename T>
__device__ void load_rows(const T* X, int N, int lo, int rows, int r, T* p, int ld) {
  const FastDiv by_rows(rows);
  for (int e = threadIdx.x; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    p[k * ld + 1 + i] = X[lo + i + (int64_t)k * N];
  }
}

// pushes this CTA's first and last rows into the neighbours' halo rows
// (panel at the same shared address in every CTA); the cluster must
// synchronise before they are read
template <typename T>
__device__ void push_halos(const Team& tm, int N, int rows, int r, T* p, int ld) {
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
template <typename T>
__device__ void load_rows_halo(const T* X, int N, int lo, int rows, int r, T* p, int ld) {
  for (int e = threadIdx.x; e < (rows + 2) * r; e += WT) {
    const int i = e % (rows + 2), k = e / (rows + 2), g = lo - 1 + i;
    p[k * ld + i] = (g >= 0 && g < N) ? X[g + (int64_t)k * N] : T(0);
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
template <typename T>
struct QrSmem {
  T* slot;  // 2 x C x r: partial dots of every CTA, alternating by column
  T* row;   // 2 x r: the pivot row
  T* part;  // (WT / 32) x r
  T* dots;  // r
  T* v1;    // r x (r + 1): pivot rows of V, v1[k LT + j], j < k
  T* tri;   // r x (r + 1): T of the compact WY form, T(i, k) at i LT + k
  T* coef;  // beta, tau, scal, flag
  T* sgn;   // r: column scales, then signs (fast forms)
  __host__ __device__ static constexpr size_t elems(int C, int r) {
    return (size_t)r * (2 * C + 2 + WT / 32 + 1) + 2 * (size_t)r * (r + 1) + 4 + r;
  }
  __device__ static QrSmem carve(T* p, int C, int r) {
    QrSmem s;
    s.slot = p;
    s.row = s.slot + 2 * C * r;
    s.part = s.row + 2 * r;
    s.dots = s.part + (WT / 32) * r;
    s.v1 = s.dots + r;
    s.tri = s.v1 + r * (r + 1);
    s.coef = s.tri + r * (r + 1);
    s.sgn = s.coef + 4;
    return s;
  }
};

__device__ __forceinline__ float two_to(float, int e) { return ldexpf(1.0f, e); }
__device__ __forceinline__ dfloat two_to(dfloat, int e) { return dfloat(ldexpf(1.0f, e), 0.0f); }
__device__ __forceinline__ double two_to(double, int e) { return __hiloint2double((e + 1023) << 20, 0); }
__device__ __forceinline__ float lead(float x) { return x; }
__device__ __forceinline__ float lead(dfloat x) { return x.hi; }
__device__ __forceinline__ float lead(double x) { return (float)x; }

// Square root and reciprocal of the reflector's scalars.  FP64: Newton steps
// from the FP32 estimates (about 12 and 5 FP64 instructions, where the library
// calls take some 25 and 12; one warp's chain of them is on the critical path
// of every column), within the FP32 exponent range, else the library's.  At
// most one unit in the last place from the correctly rounded values.
__device__ __forceinline__ float root(float x) { return sqrtf(x); }
__device__ __forceinline__ dfloat root(dfloat x) { return lri_df::sqrt(x); }
__device__ __forceinline__ double root(double x) {
  if (!(x > 1.0e-30 && x < 1.0e30)) return ::sqrt(x);
  double y = (double)rsqrtf((float)x);
  y = y * fma(-0.5 * (x * y), y, 1.5);
  y = y * fma(-0.5 * (x * y), y, 1.5);
  const double s = x * y;
  return fma(fma(-s, s, x), 0.5 * y, s);
}
__device__ __forceinline__ float reciprocal(float x) { return 1.0f / x; }
__device__ __forceinline__ dfloat reciprocal(dfloat x) { return dfloat(1.0f, 0.0f) / x; }
__device__ __forceinline__ double reciprocal(double x) {  // 1e-30 < |x| < 1e30
  double q = (double)(1.0f / (float)x);
  q = fma(q, fma(-x, q, 1.0), q);
  return fma(q, fma(-x, q, 1.0), q);
}

// A reflector's column x below the pivot alpha: whether alpha^2 + x^T x (xn2 =
// x^T x) is so small that squares have lost bits at the end of the type's
// exponent range.  (Integer tests: an FP64 comparison in every thread would
// show in every column.)
__device__ __forceinline__ bool squares_lost(float alpha, float xn2) {
  return fabsf(alpha) < 0x1p-50f && xn2 < 0x1p-100f;
}
__device__ __forceinline__ bool squares_lost(dfloat alpha, dfloat xn2) {
  return fabsf(alpha.hi) < 0x1p-45f && xn2.hi < 0x1p-90f;
}
__device__ __forceinline__ bool squares_lost(double alpha, double xn2) {  // 2^-450, 2^-900
  return (__double2hiint(alpha) & 0x7fffffff) < (1023 - 450) << 20 &&
         (__double2hiint(xn2) & 0x7fffffff) < (1023 - 900) << 20;
}
// magnitude as an integer that grows with it, and the power of two that brings
// it near 1 (0 for zero and for values that are not finite)
__device__ __forceinline__ int size_key(float x) { return __float_as_int(x) & 0x7fffffff; }
__device__ __forceinline__ int size_key(dfloat x) { return size_key(x.hi); }
__device__ __forceinline__ int size_key(double x) { return __double2hiint(x) & 0x7fffffff; }
template <typename T>
__device__ __forceinline__ int scale_exponent(int key) {
  constexpr bool F64 = std::is_same<T, double>::value;
  constexpr int mant = F64 ? 20 : 23, bias = F64 ? 1023 : 127, most = F64 ? 1000 : 120;
  if (key == 0 || key >= (2 * bias + 1) << mant) return 0;
  return max(-most, min(most, bias - (key >> mant)));
}

// The dots of column k again (s.dots) with the column scaled by a power of two
// from the largest entry over the cluster, pivot included; returns the
// exponent (0: a zero column, nothing changed).  `slot` holds this column's
// partial dots, `other` the next one's (free).  The same on every thread; ends
// with a barrier.
template <typename T>
__device__ __noinline__ int rescaled_dots(const Team& tm, int rows, int r, T* a, int ld, int k, int i0, T alpha,
                                          T* slot, T* other, const QrSmem<T>& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T* x = a + k * ld;
  int* wmax = reinterpret_cast<int*>(s.part);
  int* all = reinterpret_cast<int*>(other);
  int key = size_key(alpha);
  for (int i = i0 + tid; i < rows; i += WT) key = max(key, size_key(x[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
  if (lane == 0) wmax[warp] = key;
  __syncthreads();
  if (tid < tm.C) {
#pragma unroll
    for (int w = 0; w < WT / 32; ++w) key = max(key, wmax[w]);
    tm.at(all, tid)[tm.q] = key;
  }
  tm.barrier();
  key = all[0];
  for (int c = 1; c < tm.C; ++c) key = max(key, all[c]);
  const int up = scale_exponent<T>(key);
  if (up != 0) {
    const T f = two_to(T(0), up);
    for (int i = i0 + tid; i < rows; i += WT) x[i] = x[i] * f;
    __syncthreads();
    for (int j = warp; j < r; j += WT / 32) {
      T p = T(0);
      for (int i = i0 + lane; i < rows; i += 32) p = fma(x[i], a[j * ld + i], p);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) p += shfl_xor(p, o);
      for (int c = lane; c < tm.C; c += 32) tm.at(slot, c)[tm.q * r + j] = p;
    }
  }
  tm.barrier();
  if (up != 0) {
    if (tid < r) {
      T p = slot[tid];
      for (int c = 1; c < tm.C; ++c) p += slot[c * r + tid];
      s.dots[tid] = p;
    }
    __syncthreads();
  }
  return up;
}

// The reflectors of the columns from k0 on.  A column whose squares leave the
// exponent range (seen by the warp that forms the scalars, so that the others
// read a flag beside them) ends the plain form, which returns it with nothing of
// it changed; the safe form scales such columns.  Returns r at the end.
template <typename T, bool POS, bool SAFE>
__device__ __forceinline__ int qr_columns(const Team& tm, int lo, int rows, int r, T* a, int ld, T* R, int ldr,
                                          const QrSmem<T>& s, int R0, int k0) {
  constexpr bool F64 = std::is_same<T, double>::value;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int LT = r + 1;
  const int jw = r <= 8 ? 8 : (r <= 16 ? 16 : 32), ncls = WT / jw, cls = tid / jw;
  for (int k = k0; k < r; ++k) {
    T* slot = s.slot + (k & 1) * tm.C * r;
    T* row = s.row + (k & 1) * r;
    T* x = a + k * ld;
    const int i0 = max(0, k + 1 - lo);  // rows below the pivot
    // partial dots: lanes along the columns (jw per row class), a warp's row
    // classes combined by shuffles
    for (int jb = 0; jb < r; jb += jw) {
      const int j = jb + (lane & (jw - 1));
      const T* aj = a + min(j, r - 1) * ld;
      T p = T(0);
      if constexpr (F64) {
        for (int i = i0 + cls; i < rows; i += ncls) p = fma(x[i], aj[i], p);
      } else {
        for (int ib = i0 + cls; ib < rows; ib += 8 * ncls) {
          T q = T(0);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int i = ib + u * ncls;
            if (i < rows) q = fma_acc(x[i], aj[i], q);
          }
          p += renorm(q);
        }
      }
      for (int o = jw; o < 32; o <<= 1) p += shfl_xor(p, o);
      if (lane < jw && j < r) s.part[warp * r + j] = p;
    }
    if (tm.q == k / R0)
      for (int e = tid; e < r * tm.C; e += WT) tm.at(row, e / r)[e % r] = a[(e % r) * ld + (k - lo)];
    __syncthreads();
    if (tid < r) {
      T p = T(0);
#pragma unroll
      for (int w = 0; w < WT / 32; ++w) p += s.part[w * r + tid];
      if (tm.C == 1) s.dots[tid] = p;
      else
        for (int c = 0; c < tm.C; ++c) tm.at(slot, c)[tm.q * r + tid] = p;
    }
    tm.barrier();
    if (tm.C > 1) {
      // totals: four lanes per column
      for (int j0 = 0; j0 < r; j0 += WT / 4) {
        const int j = j0 + (tid >> 2);
        T p = T(0);
        if (j < r)
          for (int c = tid & 3; c < tm.C; c += 4) p += slot[c * r + j];
        p += shfl_xor(p, 1);
        p += shfl_xor(p, 2);
        if (j < r && (tid & 3) == 0) s.dots[j] = p;
      }
      __syncthreads();
    }
    int up = 0;
    if constexpr (SAFE) {
      if (squares_lost(row[k], s.dots[k]))
        up = rescaled_dots(tm, rows, r, a, ld, k, i0, row[k], slot, s.slot + ((k + 1) & 1) * tm.C * r, s);
    }
    if (warp == 0) {
      const T xn2 = s.dots[k], alpha = SAFE && up ? row[k] * two_to(T(0), up) : row[k];
      T beta = alpha, tau = T(0), scal = T(0);
      if (xn2 > T(0)) {
        beta = -copysign(root(fma(alpha, alpha, xn2)), alpha);
        const T d = alpha - beta, bd = beta * d;
        if (F64 && lead(bd) < -1.0e-30f && lead(bd) > -1.0e30f) {
          // one reciprocal for both, 1 / (beta (alpha - beta))
          const T q = reciprocal(bd);
          tau = -(d * d) * q;
          scal = q * beta;
        } else {
          tau = (beta - alpha) / beta;
          scal = T(1) / d;
        }
      }
      if (lane == 0) {
        s.coef[0] = SAFE && up ? beta * two_to(T(0), -up) : beta;
        s.coef[1] = tau;
        s.coef[2] = scal;
        if constexpr (!SAFE) s.coef[3] = squares_lost(alpha, xn2) ? T(1) : T(0);
        if constexpr (!F64) s.sgn[k] = (POS && lead(beta) < 0.0f) ? T(-1.0f) : T(1.0f);
      }
    }
    __syncthreads();
    if (!SAFE && size_key(s.coef[3]) != 0) return k;
    const T beta = s.coef[0], tau = s.coef[1], scal = s.coef[2];
    // w_j (trailing columns) and z_j = -tau V_j^T v_k (earlier reflectors)
    if (tid < r) {
      const int j = tid;
      const T rk = row[j];
      const T t = (j != k) ? tau * fma(scal, s.dots[j], rk) : T(0);
      if (j < k) {
        s.v1[k * LT + j] = rk;
        s.tri[j * LT + k] = -t;
      }
      if (j == k) s.tri[k * LT + k] = tau;
      if (F64 && R && tm.q == 0) R[k + (int64_t)j * ldr] = (j > k) ? rk - t : ((j == k) ? beta : T(0));
      s.dots[j] = t;
    }
    __syncthreads();
    // trailing update, the reflector stored in column k
    const int ib = max(0, k - lo), nr = rows - ib, nj = r - k - 1;
    if (tau != T(0) && nr > 0) {
      if (nr >= WT / 2) {
        // a row per thread
        for (int i = ib + tid; i < rows; i += WT) {
          T vi = T(1);
          if (lo + i > k) {
            vi = x[i] * scal;
            x[i] = vi;
          }
#pragma unroll 4
          for (int j = k + 1; j < r; ++j) a[j * ld + i] = fma(-vi, s.dots[j], a[j * ld + i]);
        }
      } else {
        const FastDiv by_nr(nr);
        for (int e = tid; e < nr * nj; e += WT) {
          const int q = by_nr.div(e), i = ib + e - q * nr, j = k + 1 + q;
          const T vi = (lo + i == k) ? T(1) : x[i] * scal;
          a[j * ld + i] = fma(-vi, s.dots[j], a[j * ld + i]);
        }
        __syncthreads();
        for (int i = i0 + tid; i < rows; i += WT) x[i] = x[i] * scal;
      }
    }
    __syncthreads();
  }
  return r;
}

// Householder QR (LAPACK signs; POS: a positive diagonal of R) of an N x r
// panel whose rows [lo, lo + rows) are this CTA's a[k ld + i]; the explicit Q
// goes to qout (ld ldq) and, when R is given, the factor to R (global, ld
// ldr, zeros below; not with the scaled columns of the FP32-based types).  One
// cluster barrier per column: a single pass forms x^T A for every column (the
// trailing ones, and the earlier reflectors for the compact WY form), its
// partials and the pivot row are pushed to every CTA, and every CTA derives
// the reflector from the same sums.  Q = [I; 0] - V (T V1^T), T from those
// products, replaces the backward accumulation: N r^2 / 2 multiply-adds and
// no further barrier.  a is overwritten.
// float and dfloat columns are first scaled by powers of two to a largest
// entry in [1, 2) (Q does not change), so that the squares of graded columns
// stay inside the FP32 exponent range; their dots are summed in runs of eight
// rows.
// The plain form is left at a column that it cannot take (see qr_columns), and
// the safe one goes on from there.  Two functions without calls of their own:
// with the scaling's call inside the plain one an FP64 ensemble's step took 5 %
// longer (18.3 against 17.5 ms), like this 0.2 %.
template <typename T, bool POS, bool SAFE>
__device__ __forceinline__ int qr_form(const Team& tm, int N, int lo, int rows, int r, T* a, int ld, T* qout, int ldq,
                                       T* R, int ldr, const QrSmem<T>& s, int k0) {
  constexpr bool F64 = std::is_same<T, double>::value;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int LT = r + 1;
  const int R0 = tm.rows_per(N);
  const FastDiv by_rows(rows);
  if constexpr (!SAFE)
    for (int e = tid; e < r * LT; e += WT) s.tri[e] = s.v1[e] = T(0);
  if constexpr (SAFE) {
    tm.barrier();  // every CTA is past its reads of column k0's partial dots
  } else if constexpr (!F64) {
    // column maxima: warps take columns, every CTA learns all (slot 0 of both buffers)
    for (int j = warp; j < r; j += WT / 32) {
      float m = 0.0f;
      for (int i = lane; i < rows; i += 32) m = fmaxf(m, fabsf(lead(a[j * ld + i])));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      for (int c = lane; c < tm.C; c += 32) tm.at(s.slot, c)[tm.q * r + j] = T(m);
    }
    tm.barrier();
    if (tid < r) {
      float m = 0.0f;
      for (int c = 0; c < tm.C; ++c) m = fmaxf(m, lead(s.slot[c * r + tid]));
      int e = 0;
      if (m > 0.0f && m < 3.0e38f) frexpf(m, &e);
      s.sgn[tid] = two_to(T(0), max(-120, min(120, 1 - e)));
    }
    __syncthreads();
    for (int e = tid; e < rows * r; e += WT) {
      const int k = by_rows.div(e), i = e - k * rows;
      a[k * ld + i] = a[k * ld + i] * s.sgn[k];
    }
    tm.barrier();  // the slots are reused
  } else {
    __syncthreads();
  }
  const int done = qr_columns<T, POS, SAFE>(tm, lo, rows, r, a, ld, R, ldr, s, R0, k0);
  if (!SAFE && done < r) return done;
  // T: column k is T[:, 0:k] z_k (z_k sits in column k), diagonal tau; eight
  // lanes per row
  constexpr int TU = WR_MAX * 8 / WT;
  for (int k = 1; k < r; ++k) {
    T v[TU];
#pragma unroll
    for (int u = 0; u < TU; ++u) {
      const int i = (tid + u * WT) >> 3;
      T p = T(0);
      if (u * (WT / 8) < r) {  // uniform
        if (i < k)
          for (int l = i + (tid & 7); l < k; l += 8) p = fma(s.tri[i * LT + l], s.tri[l * LT + k], p);
        p += shfl_xor(p, 1);
        p += shfl_xor(p, 2);
        p += shfl_xor(p, 4);
      }
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
  // X = T V1^T (V1 unit lower triangular), X(i, j) at j LT + i for i <= j: the
  // result takes the places of T's transpose
  for (int e = tid; e < r * r; e += WT) {
    const int i = e % r, j = e / r;
    if (i > j) continue;
    T p = s.tri[i * LT + j];
    for (int l = i; l < j; ++l) p = fma(s.tri[i * LT + l], s.v1[j * LT + l], p);
    if (i < j) s.tri[j * LT + i] = p;  // strictly lower entries: T has none there
    else s.tri[j * LT + r] = p;        // the diagonal: the spare column
  }
  // explicit V: zeros above the unit diagonal
  for (int e = tid; e < min(rows, max(0, r - lo)) * r; e += WT) {
    const int i = e / r, k = e - i * r;
    if (lo + i <= k) a[k * ld + i] = (lo + i == k) ? T(1) : T(0);
  }
  __syncthreads();
  if constexpr (F64) {
    for (int e = tid; e < rows * r; e += WT) {
      const int j = by_rows.div(e), i = e - j * rows;
      T p = (lo + i == j) ? T(1) : T(0);
      for (int k = 0; k < j; ++k) p = fma(-a[k * ld + i], s.tri[j * LT + k], p);
      qout[(int64_t)j * ldq + i] = fma(-a[j * ld + i], s.tri[j * LT + r], p);
    }
  } else {
    // four columns per thread share the loads of V
    const int ng = (r + 3) >> 2;
    for (int e = tid; e < rows * ng; e += WT) {
      const int g = by_rows.div(e), i = e - g * rows, j0 = 4 * g, kn = min(r, j0 + 4);
      T p[4] = {T(0), T(0), T(0), T(0)};
      for (int k = 0; k < j0; ++k) {
        const T v = a[k * ld + i];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = fma_acc(v, s.tri[min(j0 + u, r - 1) * LT + k], p[u]);
      }
      for (int k = j0; k < kn; ++k) {
        const T v = a[k * ld + i];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k <= j0 + u && j0 + u < r) p[u] = fma_acc(v, s.tri[(j0 + u) * LT + ((k == j0 + u) ? r : k)], p[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + u < r) {
          T q = ((lo + i == j0 + u) ? T(1) : T(0)) - renorm(p[u]);
          if constexpr (POS) q = q * s.sgn[j0 + u];
          qout[(int64_t)(j0 + u) * ldq + i] = q;
        }
    }
  }
  __syncthreads();
  return r;
}

template <typename T, bool POS>
__device__ __noinline__ int qr_plain(const Team& tm, int N, int lo, int rows, int r, T* a, int ld, T* qout, int ldq,
                                     T* R, int ldr, const QrSmem<T>& s) {
  return qr_form<T, POS, false>(tm, N, lo, rows, r, a, ld, qout, ldq, R, ldr, s, 0);
}
template <typename T, bool POS>
__device__ __noinline__ void qr_safe(const Team& tm, int N, int lo, int rows, int r, T* a, int ld, T* qout, int ldq,
                                     T* R, int ldr, const QrSmem<T>& s, int k0) {
  qr_form<T, POS, true>(tm, N, lo, rows, r, a, ld, qout, ldq, R, ldr, s, k0);
}

template <typename T, bool POS = false>
__device__ __forceinline__ void qr(const Team& tm, int N, int lo, int rows, int r, T* a, int ld, T* qout, int ldq,
                                   T* R, int ldr, const QrSmem<T>& s) {
  const int done = qr_plain<T, POS>(tm, N, lo, rows, r, a, ld, qout, ldq, R, ldr, s);
  if (done < r) qr_safe<T, POS>(tm, N, lo, rows, r, a, ld, qout, ldq, R, ldr, s, done);
}

}  // namespace wide
}  // namespace lri
