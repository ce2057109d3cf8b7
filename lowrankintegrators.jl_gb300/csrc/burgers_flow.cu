// burgers_flow.cu - substep flows of the large Burgers engine (stream.cu) at
// low rank, every RK stage of a flow inside one launch (L and S flows) or a
// few (K flow).
//
// One stage at rank 16 is 1 to 3 us of arithmetic; as separate launches the
// 768 stages of a step (64 RK4 substeps, three flows) were bound by the
// launches themselves: each reloaded the flow tensor, and the S stage read
// n x 2r panels to change a 2r x 2r core.  A step at n = 4096, m = 16384,
// rank 16: 16.0 ms with one launch per stage (S rows 38 us, finish 4 us, K and
// L stages 14 us each), 4.5 ms with the flows below.
#include "burgers_flow.h"

#include <cooperative_groups.h>

namespace lri {
namespace {

namespace cg = cooperative_groups;

constexpr int FL_NT = 256;

__device__ __forceinline__ void fl_ld4(const float* p, float* v) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void fl_ld4(const double* p, double* v) {
  const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
  v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void fl_ld2(const float* p, float* v) {
  const float2 x = *reinterpret_cast<const float2*>(p);
  v[0] = x.x; v[1] = x.y;
}
__device__ __forceinline__ void fl_ld2(const double* p, double* v) {
  const double2 x = *reinterpret_cast<const double2*>(p);
  v[0] = x.x; v[1] = x.y;
}

// active column j of an augmented panel (the first r of each half of 2R)
__device__ __forceinline__ int fl_act(int j, int r, int R) { return (j < r) ? j : R + (j - r); }

// row stride of the pair-major tensor in shared memory
__host__ __device__ constexpr int fl_kpp(int kap) { return kap + 4; }

// Four consecutive columns c0 .. c0 + 3 of one row of
//   sum_{a <= b} KR(P, Q)_ab T'[p(a,b), c],  KR(P, Q)_ab = (P_a Q_b + P_b Q_a) / 2
// (SAME: P == Q); the row's values in registers (zero beyond ka), T'
// pair-major in shared memory, tpt[p kpp + c], zero beyond the active
// columns.  Each 16-byte tensor load serves 4 (8) multiply-adds and is the
// loop's only shared-memory read; a warp's threads share c0, so the tensor
// reads are broadcasts.
template <typename T, int KMAX, bool SAME>
__device__ __forceinline__ void kr_row4(int ka, int kpp, const T (&pv)[KMAX], const T (&qv)[KMAX], const T* tpt,
                                        int c0, T (&acc)[4]) {
  const T* tp = tpt + c0;
#pragma unroll
  for (int a = 0; a < KMAX; ++a) {
    if (a < ka) {
      T g1[4] = {T(0), T(0), T(0), T(0)}, g2[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
      for (int b = a; b < KMAX; ++b) {
        if (b < ka) {
          T t[4];
          fl_ld4(tp, t);
          tp += kpp;
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            g1[v] = fma(qv[b], t[v], g1[v]);
            if (!SAME) g2[v] = fma(pv[b], t[v], g2[v]);
          }
        }
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        if (SAME) acc[v] = fma(qv[a], g1[v], acc[v]);
        else acc[v] = fma(T(0.5), fma(pv[a], g1[v], qv[a] * g2[v]), acc[v]);
      }
    }
  }
}

// the packed tensor's active block, pair-major: tpt[p kpp + c] = Tp[p + c PP]
// for c < ka, zero for ka <= c < kpp; global reads run along the pairs
template <typename T>
__device__ __forceinline__ void load_tensor(int ka, int kap, const T* __restrict__ Tp, int PP, T* tpt) {
  const int np = ka * (ka + 1) / 2, kpp = fl_kpp(kap), total = np * kpp;
  constexpr int U = 8;  // loads in flight per thread
  for (int e0 = threadIdx.x; e0 < total; e0 += U * blockDim.x) {
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * blockDim.x;
      const int pp = e % np, c = e / np;
      v[u] = (e < total && c < ka) ? Tp[pp + (int64_t)c * PP] : T(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * blockDim.x;
      if (e < total) tpt[(e % np) * kpp + e / np] = v[u];
    }
  }
}

// One stage of an explicit RK scheme (sub-diagonal a) with derivative v:
// a = (first ? 0 : a) + b v; returns the next stage's input y + h a_{s+1} v,
// or after the last stage the new y += h a.
template <typename T>
__device__ __forceinline__ T rk_next(const Scheme& sc, int s, T h, T v, T& y, T& a) {
  const T b = T(sc.b[s]);
  a = (s == 0) ? b * v : fma(b, v, a);
  if (s + 1 < sc.nstages) return fma(h * T(sc.a[s + 1]), v, y);
  y = fma(h, a, y);
  return y;
}

// ---------------------------------------------------------------------------
// L flow: the rows are independent ODEs, so a CTA takes FL_ROWS rows through
// every stage of every substep: the tensor and the stage inputs stay in
// shared memory, y and the accumulator in registers (four columns of one row
// per item, KMAX / 16 items per thread), one barrier per stage.  Bound by the
// tensor's shared-memory broadcasts, which feed four multiply-adds each.
// ---------------------------------------------------------------------------
constexpr int FL_ROWS = 64;

template <typename T, int KMAX>
__global__ void __launch_bounds__(FL_NT) l_flow_kernel(int M, int R, const int32_t* __restrict__ rank, T* y,
                                                       const T* __restrict__ nu, const double* __restrict__ Axx,
                                                       const T* __restrict__ Tp, int PP, int nonlin,
                                                       const __grid_constant__ Scheme sc, double hd,
                                                       uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int ka = min(R, (int)*rank);
  if (ka > KMAX) {
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(status, ST_BAD_SHAPE);
    return;
  }
  const T h = T(hd);
  constexpr int IT = KMAX / 16;  // items per thread: FL_ROWS * KMAX / 4 = IT * FL_NT
  const int np = ka * (ka + 1) / 2, kap = (ka + 3) & ~3, ncg = kap / 4, kpp = fl_kpp(kap), ld = KMAX | 1;
  T* tpt = sm;                               // np x kpp
  T* as = tpt + (nonlin ? np * kpp : 0);     // ka x kap: as[a kap + c] = A_xx(a, c)
  T* zs = as + KMAX * KMAX;                  // 2 x FL_ROWS x ld
  const int j0 = blockIdx.x * FL_ROWS, rows = min(FL_ROWS, M - j0);
  if (nonlin) load_tensor(ka, kap, Tp, PP, tpt);
  for (int e = threadIdx.x; e < ka * kap; e += FL_NT) {
    const int a = e / kap, c = e - (e / kap) * kap;
    as[e] = (c < ka) ? T(Axx[a + (int64_t)c * R]) : T(0);
  }
  for (int e = threadIdx.x; e < FL_ROWS * KMAX; e += FL_NT) {
    const int jj = e % FL_ROWS, a = e / FL_ROWS;
    zs[jj * ld + a] = (jj < rows && a < ka) ? y[(j0 + jj) + (int64_t)a * M] : T(0);
  }
  __syncthreads();
  T yv[IT][4], av[IT][4], nj[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = threadIdx.x + it * FL_NT, jj = e % FL_ROWS, c0 = 4 * (e / FL_ROWS);
    nj[it] = (jj < rows) ? nu[j0 + jj] : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      yv[it][q] = zs[jj * ld + c0 + q];
      av[it][q] = T(0);
    }
  }
  T* cur = zs;
  T* nxt = zs + FL_ROWS * ld;
  for (int sub = 0; sub < sc.nsub; ++sub)
    for (int s = 0; s < sc.nstages; ++s) {
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int e = threadIdx.x + it * FL_NT, jj = e % FL_ROWS, cgi = e / FL_ROWS, c0 = 4 * cgi;
        if (cgi < ncg) {
          T z[KMAX];
#pragma unroll
          for (int k = 0; k < KMAX; ++k) z[k] = cur[jj * ld + k];
          T lin[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
          for (int a = 0; a < KMAX; ++a)
            if (a < ka) {
              T t[4];
              fl_ld4(as + a * kap + c0, t);
#pragma unroll
              for (int q = 0; q < 4; ++q) lin[q] = fma(z[a], t[q], lin[q]);
            }
          T kr[4] = {T(0), T(0), T(0), T(0)};
          if (nonlin) kr_row4<T, KMAX, true>(ka, kpp, z, z, tpt, c0, kr);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            nxt[jj * ld + c0 + q] = rk_next(sc, s, h, fma(nj[it], lin[q], kr[q]), yv[it][q], av[it][q]);
        }
      }
      __syncthreads();
      T* t = cur;
      cur = nxt;
      nxt = t;
    }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = threadIdx.x + it * FL_NT, jj = e % FL_ROWS, c0 = 4 * (e / FL_ROWS);
    if (jj < rows)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (c0 + q < ka) y[(j0 + jj) + (int64_t)(c0 + q) * M] = yv[it][q];
  }
}

// ---------------------------------------------------------------------------
// K flow: a stage couples a row to its two neighbours (periodic), so a CTA
// takes a tile of FL_ROWS rows through `q` substeps with nstages * q halo
// rows on each side: every stage makes the outermost row of each side stale,
// and the rows left after the launch are exact.  Two barriers per stage (the
// quadratic term is formed for every row before its Dx).  Halo rows are
// recomputed by the neighbouring CTAs instead of exchanged: no CTA waits for
// another, at FL_ROWS / (FL_ROWS - 2 nstages q) times the arithmetic.
// ---------------------------------------------------------------------------
template <typename T, int KMAX>
__global__ void __launch_bounds__(FL_NT) k_flow_kernel(int N, int R, const int32_t* __restrict__ rank,
                                                       const T* __restrict__ yin, T* __restrict__ yout,
                                                       const double* __restrict__ Nnu, const T* __restrict__ Tp,
                                                       int PP, double ih2d, double ihxd, double alphad, double betad,
                                                       const __grid_constant__ Scheme sc, double hd, int q,
                                                       uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int ka = min(R, (int)*rank);
  if (ka > KMAX) {
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(status, ST_BAD_SHAPE);
    return;
  }
  const T ih2 = T(ih2d), ihx = T(ihxd), alpha = T(alphad), beta = T(betad), h = T(hd);
  constexpr int IT = KMAX / 16;
  const int np = ka * (ka + 1) / 2, kap = (ka + 3) & ~3, ncg = kap / 4, kpp = fl_kpp(kap);
  constexpr int ld = KMAX | 1;
  const bool nonlin = alpha != T(0) || beta != T(0);
  T* tpt = sm;                               // np x kpp
  T* ns = tpt + (nonlin ? np * kpp : 0);     // ka x kap: ns[a kap + c] = N_nu(a, c)
  T* zs = ns + KMAX * KMAX;                  // 2 x (FL_ROWS + 2) x ld, a zero row on each side
  T* ks = zs + 2 * (FL_ROWS + 2) * ld;       // (FL_ROWS + 2) x ld: KR(z, z) T'
  const int H = sc.nstages * q, BM = FL_ROWS - 2 * H;
  const int i0 = blockIdx.x * BM, rows = min(BM, N - i0);
  if (nonlin) load_tensor(ka, kap, Tp, PP, tpt);
  for (int e = threadIdx.x; e < ka * kap; e += FL_NT) {
    const int a = e / kap, c = e - (e / kap) * kap;
    ns[e] = (c < ka) ? T(Nnu[a + (int64_t)c * R]) : T(0);
  }
  for (int e = threadIdx.x; e < 3 * 2 * ld; e += FL_NT) {
    const int b = e / (2 * ld), x = e - b * 2 * ld;
    zs[b * (FL_ROWS + 2) * ld + ((x < ld) ? x : (FL_ROWS + 1) * ld + x - ld)] = T(0);
  }
  for (int e = threadIdx.x; e < FL_ROWS * KMAX; e += FL_NT) {
    const int ii = e % FL_ROWS, a = e / FL_ROWS;
    int g = (i0 - H + ii) % N;
    if (g < 0) g += N;
    zs[(ii + 1) * ld + a] = (a < ka) ? yin[g + (int64_t)a * N] : T(0);
  }
  __syncthreads();
  T yv[IT][4], av[IT][4];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = threadIdx.x + it * FL_NT, ii = e % FL_ROWS, c0 = 4 * (e / FL_ROWS);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      yv[it][u] = zs[(ii + 1) * ld + c0 + u];
      av[it][u] = T(0);
    }
  }
  T* cur = zs;
  T* nxt = zs + (FL_ROWS + 2) * ld;
  for (int sub = 0; sub < q; ++sub)
    for (int s = 0; s < sc.nstages; ++s) {
      if (beta != T(0)) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
          const int e = threadIdx.x + it * FL_NT, ii = e % FL_ROWS, cgi = e / FL_ROWS, c0 = 4 * cgi;
          if (cgi < ncg) {
            T z[KMAX];
#pragma unroll
            for (int k = 0; k < KMAX; ++k) z[k] = cur[(ii + 1) * ld + k];
            T kr[4] = {T(0), T(0), T(0), T(0)};
            kr_row4<T, KMAX, true>(ka, kpp, z, z, tpt, c0, kr);
#pragma unroll
            for (int u = 0; u < 4; ++u) ks[(ii + 1) * ld + c0 + u] = kr[u];
          }
        }
        __syncthreads();
      }
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int e = threadIdx.x + it * FL_NT, ii = e % FL_ROWS, cgi = e / FL_ROWS, c0 = 4 * cgi;
        if (cgi < ncg) {
          const T* zm = cur + ii * ld;
          const T* z0 = zm + ld;
          const T* zp = z0 + ld;
          T v[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
          for (int a = 0; a < KMAX; ++a)
            if (a < ka) {
              const T d2 = ih2 * ((zm[a] + zp[a]) - T(2) * z0[a]);
              T t[4];
              fl_ld4(ns + a * kap + c0, t);
#pragma unroll
              for (int u = 0; u < 4; ++u) v[u] = fma(d2, t[u], v[u]);
            }
          if (alpha != T(0)) {
            T d1[KMAX], zv[KMAX];
#pragma unroll
            for (int k = 0; k < KMAX; ++k) {
              d1[k] = ihx * (zp[k] - zm[k]);
              zv[k] = z0[k];
            }
            T kr[4] = {T(0), T(0), T(0), T(0)};
            kr_row4<T, KMAX, false>(ka, kpp, d1, zv, tpt, c0, kr);
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = fma(alpha, kr[u], v[u]);
          }
          if (beta != T(0))
#pragma unroll
            for (int u = 0; u < 4; ++u)
              v[u] = fma(beta * ihx, ks[(ii + 2) * ld + c0 + u] - ks[ii * ld + c0 + u], v[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            nxt[(ii + 1) * ld + c0 + u] = rk_next(sc, s, h, v[u], yv[it][u], av[it][u]);
        }
      }
      __syncthreads();
      T* t = cur;
      cur = nxt;
      nxt = t;
    }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int e = threadIdx.x + it * FL_NT, ii = e % FL_ROWS, c0 = 4 * (e / FL_ROWS);
    if (ii >= H && ii < H + rows)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + u < ka) yout[(i0 + ii - H) + (int64_t)(c0 + u) * N] = yv[it][u];
  }
  // inactive columns: unchanged
  for (int e = threadIdx.x; e < rows * (R - ka); e += FL_NT) {
    const int64_t o = (i0 + e % rows) + (int64_t)(ka + e / rows) * N;
    yout[o] = yin[o];
  }
}

// ---------------------------------------------------------------------------
// S flow on the 2r x 2r core.  With A = Uhat Z,
//   Uhat^T [alpha KR(Dx A, A) + beta Dx KR(A, A)] T' (column c)
//     = sum_{p <= q} W'[pq, :] (Z T_c Z^T)_pq,
// T_c the symmetric slices of Vhat's tensor (T' holds them packed, the
// off-diagonal pairs doubled) and W' Uhat's packed tensor
// (alpha sym((Dx U)_p U_q) U_d - beta U_p U_q (Dx U)_d summed over the grid:
// Dx^T = -Dx), formed once per step.  A stage then costs O((2r)^4)
// independent of n: at r = 16, 2.6 M multiply-adds against 69 M and a
// 30-row-tile launch of 38 us for n = 4096.
// One cluster of SF_C CTAs takes the core through every stage; a CTA owns
// SF_CPC columns c (slices T_c, the columns of N_nu, y and the accumulator in
// registers), reads W' from its shared memory, and sends its columns of the
// next stage input to every CTA's copy of Z through distributed shared
// memory (two copies in turn, one cluster barrier per stage).
// ---------------------------------------------------------------------------
constexpr int SF_C = 16;
constexpr int SF_CPC = FLOW_KMAX / SF_C;  // 2
constexpr int SF_LD = 36;                 // row stride of the 32 x 32 tiles (16-byte aligned rows)
static_assert(SF_C * SF_CPC == FLOW_KMAX && SF_CPC == 2, "two columns per CTA");

template <typename T>
struct SFlowSmem {
  T z[2][FLOW_KMAX * SF_LD];              // z[k SF_LD + p] = Z(p, k)
  T tc[SF_CPC][FLOW_KMAX * SF_LD];        // T_c(a, b)
  T m1[SF_CPC][FLOW_KMAX * SF_LD];        // (T_c Z^T)(a, q)
  T g[FLOW_KMAX * (FLOW_KMAX + 1) / 2][SF_CPC];  // (Z T_c Z^T) packed pairs
  T w[FLOW_KMAX * (FLOW_KMAX + 1) / 2 * FLOW_KMAX];  // W'[pq, d]
  T red[8][SF_CPC][32];
  T ax[FLOW_KMAX * 33];                   // A_xx(d, k) at k 33 + d
  T nn[SF_CPC][32];                       // N_nu(k, c)
  T t1[SF_CPC][32];                       // (Z N_nu)(k, c)
};

template <typename T>
__global__ void __launch_bounds__(FL_NT, 1) s_flow_kernel(int R, const int32_t* __restrict__ rank, double* Zg,
                                                          const double* __restrict__ Nnu,
                                                          const double* __restrict__ Axx, const T* __restrict__ Tp,
                                                          const T* __restrict__ Wp, int PP, int nonlin,
                                                          const __grid_constant__ Scheme sc, double h,
                                                          uint32_t* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  SFlowSmem<T>& sm = *reinterpret_cast<SFlowSmem<T>*>(smraw);
  cg::cluster_group cl = cg::this_cluster();
  const int r = min(R, (int)*rank), ka = 2 * r, w2 = 2 * R;
  if (ka > FLOW_KMAX) {  // the same in every CTA of the cluster
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(status, ST_BAD_SHAPE);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int np = ka * (ka + 1) / 2, kap = (ka + 3) & ~3;
  const int cb = blockIdx.x * SF_CPC;  // this CTA's columns cb, cb + 1
  for (int e = tid; e < FLOW_KMAX * SF_LD; e += FL_NT) {
    const int k = e / SF_LD, p = e - (e / SF_LD) * SF_LD;
    const bool in = k < ka && p < ka;
    sm.z[0][e] = in ? T(Zg[fl_act(p, r, R) + (int64_t)fl_act(k, r, R) * w2]) : T(0);
    sm.z[1][e] = T(0);
    for (int u = 0; u < SF_CPC; ++u) {
      T v = T(0);
      if (nonlin && in && cb + u < ka) {
        const int a = min(k, p), b = max(k, p);
        v = Tp[a * ka - a * (a - 1) / 2 + (b - a) + (int64_t)(cb + u) * PP] * ((a == b) ? T(1) : T(0.5));
      }
      sm.tc[u][e] = v;
      sm.m1[u][e] = T(0);
    }
  }
  if (nonlin)
    for (int e = tid; e < np * 32; e += FL_NT) {
      const int d = e / np, pq = e - (e / np) * np;
      sm.w[pq * 32 + d] = (d < ka) ? Wp[pq + (int64_t)d * PP] : T(0);
    }
  for (int e = tid; e < 32 * 32; e += FL_NT) {
    const int d = e & 31, k = e >> 5;
    sm.ax[k * 33 + d] = (d < ka && k < ka) ? T(Axx[fl_act(d, r, R) + (int64_t)fl_act(k, r, R) * w2]) : T(0);
  }
  if (tid < 32 * SF_CPC) {
    const int u = tid >> 5, k = tid & 31;
    sm.nn[u][k] = (k < ka && cb + u < ka) ? T(Nnu[fl_act(k, r, R) + (int64_t)fl_act(cb + u, r, R) * w2]) : T(0);
  }
  // the entry (d, c) of the state this thread carries (tid < 64)
  const int du = tid >> 5, dd = tid & 31;
  const bool own = tid < 32 * SF_CPC && dd < ka && cb + du < ka;
  double y = own ? Zg[fl_act(dd, r, R) + (int64_t)fl_act(cb + du, r, R) * w2] : 0.0, acc = 0.0;
  // every CTA has read Z and zeroed its copies before a neighbour writes to them
  cl.sync();
  const int u = tid >> 7, t = tid & 127;  // column and tile of the 32 x 32 products
  const int ct = 4 * (t & 7), rt = 2 * (t >> 3);
  int cur = 0;
  for (int sub = 0; sub < sc.nsub; ++sub)
    for (int s = 0; s < sc.nstages; ++s) {
      const T* z = sm.z[cur];
      if (nonlin && rt < kap && ct < kap) {
        // M1 = T_c Z^T: rows a = rt, rt + 1, columns q = ct .. ct + 3
        T a0[4] = {T(0), T(0), T(0), T(0)}, a1[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
        for (int b = 0; b < ka; ++b) {
          T x[2], v[4];
          fl_ld2(sm.tc[u] + b * SF_LD + rt, x);
          fl_ld4(z + b * SF_LD + ct, v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a0[i] = fma(x[0], v[i], a0[i]);
            a1[i] = fma(x[1], v[i], a1[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sm.m1[u][rt * SF_LD + ct + i] = a0[i];
          sm.m1[u][(rt + 1) * SF_LD + ct + i] = a1[i];
        }
      }
      if (tid < 32 * SF_CPC) {
        T x = T(0);
        for (int k = 0; k < ka; ++k) x = fma(z[k * SF_LD + dd], sm.nn[du][k], x);
        sm.t1[du][dd] = x;
      }
      __syncthreads();
      if (nonlin && rt <= ct + 3 && rt < ka && ct < kap) {
        // G = Z M1 on the pairs p <= q
        T a0[4] = {T(0), T(0), T(0), T(0)}, a1[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
        for (int a = 0; a < ka; ++a) {
          T x[2], v[4];
          fl_ld2(z + a * SF_LD + rt, x);
          fl_ld4(sm.m1[u] + a * SF_LD + ct, v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a0[i] = fma(x[0], v[i], a0[i]);
            a1[i] = fma(x[1], v[i], a1[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int q = ct + i;
          if (rt <= q && q < ka) sm.g[rt * ka - rt * (rt - 1) / 2 + q - rt][u] = a0[i];
          if (rt + 1 <= q && q < ka) sm.g[(rt + 1) * ka - (rt + 1) * rt / 2 + q - rt - 1][u] = a1[i];
        }
      }
      T lin = T(0);
      if (tid < 32 * SF_CPC)
        for (int k = 0; k < ka; ++k) lin = fma(sm.ax[k * 33 + dd], sm.t1[du][k], lin);
      __syncthreads();
      if (nonlin) {
        T a0 = T(0), a1 = T(0);
        const int lo = warp * np / 8, hi = (warp + 1) * np / 8;
#pragma unroll 4
        for (int pq = lo; pq < hi; ++pq) {
          const T wv = sm.w[pq * 32 + lane];
          T gv[2];
          fl_ld2(sm.g[pq], gv);
          a0 = fma(wv, gv[0], a0);
          a1 = fma(wv, gv[1], a1);
        }
        sm.red[warp][0][lane] = a0;
        sm.red[warp][1][lane] = a1;
        __syncthreads();
      }
      if (own) {
        double v = (double)lin;
        if (nonlin)
#pragma unroll
          for (int k = 0; k < 8; ++k) v += (double)sm.red[k][du][dd];
        const T zn = T(rk_next<double>(sc, s, h, v, y, acc));
#pragma unroll
        for (int c = 0; c < SF_C; ++c) cl.map_shared_rank(sm.z[cur ^ 1], c)[(cb + du) * SF_LD + dd] = zn;
      }
      cl.sync();
      cur ^= 1;
    }
  if (own) Zg[fl_act(dd, r, R) + (int64_t)fl_act(cb + du, r, R) * w2] = y;
}

// dynamic shared memory at active widths up to K
template <typename T, int K>
constexpr size_t l_flow_smem() {
  return sizeof(T) * ((size_t)K * (K + 1) / 2 * fl_kpp(K) + K * K + 2 * FL_ROWS * (K | 1));
}
template <typename T, int K>
constexpr size_t k_flow_smem() {
  return sizeof(T) * ((size_t)K * (K + 1) / 2 * fl_kpp(K) + K * K + 3 * (FL_ROWS + 2) * (K | 1));
}
static_assert(k_flow_smem<double, FLOW_KMAX>() <= 227 * 1024 && l_flow_smem<double, FLOW_KMAX>() <= 227 * 1024 &&
                  sizeof(SFlowSmem<double>) <= 227 * 1024,
              "flow kernels exceed an SM's shared memory");

template <typename T, int KMAX>
cudaError_t k_flow_run(int N, int R, const int32_t* rank, T* y, T* tmp, const double* Nnu, const T* Tp, int PP,
                       double ih2, double ihx, double alpha, double beta, const Scheme& sc, double h, int sms,
                       uint32_t* status, cudaStream_t st) {
  constexpr size_t smem = k_flow_smem<T, KMAX>();
  static std::atomic<uint64_t> done{0};
  cudaError_t e = set_smem_limit(k_flow_kernel<T, KMAX>, (int)smem, done);
  if (e != cudaSuccess) return e;
  // Substeps per launch: as many as the halo leaves half of the tile's rows
  // for (4 at RK4) while the tiles still run at once, else half as many,
  // which recompute less (n = 4096: 128 tiles of 32 rows, 16 launches).
  int q = FL_ROWS / 4 / sc.nstages;
  if ((N + FL_ROWS / 2 - 1) / (FL_ROWS / 2) > sms) q = (q + 1) / 2;
  const int launches = (sc.nsub + q - 1) / q;
  // the panels alternate; an odd count starts from a copy so that y ends in place
  T* a = y;
  T* b = tmp;
  if (launches & 1) {
    e = cudaMemcpyAsync(tmp, y, sizeof(T) * (size_t)N * R, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    a = tmp;
    b = y;
  }
  for (int k = 0, left = sc.nsub; k < launches; ++k) {
    const int qk = left < q ? left : q;
    const int BM = FL_ROWS - 2 * sc.nstages * qk;
    k_flow_kernel<T, KMAX><<<(N + BM - 1) / BM, FL_NT, smem, st>>>(N, R, rank, a, b, Nnu, Tp, PP, ih2, ihx, alpha,
                                                                   beta, sc, h, qk, status);
    left -= qk;
    T* t = a;
    a = b;
    b = t;
  }
  return cudaGetLastError();
}

template <typename T, int KMAX>
cudaError_t l_flow_run(int M, int R, const int32_t* rank, T* y, const T* nu, const double* Axx, const T* Tp, int PP,
                       int nonlin, const Scheme& sc, double h, uint32_t* status, cudaStream_t st) {
  constexpr size_t smem = l_flow_smem<T, KMAX>();
  static std::atomic<uint64_t> done{0};
  cudaError_t e = set_smem_limit(l_flow_kernel<T, KMAX>, (int)smem, done);
  if (e != cudaSuccess) return e;
  l_flow_kernel<T, KMAX><<<(M + FL_ROWS - 1) / FL_ROWS, FL_NT, smem, st>>>(M, R, rank, y, nu, Axx, Tp, PP, nonlin,
                                                                          sc, h, status);
  return cudaGetLastError();
}

}  // namespace

template <typename T>
cudaError_t burgers_k_flow(int kmax, int N, int R, const int32_t* rank, T* y, T* tmp, const double* Nnu, const T* Tp,
                           int PP, double ih2, double ihx, double alpha, double beta, const Scheme& sc, double h,
                           int sms, uint32_t* status, cudaStream_t st) {
  return kmax <= 16 ? k_flow_run<T, 16>(N, R, rank, y, tmp, Nnu, Tp, PP, ih2, ihx, alpha, beta, sc, h, sms, status, st)
                    : k_flow_run<T, 32>(N, R, rank, y, tmp, Nnu, Tp, PP, ih2, ihx, alpha, beta, sc, h, sms, status, st);
}

template <typename T>
cudaError_t burgers_l_flow(int kmax, int M, int R, const int32_t* rank, T* y, const T* nu, const double* Axx,
                           const T* Tp, int PP, int nonlin, const Scheme& sc, double h, uint32_t* status,
                           cudaStream_t st) {
  return kmax <= 16 ? l_flow_run<T, 16>(M, R, rank, y, nu, Axx, Tp, PP, nonlin, sc, h, status, st)
                    : l_flow_run<T, 32>(M, R, rank, y, nu, Axx, Tp, PP, nonlin, sc, h, status, st);
}

template <typename T>
cudaError_t burgers_s_flow(int R, const int32_t* rank, double* Z, const double* Nnu, const double* Axx, const T* Tp,
                           const T* Wp, int PP, int nonlin, const Scheme& sc, double h, uint32_t* status,
                           cudaStream_t st) {
  static std::atomic<uint64_t> done{0}, wide{0};
  cudaError_t e = set_smem_limit(s_flow_kernel<T>, (int)sizeof(SFlowSmem<T>), done);
  if (e != cudaSuccess) return e;
  // clusters of 16 need the kernel's opt-in (per device, as set_smem_limit)
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  const uint64_t bit = (dev < 64) ? (uint64_t(1) << dev) : 0;
  if (!bit || !(wide.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(s_flow_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    if (bit) wide.fetch_or(bit, std::memory_order_acq_rel);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(SF_C, 1, 1);
  cfg.blockDim = dim3(FL_NT, 1, 1);
  cfg.dynamicSmemBytes = sizeof(SFlowSmem<T>);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = SF_C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, s_flow_kernel<T>, R, rank, Z, Nnu, Axx, Tp, Wp, PP, nonlin, sc, h, status);
  return e != cudaSuccess ? e : cudaGetLastError();
}

#define LRI_FLOW_INST(T)                                                                                             \
  template cudaError_t burgers_k_flow<T>(int, int, int, const int32_t*, T*, T*, const double*, const T*, int, double,    \
                                         double, double, double, const Scheme&, double, int, uint32_t*,            \
                                         cudaStream_t);                                                             \
  template cudaError_t burgers_l_flow<T>(int, int, int, const int32_t*, T*, const T*, const double*, const T*, int, int, \
                                         const Scheme&, double, uint32_t*, cudaStream_t);                           \
  template cudaError_t burgers_s_flow<T>(int, const int32_t*, double*, const double*, const double*, const T*,      \
                                         const T*, int, int, const Scheme&, double, uint32_t*, cudaStream_t);
LRI_FLOW_INST(float)
LRI_FLOW_INST(double)
#undef LRI_FLOW_INST

}  // namespace lri
