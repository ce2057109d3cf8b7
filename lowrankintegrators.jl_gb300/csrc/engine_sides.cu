// engine_sides.cu - BUG steps of double-float Sylvester batches with the panels
// of a side in shared memory.
//
// A step is two launches: sides_kernel takes every (instance, side) pair - the
// K and L steps read only the old factors - and core_kernel (engine_df.cu)
// every instance's S step.  A side runs on one CTA, or on a cluster of 2 to 16
// CTAs that split its rows where its three panels would not leave room for
// two CTAs on an SM.  The work is grouped into classes by cluster size and
// shared memory, one launch each.
//
// Against one CTA per instance with the panels in global scratch (bug_step):
// every stage, Gram pass and triangular solve re-staged its panel through L2;
// here they read shared memory in place, and both sides run at once.  Batches
// of 300 uneven members (n, m to 1024, r 6 to 30): 3.4 -> 1.9 ms per step; of
// 366 graded members at n = m = 256, r 23 to 32: 2.6 -> 1.9 ms, most of it
// FP32 issue of the 12-instruction multiply-adds (QR a third).
#include <algorithm>

#include "engine_api.h"
#include "wide.cuh"

namespace lri {
namespace {

using wide::FastDiv;
using wide::lanes_for;
using wide::load_rows;
using wide::load_rows_halo;
using wide::push_halos;
using wide::QrSmem;
using wide::reduce_parts;
using wide::Team;
using wide::WT;

// small-scratch block indices shared with the instance engine (engine_impl.cuh)
enum : int { SB_GU = 0, SB_GV = 2, SB_M = 4, SB_N = 5, SB_NEWU = 13, SB_NEWV = 14 };

__host__ __device__ inline int side_ld(int N, int C) { return ((N + C - 1) / C + 2) | 1; }
// bytes of the small area: the r x rp matrix of the substep or the Gram partials
// (two r x r matrices), and the tridiagonal rows
__host__ __device__ inline size_t side_small_bytes(int r) {
  const size_t rp = (r + 3) & ~3, mat = 8 * (r * rp), part = 16 * (size_t)r * r;
  return mat > part ? mat : part;
}
// the QR's scratch: two r x r matrices, then the factor and its vectors
// (CholSmem), or a Householder QR's scratch in the place of the latter
__host__ __device__ inline size_t qr_bytes(int C, int r) {
  const int rp = (r + 3) & ~3;
  const size_t ch = 8 * ((size_t)r * rp + rp) + 4 * ((size_t)r * C + r) + 16;
  const size_t hh = sizeof(dfloat) * QrSmem<dfloat>::elems(C, r);
  return ch > hh ? ch : hh;
}
// it lies in the two panels that are free during the QR where it fits
__host__ __device__ inline bool qr_overlaid(int N, int C, int r) {
  const size_t panel = 8 * (size_t)r * side_ld(N, C);
  return 16 * (size_t)r * r <= panel - 16 && qr_bytes(C, r) <= panel - 16;
}
__host__ __device__ inline size_t side_bytes(int N, int r, int C) {
  const int R0 = (N + C - 1) / C;
  return 24 * (size_t)r * side_ld(N, C) + 16 + side_small_bytes(r) + 24 * (size_t)R0 + 16 +
         (qr_overlaid(N, C, r) ? 0 : 16 * (size_t)r * r + qr_bytes(C, r) + 16);
}

// out(i, c) = sum_k w(i, k) M(k, c) for this CTA's rows: a row by four columns per
// thread, w column-major with odd stride (conflict-free), M row-major
// (broadcast 16-byte loads); epi(i, c0, acc) gets four columns.
template <class E>
__device__ __forceinline__ void panel_mul(int rows, int r, const dfloat* w, int ld, const dfloat* M, int rp,
                                          const E& epi) {
  const int ng = rp >> 2;
  const FastDiv by(rows);
  for (int e = threadIdx.x; e < rows * ng; e += WT) {
    const int g = by.div(e), i = e - g * rows;
    dfloat acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = dfloat(0.0f, 0.0f);
    const dfloat* m = M + 4 * g;
#pragma unroll 4
    for (int k = 0; k < r; ++k) {
      const dfloat x = w[k * ld + i];
      dfloat v[4];
      ld4(m + k * rp, v);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = lri_df::fma_acc(x, v[u], acc[u]);
    }
    epi(i, 4 * g, acc);
  }
}

// Two products over this CTA's rows in double-float, M = Q^T X and P = Q^T Y:
// part[o] and part[r r + o], o = a + c r
__device__ __forceinline__ void gram_pair(int rows, int r, const dfloat* Q, const dfloat* X, const dfloat* Y, int ld,
                                          bool both, dfloat* part) {
  const int rr = r * r, L = lanes_for(rr), per = WT / L, l = threadIdx.x & (L - 1);
  const FastDiv by(r);
  for (int o0 = 0; o0 < rr; o0 += per) {
    const int o = o0 + threadIdx.x / L;
    dfloat sx(0.0f, 0.0f), sy(0.0f, 0.0f);
    if (o < rr) {
      const int c = by.div(o), a = o - c * r;
      const dfloat* q = Q + a * ld;
      const dfloat* x = X + c * ld;
      const dfloat* y = Y + c * ld;
      int cnt = 0;
#pragma unroll 4
      for (int i = l; i < rows; i += L) {
        const dfloat qv = q[i];
        if (both) sx = lri_df::fma_acc(qv, x[i], sx);
        sy = lri_df::fma_acc(qv, y[i], sy);
        if ((++cnt & 31) == 0) {
          sx = renorm(sx);
          sy = renorm(sy);
        }
      }
      sx = renorm(sx);
      sy = renorm(sy);
    }
    for (int s = L >> 1; s > 0; s >>= 1) {
      if (both) sx += shfl_xor(sx, s);
      sy += shfl_xor(sy, s);
    }
    if (o < rr && l == 0) {
      if (both) part[o] = sx;
      part[rr + o] = sy;
    }
  }
}

// ---------------------------------------------------------------------------
// QR of a side's panel by CholeskyQR (a positive diagonal of R) on shared
// memory: three cluster barriers per pass instead of one per column.  The
// columns are first scaled by powers of two (Q does not change).  Every pass:
// the upper Gram triangle, a Cholesky factor in every CTA, a row-wise
// triangular solve (backward stable).  Two passes while the factor's diagonal
// shows kappa(K) <= 1e6, else three with a shifted first one (Fukaya et al.
// 2020).  Returns false on a breakdown (a holds the panel or a previous
// pass's result); the caller falls back to Householder.
// ---------------------------------------------------------------------------
struct CholSmem {
  dfloat* G;    // r x r: Gram matrix, packed sums before
  dfloat* gs;   // r x r: partial sums
  dfloat* Rt;   // r x rp: the factor, row-major
  dfloat* inv;  // rp: inverse diagonal
  float* top;   // C x r: column maxima; then the factor's outcome
  float* sgn;   // r: column scales
};

// packed upper-triangle index o (by columns) -> (a, c), a <= c
__device__ __forceinline__ void packed_pair(int o, int& a, int& c) {
  c = (int)((sqrtf(8.0f * (float)o + 1.0f) - 1.0f) * 0.5f);
  while (c * (c + 1) / 2 > o) --c;
  while ((c + 1) * (c + 2) / 2 <= o) ++c;
  a = o - c * (c + 1) / 2;
}

// 1 / sqrt(d) in double-float from the FP32 estimate y: with e = 1 - d y^2,
// y (1 - e)^(-1/2) = y + y (e / 2 + 3 e^2 / 8 + ...)
__device__ __forceinline__ dfloat rsqrt_df(dfloat d) {
  const float y = rsqrtf(d.hi);
  const dfloat dy = d * dfloat(y, 0.0f);  // d y
  const float p = dy.hi * y, e = fmaf(dy.hi, y, -p);
  const float res = ((1.0f - p) - e) - dy.lo * y;  // 1 - d y^2 (1 - p is exact: p is within 2^-20 of 1)
  return lri_df::fast_two_sum(y, y * res * fmaf(0.375f, res, 0.5f));
}

// Cholesky factor G = R^T R of the upper triangle of G (r x r, column-major in
// shared memory) plus shift I, into Rt (row-major, zero below the diagonal)
// and inv; G is kept.  The entries stay in registers; per step the pivot row
// goes through shared memory (one barrier) and the trailing entries take
// v_ij -= g_i (g_j / d); rows are scaled by 1 / sqrt(d) at the end.  False on a
// non-positive pivot.
__device__ __noinline__ bool chol_rows(int r, const dfloat* G, dfloat shift, const CholSmem& s) {
  constexpr int EU = (wide::WR_MAX * (wide::WR_MAX + 1) / 2 + WT - 1) / WT;
  const int tid = threadIdx.x, np = r * (r + 1) / 2, rp = (r + 3) & ~3;
  dfloat v[EU];
  int ij[EU];  // i | j << 8, i <= j
#pragma unroll
  for (int u = 0; u < EU; ++u) {
    const int o = tid + u * WT;
    ij[u] = 255;
    v[u] = dfloat(0.0f, 0.0f);
    if (o < np) {
      int a, c;
      packed_pair(o, a, c);
      ij[u] = a | (c << 8);
      v[u] = G[a + c * r];
      if (a == c) v[u] += shift;
    }
  }
  for (int e = tid; e < r * rp; e += WT) s.Rt[e] = dfloat(0.0f, 0.0f);
  __syncthreads();
  bool ok = true;
  for (int k = 0; k < r; ++k) {
    dfloat* row = s.Rt + k * rp;  // unscaled until the end
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      if (u * WT >= np) break;
      if ((ij[u] & 255) == k) row[ij[u] >> 8] = v[u];
    }
    __syncthreads();
    const dfloat d = row[k];
    ok = ok && d.hi > 0.0f;
    // 1 / d from the FP32 reciprocal, one Newton step
    const float q = (d.hi > 0.0f) ? 1.0f / d.hi : 1.0f;
    const float p = q * d.hi, res = ((1.0f - p) - fmaf(q, d.hi, -p)) - q * d.lo;
    const dfloat id = lri_df::fast_two_sum(q, q * fmaf(res, res, res));
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      if (u * WT >= np) break;
      const int i = ij[u] & 255, j = ij[u] >> 8;
      if (i > k && i < 255) v[u] = fma(-row[i], row[j] * id, v[u]);
    }
  }
  __syncthreads();
  for (int j = tid; j < rp; j += WT) {
    const dfloat d = (j < r) ? s.Rt[j * rp + j] : dfloat(0.0f, 0.0f);
    s.inv[j] = (d.hi > 0.0f) ? rsqrt_df(d) : dfloat(0.0f, 0.0f);
  }
  __syncthreads();
  for (int e = tid; e < r * rp; e += WT) s.Rt[e] = s.Rt[e] * s.inv[e / rp];
  __syncthreads();
  return ok;
}

__device__ __noinline__ bool cholqr(const Team& tm, int N, int lo, int rows, int r, dfloat* a, int ld,
                                    const CholSmem& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rp = (r + 3) & ~3, np = r * (r + 1) / 2;
  const FastDiv by_rows(rows);
  // column scales from the maxima over the cluster
  for (int j = warp; j < r; j += WT / 32) {
    float m = 0.0f;
    for (int i = lane; i < rows; i += 32) m = fmaxf(m, fabsf(a[j * ld + i].hi));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    for (int c = lane; c < tm.C; c += 32) tm.at(s.top, c)[tm.q * r + j] = m;
  }
  tm.barrier();
  if (tid < r) {
    float m = 0.0f;
    for (int c = 0; c < tm.C; ++c) m = fmaxf(m, s.top[c * r + tid]);
    int e = 0;
    if (m > 0.0f && m < 3.0e38f) frexpf(m, &e);
    s.sgn[tid] = ldexpf(1.0f, max(-120, min(120, 1 - e)));
  }
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    a[k * ld + i] = dfloat(a[k * ld + i].hi * s.sgn[k], a[k * ld + i].lo * s.sgn[k]);
  }
  __syncthreads();
  int npass = 2;
  for (int pass = 0; pass < npass; ++pass) {
    // upper triangle of the Gram matrix, packed by columns in gs
    const int L = lanes_for(np), per = WT / L, l = tid & (L - 1);
    for (int o0 = 0; o0 < np; o0 += per) {
      const int o = o0 + tid / L;
      dfloat sum(0.0f, 0.0f);
      if (o < np) {
        int ra, c;
        packed_pair(o, ra, c);
        const dfloat* x = a + ra * ld;
        const dfloat* y = a + c * ld;
        int cnt = 0;
#pragma unroll 4
        for (int i = l; i < rows; i += L) {
          sum = lri_df::fma_acc(x[i], y[i], sum);
          if ((++cnt & 31) == 0) sum = renorm(sum);
        }
        sum = renorm(sum);
      }
      for (int q = L >> 1; q > 0; q >>= 1) sum += shfl_xor(sum, q);
      if (o < np && l == 0) s.gs[o] = sum;
    }
    __syncthreads();
    // the sums to the first CTA, which factors and sends R, its inverse diagonal
    // and the outcome (flag: 0 breakdown, 1 fine, 2 shifted) to the others
    reduce_parts(tm, s.gs, np, [&](int o, dfloat v) {
      int ra, c;
      packed_pair(o, ra, c);
      tm.at(s.G, 0)[ra + c * r] = v;
    });
    if (tm.q == 0) {
      bool ok = chol_rows(r, s.G, dfloat(0.0f, 0.0f), s);
      int flag = ok;
      if (pass == 0) {
        float imax = 0.0f, imin = 3.0e38f;
        for (int j = 0; j < r; ++j) {
          imax = fmaxf(imax, s.inv[j].hi);
          imin = fminf(imin, s.inv[j].hi);
        }
        if (!ok || !(imax <= 1.0e6f * imin)) {
          // shift 11 (N r + r (r + 1)) u trace(G), u = 2^-44 for the double-float arithmetic
          dfloat tr(0.0f, 0.0f);
          for (int j = 0; j < r; ++j) tr += s.G[j + j * r];
          __syncthreads();
          ok = chol_rows(r, s.G, tr * dfloat(11.0 * ((double)N * r + (double)r * (r + 1)) * 5.7e-14), s);
          flag = ok ? 2 : 0;
        }
      }
      for (int c = 1; c < tm.C; ++c)
        for (int e = tid; e < r * rp + rp; e += WT) tm.at(s.Rt, c)[e] = s.Rt[e];  // inv follows Rt
      if (tid < tm.C) tm.at(s.top, tid)[0] = (float)flag;
    }
    tm.barrier();
    const int flag = (int)s.top[0];
    if (flag == 2) npass = 3;
    const bool ok = flag != 0;
    if (!ok) return false;
    // X <- X R^-1: four lanes per row, one column of a block of four each
    for (int i0 = 0; i0 < rows; i0 += WT / 4) {
      const int i = i0 + (tid >> 2), u = tid & 3;
      const bool in = i < rows;
      dfloat* x = a + (in ? i : 0);
      for (int jb = 0; jb < r; jb += 4) {
        const dfloat* R = s.Rt + jb + u;
        dfloat acc(0.0f, 0.0f), acc2(0.0f, 0.0f);
#pragma unroll 2
        for (int k = 0; k < jb; k += 2) {
          acc = lri_df::fma_acc(x[k * ld], R[k * rp], acc);
          acc2 = lri_df::fma_acc(x[(k + 1) * ld], R[(k + 1) * rp], acc2);
        }
        const int j = jb + u;
        dfloat sum = renorm(acc) + renorm(acc2), xj(0.0f, 0.0f);
        const dfloat kj = (j < r) ? x[j * ld] : dfloat(0.0f, 0.0f);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if (u == v) xj = (kj - sum) * s.inv[min(j, rp - 1)];
          const dfloat xv(__shfl_sync(0xffffffffu, xj.hi, (lane & ~3) | v), __shfl_sync(0xffffffffu, xj.lo, (lane & ~3) | v));
          if (u > v && jb + v < r) sum = fma(xv, R[(jb + v) * rp], sum);
        }
        __syncwarp();
        if (in && j < r) x[j * ld] = xj;
        __syncwarp();
      }
    }
    __syncthreads();
  }
  return true;
}

__global__ void __launch_bounds__(WT, 2)
    sides_kernel(const __grid_constant__ StepArgs<dfloat> g, const int32_t* __restrict__ items, int C) {
  using T = dfloat;
  extern __shared__ __align__(16) unsigned char smraw[];
  Team tm{wide::cg::this_cluster(), (int)wide::cg::this_cluster().block_rank(), C};
  const int tid = threadIdx.x, item = items[blockIdx.x / C], inst = item >> 1;
  const bool kside = (item & 1) == 0;
  const InstDesc d = g.inst[inst];
  const int r = g.rank[inst], W = d.wcap;
  if (r < 1 || r > d.rcap) {  // the same in every CTA of the cluster
    if (tid == 0) atomicOr(g.status, ST_BAD_SHAPE);
    return;
  }
  const int N = kside ? d.n : d.m, No = kside ? d.m : d.n;
  T* X = kside ? g.U + d.offU : g.V + d.offV;
  const T* Xo = kside ? g.V + d.offV : g.U + d.offU;
  const T* S = g.S + d.offS;
  const T* tri = kside ? g.opA + d.offA : g.opB + d.offB;
  const int64_t bs = ((int64_t)W * W + 3) & ~int64_t(3);
  T* small = g.small + d.offSmall;
  auto blk = [&](int i) { return small + i * bs; };
  T* Po = blk(kside ? SB_GV : SB_GU) + (int64_t)r * W;  // P of the other (old) basis
  const bool fresh = g.proj_valid[inst] == 0;
  const int R0 = tm.rows_per(N), lo = tm.lo(N), rows = tm.hi(N) - lo, ld = side_ld(N, C), rp = (r + 3) & ~3, rr = r * r;
  T* p0 = reinterpret_cast<T*>(smraw);
  T* p1 = p0 + r * ld;
  T* p2 = p1 + r * ld;
  auto align16 = [](unsigned char* p) {
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15));
  };
  unsigned char* mp = align16(reinterpret_cast<unsigned char*>(p2 + r * ld));
  T* mat = reinterpret_cast<T*>(mp);               // r x rp, row-major
  dfloat* part = reinterpret_cast<dfloat*>(mp);    // Gram partials (never beside mat)
  T* ts = reinterpret_cast<T*>(mp + side_small_bytes(r));  // sub, dia, sup of this CTA's rows (zero outside)
  const FastDiv by_rows(rows);
  if (C > 1) tm.cl.sync();  // every CTA runs before any distributed access
  if (fresh) {
    // P = Xo^T (To Xo) of the other basis, in blocks of at most R0 rows
    const T* to = kside ? g.opB + d.offB : g.opA + d.offA;
    const int lo2 = tm.lo(No), hi2 = tm.hi(No);
    dfloat* sum = part;
    for (int e = tid; e < rr; e += WT) sum[e] = dfloat(0.0f, 0.0f);
    for (int b = lo2; b < hi2; b += R0) {
      const int nb = min(R0, hi2 - b);
      const FastDiv by_nb(nb);
      __syncthreads();
      load_rows_halo(Xo, No, b, nb, r, p0, ld);
      __syncthreads();
      for (int e = tid; e < nb * r; e += WT) {
        const int k = by_nb.div(e), i = e - k * nb, gi = b + i;
        const T* w = p0 + k * ld + i;
        const T cs = gi > 0 ? to[gi] : T(0), cp = gi + 1 < No ? to[2 * No + gi] : T(0);
        p1[k * ld + 1 + i] = fma(cs, w[0], fma(cp, w[2], to[No + gi] * w[1]));
      }
      __syncthreads();
      gram_pair(nb, r, p0 + 1, p0 + 1, p1 + 1, ld, false, part);
      __syncthreads();
      for (int e = tid; e < rr; e += WT) sum[e] += part[rr + e];
    }
    __syncthreads();
    reduce_parts(tm, sum, rr, [&](int e, dfloat s) {
      Po[e % r + (int64_t)(e / r) * W] = s;
    });
  }
  // zero halo rows at the ends of the domain (never pushed to)
  for (int e = tid; e < 3 * r; e += WT) {
    T* p = (e < r) ? p0 : (e < 2 * r ? p1 : p2);
    const int k = e % r;
    p[k * ld] = T(0);
    p[k * ld + 1 + R0] = T(0);
    p[k * ld + 1 + rows] = T(0);
  }
  // K0 = X C, C = S (K) or S^T (L)
  for (int e = tid; e < r * rp; e += WT) {
    const int k = e / rp, c = e - k * rp;
    mat[e] = (c < r) ? (kside ? S[k + (int64_t)c * d.rcap] : S[c + (int64_t)k * d.rcap]) : T(0);
  }
  for (int i = tid; i < rows; i += WT) {
    const int gi = lo + i;
    ts[i] = gi > 0 ? tri[gi] : T(0);
    ts[R0 + i] = tri[N + gi];
    ts[2 * R0 + i] = gi + 1 < N ? tri[2 * N + gi] : T(0);
  }
  load_rows(X, N, lo, rows, r, p1, ld);
  __syncthreads();
  panel_mul(rows, r, p1 + 1, ld, mat, rp, [&](int i, int c0, const T (&acc)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u < r) p0[(c0 + u) * ld + 1 + i] = p2[(c0 + u) * ld + 1 + i] = renorm(acc[u]);
  });
  __syncthreads();
  for (int e = tid; e < r * rp; e += WT) {
    const int k = e / rp, c = e - k * rp;
    mat[e] = (c < r) ? Po[c + (int64_t)k * W] : T(0);  // P(c, k)
  }
  T* win = p0;
  T* wout = p1;
  if (C > 1) tm.cl.sync();  // the zero halo rows of every CTA are set
  if (C > 1) push_halos(tm, N, rows, r, win, ld);
  tm.barrier();
  // Horner form of the substep flow: w <- g_j y + h (T w + w P^T)
  const Scheme& sc = kside ? g.sK : g.sL;
  const T h = T(g.dt / sc.nsub);
  for (int sub = 0; sub < sc.nsub; ++sub) {
    T hw = h * T(sc.gam[sc.nstages]);
    for (int j = sc.nstages - 1; j >= 0; --j) {
      const T gj = (j == 0) ? T(1) : T(sc.gam[j]);
      const bool up = tm.q > 0, dn = tm.q + 1 < C && lo + rows < N;
      panel_mul(rows, r, win + 1, ld, mat, rp, [&](int i, int c0, const T (&acc)[4]) {
        const T cs = ts[i], cd = ts[R0 + i], cp = ts[2 * R0 + i];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u;
          if (c >= r) break;
          const T* w = win + c * ld + i;
          const T tz = fma(cs, w[0], fma(cp, w[2], cd * w[1]));
          const T v = fma(hw, tz + renorm(acc[u]), gj * p2[c * ld + 1 + i]);
          wout[c * ld + 1 + i] = v;
          if (j == 0) p2[c * ld + 1 + i] = v;  // the next substep's base
          if (C > 1) {
            if (i == 0 && up) tm.at(wout, tm.q - 1)[c * ld + 1 + R0] = v;
            if (i == rows - 1 && dn) tm.at(wout, tm.q + 1)[c * ld] = v;
          }
        }
      });
      tm.barrier();
      T* t = win;
      win = wout;
      wout = t;
      hw = h;
    }
  }
  {
    // scratch in the two free panels, or behind the small area
    const bool over = qr_overlaid(N, C, r);
    unsigned char* tail = reinterpret_cast<unsigned char*>(ts + 3 * R0);
    unsigned char* m2 = align16(over ? reinterpret_cast<unsigned char*>(wout) : tail);
    unsigned char* fac = align16(over ? reinterpret_cast<unsigned char*>(p2) : m2 + 16 * (size_t)rr);
    CholSmem cs;
    cs.G = reinterpret_cast<dfloat*>(m2);
    cs.gs = cs.G + rr;
    cs.Rt = reinterpret_cast<dfloat*>(fac);
    cs.inv = cs.Rt + r * rp;
    cs.top = reinterpret_cast<float*>(cs.inv + rp);
    cs.sgn = cs.top + r * C;
    const QrSmem<T> qs = QrSmem<T>::carve(reinterpret_cast<T*>(fac), C, r);
    if (!cholqr(tm, N, lo, rows, r, win + 1, ld, cs)) {  // uniform over the cluster
      tm.barrier();
      wide::qr<T, true>(tm, N, lo, rows, r, win + 1, ld, wout + 1, ld, static_cast<T*>(nullptr), 0, qs);
      T* t = win;
      win = wout;
      wout = t;
    }
  }
  // basis change Q^T X0 and the new basis's projection Q^T (T Q)
  T* Q = win;
  win = wout;
  // (the QR's scratch may have overwritten the panel's halo rows)
  for (int k = tid; k < r; k += WT) {
    if (tm.q == 0) Q[k * ld] = T(0);
    if (lo + rows == N) Q[k * ld + 1 + rows] = T(0);
  }
  load_rows(X, N, lo, rows, r, win, ld);
  if (C > 1) {
    push_halos(tm, N, rows, r, Q, ld);
    tm.cl.sync();
  }
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    const T* w = Q + k * ld + i;
    p2[k * ld + 1 + i] = fma(ts[i], w[0], fma(ts[2 * R0 + i], w[2], ts[R0 + i] * w[1]));
  }
  __syncthreads();
  gram_pair(rows, r, Q + 1, win + 1, p2 + 1, ld, true, part);
  dfloat* Mo = blk(kside ? SB_M : SB_N);
  dfloat* Pn = blk(kside ? SB_NEWU : SB_NEWV);
  __syncthreads();
  reduce_parts(tm, part, 2 * rr, [&](int e, dfloat s) {
    ((e < rr) ? Mo : Pn)[e % r + (int64_t)((e / r) % r) * W] = s;
  });
  // in place where nobody else reads these rows, else to the workspace (the
  // other side of a first step reads the old basis; core_kernel copies)
  T* dst = !fresh ? X : g.work + (kside ? d.offWK : d.offWL);
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    dst[lo + i + (int64_t)k * N] = Q[k * ld + 1 + i];
  }
}

}  // namespace

// Classes by cluster size (the largest first) and by whether two CTAs fit an SM,
// longest work first inside a class.
bool group_sides(std::vector<SideItem>& v, SidesPlan* p, std::vector<int32_t>* items) {
  auto group = [](const SideItem& x) { return 2 * x.C + (x.smem > kHalfSmem ? 1 : 0); };
  std::stable_sort(v.begin(), v.end(), [&](const SideItem& a, const SideItem& b) {
    const int ga = group(a), gb = group(b);
    return ga != gb ? ga > gb : a.cost > b.cost;
  });
  p->nclass = 0;
  items->clear();
  for (size_t i = 0; i < v.size(); ++i) {
    if (i == 0 || group(v[i]) != group(v[i - 1])) {
      if (p->nclass == SidesPlan::kMaxClass) return false;
      p->cls[p->nclass++] = {v[i].C, (int32_t)i, 0, 0};
    }
    SidesPlan::Class& c = p->cls[p->nclass - 1];
    ++c.count;
    c.smem = std::max(c.smem, v[i].smem);
    items->push_back(v[i].id);
  }
  return true;
}

// Double-float sides: the smallest cluster whose panels leave room for two CTAs
// on an SM (they hide each other's barriers); where the batch leaves SMs idle,
// larger clusters down to 32 rows per CTA.
//
// The step kernel (one CTA per instance, three per SM, panels through L2) is
// the better one for batches that fill the GPU with tall panels of high rank:
// a side that needs a cluster pays for its barriers and for the QR's r x r work
// on every CTA.  Costs in units of the work N r (r + 8) at the step kernel's
// full rate, at which one CTA alone runs 1/230: the step kernel takes its
// total, but at least its longest instance; sides take 0.75 of a panel on one
// CTA or two and 1.35 on more.  Members of n, m to 1024, step kernel
// against sides per step: r 23 to 32, 350: 4.5, 3.8 ms; 700: 6.3, 7.4 ms; 1400:
// 10.8, 14.4 ms; r 4 to 32, 1000: 5.1, 5.4 ms; n, m to 512, r 4 to 24, 1000: 2.3,
// 1.8 ms; n = m = 256, r 23 to 32, 366: 2.6, 1.9 ms.
bool sides_plan(SidesPlan* p, int count, const int64_t* n, const int64_t* m, const int64_t* r, int sms,
                std::vector<int32_t>* items) {
  std::vector<SideItem> v;
  double total = 0.0, longest = 0.0, by_sides = 0.0;
  for (int i = 0; i < count; ++i) {
    if (r[i] > wide::WR_MAX) return false;
    const double rr = (double)r[i] * ((double)r[i] + 8.0);
    for (int s = 0; s < 2; ++s) {
      const int N = (int)(s ? m[i] : n[i]), ri = (int)r[i];
      int C = 1;
      while (C < wide::WC_MAX && side_bytes(N, ri, C) > kHalfSmem) C *= 2;
      by_sides += N * rr * (C <= 2 ? 0.75 : 1.35);
      while (C < wide::WC_MAX && 4 * (int64_t)C * count <= sms && N >= 64 * C) C *= 2;
      if (side_bytes(N, ri, C) > kWideSmemMax) return false;
      v.push_back({(int32_t)(2 * i + s), C, side_bytes(N, ri, C), N * rr / C});
    }
    total += (double)(n[i] + m[i]) * rr;
    longest = std::max(longest, (double)(n[i] + m[i]) * rr);
  }
  if (by_sides > std::max(total, 230.0 * longest)) return false;
  return group_sides(v, p, items);
}

cudaError_t launch_sides_class(const StepArgs<dfloat>& g, const SidesPlan& p, int k, const int32_t* items,
                               cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  const SidesPlan::Class& c = p.cls[k];
  cudaError_t e = wide::cluster_attributes(sides_kernel, done);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  wide::cluster_config(cfg, attr, c.C * c.count, c.C, c.smem, st);
  return cudaLaunchKernelEx(&cfg, sides_kernel, g, items + c.first, (int)c.C);
}

}  // namespace lri
