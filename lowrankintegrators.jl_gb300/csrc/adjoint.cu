// adjoint.cu - discrete adjoint of the BUG step (FP64, Sylvester flow).
//
// One CTA per instance (or, for small batches, one 2-CTA cluster: the K side
// on one SM, the L side on another) reverses one BUG step: given the step's input factors
// (U0, S0, V0) and the adjoints of its outputs (U1_bar, S1_bar, V1_bar), it
// recomputes the step in stage form keeping every intermediate (RK stage
// inputs, Q and R of both QRs, M, N, the projections, the S-stage inputs)
// and sweeps back through it, producing (U0_bar, S0_bar, V0_bar) in place and
// accumulating theta_bar for a diagonal shift theta of the left operator A.
// Forward step (src/integrators/unconventional.jl:133-157), F = A X + X B^T:
//   K' = A K G_V + K P_V^T   from K0 = U0 S0      U1 = Q(K1), M = U1^T U0
//   L' = B L G_U + L P_U^T   from L0 = V0 S0^T    V1 = Q(L1), N = V1^T V0
//   S' = Pu S Gv + Gu S Pv^T from M S0 N^T on (U1, V1)
// with G_X = X^T X and P_X = X^T T X.  The reference has no derivative; the
// reverse sweep is the exact adjoint of this discrete map (RK stages in
// reverse, thin-QR adjoint A_bar = (Q_bar + Q copyltu(-Q_bar^T Q)) R^{-T}).
#include <cooperative_groups.h>

#include "engine_impl.cuh"
#include "wide.cuh"

namespace cg = cooperative_groups;

namespace lri {
namespace {

constexpr int kAdjMaxStages = 16;  // nstages * nsub of any substep scheme

// small-block indices (W x W doubles each, ld W)
enum : int {
  A_GV = 0, A_PV = 1, A_GU = 2, A_PU = 3, A_GU1 = 4, A_PU1 = 5, A_GV1 = 6, A_PV1 = 7, A_M = 8, A_N = 9, A_RK = 10,
  A_RL = 11, A_CPU = 12, A_CGV = 13, A_CGU = 14, A_CPV = 15, A_KG = 16, A_KP = 17, A_LG = 18, A_LP = 19, A_MB = 20,
  A_NB = 21, A_S0B = 22, A_SB = 23, A_SYB = 24, A_SKB = 25, A_SZB = 26, A_T1 = 27, A_T2 = 28, A_T3 = 29,
  A_ZERO = 30, A_X1 = 31, A_X2 = 32, A_SACC = 33, A_SK = 34, A_SST = 35,  // A_SST .. A_SST + 15: S stage inputs
  A_COUNT = A_SST + kAdjMaxStages
};
// panels per side: stage inputs, then
enum : int { P_Y1 = 0, P_Q = 1, P_YB = 2, P_KB = 3, P_ZB = 4, P_T1 = 5, P_T2 = 6, P_XB = 7, P_COUNT = 8 };

struct AdjArgs {
  const InstDesc* inst;
  const int64_t* adj_off;  // per-instance adjoint workspace offset
  const int64_t* th_off;   // per-instance theta_bar offset
  const double* U0;
  const double* S0;
  const double* V0;
  double* Ub;
  double* Sb;
  double* Vb;
  double* thb;
  const double* opA;
  const double* opB;
  double* work;
  Scheme sK, sL, sS;
  double dt;
  int split;  // 1: one 2-CTA cluster per instance (K side on CTA 0, L side on CTA 1)
};

struct AdjSide {
  int N;
  const double* X0;   // the side's input basis (U0 or V0), ld N
  const double* tri;  // its operator (A or B)
  double* triT;       // transposed operator coefficients (3N)
  double* Z;          // stage inputs, ns*nsub panels N x r
  double* P[P_COUNT];
};

__device__ __forceinline__ double* blkp(double* small, int W, int i) { return small + (int64_t)i * W * W; }

// T^T of a tridiagonal T = [sub | dia | sup]: sub'[i] = sup[i-1], sup'[i] = sub[i+1].
__device__ void tri_transpose(int N, const double* tri, double* triT) {
  for (int i = threadIdx.x; i < N; i += NT) {
    triT[i] = (i > 0) ? tri[2 * N + i - 1] : 0.0;
    triT[N + i] = tri[N + i];
    triT[2 * N + i] = (i + 1 < N) ? tri[i + 1] : 0.0;
  }
  __syncthreads();
}

__device__ void panel_copy(int64_t len, const double* x, double* y) {
  for (int64_t o = threadIdx.x; o < len; o += NT) y[o] = x[o];
  __syncthreads();
}

// y = a * x (+ b * z when z != nullptr)
__device__ void panel_axpby(int64_t len, double a, const double* x, double b, const double* z, double* y) {
  for (int64_t o = threadIdx.x; o < len; o += NT) y[o] = z ? fma(b, z[o], a * x[o]) : a * x[o];
  __syncthreads();
}

// y += a * x
__device__ void panel_add(int64_t len, double a, const double* x, double* y) {
  for (int64_t o = threadIdx.x; o < len; o += NT) y[o] = fma(a, x[o], y[o]);
  __syncthreads();
}

// out[i] += sum_j X(i, j) Y(i, j)   (N x r panels, ld N)
__device__ void rowdot_add(int N, int r, const double* X, const double* Y, double* out) {
  for (int i = threadIdx.x; i < N; i += NT) {
    double s = 0.0;
    for (int j = 0; j < r; ++j) s = fma(X[i + (int64_t)j * N], Y[i + (int64_t)j * N], s);
    out[i] += s;
  }
  __syncthreads();
}

// C <- C R^{-T} row by row (back substitution; R upper triangular, ld ldr)
__device__ void solve_rt_rows(int N, int r, double* C, const double* R, int ldr) {
  for (int i = threadIdx.x; i < N; i += NT) {
    for (int k = r - 1; k >= 0; --k) {
      double s = C[i + (int64_t)k * N];
      for (int j = k + 1; j < r; ++j) s = fma(-C[i + (int64_t)j * N], R[k + (int64_t)j * ldr], s);
      C[i + (int64_t)k * N] = s / R[k + (int64_t)k * ldr];
    }
  }
  __syncthreads();
}

__device__ void small_transpose(int r, const double* X, int W, double* Y) {
  for (int o = threadIdx.x; o < r * r; o += NT) {
    const int i = o % r, j = o / r;
    Y[j + (int64_t)i * W] = X[i + (int64_t)j * W];
  }
  __syncthreads();
}

// Y = X + X^T
__device__ void small_sym(int r, const double* X, int W, double* Y) {
  for (int o = threadIdx.x; o < r * r; o += NT) {
    const int i = o % r, j = o / r;
    Y[i + (int64_t)j * W] = X[i + (int64_t)j * W] + X[j + (int64_t)i * W];
  }
  __syncthreads();
}

// out (N x r) = L(z) = T z G + z P^T     (Gm = G, Pm = P; pass transposes for L^T)
__device__ void apply_op(int N, int r, const double* z, const double* tri, const double* Gm, const double* Pm, int W,
                         double* out, Smem<double>& sm) {
  tile_gemm<double>(N, 2 * r, r, sm.stage, LoadStencilAug<double>{z, N, N, r, tri}, LoadGP<double>{Gm, Pm, W, r},
                    EpiStore<double>{out, N});
}

// Xb += [T X | X] [C1^T ; C2] + [T^T X | X] [C1 ; 0] with C2 symmetric:
// the adjoint of G = X^T X (C2 = Gbar + Gbar^T) and P = X^T T X (C1 = Pbar).
__device__ void proj_adjoint(int N, int r, const double* X, const double* tri, const double* triT, const double* C1,
                             const double* C2, double* small, int W, double* Xb, Smem<double>& sm) {
  double* C1t = blkp(small, W, A_X1);
  small_transpose(r, C1, W, C1t);
  tile_gemm<double>(N, 2 * r, r, sm.stage, LoadStencilAug<double>{X, N, N, r, tri}, LoadGP<double>{C1t, C2, W, r},
                    EpiAdd<double>{Xb, N});
  tile_gemm<double>(N, 2 * r, r, sm.stage, LoadStencilAug<double>{X, N, N, r, triT},
                    LoadGP<double>{C1, blkp(small, W, A_ZERO), W, r}, EpiAdd<double>{Xb, N});
}

// Stage-form RK of y' = T y G + y P^T from y0 (panel Z[0]); the stage
// inputs stay in Z[sub*ns + s]; the result goes to out.
__device__ void rk_forward(const AdjSide& sd, int r, const double* Gm, const double* Pm, int W, const Scheme& sc,
                           double dt, double* out, Smem<double>& sm) {
  const int N = sd.N, ns = sc.nstages;
  const int64_t len = (int64_t)N * r;
  const double h = dt / sc.nsub;
  double* k = sd.P[P_T1];
  double* acc = sd.P[P_T2];
  for (int sub = 0; sub < sc.nsub; ++sub) {
    const double* y = sd.Z + (int64_t)(sub * ns) * len;
    for (int s = 0; s < ns; ++s) {
      const double* z = sd.Z + (int64_t)(sub * ns + s) * len;
      apply_op(N, r, z, sd.tri, Gm, Pm, W, k, sm);
      if (s == 0) panel_axpby(len, sc.b[0], k, 0.0, nullptr, acc);
      else panel_add(len, sc.b[s], k, acc);
      if (s + 1 < ns) panel_axpby(len, 1.0, y, h * sc.a[s + 1], k, sd.Z + (int64_t)(sub * ns + s + 1) * len);
    }
    double* ynext = (sub + 1 < sc.nsub) ? sd.Z + (int64_t)((sub + 1) * ns) * len : out;
    panel_axpby(len, 1.0, y, h, acc, ynext);
  }
}

// Reverse of rk_forward: on entry P[P_YB] holds y1_bar, on exit y0_bar.
// Accumulates Gbar += (T z)^T kbar, Pbar += kbar^T z per stage, and
// theta_bar[i] += kbar(i,:) . (z G)(i,:) when thb != nullptr.
__device__ void rk_reverse(const AdjSide& sd, int r, const double* Gm, const double* GmT, const double* PmT, int W,
                           const Scheme& sc, double dt, double* Gbar, double* Pbar, double* thb, Smem<double>& sm) {
  const int N = sd.N, ns = sc.nstages;
  const int64_t len = (int64_t)N * r;
  const double h = dt / sc.nsub;
  double* yb = sd.P[P_YB];
  double* kb = sd.P[P_KB];
  double* zb = sd.P[P_ZB];
  double* ybn = sd.P[P_T2];
  double* tmp = sd.P[P_T1];
  for (int sub = sc.nsub - 1; sub >= 0; --sub) {
    panel_copy(len, yb, ybn);
    for (int s = ns - 1; s >= 0; --s) {
      const double* z = sd.Z + (int64_t)(sub * ns + s) * len;
      // kbar_s = h b_s ybar' + h a_{s+1} zbar_{s+1}
      panel_axpby(len, h * sc.b[s], ybn, h * ((s + 1 < ns) ? sc.a[s + 1] : 0.0), (s + 1 < ns) ? zb : nullptr, kb);
      tile_gram<double>(N, r, r, sm.stage, RowLoadStencil<double>{z, N, N, r, sd.tri}, RowLoadPanel<double>{kb, N, r},
                        Gbar, W, 1.0, 1.0);
      tile_gram<double>(N, r, r, sm.stage, RowLoadPanel<double>{kb, N, r}, RowLoadPanel<double>{z, N, r}, Pbar, W,
                        1.0, 1.0);
      if (thb) {
        tile_gemm<double>(N, r, r, sm.stage, LoadPanel<double>{z, N}, LoadSmall<double>{Gm, W, false},
                          EpiStore<double>{tmp, N});
        rowdot_add(N, r, kb, tmp, thb);
      }
      // zbar_s = T^T kbar G^T + kbar P
      apply_op(N, r, kb, sd.triT, GmT, PmT, W, zb, sm);
      panel_add(len, 1.0, zb, yb);
    }
  }
}

// Thin-QR adjoint in place: Xb <- (Xb + Q copyltu(-Xb^T Q)) R^{-T}.
__device__ void qr_adjoint(int N, int r, const double* Q, const double* R, double* Xb, double* small, int W,
                           Smem<double>& sm) {
  double* Mx = blkp(small, W, A_T1);
  double* Cl = blkp(small, W, A_T2);
  tile_gram<double>(N, r, r, sm.stage, RowLoadPanel<double>{Xb, N, r}, RowLoadPanel<double>{Q, N, r}, Mx, W, -1.0,
                    0.0);
  for (int o = threadIdx.x; o < r * r; o += NT) {
    const int i = o % r, j = o / r;
    Cl[i + (int64_t)j * W] = (i >= j) ? Mx[i + (int64_t)j * W] : Mx[j + (int64_t)i * W];
  }
  __syncthreads();
  tile_gemm<double>(N, r, r, sm.stage, LoadPanel<double>{Q, N}, LoadSmall<double>{Cl, W, false},
                    EpiAdd<double>{Xb, N});
  solve_rt_rows(N, r, Xb, R, W);
}

__device__ void small_zero(int r, double* X, int W) {
  for (int o = threadIdx.x; o < r * r; o += NT) X[(o % r) + (int64_t)(o / r) * W] = 0.0;
  __syncthreads();
}

// S-step stage derivative: out = Pu z Gv + Gu z Pv^T
__device__ void s_op(int r, const double* z, double* small, int W, double* out) {
  double* t1 = blkp(small, W, A_T3);
  small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_PU1), W, false, z, W, false, 0.0, t1, W);
  small_gemm<double>(r, r, r, 1.0, t1, W, false, blkp(small, W, A_GV1), W, false, 0.0, out, W);
  small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_GU1), W, false, z, W, false, 0.0, t1, W);
  small_gemm<double>(r, r, r, 1.0, t1, W, false, blkp(small, W, A_PV1), W, true, 1.0, out, W);
}

// One instance per CTA, or (split) per 2-CTA thread-block cluster: CTA 0
// takes the K side (U), CTA 1 the L side (V), in four phases separated by
// cluster barriers (every thread of both CTAs reaches all three):
//   1. forward recomputation of each side's substep, QR, basis change and
//      projections;
//   2. (CTA 0) the S step forward and reversed, Mbar, Nbar, S0bar;
//   3. each side's QR adjoint and RK reversal (the gradients of its
//      projection coefficients, its part of S0bar);
//   4. each side adds the adjoint of the other side's projections of its own
//      basis (K step -> G_V, P_V; L step -> G_U, P_U) and writes its output;
//      CTA 1 sums S0bar.
// Scratch blocks: the K side uses `small`, the L side `small1` (disjoint),
// so the halves never write the same block.  Without a cluster the same
// phases run one after the other in one CTA.
__global__ void __launch_bounds__(NT, 3) adjoint_step_kernel(AdjArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<double>& sm = *reinterpret_cast<Smem<double>*>(smem_raw);
  const bool split = g.split != 0;
  const int inst = split ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int crank = split ? (int)cg::this_cluster().block_rank() : 0;
  const bool doK = !split || crank == 0;
  const bool doL = !split || crank == 1;
  auto phase_end = [&]() {
    if (split) {
      __threadfence();
      cg::this_cluster().sync();
    }
  };
  const InstDesc d = g.inst[inst];
  const int n = d.n, m = d.m, r = d.rcap, W = d.rcap, ldS = d.rcap;
  const double* U0 = g.U0 + d.offU;
  const double* S0 = g.S0 + d.offS;
  const double* V0 = g.V0 + d.offV;
  double* Ub = g.Ub + d.offU;
  double* Sb = g.Sb + d.offS;
  double* Vb = g.Vb + d.offV;
  double* thb = g.thb + g.th_off[inst];
  double* w = g.work + g.adj_off[inst];
  // workspace: small blocks | L-side scratch blocks | K side (triT, stage panels, panels) | L side
  double* small = w;
  w += (int64_t)A_COUNT * W * W;
  double* small1 = w;
  w += (int64_t)A_COUNT * W * W;
  AdjSide K, L;
  K.N = n;
  K.X0 = U0;
  K.tri = g.opA + d.offA;
  K.triT = w;
  w += 3 * (int64_t)n;
  K.Z = w;
  w += (int64_t)(g.sK.nstages * g.sK.nsub) * n * r;
  for (int p = 0; p < P_COUNT; ++p) {
    K.P[p] = w;
    w += (int64_t)n * r;
  }
  L.N = m;
  L.X0 = V0;
  L.tri = g.opB + d.offB;
  L.triT = w;
  w += 3 * (int64_t)m;
  L.Z = w;
  w += (int64_t)(g.sL.nstages * g.sL.nsub) * m * r;
  for (int p = 0; p < P_COUNT; ++p) {
    L.P[p] = w;
    w += (int64_t)m * r;
  }
  Inst<double> I;
  I.n = n;
  I.m = m;
  I.rcap = r;
  I.W = W;
  I.inst = inst;
  const double* U1 = K.P[P_Q];
  const double* V1 = L.P[P_Q];
  double* T1s = blkp(small, W, A_T1);
  double* T2s = blkp(small, W, A_T2);

  // ---------------- phase 1: forward recomputation of both sides ----------------
  if (doK) {
    tri_transpose(n, K.tri, K.triT);
    small_zero(r, blkp(small, W, A_ZERO), W);
    projections<double>(I, V0, m, r, L.tri, blkp(small, W, A_GV), sm);  // G_V, P_V (adjacent blocks)
    // K step: K0 = U0 S0 -> K1 -> U1 = Q, RK
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{U0, n}, LoadSmall<double>{S0, ldS, false},
                      EpiStore<double>{K.Z, n});
    rk_forward(K, r, blkp(small, W, A_GV), blkp(small, W, A_PV), W, g.sK, g.dt, K.P[P_Y1], sm);
    qr_panel<double>(K.P[P_Y1], n, r, K.P[P_Q], blkp(small, W, A_RK), W, sm);
    tile_gram<double>(n, r, r, sm.stage, RowLoadPanel<double>{K.P[P_Q], n, r}, RowLoadPanel<double>{U0, n, r},
                      blkp(small, W, A_M), W, 1.0, 0.0);
    projections<double>(I, U1, n, r, K.tri, blkp(small, W, A_GU1), sm);  // Gu1, Pu1
  }
  if (doL) {
    tri_transpose(m, L.tri, L.triT);
    small_zero(r, blkp(small1, W, A_ZERO), W);
    projections<double>(I, U0, n, r, K.tri, blkp(small, W, A_GU), sm);  // G_U, P_U
    // L step: L0 = V0 S0^T -> L1 -> V1, RL
    tile_gemm<double>(m, r, r, sm.stage, LoadPanel<double>{V0, m}, LoadSmall<double>{S0, ldS, true},
                      EpiStore<double>{L.Z, m});
    rk_forward(L, r, blkp(small, W, A_GU), blkp(small, W, A_PU), W, g.sL, g.dt, L.P[P_Y1], sm);
    qr_panel<double>(L.P[P_Y1], m, r, L.P[P_Q], blkp(small, W, A_RL), W, sm);
    tile_gram<double>(m, r, r, sm.stage, RowLoadPanel<double>{L.P[P_Q], m, r}, RowLoadPanel<double>{V0, m, r},
                      blkp(small, W, A_N), W, 1.0, 0.0);
    projections<double>(I, V1, m, r, L.tri, blkp(small, W, A_GV1), sm);  // Gv1, Pv1
  }
  phase_end();

  // ---------------- phase 2: the S step, forward and reversed ----------------
  double* Mb = blkp(small, W, A_MB);
  double* Nb = blkp(small, W, A_NB);
  double* S0b = blkp(small, W, A_S0B);
  if (doK) {
    // S~0 = M S0 N^T into the first stage input
    small_gemm<double>(r, r, r, 1.0, S0, ldS, false, blkp(small, W, A_N), W, true, 0.0, T1s, W);
    small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_M), W, false, T1s, W, false, 0.0, blkp(small, W, A_SST), W);
    {
      const int ns = g.sS.nstages;
      const double h = g.dt / g.sS.nsub;
      double* kS = blkp(small, W, A_SK);
      double* acc = blkp(small, W, A_SACC);
      for (int sub = 0; sub < g.sS.nsub; ++sub) {
        const double* y = blkp(small, W, A_SST + sub * ns);
        for (int s = 0; s < ns; ++s) {
          s_op(r, blkp(small, W, A_SST + sub * ns + s), small, W, kS);
          for (int o = threadIdx.x; o < r * r; o += NT) {
            const int64_t e = (o % r) + (int64_t)(o / r) * W;
            acc[e] = (s == 0) ? g.sS.b[0] * kS[e] : fma(g.sS.b[s], kS[e], acc[e]);
            if (s + 1 < ns) blkp(small, W, A_SST + sub * ns + s + 1)[e] = fma(h * g.sS.a[s + 1], kS[e], y[e]);
          }
          __syncthreads();
        }
        if (sub + 1 < g.sS.nsub) {
          double* yn = blkp(small, W, A_SST + (sub + 1) * ns);
          for (int o = threadIdx.x; o < r * r; o += NT) {
            const int64_t e = (o % r) + (int64_t)(o / r) * W;
            yn[e] = fma(h, acc[e], y[e]);
          }
          __syncthreads();
        }
      }
    }
    // S step reversed: Sbar = S1_bar -> S~0_bar; coefficient gradients cPu, cGv, cGu, cPv
    double* Sbar = blkp(small, W, A_SB);
    for (int o = threadIdx.x; o < r * r; o += NT)
      Sbar[(o % r) + (int64_t)(o / r) * W] = Sb[(o % r) + (int64_t)(o / r) * ldS];
    for (int b = A_CPU; b <= A_LP; ++b) small_zero(r, blkp(small, W, b), W);
    {
      const int ns = g.sS.nstages;
      const double h = g.dt / g.sS.nsub;
      double* ybn = blkp(small, W, A_SYB);
      double* kb = blkp(small, W, A_SKB);
      double* zb = blkp(small, W, A_SZB);
      double* t3 = blkp(small, W, A_T3);
      for (int sub = g.sS.nsub - 1; sub >= 0; --sub) {
        copy_mat<double>(r, r, Sbar, W, ybn, W);
        for (int s = ns - 1; s >= 0; --s) {
          const double* z = blkp(small, W, A_SST + sub * ns + s);
          for (int o = threadIdx.x; o < r * r; o += NT) {
            const int64_t e = (o % r) + (int64_t)(o / r) * W;
            kb[e] = h * g.sS.b[s] * ybn[e] + ((s + 1 < ns) ? h * g.sS.a[s + 1] * zb[e] : 0.0);
          }
          __syncthreads();
          // cPu += kb Gv1^T z^T ; cGv += (Pu1 z)^T kb ; cGu += kb Pv1 z^T ; cPv += kb^T Gu1 z
          small_gemm<double>(r, r, r, 1.0, kb, W, false, blkp(small, W, A_GV1), W, true, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, t3, W, false, z, W, true, 1.0, blkp(small, W, A_CPU), W);
          small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_PU1), W, false, z, W, false, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, t3, W, true, kb, W, false, 1.0, blkp(small, W, A_CGV), W);
          small_gemm<double>(r, r, r, 1.0, kb, W, false, blkp(small, W, A_PV1), W, false, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, t3, W, false, z, W, true, 1.0, blkp(small, W, A_CGU), W);
          small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_GU1), W, false, z, W, false, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, kb, W, true, t3, W, false, 1.0, blkp(small, W, A_CPV), W);
          // zb = Pu1^T kb Gv1^T + Gu1^T kb Pv1
          small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_PU1), W, true, kb, W, false, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, t3, W, false, blkp(small, W, A_GV1), W, true, 0.0, zb, W);
          small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_GU1), W, true, kb, W, false, 0.0, t3, W);
          small_gemm<double>(r, r, r, 1.0, t3, W, false, blkp(small, W, A_PV1), W, false, 1.0, zb, W);
          for (int o = threadIdx.x; o < r * r; o += NT) {
            const int64_t e = (o % r) + (int64_t)(o / r) * W;
            Sbar[e] += zb[e];
          }
          __syncthreads();
        }
      }
    }
    // S~0 = M S0 N^T:  Mb = St0b N S0^T, Nb = St0b^T M S0, S0b = M^T St0b N
    small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_N), W, false, S0, ldS, true, 0.0, T1s, W);
    small_gemm<double>(r, r, r, 1.0, Sbar, W, false, T1s, W, false, 0.0, Mb, W);
    small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_M), W, false, S0, ldS, false, 0.0, T1s, W);
    small_gemm<double>(r, r, r, 1.0, Sbar, W, true, T1s, W, false, 0.0, Nb, W);
    small_gemm<double>(r, r, r, 1.0, Sbar, W, false, blkp(small, W, A_N), W, false, 0.0, T1s, W);
    small_gemm<double>(r, r, r, 1.0, blkp(small, W, A_M), W, true, T1s, W, false, 0.0, S0b, W);
  }
  phase_end();

  // ---------------- phase 3: QR adjoints and RK reversals of both sides ----------------
  const int64_t lenK = (int64_t)n * r, lenL = (int64_t)m * r;
  if (doK) {
    // U1_bar (panel K.P[P_YB]) = U1_bar(out) + U0 Mb^T + adjoint of Gu1, Pu1; theta_bar from Pu1
    for (int64_t o = threadIdx.x; o < lenK; o += NT) K.P[P_YB][o] = Ub[o];
    __syncthreads();
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{U0, n}, LoadSmall<double>{Mb, W, true},
                      EpiAdd<double>{K.P[P_YB], n});
    small_sym(r, blkp(small, W, A_CGU), W, T2s);
    proj_adjoint(n, r, U1, K.tri, K.triT, blkp(small, W, A_CPU), T2s, small, W, K.P[P_YB], sm);
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{U1, n},
                      LoadSmall<double>{blkp(small, W, A_CPU), W, true}, EpiStore<double>{K.P[P_T1], n});
    rowdot_add(n, r, K.P[P_T1], U1, thb);
    // U0_bar accumulator (panel P_XB): U1 Mb
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{U1, n}, LoadSmall<double>{Mb, W, false},
                      EpiStore<double>{K.P[P_XB], n});
    // K step: K1_bar = qr_adjoint(U1_bar); RK reverse -> K0_bar
    qr_adjoint(n, r, U1, blkp(small, W, A_RK), K.P[P_YB], small, W, sm);
    small_transpose(r, blkp(small, W, A_GV), W, blkp(small, W, A_T1));
    small_transpose(r, blkp(small, W, A_PV), W, blkp(small, W, A_T2));
    // L^T(X) = A^T X G_V^T + X P_V : apply_op with (G^T, P^T) gives [G^T ; P]
    rk_reverse(K, r, blkp(small, W, A_GV), blkp(small, W, A_T1), blkp(small, W, A_T2), W, g.sK, g.dt,
               blkp(small, W, A_KG), blkp(small, W, A_KP), thb, sm);
    // U0_bar += K0_bar S0^T ; S0_bar += U0^T K0_bar
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{K.P[P_YB], n}, LoadSmall<double>{S0, ldS, true},
                      EpiAdd<double>{K.P[P_XB], n});
    tile_gram<double>(n, r, r, sm.stage, RowLoadPanel<double>{U0, n, r}, RowLoadPanel<double>{K.P[P_YB], n, r}, S0b,
                      W, 1.0, 1.0);
  }
  if (doL) {
    double* T2l = blkp(small1, W, A_T2);
    // V1_bar (panel L.P[P_YB]) = V1_bar(out) + V0 Nb^T + adjoint of Gv1, Pv1
    for (int64_t o = threadIdx.x; o < lenL; o += NT) L.P[P_YB][o] = Vb[o];
    __syncthreads();
    tile_gemm<double>(m, r, r, sm.stage, LoadPanel<double>{V0, m}, LoadSmall<double>{Nb, W, true},
                      EpiAdd<double>{L.P[P_YB], m});
    small_sym(r, blkp(small, W, A_CGV), W, T2l);
    proj_adjoint(m, r, V1, L.tri, L.triT, blkp(small, W, A_CPV), T2l, small1, W, L.P[P_YB], sm);
    // V0_bar accumulator: V1 Nb
    tile_gemm<double>(m, r, r, sm.stage, LoadPanel<double>{V1, m}, LoadSmall<double>{Nb, W, false},
                      EpiStore<double>{L.P[P_XB], m});
    // L step: L1_bar = qr_adjoint(V1_bar); RK reverse -> L0_bar
    qr_adjoint(m, r, V1, blkp(small, W, A_RL), L.P[P_YB], small1, W, sm);
    small_transpose(r, blkp(small, W, A_GU), W, blkp(small1, W, A_T1));
    small_transpose(r, blkp(small, W, A_PU), W, blkp(small1, W, A_T2));
    rk_reverse(L, r, blkp(small, W, A_GU), blkp(small1, W, A_T1), blkp(small1, W, A_T2), W, g.sL, g.dt,
               blkp(small, W, A_LG), blkp(small, W, A_LP), nullptr, sm);
    // V0_bar += L0_bar S0 ; this side's part of S0_bar: L0_bar^T V0
    tile_gemm<double>(m, r, r, sm.stage, LoadPanel<double>{L.P[P_YB], m}, LoadSmall<double>{S0, ldS, false},
                      EpiAdd<double>{L.P[P_XB], m});
    tile_gram<double>(m, r, r, sm.stage, RowLoadPanel<double>{L.P[P_YB], m, r}, RowLoadPanel<double>{V0, m, r},
                      blkp(small1, W, A_S0B), W, 1.0, 0.0);
  }
  phase_end();

  // ---------------- phase 4: cross-side projection adjoints, outputs ----------------
  if (doK) {
    // U0_bar += adjoint of G_U, P_U (L step) ; theta_bar from P_U
    small_sym(r, blkp(small, W, A_LG), W, T2s);
    proj_adjoint(n, r, U0, K.tri, K.triT, blkp(small, W, A_LP), T2s, small, W, K.P[P_XB], sm);
    tile_gemm<double>(n, r, r, sm.stage, LoadPanel<double>{U0, n}, LoadSmall<double>{blkp(small, W, A_LP), W, true},
                      EpiStore<double>{K.P[P_T1], n});
    rowdot_add(n, r, K.P[P_T1], U0, thb);
    for (int64_t o = threadIdx.x; o < lenK; o += NT) Ub[o] = K.P[P_XB][o];
  }
  if (doL) {
    // V0_bar += adjoint of G_V, P_V (K step)
    double* T2l = blkp(small1, W, A_T2);
    small_sym(r, blkp(small, W, A_KG), W, T2l);
    proj_adjoint(m, r, V0, L.tri, L.triT, blkp(small, W, A_KP), T2l, small1, W, L.P[P_XB], sm);
    for (int64_t o = threadIdx.x; o < lenL; o += NT) Vb[o] = L.P[P_XB][o];
    const double* S0bl = blkp(small1, W, A_S0B);
    for (int o = threadIdx.x; o < r * r; o += NT) {
      const int64_t e = (o % r) + (int64_t)(o / r) * W;
      Sb[(o % r) + (int64_t)(o / r) * ldS] = S0b[e] + S0bl[e];
    }
  }
}

// ---------------------------------------------------------------------------
// The same reversal of small batches on thread-block clusters (wide.cuh): four
// launches, the phases above.  adj_fwd, adj_rev and adj_out give each side of
// an instance a cluster whose CTAs split its rows (panels in shared memory,
// the stage inputs in the workspace); adj_core splits the core's entries over
// one cluster.  The products with a Gram matrix take its FP32 form where the
// forward steps do (below_2_100 in wide.cuh).  One reverse step at n = m =
// 2048, r = 32: 37.0 ms on a 2-CTA pair, 2.0 ms here (adj_fwd 0.63, adj_core
// 0.18, adj_rev 1.02, adj_out 0.15), bound by FP64 issue on 32 SMs.
// ---------------------------------------------------------------------------
using wide::load_rows;
using wide::load_rows_halo;
using wide::outputs;
using wide::push_halos;
using wide::QrSmem;
using wide::reduce_parts;
using wide::Team;
using wide::Tri;
using wide::WT;

// One side of an instance and its workspace (the layout of adjoint_step_kernel).
struct WideAdj {
  int n, m, r, W, N, No;
  bool kside;
  const double* X0;   // this side's input basis
  const double* Xo;   // the other side's
  const double* S0;
  double* Xb;         // the adjoint of this side's basis (in: output's, out: input's)
  double* Sb;
  double* thb;
  const double* tri;
  const double* trio;
  double* small;
  double* small1;
  double* Z;          // stage inputs
  double* Q;
  double* xb;
};

__device__ void wide_adj(const AdjArgs& g, int inst, bool kside, WideAdj& s) {
  const InstDesc d = g.inst[inst];
  const int n = d.n, m = d.m, r = d.rcap;
  s.n = n; s.m = m; s.r = s.W = r; s.kside = kside;
  s.N = kside ? n : m;
  s.No = kside ? m : n;
  s.X0 = kside ? g.U0 + d.offU : g.V0 + d.offV;
  s.Xo = kside ? g.V0 + d.offV : g.U0 + d.offU;
  s.S0 = g.S0 + d.offS;
  s.Xb = kside ? g.Ub + d.offU : g.Vb + d.offV;
  s.Sb = g.Sb + d.offS;
  s.thb = g.thb + g.th_off[inst];
  s.tri = kside ? g.opA + d.offA : g.opB + d.offB;
  s.trio = kside ? g.opB + d.offB : g.opA + d.offA;
  double* w = g.work + g.adj_off[inst];
  s.small = w;
  s.small1 = w + (int64_t)A_COUNT * r * r;
  w += 2 * (int64_t)A_COUNT * r * r;
  const int64_t lenK = (int64_t)n * r, nsK = g.sK.nstages * g.sK.nsub, nsL = g.sL.nstages * g.sL.nsub;
  if (!kside) w += 3 * (int64_t)n + (nsK + P_COUNT) * lenK;
  w += 3 * (int64_t)s.N;
  s.Z = w;
  const int64_t len = (int64_t)s.N * r;
  w += (kside ? nsK : nsL) * len;
  s.Q = w + P_Q * len;
  s.xb = w + P_XB * len;
}

// shared memory in doubles: panels, then the small matrices
__host__ __device__ inline size_t adj_ld(int N, int C) { return (size_t)((((N + C - 1) / C) + 2) | 1); }
__host__ __device__ inline size_t adj_misc(int N, int r, int C) {
  const size_t R0 = (N + C - 1) / C, rr = (size_t)r * r;
  return 4 * rr + (rr + 1) / 2 + (size_t)r * R0 / 2 + 1;  // P, three partials, E, the FP32 copy
}
__host__ inline size_t adj_fwd_doubles(int N, int r, int C) {
  return 4 * adj_ld(N, C) * r + adj_misc(N, r, C) + QrSmem<double>::elems(C, r);
}
__host__ inline size_t adj_rev_doubles(int N, int r, int C) { return 5 * adj_ld(N, C) * r + adj_misc(N, r, C) + r; }

// C E-form operands: Ps[k r + c] = P(c, k) (or P(k, c) with pt), Es = G - I (or
// its transpose with gt); true when the full product is needed
__device__ bool load_ep(int r, int W, const double* G, const double* P, bool gt, bool pt, double* Ps, float* Es) {
  int full = 0;
  for (int e = threadIdx.x; e < r * r; e += WT) {
    const int k = e / r, c = e % r;
    Ps[e] = pt ? P[k + (int64_t)c * W] : P[c + (int64_t)k * W];
    const double ev = (gt ? G[c + (int64_t)k * W] : G[k + (int64_t)c * W]) - ((k == c) ? 1.0 : 0.0);
    Es[e] = (float)ev;
    if (!(fabs(ev) <= 0x1p-36)) full = 1;  // NaN included
  }
  return __syncthreads_or(full) != 0;
}

__global__ void __launch_bounds__(WT, 1) adj_fwd(const __grid_constant__ AdjArgs g, int C) {
  extern __shared__ __align__(16) double dsm[];
  Team tm{cg::this_cluster(), (int)cg::this_cluster().block_rank(), C};
  const int ci = blockIdx.x / C, tid = threadIdx.x;
  WideAdj s;
  wide_adj(g, ci >> 1, (ci & 1) == 0, s);
  const int r = s.r, W = s.W, N = s.N, No = s.No, rr = r * r;
  const int R0 = tm.rows_per(N), lo = tm.lo(N), rows = tm.hi(N) - lo, ld = (int)adj_ld(N, C);
  const int64_t len = (int64_t)N * r;
  const Tri T{s.tri, N, lo};
  const wide::FastDiv by_rows(rows);
  double* p0 = dsm;
  double* p1 = p0 + (size_t)r * ld;
  double* y = p1 + (size_t)r * ld;
  double* acc = y + (size_t)r * ld;
  double* misc = acc + (size_t)r * ld;
  const QrSmem<double> qs = QrSmem<double>::carve(misc + adj_misc(N, r, C), C, r);
  double* Gg = blkp(s.small, W, s.kside ? A_GV : A_GU);  // G, then P
  tm.cl.sync();  // every CTA runs before any distributed access
  {
    // projections of the other input basis, in blocks of at most R0 rows
    const int lo2 = tm.lo(No), hi2 = tm.hi(No);
    double* part = misc;
    for (int e = tid; e < 2 * rr; e += WT) part[e] = 0.0;
    for (int b = lo2; b < hi2; b += R0) {
      const int nb = min(R0, hi2 - b);
      __syncthreads();
      load_rows_halo(s.Xo, No, b, nb, r, p0, ld);
      __syncthreads();
      const Tri To{s.trio, No, b};
      for (int e = tid; e < nb * r; e += WT) p1[(e / nb) * ld + 1 + e % nb] = To.mul(p0, ld, e % nb, e / nb);
      __syncthreads();
      for (int o = tid; o < 2 * rr; o += WT) {
        const int a = o % r, c = (o / r) % r;
        if (o < rr && a > c) continue;  // G is symmetric
        const double* x = (o < rr) ? p0 : p1;
        double v = part[o];
        for (int i = 1; i <= nb; ++i) v = fma(p0[a * ld + i], x[c * ld + i], v);
        part[o] = v;
      }
    }
    __syncthreads();
    reduce_parts(tm, part, 2 * rr, [&](int e, double v) {
      const int a = e % r, c = (e / r) % r;
      if (e >= rr) Gg[(int64_t)W * W + a + (int64_t)c * W] = v;
      else if (a <= c) Gg[a + (int64_t)c * W] = Gg[c + (int64_t)a * W] = v;
    });
  }
  // zero halo rows at the ends of the domain (never pushed to)
  for (int e = tid; e < 2 * r; e += WT) {
    double* p = (e < r) ? p0 : p1;
    const int k = e % r;
    p[k * ld] = 0.0;
    p[k * ld + 1 + R0] = 0.0;
    if (rows < R0) p[k * ld + 1 + rows] = 0.0;
  }
  // K0 = U0 S0 (L0 = V0 S0^T)
  double* Ps = misc;
  for (int e = tid; e < rr; e += WT) {
    const int k = e / r, c = e % r;
    Ps[e] = s.kside ? s.S0[k + (int64_t)c * r] : s.S0[c + (int64_t)k * r];
  }
  load_rows(s.X0, N, lo, rows, r, p1, ld);
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    double v = 0.0;
    for (int k = 0; k < r; ++k) v = fma(p1[k * ld + 1 + i], Ps[k * r + c], v);
    p0[c * ld + 1 + i] = y[c * ld + 1 + i] = v;
    s.Z[lo + i + (int64_t)c * N] = v;
  }
  __syncthreads();
  float* Es = reinterpret_cast<float*>(misc + 4 * rr);
  float* tf = reinterpret_cast<float*>(misc + 4 * rr + (rr + 1) / 2);
  const bool full = load_ep(r, W, Gg, Gg + (int64_t)W * W, false, false, Ps, Es);
  tm.cl.sync();  // the zero halo rows of every CTA are set
  push_halos(tm, N, rows, r, p0, ld);
  tm.cl.sync();
  // stage-form RK of y' = T y G + y P^T, every stage input to the workspace
  const Scheme& sc = s.kside ? g.sK : g.sL;
  const double h = g.dt / sc.nsub;
  double* win = p0;
  double* wout = p1;
  for (int sub = 0; sub < sc.nsub; ++sub)
    for (int st = 0; st < sc.nstages; ++st) {
      int big = full, reaches = 0;
      if (!full) {
        for (int e = tid; e < rows * r; e += WT) {
          const int k = by_rows.div(e), i = e - k * rows;
          const double tw = T.mul(win, ld, i, k);
          wout[k * ld + 1 + i] = tw;
          tf[e] = (float)tw;
          big |= !wide::below_2_100(tw);
          reaches |= wide::reaches_2_m80(tw);
        }
        big = wide::out_of_f32(big, reaches);
      }
      const bool last = st + 1 == sc.nstages, end = last && sub + 1 == sc.nsub;
      const double bs = sc.b[st], ha = last ? 0.0 : h * sc.a[st + 1];
      double* Zn = s.Z + (int64_t)(sub * sc.nstages + st + 1) * len;
      for (int e = tid; e < rows * r; e += WT) {
        const int c = by_rows.div(e), i = e - c * rows, o = c * ld + 1 + i;
        double v;
        if (!big) {
          float ef = 0.0f;
          for (int k = 0; k < r; ++k) ef = fmaf(tf[k * rows + i], Es[k * r + c], ef);
          v = wout[o] + (double)ef;
        } else {
          v = 0.0;
          for (int k = 0; k < r; ++k) v = fma(T.mul(win, ld, i, k), Gg[k + (int64_t)c * W], v);
        }
        for (int k = 0; k < r; ++k) v = fma(win[k * ld + 1 + i], Ps[k * r + c], v);
        const double a = (st == 0) ? bs * v : fma(bs, v, acc[o]);
        acc[o] = a;
        double z;
        if (last) y[o] = z = fma(h, a, y[o]);
        else z = fma(ha, v, y[o]);
        wout[o] = z;
        if (!end) Zn[lo + i + (int64_t)c * N] = z;
        if (i == 0 && tm.q > 0) tm.at(wout, tm.q - 1)[c * ld + 1 + R0] = z;
        if (i == rows - 1 && tm.q + 1 < C && lo + rows < N) tm.at(wout, tm.q + 1)[c * ld] = z;
      }
      tm.cl.sync();
      double* t = win;
      win = wout;
      wout = t;
    }
  wide::qr<double>(tm, N, lo, rows, r, win + 1, ld, wout + 1, ld, blkp(s.small, W, s.kside ? A_RK : A_RL), W, qs);
  // M = Q^T X0 and the projections of Q
  double* Q = wout;
  double* part = misc;
  load_rows(s.X0, N, lo, rows, r, win, ld);
  push_halos(tm, N, rows, r, Q, ld);
  tm.cl.sync();
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    y[k * ld + 1 + i] = T.mul(Q, ld, i, k);
    s.Q[lo + i + (int64_t)k * N] = Q[k * ld + 1 + i];
  }
  __syncthreads();
  outputs(3 * rr, rows, [&](int o, int l, int L) {
    const int a = o % r, c = (o / r) % r, w = o / rr;
    if (w == 1 && a > c) return 0.0;
    const double* x = (w == 0) ? win : (w == 1 ? Q : y);
    double v = 0.0;
    for (int i = 1 + l; i <= rows; i += L) v = fma(Q[a * ld + i], x[c * ld + i], v);
    return v;
  }, [&](int o, double v) { part[o] = v; });
  double* Mo = blkp(s.small, W, s.kside ? A_M : A_N);
  double* Gn = blkp(s.small, W, s.kside ? A_GU1 : A_GV1);
  double* Pn = blkp(s.small, W, s.kside ? A_PU1 : A_PV1);
  reduce_parts(tm, part, 3 * rr, [&](int e, double v) {
    const int a = e % r, c = (e / r) % r, w = e / rr;
    if (w == 0) Mo[a + (int64_t)c * W] = v;
    else if (w == 2) Pn[a + (int64_t)c * W] = v;
    else if (a <= c) Gn[a + (int64_t)c * W] = Gn[c + (int64_t)a * W] = v;
  });
}

// C = alpha op(A) op(B) over this CTA's share of the entries (r x r, ld W);
// fin(entry offset, value) stores it
template <class F>
__device__ __forceinline__ void dgemm(const Team& tm, int r, int W, const double* A, bool ta, const double* B, bool tb,
                                      const F& fin) {
  const int per = (r * r + tm.C - 1) / tm.C, e0 = tm.q * per, e1 = min(r * r, e0 + per);
  outputs(max(0, e1 - e0), r, [&](int o, int l, int L) {
    const int i = (e0 + o) % r, j = (e0 + o) / r;
    double v = 0.0;
    for (int k = l; k < r; k += L)
      v = fma(ta ? A[k + (int64_t)i * W] : A[i + (int64_t)k * W], tb ? B[j + (int64_t)k * W] : B[k + (int64_t)j * W], v);
    return v;
  }, [&](int o, double v) { fin((e0 + o) % r + (int64_t)((e0 + o) / r) * W, v); },
          wide::lanes_for(max(1, e1 - e0)));  // (operands from L2: latency, not FP64 issue)
}

// Phase 2: the S step forward and reversed; entries split over one cluster,
// intermediates in the scratch blocks, a cluster barrier after each group of
// independent products.
__global__ void __launch_bounds__(WT, 1) adj_core(const __grid_constant__ AdjArgs g, int C) {
  Team tm{cg::this_cluster(), (int)cg::this_cluster().block_rank(), C};
  WideAdj s;
  wide_adj(g, blockIdx.x / C, true, s);
  const int r = s.r, W = s.W;
  auto B = [&](int i) { return blkp(s.small, W, i); };
  auto t = [&](int i) { return blkp(s.small1, W, A_SST + i); };  // the L side's copy: scratch here
  auto put = [](double* d) { return [d](int64_t e, double v) { d[e] = v; }; };
  const double* S0 = s.S0;  // ld r = W
  const Scheme& sc = g.sS;
  const int ns = sc.nstages;
  const double h = g.dt / sc.nsub;
  dgemm(tm, r, W, S0, false, B(A_N), true, put(t(0)));
  tm.sync();
  dgemm(tm, r, W, B(A_M), false, t(0), false, put(B(A_SST)));
  tm.sync();
  double* acc = B(A_SACC);
  for (int sub = 0; sub < sc.nsub; ++sub) {
    const double* y = B(A_SST + sub * ns);
    for (int st = 0; st < ns; ++st) {
      const double* z = B(A_SST + sub * ns + st);
      dgemm(tm, r, W, B(A_PU1), false, z, false, put(t(0)));
      dgemm(tm, r, W, B(A_GU1), false, z, false, put(t(1)));
      tm.sync();
      double* k1 = t(2);
      dgemm(tm, r, W, t(0), false, B(A_GV1), false, put(k1));
      __syncthreads();  // k1's entries may be another thread's of this CTA
      dgemm(tm, r, W, t(1), false, B(A_PV1), true, [&](int64_t e, double v) {
        v += k1[e];
        const double a = (st == 0) ? sc.b[0] * v : fma(sc.b[st], v, acc[e]);
        acc[e] = a;
        if (st + 1 < ns) B(A_SST + sub * ns + st + 1)[e] = fma(h * sc.a[st + 1], v, y[e]);
        else if (sub + 1 < sc.nsub) B(A_SST + (sub + 1) * ns)[e] = fma(h, a, y[e]);
      });
      tm.sync();
    }
  }
  // reversed: Sbar = S1_bar -> S~0_bar, coefficient gradients
  double* Sbar = B(A_SB);
  double* ybn = B(A_SYB);
  double* kb = B(A_SKB);
  double* zb = B(A_SZB);
  const int per = (r * r + C - 1) / C, e0 = tm.q * per, e1 = min(r * r, e0 + per);
  for (int o = e0 + threadIdx.x; o < e1; o += WT) {
    const int64_t e = o % r + (int64_t)(o / r) * W;
    Sbar[e] = s.Sb[e];
    for (int b = A_CPU; b <= A_CPV; ++b) B(b)[e] = 0.0;
  }
  __syncthreads();
  for (int sub = sc.nsub - 1; sub >= 0; --sub) {
    for (int st = ns - 1; st >= 0; --st) {
      const double* z = B(A_SST + sub * ns + st);
      for (int o = e0 + threadIdx.x; o < e1; o += WT) {
        const int64_t e = o % r + (int64_t)(o / r) * W;
        if (st == ns - 1) ybn[e] = Sbar[e];
        kb[e] = h * sc.b[st] * ybn[e] + ((st + 1 < ns) ? h * sc.a[st + 1] * zb[e] : 0.0);
      }
      tm.sync();
      dgemm(tm, r, W, kb, false, B(A_GV1), true, put(t(0)));
      dgemm(tm, r, W, B(A_PU1), false, z, false, put(t(1)));
      dgemm(tm, r, W, kb, false, B(A_PV1), false, put(t(2)));
      dgemm(tm, r, W, B(A_GU1), false, z, false, put(t(3)));
      dgemm(tm, r, W, B(A_PU1), true, kb, false, put(t(4)));
      dgemm(tm, r, W, B(A_GU1), true, kb, false, put(t(5)));
      tm.sync();
      auto add = [](double* d) { return [d](int64_t e, double v) { d[e] += v; }; };
      dgemm(tm, r, W, t(0), false, z, true, add(B(A_CPU)));
      dgemm(tm, r, W, t(1), true, kb, false, add(B(A_CGV)));
      dgemm(tm, r, W, t(2), false, z, true, add(B(A_CGU)));
      dgemm(tm, r, W, kb, true, t(3), false, add(B(A_CPV)));
      dgemm(tm, r, W, t(4), false, B(A_GV1), true, put(t(6)));
      __syncthreads();
      dgemm(tm, r, W, t(5), false, B(A_PV1), false, [&](int64_t e, double v) {
        v += t(6)[e];
        zb[e] = v;
        Sbar[e] += v;
      });
      tm.sync();  // kb is rewritten next
    }
  }
  // S~0 = M S0 N^T:  Mb = St0b N S0^T, Nb = St0b^T M S0, S0b = M^T St0b N
  dgemm(tm, r, W, B(A_N), false, S0, true, put(t(0)));
  dgemm(tm, r, W, B(A_M), false, S0, false, put(t(1)));
  dgemm(tm, r, W, Sbar, false, B(A_N), false, put(t(2)));
  tm.sync();
  dgemm(tm, r, W, Sbar, false, t(0), false, put(B(A_MB)));
  dgemm(tm, r, W, Sbar, true, t(1), false, put(B(A_NB)));
  dgemm(tm, r, W, B(A_M), true, t(2), false, put(B(A_S0B)));
}

// out(i, c) of this CTA's rows: x + sum_k [T X](i, k) C1(c, k) + X(i, k) C2(k, c) +
// [T^T X](i, k) C1(k, c), the adjoint of G = X^T X (C2 = Gbar + Gbar^T) and P = X^T T X
// (C1 = Pbar); C1s, C2s at k r + c
__device__ __forceinline__ double proj_adj(const double* X, const double* TX, const double* TtX, int ld, int r, int i,
                                           int c, const double* C1s, const double* C2s, double x) {
  for (int k = 0; k < r; ++k) {
    const int o = k * ld + 1 + i;
    x = fma(TX[o], C1s[c * r + k], x);
    x = fma(X[o], C2s[k * r + c], x);
    x = fma(TtX[o], C1s[k * r + c], x);
  }
  return x;
}

// theta_bar[lo + i] += sum_c X(i, c) sum_k X(i, k) C1(c, k)
__device__ void theta_proj(const Team& tm, int rows, int lo, int r, const double* X, int ld, const double* C1s,
                           double* scr, double* thb) {
  const wide::FastDiv by_rows(rows);
  for (int e = threadIdx.x; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    double v = 0.0;
    for (int k = 0; k < r; ++k) v = fma(X[k * ld + 1 + i], C1s[c * r + k], v);
    scr[c * ld + 1 + i] = v * X[c * ld + 1 + i];
  }
  __syncthreads();
  outputs(rows, r, [&](int i, int l, int L) {
    double v = 0.0;
    for (int c = l; c < r; c += L) v += scr[c * ld + 1 + i];
    return v;
  }, [&](int i, double v) { thb[lo + i] += v; });
  __syncthreads();
}

// small matrix (ld W) to Ms[k r + c]; sym: M + M^T
__device__ __forceinline__ void load_small(int r, int W, const double* M, bool sym, double* Ms) {
  for (int e = threadIdx.x; e < r * r; e += WT) {
    const int k = e / r, c = e % r;
    Ms[e] = M[k + (int64_t)c * W] + (sym ? M[c + (int64_t)k * W] : 0.0);
  }
}

__global__ void __launch_bounds__(WT, 1) adj_rev(const __grid_constant__ AdjArgs g, int C) {
  extern __shared__ __align__(16) double dsm[];
  Team tm{cg::this_cluster(), (int)cg::this_cluster().block_rank(), C};
  const int ci = blockIdx.x / C, tid = threadIdx.x;
  WideAdj s;
  wide_adj(g, ci >> 1, (ci & 1) == 0, s);
  const int r = s.r, W = s.W, N = s.N, rr = r * r;
  const int lo = tm.lo(N), rows = tm.hi(N) - lo, ld = (int)adj_ld(N, C);
  const int64_t len = (int64_t)N * r;
  const Tri T{s.tri, N, lo};
  const wide::FastDiv by_rows(rows);
  double* p0 = dsm;
  double* p1 = p0 + (size_t)r * ld;
  double* yb = p1 + (size_t)r * ld;
  double* p3 = yb + (size_t)r * ld;
  double* p4 = p3 + (size_t)r * ld;
  double* misc = p4 + (size_t)r * ld;
  double* inv = misc + adj_misc(N, r, C);
  tm.cl.sync();
  // Q_bar = output's adjoint + X0 Mb^T + adjoint of the projections of Q; the
  // first part of X0_bar: Q Mb
  double* Mb = misc;
  double* C1s = misc + rr;
  double* C2s = misc + 2 * rr;
  load_small(r, W, blkp(s.small, W, s.kside ? A_MB : A_NB), false, Mb);
  load_small(r, W, blkp(s.small, W, s.kside ? A_CPU : A_CPV), false, C1s);
  load_small(r, W, blkp(s.small, W, s.kside ? A_CGU : A_CGV), true, C2s);
  load_rows_halo(s.Q, N, lo, rows, r, p0, ld);
  load_rows(s.X0, N, lo, rows, r, p1, ld);
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    p3[k * ld + 1 + i] = T.mul(p0, ld, i, k);
    p4[k * ld + 1 + i] = T.mul_t(p0, ld, i, k);
  }
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    double v = s.Xb[lo + i + (int64_t)c * N], x = 0.0;
    for (int k = 0; k < r; ++k) {
      v = fma(p1[k * ld + 1 + i], Mb[c * r + k], v);
      x = fma(p0[k * ld + 1 + i], Mb[k * r + c], x);
    }
    yb[c * ld + 1 + i] = proj_adj(p0, p3, p4, ld, r, i, c, C1s, C2s, v);
    s.xb[lo + i + (int64_t)c * N] = x;
  }
  __syncthreads();
  if (s.kside) theta_proj(tm, rows, lo, r, p0, ld, C1s, p1, s.thb);
  // QR adjoint: yb <- (yb + Q copyltu(-yb^T Q)) R^-T
  {
    double* part = misc + 2 * rr;
    __syncthreads();
    outputs(rr, rows, [&](int o, int l, int L) {
      const int a = o % r, c = o / r;
      double v = 0.0;
      for (int i = 1 + l; i <= rows; i += L) v = fma(-yb[a * ld + i], p0[c * ld + i], v);
      return v;
    }, [&](int o, double v) { part[o] = v; });
    double* Mx = blkp(s.kside ? s.small : s.small1, W, A_T1);
    reduce_parts(tm, part, rr, [&](int e, double v) { Mx[e % r + (int64_t)(e / r) * W] = v; });
    const double* R = blkp(s.small, W, s.kside ? A_RK : A_RL);
    double* Cl = misc;
    double* Rs = misc + rr;  // Rs[k r + j] = R(k, j)
    for (int e = tid; e < rr; e += WT) {
      const int k = e / r, c = e % r;
      Cl[e] = (k >= c) ? Mx[k + (int64_t)c * W] : Mx[c + (int64_t)k * W];
      Rs[e] = R[k + (int64_t)c * W];
    }
    if (tid < r) inv[tid] = 1.0 / R[tid + (int64_t)tid * W];
    __syncthreads();
    for (int e = tid; e < rows * r; e += WT) {
      const int c = by_rows.div(e), i = e - c * rows;
      double v = yb[c * ld + 1 + i];
      for (int k = 0; k < r; ++k) v = fma(p0[k * ld + 1 + i], Cl[k * r + c], v);
      yb[c * ld + 1 + i] = v;
    }
    __syncthreads();
    // back substitution along each row, two lanes per row
    for (int i0 = 0; i0 < rows; i0 += WT / 2) {
      const int i = i0 + (tid >> 1), l = tid & 1;
      const bool in = i < rows;
      for (int k = r - 1; k >= 0; --k) {
        double v = 0.0;
        if (in)
          for (int j = k + 1 + l; j < r; j += 2) v = fma(yb[j * ld + 1 + i], Rs[k * r + j], v);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if (in && l == 0) yb[k * ld + 1 + i] = (yb[k * ld + 1 + i] - v) * inv[k];
        __syncwarp();
      }
    }
    __syncthreads();
  }
  // RK reversal: kb = h b_s yb' + h a_{s+1} zb_{s+1}; Gbar += (T z)^T kb,
  // Pbar += kb^T z, theta_bar += kb . (z G); zb = T^T kb G^T + kb P; yb += zb
  const double* Gg = blkp(s.small, W, s.kside ? A_GV : A_GU);
  double* Ps = misc;
  double* part = misc + rr;
  float* Es = reinterpret_cast<float*>(misc + 4 * rr);
  float* tf = reinterpret_cast<float*>(misc + 4 * rr + (rr + 1) / 2);
  const bool full = load_ep(r, W, Gg, Gg + (int64_t)W * W, true, true, Ps, Es);
  for (int e = tid; e < 3 * rr; e += WT) part[e] = 0.0;
  const Scheme& sc = s.kside ? g.sK : g.sL;
  const double h = g.dt / sc.nsub;
  double* kb = p0;
  double* ybn = p1;
  double* z = p4;
  // kb's halo rows: zero at the ends of the domain (no neighbour pushes there)
  tm.cl.sync();  // every CTA is past its reads of Q's halo rows
  for (int e = tid; e < r; e += WT) {
    kb[e * ld] = 0.0;
    kb[e * ld + 1 + tm.rows_per(N)] = 0.0;
    kb[e * ld + 1 + rows] = 0.0;
  }
  tm.cl.sync();
  for (int sub = sc.nsub - 1; sub >= 0; --sub) {
    for (int e = tid; e < rows * r; e += WT) {
      const int q = by_rows.div(e), o = q * ld + 1 + e - q * rows;
      ybn[o] = yb[o];
    }
    for (int st = sc.nstages - 1; st >= 0; --st) {
      const double hb = h * sc.b[st], ha = (st + 1 < sc.nstages) ? h * sc.a[st + 1] : 0.0;
      for (int e = tid; e < rows * r; e += WT) {  // every thread its own entries
        const int q = by_rows.div(e), o = q * ld + 1 + e - q * rows;
        kb[o] = (st + 1 < sc.nstages) ? fma(ha, p3[o], hb * ybn[o]) : hb * ybn[o];
      }
      load_rows_halo(s.Z + (int64_t)(sub * sc.nstages + st) * len, N, lo, rows, r, z, ld);
      __syncthreads();
      push_halos(tm, N, rows, r, kb, ld);
      int zbig = full, zreaches = 0;
      for (int e = tid; e < rows * r; e += WT) {
        const int q = by_rows.div(e), o = q * ld + 1 + e - q * rows;
        p3[o] = T.mul(z, ld, e % rows, e / rows);
        zbig |= !wide::below_2_100(z[o]);
        zreaches |= wide::reaches_2_m80(z[o]);
      }
      tm.cl.sync();
      outputs(2 * rr, rows, [&](int o, int l, int L) {
        const int a = o % r, c = (o / r) % r;
        const double* x = (o < rr) ? p3 : kb;
        const double* y = (o < rr) ? kb : z;
        double v = 0.0;
        for (int i = 1 + l; i <= rows; i += L) v = fma(x[a * ld + i], y[c * ld + i], v);
        return v;
      }, [&](int o, double v) { part[o] += v; });
      zbig = wide::out_of_f32(zbig, zreaches);  // T z is consumed
      if (s.kside) {
        for (int e = tid; e < rows * r; e += WT) {
          const int c = by_rows.div(e), i = e - c * rows;
          double v;
          if (!zbig) {
            float ef = 0.0f;  // Es holds the transpose of G - I
            for (int k = 0; k < r; ++k) ef = fmaf((float)z[k * ld + 1 + i], Es[c * r + k], ef);
            v = z[c * ld + 1 + i] + (double)ef;
          } else {
            v = 0.0;
            for (int k = 0; k < r; ++k) v = fma(z[k * ld + 1 + i], Gg[k + (int64_t)c * W], v);
          }
          p3[c * ld + 1 + i] = v * kb[c * ld + 1 + i];
        }
        __syncthreads();
        outputs(rows, r, [&](int i, int l, int L) {
          double v = 0.0;
          for (int c = l; c < r; c += L) v += p3[c * ld + 1 + i];
          return v;
        }, [&](int i, double v) { s.thb[lo + i] += v; });
        __syncthreads();
      }
      int big = full, reaches = 0;
      if (!full) {
        for (int e = tid; e < rows * r; e += WT) {
          const int k = by_rows.div(e), i = e - k * rows;
          const double tk = T.mul_t(kb, ld, i, k);
          p3[k * ld + 1 + i] = tk;
          tf[e] = (float)tk;
          big |= !wide::below_2_100(tk);
          reaches |= wide::reaches_2_m80(tk);
        }
        big = wide::out_of_f32(big, reaches);
      }
      for (int e = tid; e < rows * r; e += WT) {
        const int c = by_rows.div(e), i = e - c * rows, o = c * ld + 1 + i;
        double v;
        if (!big) {
          float ef = 0.0f;
          for (int k = 0; k < r; ++k) ef = fmaf(tf[k * rows + i], Es[k * r + c], ef);
          v = p3[o] + (double)ef;
        } else {
          v = 0.0;
          for (int k = 0; k < r; ++k) v = fma(T.mul_t(kb, ld, i, k), Gg[c + (int64_t)k * W], v);
        }
        for (int k = 0; k < r; ++k) v = fma(kb[k * ld + 1 + i], Ps[k * r + c], v);
        p3[o] = v;
        yb[o] += v;
      }
      tm.cl.sync();  // kb and its halo rows are rewritten next
    }
  }
  // X0_bar += y0_bar S0^T (K) or S0 (L); S0_bar's part: X0^T y0_bar (K) or its transpose
  for (int e = tid; e < rr; e += WT) {
    const int k = e / r, c = e % r;
    Ps[e] = s.kside ? s.S0[c + (int64_t)k * r] : s.S0[k + (int64_t)c * r];
  }
  load_rows(s.X0, N, lo, rows, r, p4, ld);
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    double v = s.xb[lo + i + (int64_t)c * N];
    for (int k = 0; k < r; ++k) v = fma(yb[k * ld + 1 + i], Ps[k * r + c], v);
    s.xb[lo + i + (int64_t)c * N] = v;
  }
  outputs(rr, rows, [&](int o, int l, int L) {
    const int a = o % r, c = o / r;
    const double* x = s.kside ? p4 : yb;
    const double* y = s.kside ? yb : p4;
    double v = 0.0;
    for (int i = 1 + l; i <= rows; i += L) v = fma(x[a * ld + i], y[c * ld + i], v);
    return v;
  }, [&](int o, double v) { part[2 * rr + o] = v; });
  double* Gb = blkp(s.small, W, s.kside ? A_KG : A_LG);
  double* Pb = blkp(s.small, W, s.kside ? A_KP : A_LP);
  double* S0b = s.kside ? blkp(s.small, W, A_S0B) : blkp(s.small1, W, A_S0B);
  reduce_parts(tm, part, 3 * rr, [&](int e, double v) {
    const int64_t o = e % r + (int64_t)((e / r) % r) * W;
    if (e < rr) Gb[o] = v;
    else if (e < 2 * rr) Pb[o] = v;
    else S0b[o] = s.kside ? S0b[o] + v : v;
  });
}

__global__ void __launch_bounds__(WT, 1) adj_out(const __grid_constant__ AdjArgs g, int C) {
  extern __shared__ __align__(16) double dsm[];
  Team tm{cg::this_cluster(), (int)cg::this_cluster().block_rank(), C};
  const int ci = blockIdx.x / C, tid = threadIdx.x;
  WideAdj s;
  wide_adj(g, ci >> 1, (ci & 1) == 0, s);
  const int r = s.r, W = s.W, N = s.N, rr = r * r;
  const int lo = tm.lo(N), rows = tm.hi(N) - lo, ld = (int)adj_ld(N, C);
  const Tri T{s.tri, N, lo};
  const wide::FastDiv by_rows(rows);
  double* p0 = dsm;
  double* p3 = p0 + (size_t)r * ld;
  double* p4 = p3 + (size_t)r * ld;
  double* C1s = p4 + (size_t)r * ld;
  double* C2s = C1s + rr;
  // adjoint of the other side's projections of this side's input basis
  load_small(r, W, blkp(s.small, W, s.kside ? A_LP : A_KP), false, C1s);
  load_small(r, W, blkp(s.small, W, s.kside ? A_LG : A_KG), true, C2s);
  load_rows_halo(s.X0, N, lo, rows, r, p0, ld);
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int k = by_rows.div(e), i = e - k * rows;
    p3[k * ld + 1 + i] = T.mul(p0, ld, i, k);
    p4[k * ld + 1 + i] = T.mul_t(p0, ld, i, k);
  }
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    const int64_t o = lo + i + (int64_t)c * N;
    s.Xb[o] = proj_adj(p0, p3, p4, ld, r, i, c, C1s, C2s, s.xb[o]);
  }
  __syncthreads();
  if (s.kside) theta_proj(tm, rows, lo, r, p0, ld, C1s, p3, s.thb);
  if (!s.kside) {
    const double* a = blkp(s.small, W, A_S0B);
    const double* b = blkp(s.small1, W, A_S0B);
    for (int e = tm.q * WT + tid; e < rr; e += C * WT) {
      const int64_t o = e % r + (int64_t)(e / r) * W;
      s.Sb[o] = a[o] + b[o];
    }
  }
}

cudaError_t adj_launch(void (*kern)(const AdjArgs, int), const AdjArgs& g, int blocks, int C, size_t smem,
                       std::atomic<uint64_t>& done, cudaStream_t st) {
  cudaError_t e = wide::cluster_attributes(kern, done);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  wide::cluster_config(cfg, attr, blocks, C, smem, st);
  return cudaLaunchKernelEx(&cfg, kern, g, C);
}

}  // namespace

size_t adjoint_work_elems(int64_t n, int64_t m, int64_t r, int ns_k, int ns_l) {
  return 2 * (size_t)A_COUNT * r * r + 3 * (size_t)(n + m) + (size_t)(ns_k + P_COUNT) * n * r +
         (size_t)(ns_l + P_COUNT) * m * r;
}

int adjoint_max_stages() { return kAdjMaxStages; }

AdjointPlan adjoint_plan(int count, const int64_t* n, const int64_t* m, const int64_t* r, int sms) {
  AdjointPlan p;
  int64_t tall = 0;
  for (int i = 0; i < count; ++i) tall = std::max(tall, std::max(n[i], m[i]));
  p.C = wide_cluster(count, tall, sms);
  if (p.C < 2) return AdjointPlan{};
  for (int i = 0; i < count; ++i)
    for (int64_t N : {n[i], m[i]}) {
      const int ri = (int)r[i];
      if (ri > wide::WR_MAX) return AdjointPlan{};
      p.fwd_smem = std::max(p.fwd_smem, sizeof(double) * adj_fwd_doubles((int)N, ri, p.C));
      p.rev_smem = std::max(p.rev_smem, sizeof(double) * adj_rev_doubles((int)N, ri, p.C));
    }
  if (p.fwd_smem > kWideSmemMax || p.rev_smem > kWideSmemMax) return AdjointPlan{};
  p.fwd_smem = std::max(p.fwd_smem, (size_t)120 * 1024);  // a CTA per SM
  p.rev_smem = std::max(p.rev_smem, (size_t)120 * 1024);
  return p;
}

cudaError_t launch_adjoint_step(const InstDesc* inst, const int64_t* adj_off, const int64_t* th_off, int count,
                                const double* U0, const double* S0, const double* V0, double* Ub, double* Sb,
                                double* Vb, double* thb, const double* opA, const double* opB, double* work,
                                const Scheme& sK, const Scheme& sL, const Scheme& sS, double dt, const AdjointPlan& plan,
                                cudaStream_t st) {
  AdjArgs g{inst, adj_off, th_off, U0, S0, V0, Ub, Sb, Vb, thb, opA, opB, work, sK, sL, sS, dt, 0};
  if (plan.C) {
    static std::atomic<uint64_t> d0{0}, d1{0}, d2{0}, d3{0};
    const int C = plan.C;
    cudaError_t e = adj_launch(adj_fwd, g, 2 * C * count, C, plan.fwd_smem, d0, st);
    if (e == cudaSuccess) e = adj_launch(adj_core, g, C * count, C, 0, d1, st);
    if (e == cudaSuccess) e = adj_launch(adj_rev, g, 2 * C * count, C, plan.rev_smem, d2, st);
    if (e == cudaSuccess) e = adj_launch(adj_out, g, 2 * C * count, C, plan.rev_smem, d3, st);
    return e != cudaSuccess ? e : cudaGetLastError();
  }
  const size_t smem = sizeof(Smem<double>);
  // Batches small enough that every instance can have two SMs run the K and
  // L sides on a 2-CTA cluster each.  Its CTAs ask for more shared memory
  // than two CTAs of an SM can hold, so the pair runs on two SMs (a CTA pair
  // on one SM would share its FP64 units).
  constexpr int kSplitSmem = 120 * 1024;
  static_assert(sizeof(Smem<double>) <= kSplitSmem, "split launch smem below the kernel's");
  static std::atomic<uint64_t> attr_done{0};
  cudaError_t e = set_smem_limit(adjoint_step_kernel, kSplitSmem, attr_done);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (2 * count <= sms) {
    g.split = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * count, 1, 1);
    cfg.blockDim = dim3(NT, 1, 1);
    cfg.dynamicSmemBytes = kSplitSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, adjoint_step_kernel, g);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
  }
  adjoint_step_kernel<<<count, NT, smem, st>>>(g);
  return cudaGetLastError();
}

}  // namespace lri
