// engine_wide.cu - FP64 BUG steps (Sylvester flow and data streams) with the
// panels of a side in shared memory, each side on one CTA or spread over a
// thread-block cluster.
//
// An FP64 step of one instance is bound by the FP64 units of the SMs it runs
// on (about 1.9 multiply-adds per clock each); on one 2-CTA pair a batch of
// one leaves 150 SMs idle.  Here a step is two launches:
//   wide_sides  two clusters per instance, one per side (the K and L steps
//               read only the old factors): the side's rows are split over the
//               cluster's CTAs and stay in shared memory through the substep
//               (halo rows pushed to the neighbours through distributed
//               shared memory), the QR (wide::qr), the basis change and the
//               new basis's projections;
//   wide_core   one cluster per instance: S~0 = M S0 N^T and the S step, the
//               core's columns split over the CTAs.
// One instance, per step: 256 x 256, r = 8, 20 RK4 substeps 1056 us on a 2-CTA
// pair, 275 us here (sides 165, core 109; what is left are the 160 dependent
// stages' barriers and FP64 chains); 2048 x 2048, r = 32, 12.0 ms against 0.57
// ms (FP64 issue on 32 SMs); a 100 x 100 data step, r = 12, 754 us on one CTA,
// 86 us here.
// Same operations as bug_step / bug_step_pair of the instance engine (the
// literal form with the Gram factors), sums in a different order; the QR is
// Householder's with the same signs.
#include "engine_api.h"
#include "wide.cuh"

namespace lri {
namespace {

using wide::load_rows;
using wide::outputs;
using wide::push_halos;
using wide::QrSmem;
using wide::reduce_parts;
using wide::Team;
using wide::Tri;
using wide::WT;

// small-scratch block indices shared with the instance engine
enum : int { WB_GU = 0, WB_GV = 2, WB_M = 4, WB_N = 5, WB_NEWU = 19, WB_NEWV = 21 };

// one instance's pointers (the packed layout of the instance engine)
struct WInst {
  int n, m, W, rcap, inst, r;
  double* U;
  double* S;
  double* V;
  const double* opA;
  const double* opB;
  double* QU;  // QR outputs of steps whose sides read both old bases
  double* QV;
  double* small;
  double* Yp;
  const double* Yn;
  __device__ double* blk(int i) const { return small + (int64_t)i * (((int64_t)W * W + 3) & ~int64_t(3)); }
};

__device__ __forceinline__ bool wide_inst(const StepArgs<double>& g, int inst, WInst& I) {
  const InstDesc d = g.inst[inst];
  I.n = d.n; I.m = d.m; I.W = d.wcap; I.rcap = d.rcap; I.inst = inst;
  I.U = g.U + d.offU;
  I.S = g.S + d.offS;
  I.V = g.V + d.offV;
  I.opA = g.opA ? g.opA + d.offA : nullptr;
  I.opB = g.opB ? g.opB + d.offB : nullptr;
  I.QU = g.work + d.offWK;
  I.QV = g.work + d.offWL;
  I.small = g.small + d.offSmall;
  I.Yp = (g.op == OP_DATA) ? g.Yprev + d.offY : nullptr;
  I.Yn = (g.op == OP_DATA) ? g.Ynext + d.offY : nullptr;
  I.r = g.rank[inst];
  if (I.r < 1 || I.r > d.rcap) {
    if (threadIdx.x == 0) atomicOr(g.status, ST_BAD_SHAPE);
    return false;
  }
  return true;
}

// Shared memory of wide_sides: three panels of the cluster's rows, p[k ld + 1 +
// i] with a halo row on each side (i = -1 and i = R0), the small matrices and
// the FP32 copy of T w (later the Gram partials, or a data step's chunks), the
// QR's scratch.
__host__ __device__ inline size_t misc_doubles(int R0, int r) {
  const size_t sub = (size_t)r * R0 / 2 + 1 + 2 * (size_t)r * r + ((size_t)r * r + 1) / 2, gram = 3 * (size_t)r * r;
  const size_t data = 32 * (size_t)(R0 + r);  // data steps: a 32-column chunk of dY and of the other basis
  return sub > gram ? (sub > data ? sub : data) : (gram > data ? gram : data);
}
__host__ __device__ inline size_t side_doubles(int N, int r, int C) {
  const int R0 = (N + C - 1) / C, ld = (R0 + 2) | 1;
  return 3 * (size_t)r * ld + misc_doubles(R0, r) + QrSmem<double>::elems(C, r);
}

__global__ void __launch_bounds__(WT, 2)
    wide_sides(const __grid_constant__ StepArgs<double> g, const int32_t* __restrict__ items, int C) {
  extern __shared__ __align__(16) double dsm[];
  Team tm{wide::cg::this_cluster(), (int)wide::cg::this_cluster().block_rank(), C};
  const int item = items[blockIdx.x / C], tid = threadIdx.x;
  WInst I;
  if (!wide_inst(g, item >> 1, I)) return;  // the same in every CTA of the cluster
  const bool kside = (item & 1) == 0;
  const int r = I.r, W = I.W, N = kside ? I.n : I.m, No = kside ? I.m : I.n;
  double* X = kside ? I.U : I.V;
  const double* Xo = kside ? I.V : I.U;
  const bool sylv = g.op == OP_SYLVESTER;
  // before the first step the other basis's projections are formed here, so
  // both sides read both old bases (as in a data step)
  const bool fresh = sylv && g.proj_valid[I.inst] == 0;
  const int R0 = tm.rows_per(N), lo = tm.lo(N), rows = tm.hi(N) - lo;
  const Tri T{kside ? I.opA : I.opB, N, lo};
  const wide::FastDiv by_rows(rows);
  const int ldr = (R0 + 2) | 1;
  // carve
  double* sp = dsm;
  double* p0 = sp; sp += r * ldr;
  double* p1 = sp; sp += r * ldr;
  double* p2 = sp; sp += r * ldr;
  double* misc = sp; sp += misc_doubles(R0, r);
  const QrSmem<double> qs = QrSmem<double>::carve(sp, C, r);
  double* Go = I.blk(kside ? WB_GV : WB_GU);  // projections of the other basis
  tm.cl.sync();  // every CTA runs before any distributed access
  if (fresh) {
    // projections of the other (old) basis: G = Xo^T Xo, P = Xo^T (To Xo);
    // its rows through the panels in blocks of R0 (they may be more than this
    // side's), both halo rows from memory
    const double* to = kside ? I.opB : I.opA;
    const int lo2 = tm.lo(No), hi2 = tm.hi(No);
    double* part = misc;
    for (int e = tid; e < 2 * r * r; e += WT) part[e] = 0.0;
    __syncthreads();
    for (int b = lo2; b < hi2; b += R0) {
      const int nb = min(R0, hi2 - b);
      for (int e = tid; e < (nb + 2) * r; e += WT) {
        const int i = b - 1 + e % (nb + 2), k = e / (nb + 2);
        p0[k * ldr + e % (nb + 2)] = (i >= 0 && i < No) ? Xo[i + (int64_t)k * No] : 0.0;
      }
      __syncthreads();
      const Tri To{to, No, b};
      for (int e = tid; e < nb * r; e += WT) p1[(e / nb) * ldr + 1 + e % nb] = To.mul(p0, ldr, e % nb, e / nb);
      __syncthreads();
      for (int o = tid; o < 2 * r * r; o += WT) {
        const int a = o % r, c = (o / r) % r;
        const double* y = (o < r * r) ? p0 : p1;
        double s = part[o];
        for (int i = 1; i <= nb; ++i) s = fma(p0[a * ldr + i], y[c * ldr + i], s);
        part[o] = s;
      }
      __syncthreads();
    }
    reduce_parts(tm, part, 2 * r * r, [&](int e, double s) {
      Go[(e / (r * r)) * r * W + e % r + (int64_t)((e / r) % r) * W] = s;
    });
  }
  // zero halo rows at the ends of the domain (never pushed to)
  for (int e = tid; e < 3 * r; e += WT) {
    double* p = (e < r) ? p0 : (e < 2 * r ? p1 : p2);
    const int k = e % r;
    p[k * ldr] = 0.0;
    p[k * ldr + 1 + R0] = 0.0;
    if (rows < R0) p[k * ldr + 1 + rows] = 0.0;
  }
  // y = X C, C = S (K) or S^T (L)
  double* Cs = misc;  // Cs[k r + c]
  for (int e = tid; e < r * r; e += WT) {
    const int k = e / r, c = e % r;
    Cs[e] = kside ? I.S[k + (int64_t)c * I.rcap] : I.S[c + (int64_t)k * I.rcap];
  }
  load_rows(X, N, lo, rows, r, p1, ldr);
  __syncthreads();
  for (int e = tid; e < rows * r; e += WT) {
    const int c = by_rows.div(e), i = e - c * rows;
    double s = 0.0;
    for (int k = 0; k < r; ++k) s = fma(p1[k * ldr + 1 + i], Cs[k * r + c], s);
    p0[c * ldr + 1 + i] = s;
    p2[c * ldr + 1 + i] = s;
  }
  __syncthreads();
  double* win = p0;
  double* wout = p1;
  if (sylv) {
    double* Ps = misc;                                      // Ps[k r + c] = P(c, k)
    double* Gs = Ps + r * r;                                // Gs[k r + c] = G(k, c)
    float* Es = reinterpret_cast<float*>(Gs + r * r);       // G - I
    float* tf = reinterpret_cast<float*>(misc + 2 * r * r + (r * r + 1) / 2);  // FP32 copy of T w, [k][i]
    const double* P = Go + (int64_t)r * W;
    int full = 0;
    for (int e = tid; e < r * r; e += WT) {
      const int k = e / r, c = e % r;
      Ps[e] = P[c + (int64_t)k * W];
      const double gv = Go[k + (int64_t)c * W], ev = gv - ((k == c) ? 1.0 : 0.0);
      Gs[e] = gv;
      Es[e] = (float)ev;
      if (!(fabs(ev) <= 0x1p-36)) full = 1;  // NaN included
    }
    // (T w) G = T w + (T w) E with E applied in FP32 (see below_2_100), or the
    // full product
    full = __syncthreads_or(full);
    tm.cl.sync();  // the zero halo rows of every CTA are set
    push_halos(tm, N, rows, r, win, ldr);
    tm.cl.sync();
    const Scheme& sc = kside ? g.sK : g.sL;
    const double h = g.dt / sc.nsub;
    for (int sub = 0; sub < sc.nsub; ++sub) {
      double hw = h * sc.gam[sc.nstages];
      for (int j = sc.nstages - 1; j >= 0; --j) {
        const double gj = (j == 0) ? 1.0 : sc.gam[j];
        int big = full, reaches = 0;
        if (!full) {
          // T w into this thread's own entries of wout, its FP32 copy for the row
          for (int e = tid; e < rows * r; e += WT) {
            const int k = by_rows.div(e), i = e - k * rows;
            const double tw = T.mul(win, ldr, i, k);
            wout[k * ldr + 1 + i] = tw;
            tf[e] = (float)tw;
            big |= !wide::below_2_100(tw);
            reaches |= wide::reaches_2_m80(tw);
          }
          big = wide::out_of_f32(big, reaches);
        }
        for (int e = tid; e < rows * r; e += WT) {
          const int c = by_rows.div(e), i = e - c * rows;
          double s;
          if (!big) {
            float ef = 0.0f;
            for (int k = 0; k < r; ++k) ef = fmaf(tf[k * rows + i], Es[k * r + c], ef);
            s = wout[c * ldr + 1 + i] + (double)ef;
          } else {
            s = 0.0;
            for (int k = 0; k < r; ++k) s = fma(T.mul(win, ldr, i, k), Gs[k * r + c], s);
          }
          for (int k = 0; k < r; ++k) s = fma(win[k * ldr + 1 + i], Ps[k * r + c], s);
          s = fma(hw, s, gj * p2[c * ldr + 1 + i]);
          wout[c * ldr + 1 + i] = s;
          if (j == 0) p2[c * ldr + 1 + i] = s;  // the next substep's base
          // boundary rows to the neighbours' halos
          if (i == 0 && tm.q > 0) tm.at(wout, tm.q - 1)[c * ldr + 1 + R0] = s;
          if (i == rows - 1 && tm.q + 1 < C && lo + rows < N) tm.at(wout, tm.q + 1)[c * ldr] = s;
        }
        tm.cl.sync();
        double* t = win;
        win = wout;
        wout = t;
        hw = h;
      }
    }
  } else {
    // data: y += dY Xo (K) or dY^T Xo (L), dY = Yn - Yp, in chunks of 32
    double* dl = misc;            // dl[jj R0 + i]
    double* xo = misc + 32 * R0;  // xo[jj r + c]
    for (int j0 = 0; j0 < No; j0 += 32) {
      const int nj = min(32, No - j0);
      for (int e = tid; e < nj * rows; e += WT) {
        const int jj = kside ? e / rows : e % nj, i = kside ? e % rows : e / nj;
        const int64_t o = kside ? (lo + i) + (int64_t)(j0 + jj) * I.n : (j0 + jj) + (int64_t)(lo + i) * I.n;
        dl[jj * R0 + i] = I.Yn[o] - I.Yp[o];
      }
      for (int e = tid; e < nj * r; e += WT) xo[(e % nj) * r + e / nj] = Xo[j0 + e % nj + (int64_t)(e / nj) * No];
      __syncthreads();
      outputs(rows * r, nj, [&](int o, int l, int L) {
        const int i = o % rows, c = o / rows;
        double s = 0.0;
        for (int jj = l; jj < nj; jj += L) s = fma(dl[jj * R0 + i], xo[jj * r + c], s);
        return s;
      }, [&](int o, double v) { win[(o / rows) * ldr + 1 + o % rows] += v; });
      __syncthreads();
    }
  }
  wide::qr<double>(tm, N, lo, rows, r, win + 1, ldr, wout + 1, ldr, nullptr, 0, qs);
  // basis change X1^T X0 and, for the flow, the new basis's projections
  double* Q = wout;
  double* part = misc;
  load_rows(X, N, lo, rows, r, win, ldr);
  if (sylv) {
    push_halos(tm, N, rows, r, Q, ldr);
    tm.cl.sync();
    for (int e = tid; e < rows * r; e += WT) {
      const int k = by_rows.div(e), i = e - k * rows;
      p2[k * ldr + 1 + i] = T.mul(Q, ldr, i, k);
    }
  }
  __syncthreads();
  const int nout = (sylv ? 3 : 1) * r * r;
  outputs(nout, rows, [&](int o, int l, int L) {
    const int a = o % r, c = (o / r) % r, w = o / (r * r);
    if (w == 1 && a > c) return 0.0;  // G is symmetric
    const double* y = (w == 0) ? win : (w == 1 ? Q : p2);
    double s = 0.0;
    for (int i = 1 + l; i <= rows; i += L) s = fma(Q[a * ldr + i], y[c * ldr + i], s);
    return s;
  }, [&](int o, double v) { part[o] = v; });
  double* Mo = I.blk(kside ? WB_M : WB_N);
  double* Gn = I.blk(kside ? WB_NEWU : WB_NEWV);
  reduce_parts(tm, part, nout, [&](int e, double s) {
    const int a = e % r, c = (e / r) % r, w = e / (r * r);
    if (w == 0) Mo[a + (int64_t)c * W] = s;
    else if (w == 2) Gn[(int64_t)r * W + a + (int64_t)c * W] = s;
    else if (a <= c) {
      Gn[a + (int64_t)c * W] = s;
      Gn[c + (int64_t)a * W] = s;
    }
  });
  // the new basis: in place where nobody else reads these rows, else to the
  // workspace (wide_core copies it)
  double* dst = (sylv && !fresh) ? X : (kside ? I.QU : I.QV);
  for (int e = tid; e < rows * r; e += WT)
    dst[lo + e % rows + (int64_t)(e / rows) * N] = Q[(e / rows) * ldr + 1 + e % rows];
}

// shared memory of wide_core in doubles
__host__ __device__ inline size_t core_doubles(int r, int C) {
  const int cpc = (r + C - 1) / C;
  return 4 * (size_t)r * r + 6 * (size_t)r * cpc + 32 * (size_t)(r + 32) + (size_t)r * r;
}

__global__ void __launch_bounds__(WT, 1) wide_core(const __grid_constant__ StepArgs<double> g, int C) {
  extern __shared__ __align__(16) double dsm[];
  Team tm{wide::cg::this_cluster(), (int)wide::cg::this_cluster().block_rank(), C};
  const int tid = threadIdx.x;
  WInst I;
  if (!wide_inst(g, g.order[blockIdx.x / C], I)) return;
  const bool sylv = g.op == OP_SYLVESTER;
  const int r = I.r, W = I.W, rr = r * r;
  const int cpc = (r + C - 1) / C, c0 = min(r, tm.q * cpc), nc = min(r, c0 + cpc) - c0;  // own columns
  double* Z0 = dsm;           // Z(i, j) at i + j r, two copies in turn
  double* Z1 = Z0 + rr;
  double* PU = Z1 + rr;       // P_U(i, k) at i + k r
  double* GU = PU + rr;
  double* gv = GU + rr;       // G_V(:, c) of the own columns
  double* pv = gv + r * cpc;  // P_V(c, :)
  double* t1 = pv + r * cpc;
  double* t2 = t1 + r * cpc;
  double* yst = t2 + r * cpc;  // state and accumulator of the own columns
  double* ast = yst + r * cpc;
  double* stage = ast + r * cpc;    // data: chunks; partials
  const double* M = I.blk(WB_M);
  const double* Nn = I.blk(WB_N);
  const double* nu = I.blk(WB_NEWU);
  const double* nv = I.blk(WB_NEWV);
  const bool fresh = sylv && g.proj_valid[I.inst] == 0;  // read before the cluster barriers, set after them
  auto take_bases = [&]() {
    for (int64_t e = tm.q * WT + tid; e < (int64_t)I.n * r; e += (int64_t)C * WT) I.U[e] = I.QU[e];
    for (int64_t e = tm.q * WT + tid; e < (int64_t)I.m * r; e += (int64_t)C * WT) I.V[e] = I.QV[e];
  };
  tm.cl.sync();
  for (int e = tid; e < rr; e += WT) {
    Z1[e] = I.S[e % r + (int64_t)(e / r) * I.rcap];
    PU[e] = M[e % r + (int64_t)(e / r) * W];
  }
  for (int e = tid; e < r * nc; e += WT) gv[e] = Nn[c0 + e / r + (int64_t)(e % r) * W];  // N(c, k)
  __syncthreads();
  // S~0 = M (S0 N^T), own columns, to every CTA
  outputs(r * nc, r, [&](int o, int l, int L) {
    const int i = o % r, c = o / r;
    double s = 0.0;
    for (int k = l; k < r; k += L) s = fma(Z1[i + k * r], gv[k + c * r], s);
    return s;
  }, [&](int o, double v) { t1[o] = v; });
  __syncthreads();
  outputs(r * nc, r, [&](int o, int l, int L) {
    const int i = o % r, c = o / r;
    double s = 0.0;
    for (int k = l; k < r; k += L) s = fma(PU[i + k * r], t1[k + c * r], s);
    return s;
  }, [&](int o, double v) { yst[o] = v; });
  __syncthreads();
  if (!sylv) {
    // S += U1^T dY V1 (the exact data flow): rows of U1 and dY split over the
    // cluster, Z = dY V1 a chunk of 32 rows at a time
    const int lo = tm.lo(I.n), hi = tm.hi(I.n);
    double* zc = stage;         // zc[c 32 + i]
    double* dy = zc + 32 * r;   // dy[jj 32 + i]
    double* part = dy + 32 * 32;
    for (int e = tid; e < rr; e += WT) part[e] = 0.0;
    for (int i0 = lo; i0 < hi; i0 += 32) {
      const int ni = min(32, hi - i0);
      for (int e = tid; e < 32 * r; e += WT) zc[e] = 0.0;
      for (int j0 = 0; j0 < I.m; j0 += 32) {
        const int nj = min(32, I.m - j0);
        __syncthreads();
        for (int e = tid; e < ni * nj; e += WT) {
          const int64_t o = i0 + e % ni + (int64_t)(j0 + e / ni) * I.n;
          dy[(e / ni) * 32 + e % ni] = I.Yn[o] - I.Yp[o];
        }
        __syncthreads();
        outputs(ni * r, nj, [&](int o, int l, int L) {
          const int i = o % ni, c = o / ni;
          double s = 0.0;
          for (int jj = l; jj < nj; jj += L) s = fma(dy[jj * 32 + i], I.QV[j0 + jj + (int64_t)c * I.m], s);
          return s;
        }, [&](int o, double v) { zc[(o / ni) * 32 + o % ni] += v; });
      }
      __syncthreads();
      outputs(rr, ni, [&](int o, int l, int L) {
        const int a = o % r, c = o / r;
        double s = 0.0;
        for (int i = l; i < ni; i += L) s = fma(I.QU[i0 + i + (int64_t)a * I.n], zc[c * 32 + i], s);
        return s;
      }, [&](int o, double v) { part[o] += v; });
      __syncthreads();
    }
    // the sums of the own columns are added by their CTA
    tm.sync();
    for (int e = tid; e < r * nc; e += WT) {
      double s = yst[e];
      for (int k = 0; k < C; ++k) s += tm.at(part, k)[c0 * r + e];
      I.S[e % r + (int64_t)(c0 + e / r) * I.rcap] = s;
      if (!isfinite(s)) atomicOr(g.status, ST_NONFINITE);
    }
    // new bases and the snapshot for the next step
    take_bases();
    tm.sync();  // every CTA is past its reads of the previous snapshot and of the partials
    for (int64_t e = tm.q * WT + tid; e < (int64_t)I.n * I.m; e += (int64_t)C * WT) I.Yp[e] = I.Yn[e];
    return;
  }
  for (int e = tid; e < rr; e += WT) {
    GU[e] = nu[e % r + (int64_t)(e / r) * W];
    PU[e] = nu[(int64_t)r * W + e % r + (int64_t)(e / r) * W];
  }
  for (int e = tid; e < r * nc; e += WT) {
    gv[e] = nv[e % r + (int64_t)(c0 + e / r) * W];
    pv[e] = nv[(int64_t)r * W + c0 + e / r + (int64_t)(e % r) * W];
    const double y = yst[e];
    for (int k = 0; k < C; ++k) tm.at(Z0, k)[c0 * r + e] = y;
  }
  tm.cl.sync();
  const Scheme& sc = g.sS;
  const double h = g.dt / sc.nsub;
  double* zin = Z0;
  double* zout = Z1;
  for (int sub = 0; sub < sc.nsub; ++sub)
    for (int s = 0; s < sc.nstages; ++s) {
      // t1 = Z G_V, t2 = Z P_V^T (own columns)
      outputs(2 * r * nc, r, [&](int o, int l, int L) {
        const int e = (o < r * nc) ? o : o - r * nc, i = e % r, c = e / r;
        const double* b = (o < r * nc) ? gv : pv;
        double v = 0.0;
        for (int k = l; k < r; k += L) v = fma(zin[i + k * r], b[k + c * r], v);
        return v;
      }, [&](int o, double v) { ((o < r * nc) ? t1 : t2 - r * nc)[o] = v; });
      __syncthreads();
      const bool last = s + 1 == sc.nstages;
      const double bs = sc.b[s], ha = last ? 0.0 : h * sc.a[s + 1];
      outputs(r * nc, 2 * r, [&](int o, int l, int L) {
        const int i = o % r, c = o / r;
        double v = 0.0;
        for (int k = l; k < r; k += L) v = fma(PU[i + k * r], t1[k + c * r], fma(GU[i + k * r], t2[k + c * r], v));
        return v;
      }, [&](int o, double v) {
        const double a = (s == 0) ? bs * v : fma(bs, v, ast[o]);
        double z;
        if (last) {
          z = fma(h, a, yst[o]);
          yst[o] = z;
        } else {
          ast[o] = a;
          z = fma(ha, v, yst[o]);
        }
        for (int k = 0; k < C; ++k) tm.at(zout, k)[c0 * r + o] = z;
      });
      tm.cl.sync();
      double* t = zin;
      zin = zout;
      zout = t;
    }
  for (int e = tid; e < r * nc; e += WT) {
    const double s = yst[e];
    I.S[e % r + (int64_t)(c0 + e / r) * I.rcap] = s;
    if (!isfinite(s)) atomicOr(g.status, ST_NONFINITE);
  }
  if (fresh) take_bases();
  // the new bases' projections become the current ones
  for (int e = tm.q * WT + tid; e < 4 * rr; e += C * WT) {
    const int x = e % rr, which = e / rr;  // G_U, P_U, G_V, P_V
    const int64_t o = (which & 1) * (int64_t)r * W + x % r + (int64_t)(x / r) * W;
    I.blk(which < 2 ? WB_GU : WB_GV)[o] = (which < 2 ? nu : nv)[o];
  }
  if (tm.q == 0 && tid == 0) g.proj_valid[I.inst] = 1;
}

}  // namespace

int wide_cluster(int count, int64_t tall, int sms) {
  int C = wide::WC_MAX;
  while (C > 1 && (2 * (int64_t)C * count > sms || tall < 4 * C)) C /= 2;
  return C;
}

// Sides: the smallest cluster whose panels leave room for two CTAs on an SM;
// where the batch leaves SMs idle, larger clusters, down to four rows per CTA
// (below that the barriers outweigh the split).  Cores: a cluster only where
// SMs are idle.
// There is no rule by cost: FP64 issue bounds either form and the panels' way
// through L2 hides no other work, so sides win wherever they fit.  Per step,
// step kernel against sides: n, m 256 to 1024 with r 23 to 32, 350: 20.5, 12.6 ms;
// 700: 30.0, 25.7; 1400: 53.7, 49.9; n, m to 512 with r 4 to 24, 1000: 8.5, 4.5; n, m
// 40 to 100 with r 2 to 6, 4000: 3.6, 1.2; data instances of 100 to 512 with r 4 to
// 32, 64: 11.4, 3.5; 256: 13.7, 9.9; 1024: 24.3, 21.2; of 40 to 80 with r 2 to 8,
// 4000: 5.3, 1.8; of 1000 to 2000 with r 8 to 32, 20: 144, 25.
bool wide_plan(WidePlan* w, int count, const int64_t* n, const int64_t* m, const int64_t* r, bool data, int sms,
               std::vector<int32_t>* items) {
  std::vector<SideItem> v;
  w->core_smem = 0;
  w->C = wide::WC_MAX;
  while (w->C > 1 && (int64_t)w->C * count > sms) w->C /= 2;
  int64_t ctas = 0, tall = 0, rmax = 0;
  for (int i = 0; i < count; ++i) {
    const int ri = (int)r[i];
    if (ri > wide::WR_MAX) return false;
    rmax = std::max(rmax, r[i]);
    for (int s = 0; s < 2; ++s) {
      const int N = (int)(s ? m[i] : n[i]);
      auto bytes = [&](int C) { return sizeof(double) * side_doubles(N, ri, C); };
      int C = wide_cluster(count, N, sms);
      while (C < wide::WC_MAX && bytes(C) > kHalfSmem) C *= 2;
      if (bytes(C) > kWideSmemMax) return false;
      v.push_back({(int32_t)(2 * i + s), C, bytes(C), (double)N * ri * (ri + 8.0) / C});
      ctas += C;
      tall = std::max<int64_t>(tall, N);
    }
  }
  // (a core's columns are what its CTAs share, in a data step also its rows)
  while (w->C > 1 && (tall < 4 * w->C || (!data && rmax <= w->C / 2))) w->C /= 2;
  for (int i = 0; i < count; ++i)
    w->core_smem = std::max(w->core_smem, sizeof(double) * core_doubles((int)r[i], w->C));
  if (w->core_smem > kWideSmemMax) return false;
  // a few CTAs take an SM each, with all its FP64 units
  if (ctas <= sms)
    for (SideItem& x : v) x.smem = std::max(x.smem, (size_t)120 * 1024);
  return group_sides(v, &w->sides, items);
}

cudaError_t launch_wide_side(const StepArgs<double>& g, const WidePlan& p, int k, const int32_t* items,
                             cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  const SidesPlan::Class& c = p.sides.cls[k];
  cudaError_t e = wide::cluster_attributes(wide_sides, done);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  wide::cluster_config(cfg, attr, c.C * c.count, c.C, c.smem, st);
  return cudaLaunchKernelEx(&cfg, wide_sides, g, items + c.first, (int)c.C);
}

cudaError_t launch_wide_core(const StepArgs<double>& g, int count, const WidePlan& p, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  cudaError_t e = wide::cluster_attributes(wide_core, done);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  wide::cluster_config(cfg, attr, p.C * count, p.C, p.core_smem, st);
  return cudaLaunchKernelEx(&cfg, wide_core, g, p.C);
}

}  // namespace lri
