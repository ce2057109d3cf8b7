// burgers_panel.cu - K and L flows of the large Burgers engine at ranks 33 to
// 64 (FP32 panels) on the 5th-generation tensor cores.
//
// The quadratic term of a row z is sum_{a <= b} T'[p(a,b), c] z_a z_b.  Formed
// as (KR(z, z)) T' it needs every pair's product as an operand; here it is
//   D[c, b] = sum_{a <= b} T'[p(a,b), c] z_a,   then   sum_b D[c, b] z_b,
// so the operand is the panel itself (64 columns) and the second sum is one
// multiply-add per accumulator read.  A tile of D is 16 columns c times a
// block of 8 b (N = 128) for 128 rows; block j needs a < 8 (j + 1) only, so
// the products are 11 % above the packed pairs' count, not twice it.
//   warps 0-7  per stage: split the stage input (TF32 hi + lo) into tensor
//              memory as the A operand, the linear term on the CUDA cores
//              (FP32), drain the tiles (3 accumulators in turn), RK update;
//              y and the accumulated slope stay in registers;
//   warp 8     streams T' (both TF32 parts, laid out once per step in the
//              order of use) through a ring of 32 KB chunks;
//   warp 9     issues the MMAs: per tile lo parts first, then hi * hi, so
//              that at most 8 additions truncate at the accumulator's size.
// The L flow's rows are independent: one launch runs every stage.  The K
// flow's tiles carry a halo of one row per stage and a launch runs the
// substeps that the halo allows.  With few tiles a cluster of Q = 2 or 4
// CTAs shares a tile, each with a part of the columns c, and sends its columns
// of the next stage input to the others through distributed shared memory.
// Rank 64, 64 RK4 substeps: the L flow of 16384 rows 5.2 ms (20 us per stage)
// and the K flow of 4096 rows 2.4 ms, one after the other (each fills the
// GPU); with one launch per stage and the pairs' products as the operand the
// two took 115 us per stage, 29.5 ms.  What bounds the L flow: the MMAs (64
// cycles each, 432 per stage: 14 us); the rest is the turn from one stage to
// the next and drains that share shared memory with the MMAs' operand reads.
// Every wait is bounded (ST_TIMEOUT): a warp that gives up keeps the
// structure of the loops (all further waits return at once), copies and
// MMAs in flight are waited for, tensor memory is freed.
#include "burgers_panel.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "tc_common.cuh"

namespace lri {
namespace {

namespace cg = cooperative_groups;

constexpr int BP_ROWS = 128;
constexpr int BP_EPI = 256, BP_NT = 320;
constexpr int BP_RING = 4, BP_ACC = 3;
constexpr uint32_t BP_TILE = 128 * 32 * 4;  // 128 rows (16 c x 8 b) x 32 a: one swizzled operand chunk, 16 KB
constexpr int BP_ZS = PANEL_RMAX * BP_ROWS; // one stage input, [column][row]
constexpr int BP_CHUNKS = 9;                // chunks per 16 columns at rank 64: 36 slices of 8, 4 per chunk
constexpr size_t BP_BYTES = (size_t)4 * BP_CHUNKS * 2 * BP_TILE;
constexpr uint32_t BP_A = BP_ACC * 128;     // tensor-memory column of the A operand: hi, then lo
constexpr long long BP_WAIT = 4000000000LL;

constexpr int bp_smem(int Q) {  // ring, stage inputs, linear operator, its partial sums (Q - 1 of the own columns), control
  return BP_RING * 2 * (int)BP_TILE + 2 * BP_ZS * 4 + (PANEL_RMAX + (Q - 1) * BP_ROWS) * (PANEL_RMAX / Q) * 4 + 1024 +
         1024;
}
static_assert(bp_smem(1) <= 227 * 1024 && bp_smem(2) <= 227 * 1024 && bp_smem(4) <= 227 * 1024, "shared memory of the panel flows");

// an RK scheme in FP32 (a conversion from FP64 in the kernel holds the
// scheduler's FP64 unit for 64 cycles)
struct RkF {
  int nstages, nsub;
  float a[4], b[4];
};

struct BpArgs {
  int N, R, nsub, H;
  float ih2, ihx, alpha, beta, h;
  const int32_t* rank;
  const float* yin;
  float* yout;
  const float* nu;
  const double* lin;
  const unsigned char* b;
  uint32_t* status;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ uint32_t mapa(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// bounded wait with cluster scope: the peers' stores before their arrivals are visible
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                  uint32_t* status, long long limit) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > limit) {
      *abort_flag = 1;
      atomicOr(status, ST_TIMEOUT);
      return false;
    }
  }
}

// acc += x * w on two packed FP32 values
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t x, uint64_t w) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(w));
}
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float sum2(uint64_t v) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
  return x + y;
}

// The products of one group of 16 columns: blocks j = NJ - 1 .. 0 of 8 b's,
// j + 1 slices of 8 a's each, unrolled over the whole group.
struct BpIssue {
  uint32_t ring, tmem, idesc, full0, empty0, acc_full0, acc_empty0;
  int t, ck;  // tiles and chunks so far
};
template <int NJ, class W>
__device__ __forceinline__ bool issue_group(BpIssue& s, const W& wait) {
  constexpr int NS = NJ * (NJ + 1) / 2, NCH = (NS + 3) / 4;
  constexpr uint64_t LO = BP_TILE >> 4;  // descriptor distance of the lo part
  uint64_t cd[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) cd[c] = sw128_desc(s.ring + (uint32_t)((s.ck + c) % BP_RING) * 2 * BP_TILE);
  const uint32_t ah = s.tmem + BP_A, al = ah + 64u;
#pragma unroll
  for (int j = NJ - 1; j >= 0; --j) {
    const int s0 = NS - (j + 1) * (j + 2) / 2, s1 = s0 + j + 1, b = s.t % BP_ACC;
    if (s.t >= BP_ACC && !wait(s.acc_empty0 + 8u * b, (uint32_t)(s.t / BP_ACC - 1) & 1u)) return false;
#pragma unroll
    for (int c = (s0 + 3) / 4; c <= (s1 - 1) / 4; ++c)  // chunks that start in this block
      if (!wait(s.full0 + 8u * ((s.ck + c) % BP_RING), (uint32_t)((s.ck + c) / BP_RING) & 1u)) return false;
    tc_fence_after();
    const uint32_t d = s.tmem + 128u * b;
#pragma unroll
    for (int kk = 0; kk <= j; ++kk) {
      const uint64_t bd = cd[(s0 + kk) / 4 % 4] + 2 * ((s0 + kk) % 4);
      umma_tf32_ts(d, ah + 8u * kk, bd + LO, s.idesc, kk > 0 ? 1u : 0u);
      umma_tf32_ts(d, al + 8u * kk, bd, s.idesc, 1u);
    }
#pragma unroll
    for (int kk = 0; kk <= j; ++kk)
      umma_tf32_ts(d, ah + 8u * kk, cd[(s0 + kk) / 4 % 4] + 2 * ((s0 + kk) % 4), s.idesc, 1u);
    umma_commit(s.acc_full0 + 8u * b);
#pragma unroll
    for (int c = s0 / 4; c < (j == 0 ? NCH : s1 / 4); ++c)  // chunks that end in this block
      umma_commit(s.empty0 + 8u * ((s.ck + c) % BP_RING));
    ++s.t;
  }
  s.ck += NCH;
  return true;
}
static_assert(BP_RING == 4, "issue_group's chunk descriptors");

// MODE: the L flow, the K flow with alpha = 0, the general K flow
enum { BP_L = 0, BP_KB = 1, BP_KA = 2 };

template <int MODE, int Q>
__global__ void __launch_bounds__(BP_NT, 1) panel_flow_kernel(const BpArgs a, const __grid_constant__ RkF sc) {
  extern __shared__ unsigned char smem_raw[];
  constexpr bool KF = MODE != BP_L, KA = MODE == BP_KA;
  constexpr int NCG = 4 / Q, CW = PANEL_RMAX / Q, C8 = 8 * NCG;
  // the same offset in every CTA of the cluster
  unsigned char* base = align_1024(smem_raw);
  unsigned char* ring = base;
  float* zs = reinterpret_cast<float*>(base + BP_RING * 2 * BP_TILE);  // two stage inputs in turn
  float* as = zs + 2 * BP_ZS;                                          // linear operator, [k][own column]
  float* red = as + PANEL_RMAX * CW;                                   // [Q - 1][own column][row]
  unsigned char* ctrl = reinterpret_cast<unsigned char*>(red + (Q - 1) * CW * BP_ROWS);
  const uint32_t bar0 = smem_u32(ctrl);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (BP_RING + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * BP_RING + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * BP_RING + BP_ACC + b); };
  const uint32_t aready = bar0 + 8u * (2 * BP_RING + 2 * BP_ACC), zfull = aready + 8u, done = aready + 16u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 256);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 260);
  auto wait = [&](uint32_t bar, uint32_t par, long long limit = BP_WAIT) {
    return mbar_wait_st(bar, par, abort_flag, a.status, ST_TIMEOUT, limit);
  };

  const int r = min(min(a.R, PANEL_RMAX), (int)*a.rank), nj = (r + 7) / 8, ncg = (r + 15) / 16;
  const int q = (int)blockIdx.x % Q, i0 = (int)blockIdx.x / Q * (BP_ROWS - 2 * a.H);
  const int cg0 = q * NCG, own = max(0, min(NCG, ncg - cg0));  // this CTA's groups of 16 columns
  const int nch = (nj * (nj + 1) / 2 + 3) / 4;  // operand chunks per group
  const bool quad_b = MODE == BP_KB || a.beta != 0.0f;
  constexpr int npass = KA ? 2 : 1;  // second pass: A = Dx z
  const int stages = a.nsub * sc.nstages;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  auto grow = [&](int ii) {  // panel row of the tile's row ii
    if (!KF) return i0 + ii;
    const int g = (i0 - a.H + ii) % a.N;
    return g < 0 ? g + a.N : g;
  };
#pragma unroll 9
  for (int e = tid; e < BP_ZS; e += BP_NT) {
    const int ii = e % BP_ROWS, k = e / BP_ROWS, g = grow(ii);
    zs[e] = (k < r && g < a.N) ? a.yin[g + (int64_t)k * a.N] : 0.0f;
    zs[BP_ZS + e] = 0.0f;
  }
  for (int e = tid; e < PANEL_RMAX * CW; e += BP_NT) {
    const int k = e % PANEL_RMAX, cl = e / PANEL_RMAX, c = 16 * cg0 + cl;
    as[k * CW + cl] = (k < r && c < r) ? (float)a.lin[k + (int64_t)c * a.R] : 0.0f;
  }
  if (tid == 0) {
    for (int s = 0; s < BP_RING; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < BP_ACC; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), BP_EPI);
    }
    mbar_init(aready, BP_EPI);
    mbar_init(zfull, Q * BP_EPI / 32);
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  if (Q > 1) cg::this_cluster().sync();  // the peers' barriers and buffers stand before anything is sent
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 8) {
    // ---------------- operand stream ----------------
    if (elect_one()) {
      int last_par[BP_RING];
      for (int s = 0; s < BP_RING; ++s) last_par[s] = -1;
      const int per = own * nch, total = stages * npass * per;
      const unsigned char* src = a.b + (size_t)cg0 * nch * 2 * BP_TILE;
      bool ok = true;
      for (int it = 0, at = 0; it < total && ok; ++it) {
        const int s = it % BP_RING;
        const uint32_t par = (uint32_t)(it / BP_RING) & 1u;
        if (!(ok = wait(empty(s), par ^ 1u))) break;
        mbar_expect_tx(full(s), 2 * BP_TILE);
        bulk_load(smem_u32(ring) + (uint32_t)s * 2 * BP_TILE, src + (size_t)at * 2 * BP_TILE, 2 * BP_TILE, full(s));
        last_par[s] = (int)par;
        if (++at == per) at = 0;
      }
      if (!ok || *abort_flag) {
        for (int s = 0; s < BP_RING; ++s)
          if (last_par[s] >= 0) wait(full(s), (uint32_t)last_par[s], BP_WAIT / 4);
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---------------- MMA issuer ----------------
    if (own > 0 && elect_one()) {
      BpIssue is{smem_u32(ring), tmem, idesc_tf32(BP_ROWS, 128), full(0), empty(0), acc_full(0), acc_empty(0), 0, 0};
      bool ok = true;
      for (int it = 0; it < stages * npass && ok; ++it) {
        if (!(ok = wait(aready, (uint32_t)it & 1u))) break;
        tc_fence_after();
        for (int i = 0; i < own && ok; ++i) switch (nj) {
            case 8: ok = issue_group<8>(is, wait); break;
            case 7: ok = issue_group<7>(is, wait); break;
            case 6: ok = issue_group<6>(is, wait); break;
            case 5: ok = issue_group<5>(is, wait); break;
            case 4: ok = issue_group<4>(is, wait); break;
            case 3: ok = issue_group<3>(is, wait); break;
            case 2: ok = issue_group<2>(is, wait); break;
            default: ok = issue_group<1>(is, wait); break;
          }
      }
      umma_commit(done);
      if (!ok || *abort_flag) wait(done, 0, BP_WAIT / 4);
    }
    __syncwarp();
  } else {
    // ---------------- operand A, linear term, drains, RK update ----------------
    const int g = tid >> 7, row = tid & 127;  // tensor-memory lane = row; g: half of a tile's 16 columns
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const int rm = max(row - 1, 0), rp = min(row + 1, BP_ROWS - 1);
    const float nu = (!KF && i0 + row < a.N) ? a.nu[i0 + row] : 0.0f;
    // a column of this thread: entry e is column col(e)
    auto col = [&](int e) { return 16 * (cg0 + e / 8) + 8 * g + e % 8; };
    float y[C8], sl[C8], v[KF ? C8 : 1];
#pragma unroll
    for (int e = 0; e < C8; ++e) {
      y[e] = zs[col(e) * BP_ROWS + row];
      sl[e] = 0.0f;
    }
    int t = 0, k = 0;
    const uint32_t zbase = smem_u32(zs);
    for (int stg = 0; stg < stages; ++stg) {
      const float* cur = zs + (stg & 1) * BP_ZS;
      float* nxt = zs + ((stg + 1) & 1) * BP_ZS;
      const uint32_t nxta = zbase + (uint32_t)((stg + 1) & 1) * BP_ZS * 4;
      const bool more = stg + 1 < stages, last = k + 1 == sc.nstages;
      const float rb = sc.b[k], rha = last ? 0.0f : a.h * sc.a[k + 1];
      if (stg > 0) mbar_wait_cluster(zfull, (uint32_t)(stg - 1) & 1u, abort_flag, a.status, BP_WAIT);
      __syncwarp();
      // RK update of entry e with derivative d; the next stage's input goes to
      // every CTA of the cluster (columns beyond r: zero)
      auto update = [&](int e, float d) {
        sl[e] = (k == 0) ? rb * d : fmaf(rb, d, sl[e]);
        float z;
        if (last) z = y[e] = fmaf(a.h, sl[e], y[e]);
        else z = fmaf(rha, d, y[e]);
        if (more) {
          const int c = col(e), o = c * BP_ROWS + row;
          z = c < r ? z : 0.0f;
          nxt[o] = z;
#pragma unroll
          for (int w = 1; w < Q; ++w)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa(nxta + 4u * (uint32_t)o, (q + w) % Q)), "f"(z)
                         : "memory");
        }
      };
      // Linear term of the own columns: 4 rows x 8 columns per thread (bound by
      // shared-memory returns, of which a broadcast weight costs as much as any
      // other load), 8 warps = 8 / Q column groups x Q parts of the sum over k,
      // in four parts between the first tiles.
      const int lc = 8 * (warp % (8 / Q)), lk = warp / (8 / Q);
      float lin[8][4];
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int u = 0; u < 4; ++u) lin[e][u] = 0.0f;
      auto linear = [&](int k0, int k1) {
#pragma unroll 4
        for (int kk = k0; kk < k1; ++kk) {
          const float4 z4 = *reinterpret_cast<const float4*>(cur + kk * BP_ROWS + 4 * lane);
          const float4 w0 = *reinterpret_cast<const float4*>(as + kk * CW + lc);
          const float4 w1 = *reinterpret_cast<const float4*>(as + kk * CW + lc + 4);
          float x[4] = {z4.x, z4.y, z4.z, z4.w};
          if (KF) {
            const float zl = __shfl_up_sync(0xffffffffu, z4.w, 1), zr = __shfl_down_sync(0xffffffffu, z4.x, 1);
            x[0] = a.ih2 * ((zl + z4.y) - 2.0f * z4.x);
            x[1] = a.ih2 * ((z4.x + z4.z) - 2.0f * z4.y);
            x[2] = a.ih2 * ((z4.y + z4.w) - 2.0f * z4.z);
            x[3] = a.ih2 * ((z4.z + zr) - 2.0f * z4.w);
          }
          const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
          for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) lin[e][u] = fmaf(x[u], w[e], lin[e][u]);
        }
      };
      // the factors z_b of a block (KA: also the ones of the other quadratic sum)
      auto factors = [&](int j, int p, float (&zb)[8], float (&xb)[8]) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float* z = cur + (8 * j + u) * BP_ROWS;
          zb[u] = z[row];
          if (KA) xb[u] = p == 0 ? a.ihx * (z[rp] - z[rm]) : zb[u];
        }
      };
#pragma unroll 1
      for (int p = 0; p < npass; ++p) {
        if (own > 0) {
#pragma unroll
          for (int cc = 0; cc < 32; cc += 16) {
            float hi[16], lo[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float* z = cur + (32 * g + cc + e) * BP_ROWS;
              split((KA && p == 1) ? a.ihx * (z[rp] - z[rm]) : z[row], hi[e], lo[e]);
            }
            tmem_st16(tmem + lanes + BP_A + (uint32_t)(32 * g + cc), hi);
            tmem_st16(tmem + lanes + BP_A + 64u + (uint32_t)(32 * g + cc), lo);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          mbar_arrive(aready);
        }
#pragma unroll
        for (int i = 0; i < NCG; ++i) {
          if (i < own) {
            const bool lb = p == 0 && i == 0;
            const int parts = min(4, nj);
            uint64_t gq[8];
            float gx[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              gq[u] = 0;
              gx[u] = 0.0f;
            }
            float zb[8], xb[8];
            factors(nj - 1, p, zb, xb);
#pragma unroll 1
            for (int j = nj - 1; j >= 0; --j, ++t) {
              const int b = t % BP_ACC, part = nj - 1 - j;
              if (lb && part < parts) {
                const int k0 = r * lk / Q, k1 = r * (lk + 1) / Q;
                linear(k0 + (k1 - k0) * part / parts, k0 + (k1 - k0) * (part + 1) / parts);
                if (part + 1 == parts) {  // to its place in the next input's buffer, the other parts beside it
                  float* dst = lk == 0 ? nxt + (16 * cg0 + lc) * BP_ROWS : red + ((lk - 1) * CW + lc) * BP_ROWS;
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                    *reinterpret_cast<float4*>(dst + e * BP_ROWS + 4 * lane) =
                        make_float4(lin[e][0], lin[e][1], lin[e][2], lin[e][3]);
                }
              }
              // the next block's factors: a shared-memory read takes some 250
              // cycles beside the MMAs' operand reads
              float zn[8], xn[8];
              if (j > 0) factors(j - 1, p, zn, xn);
              const bool ok = __all_sync(0xffffffffu, wait(acc_full(b), (uint32_t)(t / BP_ACC) & 1u));
              tc_fence_after();
              if (ok) {
                float d[64];
                tmem_ld64(tmem + lanes + (uint32_t)(128 * b + 64 * g), d);
#pragma unroll
                for (int cc = 0; cc < 8; ++cc) {
                  if (!KF || p == 0)
#pragma unroll
                    for (int u = 0; u < 4; ++u) fma2(gq[cc], pack2(d[8 * cc + 2 * u], d[8 * cc + 2 * u + 1]), pack2(zb[2 * u], zb[2 * u + 1]));
                  if (KA) {
                    uint64_t x = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                      fma2(x, pack2(d[8 * cc + 2 * u], d[8 * cc + 2 * u + 1]), pack2(xb[2 * u], xb[2 * u + 1]));
                    gx[cc] += sum2(x);
                  }
                }
              }
              tc_fence_before();
              mbar_arrive(acc_empty(b));
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                zb[u] = zn[u];
                if (KA) xb[u] = xn[u];
              }
            }
            if (lb) asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int e = 8 * i + u;
              float* place = nxt + col(e) * BP_ROWS + row;
              float lv = *place;
#pragma unroll
              for (int w = 0; w < Q - 1; ++w) lv += red[(w * CW + col(e) - 16 * cg0) * BP_ROWS + row];
              if constexpr (!KF) {
                update(e, fmaf(nu, lv, sum2(gq[u])));
              } else {
                if (p == 0) {
                  v[e] = lv;
                  if (quad_b) *place = sum2(gq[u]);
                }
                if (KA) v[e] = fmaf(0.5f * a.alpha, gx[u], v[e]);
              }
            }
          }
        }
      }
      if constexpr (KF) {
        if (quad_b) {  // beta Dx of the product: the neighbours' values pass through the next input's buffer
          asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
          for (int e = 0; e < C8; ++e)
            if (e / 8 < own) {
              const float* z = nxt + col(e) * BP_ROWS;
              v[e] = fmaf(a.beta * a.ihx, z[rp] - z[rm], v[e]);
            }
          asm volatile("bar.sync 1, 256;" ::: "memory");
        }
#pragma unroll
        for (int e = 0; e < C8; ++e)
          if (e / 8 < own) update(e, v[e]);
      }
      if (++k == sc.nstages) k = 0;
      __syncwarp();
      if (more && lane == 0)
#pragma unroll
        for (int w = 0; w < Q; ++w)
          asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(zfull, w))
                       : "memory");
    }
    const int gr = grow(row);
    const bool out = KF ? (row >= a.H && row < BP_ROWS - a.H && i0 + row - a.H < a.N) : gr < a.N;
    if (out)
#pragma unroll
      for (int e = 0; e < C8; ++e) {
        if (e / 8 < own && col(e) < r) a.yout[gr + (int64_t)col(e) * a.N] = y[e];
      }
    if (KF && out && q == 0)  // inactive columns: unchanged
      for (int c = r + g; c < a.R; c += 2) a.yout[gr + (int64_t)c * a.N] = a.yin[gr + (int64_t)c * a.N];
  }
  tc_fence_before();
  if (Q > 1) cg::this_cluster().sync();  // no CTA leaves while a peer may write to it
  else __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// operand chunks in the order of use: [16 columns c][chunk][hi | lo][row = 8
// (c % 16) + b % 8][32 a, 128-byte swizzle]; slice s of 8 a's belongs to the
// block j of b's (descending) that it falls in
__global__ void __launch_bounds__(256) panel_tensor_kernel(int R, const int32_t* __restrict__ rank,
                                                           const float* __restrict__ Tp, int PP,
                                                           unsigned char* __restrict__ out) {
  const int r = min(min(R, PANEL_RMAX), (int)*rank), nj = (r + 7) / 8, ncg = (r + 15) / 16;
  const int ns = nj * (nj + 1) / 2, nch = (ns + 3) / 4;
  const int total = ncg * nch * 4096;
  for (int e = blockIdx.x * 256 + threadIdx.x; e < total; e += gridDim.x * 256) {
    const int f = e & 31, row = (e >> 5) & 127, ch = (e >> 12) % nch, grp = (e >> 12) / nch;
    int s = 4 * ch + f / 8, j = nj - 1;
    float v = 0.0f;
    if (s < ns) {
      while (s > j) s -= j-- + 1;
      const int pa = 8 * s + (f & 7), pb = 8 * j + (row & 7), c = 16 * grp + row / 8;
      if (pa <= pb && pb < r && c < r) v = Tp[pa * r - pa * (pa - 1) / 2 + (pb - pa) + (int64_t)c * PP];
    }
    float h, l;
    split(v, h, l);
    unsigned char* o = out + (size_t)(grp * nch + ch) * 2 * BP_TILE + row * 128 + (((f >> 2) ^ (row & 7)) << 4) +
                       (f & 3) * 4;
    *reinterpret_cast<float*>(o) = h;
    *reinterpret_cast<float*>(o + BP_TILE) = l;
  }
}

template <int MODE, int Q>
cudaLaunchConfig_t panel_config(int tiles, cudaLaunchAttribute* attr, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * Q));
  cfg.blockDim = dim3(BP_NT);
  cfg.dynamicSmemBytes = bp_smem(Q);
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = Q;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <int MODE, int Q>
cudaError_t panel_limit() {
  static std::atomic<uint64_t> done{0};
  return set_smem_limit(panel_flow_kernel<MODE, Q>, bp_smem(Q), done);
}

template <int MODE, int Q>
cudaError_t launch_panel(const BpArgs& a, const Scheme& sc, int tiles, cudaStream_t st) {
  const cudaError_t e = panel_limit<MODE, Q>();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr{};
  const cudaLaunchConfig_t cfg = panel_config<MODE, Q>(tiles, &attr, st);
  RkF rk{sc.nstages, sc.nsub, {}, {}};
  for (int k = 0; k < sc.nstages; ++k) {
    rk.a[k] = (float)sc.a[k];
    rk.b[k] = (float)sc.b[k];
  }
  return cudaLaunchKernelEx(&cfg, panel_flow_kernel<MODE, Q>, a, rk);
}

template <int MODE>
cudaError_t launch_panel(int Q, const BpArgs& a, const Scheme& sc, int tiles, cudaStream_t st) {
  return Q == 4 ? launch_panel<MODE, 4>(a, sc, tiles, st)
                : (Q == 2 ? launch_panel<MODE, 2>(a, sc, tiles, st) : launch_panel<MODE, 1>(a, sc, tiles, st));
}

// Tiles that run at once with Q CTAs each (a cluster's CTAs share one part of
// the GPU, so that fewer than sms / Q may fit).
template <int MODE, int Q>
cudaError_t panel_slots(int* n) {
  cudaError_t e = panel_limit<MODE, Q>();
  cudaLaunchAttribute attr{};
  const cudaLaunchConfig_t cfg = panel_config<MODE, Q>(1, &attr, nullptr);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(n, panel_flow_kernel<MODE, Q>, &cfg);
  if (e == cudaSuccess && *n < 1) e = cudaErrorInvalidConfiguration;
  return e;
}

// Times of the split rule (us): a stage's products for 128 rows and 64
// columns, what a stage has besides, and a launch with its tile loads.
constexpr double BP_MMA = 15.0, BP_STAGE = 5.0, BP_LAUNCH = 8.0;

struct PanelSlots {
  int n[3];  // for Q = 1, 2, 4
  double stage(int tiles, int q) const {  // us of one stage, Q = 1 << q
    return ((tiles + n[q] - 1) / n[q]) * (BP_STAGE + BP_MMA / (1 << q));
  }
};
template <int MODE>
cudaError_t panel_slots(PanelSlots* s) {
  cudaError_t e = panel_slots<MODE, 1>(&s->n[0]);
  if (e == cudaSuccess) e = panel_slots<MODE, 2>(&s->n[1]);
  if (e == cudaSuccess) e = panel_slots<MODE, 4>(&s->n[2]);
  return e;
}

}  // namespace

cudaError_t panel_flow_init(PanelFlow* p) {
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaMalloc((void**)&p->b[k], BP_BYTES);
  return e;
}

void panel_flow_free(PanelFlow* p) {
  for (unsigned char*& b : p->b) {
    cudaFree(b);
    b = nullptr;
  }
}

cudaError_t panel_flow_tensor(const PanelFlow& p, int k, int R, const int32_t* rank, const float* Tp, int PP,
                              cudaStream_t st) {
  panel_tensor_kernel<<<304, 256, 0, st>>>(R, rank, Tp, PP, p.b[k]);
  return cudaGetLastError();
}

cudaError_t panel_k_flow(const PanelFlow& p, int N, int R, const int32_t* rank, float* y, float* tmp,
                         const double* Nnu, double ih2, double ihx, double alpha, double beta, const Scheme& sc,
                         double h, uint32_t* status, cudaStream_t st) {
  // Columns split over Q CTAs and u substeps per launch: more substeps save
  // launches and recompute a wider halo, more CTAs per tile shorten a stage
  // while the tiles run at once.
  PanelSlots slots;
  const cudaError_t es = panel_slots<BP_KB>(&slots);
  if (es != cudaSuccess) return es;
  int Q = 1, u = 1;
  double best = 0.0;
  for (int q = 2; q >= 0; --q)
    for (int uu = 1; uu <= sc.nsub && (uu == 1 || uu * sc.nstages <= BP_ROWS / 4); ++uu) {
      const int BM = BP_ROWS - 2 * uu * sc.nstages;
      const double t = ((sc.nsub + uu - 1) / uu) * (BP_LAUNCH + uu * sc.nstages * slots.stage((N + BM - 1) / BM, q));
      if (best == 0.0 || t < best) {
        best = t;
        Q = 1 << q;
        u = uu;
      }
    }
  const int launches = (sc.nsub + u - 1) / u;
  // the panels alternate; an odd count starts from a copy so that y ends in place
  float* src = y;
  float* dst = tmp;
  if (launches & 1) {
    const cudaError_t e = cudaMemcpyAsync(tmp, y, sizeof(float) * (size_t)N * R, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    std::swap(src, dst);
  }
  for (int left = sc.nsub; left > 0; left -= u) {
    const int n = std::min(u, left), H = n * sc.nstages, BM = BP_ROWS - 2 * H;
    const BpArgs a{N, R, n, H, (float)ih2, (float)ihx, (float)alpha, (float)beta, (float)h, rank, src, dst, nullptr,
                   Nnu, p.b[0], status};
    const cudaError_t e = alpha != 0.0 ? launch_panel<BP_KA>(Q, a, sc, (N + BM - 1) / BM, st)
                                       : launch_panel<BP_KB>(Q, a, sc, (N + BM - 1) / BM, st);
    if (e != cudaSuccess) return e;
    std::swap(src, dst);
  }
  return cudaSuccess;
}

cudaError_t panel_l_flow(const PanelFlow& p, int M, int R, const int32_t* rank, float* y, const float* nu,
                         const double* Axx, const Scheme& sc, double h, uint32_t* status, cudaStream_t st) {
  const int tiles = (M + BP_ROWS - 1) / BP_ROWS;
  PanelSlots slots;
  const cudaError_t es = panel_slots<BP_L>(&slots);
  if (es != cudaSuccess) return es;
  int q = 0;
  for (int k = 1; k < 3; ++k)
    if (slots.stage(tiles, k) < slots.stage(tiles, q)) q = k;
  const int Q = 1 << q;
  const BpArgs a{M, R, sc.nsub, 0, 0.0f, 0.0f, 0.0f, 0.0f, (float)h, rank, y, y, nu, Axx, p.b[1], status};
  return launch_panel<BP_L>(Q, a, sc, tiles, st);
}

}  // namespace lri
