// burgers_core.cu - S flow of the large Burgers engine at ranks 17 to 64 (FP32
// panels) on the 5th-generation tensor cores.
//
// With A = Uhat Z the quadratic term of the S flow,
//   Uhat^T [alpha KR(Dx A, A) + beta Dx KR(A, A)] T'  (column c)
//     = sum_{p <= q} W'[pq, :] (Z T_c Z^T)_pq,
// needs only the 3-tensors of the two bases (T_c: symmetric slices of Vhat's,
// W': Uhat's, both formed once per step), not the n x 2r panel: at rank 64
// and n = 4096, 0.8 GFMA per stage instead of 4.3 and no panel traffic.  A
// stage is three launches (all 3xTF32 with FP32 accumulators, as the other
// tcgen05 kernels):
//   s_core_g       one CTA per column c: M1 = Z T_c (128 x 128 x 128, both
//                  operands staged by TMA), M1 split to tensor memory as the A
//                  operand of G_c = M1 Z^T, G_c's packed pairs written as row c
//                  of G; the linear part A_xx Z N_nu[:, c] on the CUDA cores
//                  meanwhile;
//   s_core_wg      W' G as a GEMM with K = pairs: 128 CTAs take 2 or 3 chunks
//                  of 32 pairs each, clusters of 8 add their tiles through
//                  distributed shared memory;
//   s_core_update  sums the 16 cluster partials, applies the RK stage to the
//                  FP64 core and writes the split of the next stage input.
// An accumulator cuts what lies below its last bit at every addition, always
// towards zero, so that a chain of K / 8 additions shortens its sum: the lo
// parts go first (their cut is 2^-11 of the others'), and M1 has an
// accumulator per chunk, G one for every other chunk and W' G one per chunk,
// at most 4, 8 and 4 additions at the sum's size.  With one chain each (16, 16
// and 12) the quadratic increment was short by 1e-6 of itself at rank 64 and
// its error up to 16 % larger than that of FP64 sums (2.3e-6 against 2.0e-6
// of it); now 4e-7 and 2.1e-6, for 0.25 ms of a 21.3 ms step.
// At rank 64 the three took 12.0 + 14.1 + 4.6 us per stage (the panel form
// 205 us: Khatri-Rao product 131, Uhat^T P2 23, five small products and
// combines 51); with each kernel's prologue and constant operands loaded while
// the one before it drains (programmatic dependent launch) a stage took 25
// us, with the accumulators above 26.
// What bounds them now: operand staging (256 KB per CTA through L2) and the
// serial chain of two 128^3 products; the MMAs themselves take about 3.5 us.
// Every mbarrier wait is bounded (ST_TIMEOUT); a CTA that gives up waits for
// its copies and MMAs in flight, frees its tensor memory and returns.
#include "burgers_core.h"

#include <cooperative_groups.h>
#include <cuda.h>

#include <atomic>

#include "tc_common.cuh"
#include "tc_pass.h"

namespace lri {
namespace {

namespace cg = cooperative_groups;

constexpr int SC_W = 128;                       // padded core width (2 r_max <= 128)
constexpr int SC_NT = 256;
constexpr uint32_t SC_TILE = SC_W * 32 * 4;     // 128 rows x 32 FP32: one swizzled operand chunk, 16 KB
constexpr int SC_RING = 3;                      // T_c chunks in flight (hi and lo each)
constexpr int SC_CTRL = 1280;                   // barriers, flags, two vectors of 128
constexpr int SC_G_SMEM = 8 * SC_TILE + 2 * SC_RING * SC_TILE + SC_CTRL + 1024;
constexpr int SC_WG_CTAS = 128, SC_WG_CL = 8;   // W' G: CTAs and CTAs per cluster
constexpr int SC_WG_CHUNKS = 3;                 // most chunks per CTA: ceil(8256 / 32 / 128)
constexpr int SC_WG_SMEM = 4 * SC_WG_CHUNKS * SC_TILE + SC_CTRL + 1024;
constexpr long long SC_WAIT = 4000000000LL;
static_assert(SC_G_SMEM <= 227 * 1024 && SC_WG_SMEM <= 227 * 1024, "shared memory of the core flow kernels");

__device__ __forceinline__ int sc_act(int j, int r, int R) { return (j < r) ? j : R + (j - r); }
__device__ __forceinline__ int sc_start(int a, int ka) { return a * ka - a * (a - 1) / 2; }

// D (+)= A B^T, both operands K-major in shared memory
__device__ __forceinline__ void umma_tf32_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// v = the sum of the accumulators at taddr, taddr + 128, ... (count of them, the
// same in every thread of the warp)
__device__ __forceinline__ void sum_blocks(uint32_t taddr, int count, float (&v)[16]) {
  float w[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = 0.0f;
  int j = 0;
  if (count >= 2) {
    tmem_ld16x2(taddr, taddr + 128u, v, w);
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] += w[q];
    j = 2;
  }
  if (j + 2 <= count) {
    float u[16];
    tmem_ld16x2(taddr + 256u, taddr + 384u, u, w);
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] += u[q] + w[q];
  } else if (j < count) {
    tmem_ld16(taddr + 128u * j, w);
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] += w[q];
  }
}

struct SGArgs {
  int R, PPp;
  const int32_t* rank;
  const float* nc;
  const float* ax;
  float* lin;
  float* gh;
  float* gl;
  uint32_t* status;
};

__global__ void __launch_bounds__(SC_NT, 1)
    s_core_g(const __grid_constant__ CUtensorMap tmZh, const __grid_constant__ CUtensorMap tmZl,
             const __grid_constant__ CUtensorMap tmTh, const __grid_constant__ CUtensorMap tmTl, const SGArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const int ka = 2 * min(a.R, (int)*a.rank), c = blockIdx.x;
  if (c >= ka) return;  // the whole CTA, before any barrier or allocation
  pdl_launch();
  const int kch = (ka + 31) / 32;
  unsigned char* base = align_1024(smem_raw);
  unsigned char* zt = base;                     // 4 chunks x (hi, lo)
  unsigned char* tt = base + 8 * SC_TILE;       // SC_RING x (hi, lo)
  unsigned char* ctrl = tt + 2 * SC_RING * SC_TILE;
  const uint32_t bar0 = smem_u32(ctrl);
  auto full = [&](int j) { return bar0 + 8u * j; };  // j < 4
  const uint32_t empty0 = bar0 + 32u, done1 = bar0 + 40u, aready = bar0 + 48u, done2 = bar0 + 56u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 64);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 68);
  float* nv = reinterpret_cast<float*>(ctrl + 128);
  float* t1 = nv + SC_W;
  auto wait = [&](uint32_t bar, long long limit = SC_WAIT) {
    return mbar_wait_st(bar, 0, abort_flag, a.status, ST_TIMEOUT, limit);
  };
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int j = 0; j < 4; ++j) mbar_init(full(j), 1);
    mbar_init(empty0, 1);
    mbar_init(done1, 1);
    mbar_init(aready, SC_NT);
    mbar_init(done2, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < SC_W) nv[tid] = a.nc[c * SC_W + tid];
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // M1: an accumulator per chunk, [128 j, 128 (j + 1)); then A hi [256, 384), A lo
  // [384, 512) and two accumulators of G, [0, 128) and [128, 256)
  const uint32_t tmem = *tmem_slot;
  const uint32_t idesc = idesc_tf32(SC_W, 32 * kch);
  auto zaddr = [&](int j, int lo) { return smem_u32(zt) + (uint32_t)(2 * j + lo) * SC_TILE; };
  auto taddr = [&](int j, int lo) { return smem_u32(tt) + (uint32_t)(2 * (j % SC_RING) + lo) * SC_TILE; };
  auto load_t = [&](int j) {
    mbar_expect_tx(full(j), 4 * SC_TILE);
    tma_load_2d(taddr(j, 0), &tmTh, 32 * j, c * SC_W, full(j));
    tma_load_2d(taddr(j, 1), &tmTl, 32 * j, c * SC_W, full(j));
  };
  auto load_z = [&](int j) {
    tma_load_2d(zaddr(j, 0), &tmZh, 32 * j, 0, full(j));
    tma_load_2d(zaddr(j, 1), &tmZl, 32 * j, 0, full(j));
  };
  int loaded = 0;
  bool mma1 = false, mma2 = false;
  if (warp == 0 && elect_one()) {
    for (; loaded < kch && loaded < SC_RING; ++loaded) load_t(loaded);
    pdl_wait();  // Z is the previous kernel's; nothing is written before it has been read
    for (int j = 0; j < loaded; ++j) load_z(j);
    bool ok = true;
    for (int j = 0; j < kch && ok; ++j) {
      if (!(ok = wait(full(j)))) break;
      tc_fence_after();
      const uint32_t d = tmem + 128u * j;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint64_t zh = sw128_desc(zaddr(j, 0) + 32u * kk), zl = sw128_desc(zaddr(j, 1) + 32u * kk);
        const uint64_t th = sw128_desc(taddr(j, 0) + 32u * kk), tl = sw128_desc(taddr(j, 1) + 32u * kk);
        umma_tf32_ss(d, zh, tl, idesc, kk > 0 ? 1u : 0u);
        umma_tf32_ss(d, zl, th, idesc, 1u);
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_tf32_ss(d, sw128_desc(zaddr(j, 0) + 32u * kk), sw128_desc(taddr(j, 0) + 32u * kk), idesc, 1u);
      if (j == 0 && kch > SC_RING) umma_commit(empty0);
      if (j == 1 && kch > SC_RING) {  // the fourth chunk takes the first one's ring slot
        if (!(ok = wait(empty0))) break;
        load_t(loaded);
        load_z(loaded++);
      }
    }
    umma_commit(done1);
    mma1 = true;
  }
  __syncwarp();
  // linear part, first factor (warps 4-7): t1 = Z N_nu[:, c], one row per thread
  if (warp >= 4) {
    const int p = tid - 128;
    float t = 0.0f;
    bool ok = true;
    for (int j = 0; j < kch && ok; ++j) {
      if (!(ok = wait(full(j)))) break;
      const unsigned char* zh = zt + (2 * j) * SC_TILE + p * 128;
      const unsigned char* zl = zh + SC_TILE;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 h = *reinterpret_cast<const float4*>(zh + ((q ^ (p & 7)) << 4));
        const float4 l = *reinterpret_cast<const float4*>(zl + ((q ^ (p & 7)) << 4));
        const float* n = nv + 32 * j + 4 * q;
        t = fmaf(h.x + l.x, n[0], t);
        t = fmaf(h.y + l.y, n[1], t);
        t = fmaf(h.z + l.z, n[2], t);
        t = fmaf(h.w + l.w, n[3], t);
      }
    }
    t1[p] = t;
    asm volatile("bar.sync 2, 128;" ::: "memory");
  }
  // M1 = Z T_c out of tensor memory, split, back as the A operand: thread =
  // row q, its warpgroup's half of the columns a
  const int g = warp >> 2, row = tid & 127;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  const bool ok1 = __syncthreads_and(wait(done1));  // uniform: the tensor-memory accesses are warp-wide
  tc_fence_after();
  if (ok1) {
#pragma unroll
    for (int cc = 0; cc < 64; cc += 16) {
      const int col = 64 * g + cc;
      if (col < 32 * kch) {
        float v[16], h[16], l[16];
        sum_blocks(tmem + lanes + (uint32_t)col, kch, v);
#pragma unroll
        for (int q = 0; q < 16; ++q) split(v[q], h[q], l[q]);
        tmem_st16(tmem + lanes + 256u + (uint32_t)col, h);
        tmem_st16(tmem + lanes + 384u + (uint32_t)col, l);
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  mbar_arrive(aready);
  if (warp == 0 && ok1 && elect_one() && wait(aready)) {
    tc_fence_after();
    for (int j = 0; j < kch; ++j)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint64_t zh = sw128_desc(zaddr(j, 0) + 32u * kk), zl = sw128_desc(zaddr(j, 1) + 32u * kk);
        const uint32_t ah = tmem + 256u + (uint32_t)(32 * j + 8 * kk), al = ah + 128u, d = tmem + 128u * (j & 1);
        umma_tf32_ts(d, ah, zl, idesc, (j > 1 || kk > 0) ? 1u : 0u);
        umma_tf32_ts(d, al, zh, idesc, 1u);
      }
    for (int j = 0; j < kch; ++j)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_tf32_ts(tmem + 128u * (j & 1), tmem + 256u + (uint32_t)(32 * j + 8 * kk),
                     sw128_desc(zaddr(j, 0) + 32u * kk), idesc, 1u);
    umma_commit(done2);
    mma2 = true;
  }
  __syncwarp();
  // linear part, second factor: lin[:, c] = A_xx t1 (the MMAs of G run meanwhile)
  if (warp >= 4) {
    const int d = tid - 128;
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
    for (int k = 0; k < 32 * kch; k += 8) {
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = a.ax[(k + q) * SC_W + d];
      s0 = fmaf(x[0], t1[k], s0); s1 = fmaf(x[1], t1[k + 1], s1);
      s2 = fmaf(x[2], t1[k + 2], s2); s3 = fmaf(x[3], t1[k + 3], s3);
      s0 = fmaf(x[4], t1[k + 4], s0); s1 = fmaf(x[5], t1[k + 5], s1);
      s2 = fmaf(x[6], t1[k + 6], s2); s3 = fmaf(x[7], t1[k + 7], s3);
    }
    a.lin[c * SC_W + d] = (s0 + s1) + (s2 + s3);
  }
  const bool ok2 = __syncthreads_and(ok1 && wait(done2));
  tc_fence_after();
  if (ok2) {
    // G_c[q, p] (symmetric): row q per thread, the pairs p <= q of column p
    // are contiguous over the lanes
    float* gh = a.gh + (int64_t)c * a.PPp;
    float* gl = a.gl + (int64_t)c * a.PPp;
#pragma unroll
    for (int cc = 0; cc < 64; cc += 16) {
      const int col = 64 * g + cc;
      if (col < 32 * kch) {
        float v[16];
        sum_blocks(tmem + lanes + (uint32_t)col, min(kch, 2), v);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int p = col + q;
          if (p <= row && row < ka) {
            float h, l;
            split(v[q], h, l);
            const int o = sc_start(p, ka) + row - p;
            gh[o] = h;
            gl[o] = l;
          }
        }
      }
    }
  }
  if (warp == 0 && elect_one() && *abort_flag) {  // let copies and MMAs in flight finish
    for (int j = 0; j < loaded; ++j) wait(full(j), SC_WAIT / 4);
    if (mma1) wait(done1, SC_WAIT / 4);
    if (mma2) wait(done2, SC_WAIT / 4);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// part[cluster][c][d] = sum over the cluster's pair chunks of W'[d, pq] G[c, pq]
__global__ void __launch_bounds__(SC_NT, 1) __cluster_dims__(SC_WG_CL, 1, 1)
    s_core_wg(const __grid_constant__ CUtensorMap tmWh, const __grid_constant__ CUtensorMap tmWl,
              const __grid_constant__ CUtensorMap tmGh, const __grid_constant__ CUtensorMap tmGl, int R,
              const int32_t* __restrict__ rank, float* __restrict__ part, uint32_t* status) {
  extern __shared__ unsigned char smem_raw[];
  cg::cluster_group cl = cg::this_cluster();
  pdl_launch();
  const int ka = 2 * min(R, (int)*rank), np = ka * (ka + 1) / 2, nch = (np + 31) / 32;
  const int k0 = (int)((int64_t)blockIdx.x * nch / SC_WG_CTAS), nk = (int)((int64_t)(blockIdx.x + 1) * nch / SC_WG_CTAS) - k0;
  // the same alignment in every CTA of the cluster: dynamic shared memory starts at one offset
  unsigned char* base = align_1024(smem_raw);
  unsigned char* ctrl = base + 4 * SC_WG_CHUNKS * SC_TILE;
  const uint32_t bar0 = smem_u32(ctrl);
  auto full = [&](int j) { return bar0 + 8u * j; };  // j < SC_WG_CHUNKS
  const uint32_t done = bar0 + 32u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 64);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 68);
  auto wait = [&](uint32_t bar, long long limit = SC_WAIT) {
    return mbar_wait_st(bar, 0, abort_flag, status, ST_TIMEOUT, limit);
  };
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int j = 0; j < SC_WG_CHUNKS; ++j) mbar_init(full(j), 1);
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp == 0 && elect_one()) {
    const uint32_t st = smem_u32(base);
    for (int j = 0; j < nk; ++j) {
      const uint32_t s = st + (uint32_t)(4 * j) * SC_TILE;
      mbar_expect_tx(full(j), 4 * SC_TILE);
      tma_load_2d(s, &tmWh, 32 * (k0 + j), 0, full(j));
      tma_load_2d(s + SC_TILE, &tmWl, 32 * (k0 + j), 0, full(j));
    }
    pdl_wait();  // G is the previous kernel's
    for (int j = 0; j < nk; ++j) {
      const uint32_t s = st + (uint32_t)(4 * j) * SC_TILE;
      tma_load_2d(s + 2 * SC_TILE, &tmGh, 32 * (k0 + j), 0, full(j));
      tma_load_2d(s + 3 * SC_TILE, &tmGl, 32 * (k0 + j), 0, full(j));
    }
    const uint32_t idesc = idesc_tf32(SC_W, SC_W);
    bool ok = true;
    for (int j = 0; j < nk && ok; ++j) {
      if (!(ok = wait(full(j)))) break;
      tc_fence_after();
      const uint32_t s = st + (uint32_t)(4 * j) * SC_TILE, d = tmem + 128u * j;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint64_t wh = sw128_desc(s + 32u * kk), wl = sw128_desc(s + SC_TILE + 32u * kk);
        const uint64_t gh = sw128_desc(s + 2 * SC_TILE + 32u * kk), gl = sw128_desc(s + 3 * SC_TILE + 32u * kk);
        umma_tf32_ss(d, wh, gl, idesc, kk > 0 ? 1u : 0u);
        umma_tf32_ss(d, wl, gh, idesc, 1u);
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_tf32_ss(d, sw128_desc(s + 32u * kk), sw128_desc(s + 2 * SC_TILE + 32u * kk), idesc, 1u);
    }
    umma_commit(done);
    if (*abort_flag) {
      for (int j = 0; j < nk; ++j) wait(full(j), SC_WAIT / 4);
      wait(done, SC_WAIT / 4);
    }
  }
  __syncwarp();
  const bool ok = __syncthreads_and(wait(done));
  tc_fence_after();
  // the tile, [c][d], over the operands (every MMA has read them)
  float* tile = reinterpret_cast<float*>(base);
  const int g = warp >> 2, row = tid & 127;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
#pragma unroll
  for (int cc = 0; cc < 64; cc += 16) {
    const int col = 64 * g + cc;
    float v[16];
    sum_blocks(tmem + lanes + (uint32_t)col, ok ? nk : 0, v);
#pragma unroll
    for (int q = 0; q < 16; ++q) tile[(col + q) * SC_W + row] = v[q];
  }
  tc_fence_before();
  cl.sync();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
  // this CTA's eighth of the columns: the cluster's tiles in rank order
  const int per = SC_W * SC_W / SC_WG_CL / 4;  // float4 per CTA
  float4* dst = reinterpret_cast<float4*>(part) + (int64_t)(blockIdx.x / SC_WG_CL) * (SC_W * SC_W / 4);
  for (int e = tid; e < per; e += SC_NT) {
    const int o = (int)cl.block_rank() * per + e;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < SC_WG_CL; ++k) {
      const float4 x = reinterpret_cast<const float4*>(cl.map_shared_rank(tile, k))[o];
      s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
    }
    dst[o] = s;
  }
  cl.sync();  // no CTA leaves while its tile may be read
}

// RK stage on the FP64 core with derivative lin + sum of the partials, and the
// split of the next stage's input (zero outside the active block)
__global__ void __launch_bounds__(256) s_core_update(int R, const int32_t* __restrict__ rank,
                                                     const float* __restrict__ lin, const float* __restrict__ part,
                                                     double* __restrict__ y, double* __restrict__ acc, double b,
                                                     double ha, double h, int first, int last,
                                                     float* __restrict__ zh, float* __restrict__ zl) {
  pdl_launch();
  pdl_wait();
  const int r = min(R, (int)*rank), ka = 2 * r, w = 2 * R;
  const int e = blockIdx.x * 256 + threadIdx.x, d = e & (SC_W - 1), c = e / SC_W;
  if (d >= ka || c >= ka) return;
  double v = (double)lin[e];
#pragma unroll
  for (int z = 0; z < SC_WG_CTAS / SC_WG_CL; ++z) v += (double)part[z * SC_W * SC_W + e];
  const int64_t o = sc_act(d, r, R) + (int64_t)sc_act(c, r, R) * w;
  const double s = first ? b * v : fma(b, v, acc[o]);
  double zn;
  if (last) {
    zn = fma(h, s, y[o]);
    y[o] = zn;
  } else {
    acc[o] = s;
    zn = fma(ha, v, y[o]);
  }
  float hi, lo;
  split((float)zn, hi, lo);
  zh[d * SC_W + c] = hi;
  zl[d * SC_W + c] = lo;
}

// operands of the step: T_c expanded from the packed tensor (the off-diagonal
// pairs hold twice the entry), W' as rows of pairs, N_nu, A_xx and Z, zero
// outside the active block
__global__ void __launch_bounds__(256) s_core_setup(int R, const int32_t* __restrict__ rank, SCore s, int PP,
                                                    const float* __restrict__ Tp, const float* __restrict__ Wp,
                                                    const double* __restrict__ Nnu, const double* __restrict__ Axx,
                                                    const double* __restrict__ Z) {
  const int r = min(R, (int)*rank), ka = 2 * r, w = 2 * R, np = ka * (ka + 1) / 2;
  const int64_t step = (int64_t)gridDim.x * blockDim.x, t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t e = t0; e < (int64_t)ka * SC_W * SC_W; e += step) {
    const int b = (int)(e & (SC_W - 1)), a = (int)(e / SC_W) & (SC_W - 1), c = (int)(e / (SC_W * SC_W));
    float v = 0.0f;
    if (a < ka && b < ka) {
      const int lo = min(a, b), hi = max(a, b);
      v = Tp[sc_start(lo, ka) + hi - lo + (int64_t)c * PP] * ((a == b) ? 1.0f : 0.5f);
    }
    split(v, s.th[e], s.tl[e]);
  }
  for (int64_t e = t0; e < (int64_t)SC_W * s.PPp; e += step) {
    const int d = (int)(e / s.PPp), p = (int)(e - (int64_t)d * s.PPp);
    const float v = (d < ka && p < np) ? Wp[p + (int64_t)d * PP] : 0.0f;
    split(v, s.wh[e], s.wl[e]);
  }
  for (int64_t e = t0; e < SC_W * SC_W; e += step) {
    const int x = (int)(e & (SC_W - 1)), q = (int)(e / SC_W);
    const bool in = x < ka && q < ka;
    s.nc[e] = in ? (float)Nnu[sc_act(x, r, R) + (int64_t)sc_act(q, r, R) * w] : 0.0f;
    s.ax[e] = in ? (float)Axx[sc_act(x, r, R) + (int64_t)sc_act(q, r, R) * w] : 0.0f;
    split(in ? (float)Z[sc_act(q, r, R) + (int64_t)sc_act(x, r, R) * w] : 0.0f, s.zh[e], s.zl[e]);
  }
}

}  // namespace

bool s_core_supported(int R) { return 2 * R <= SC_W && tc_encoder_available(); }

cudaError_t s_core_init(SCore* s, int R) {
  s->R = R;
  s->PPp = (R * (2 * R + 1) + 3) & ~3;
  const size_t z = SC_W * SC_W, t = (size_t)2 * R * SC_W * SC_W, p = (size_t)SC_W * s->PPp;
  float** dst[] = {&s->zh, &s->zl, &s->th, &s->tl, &s->wh, &s->wl, &s->gh, &s->gl, &s->nc, &s->ax, &s->lin, &s->part};
  const size_t len[] = {z, z, t, t, p, p, p, p, z, z, z, z * (SC_WG_CTAS / SC_WG_CL)};
  for (int k = 0; k < 12; ++k) {
    cudaError_t e = cudaMalloc((void**)dst[k], sizeof(float) * len[k]);
    // rows of G beyond the active columns and pairs beyond the active ones
    // meet zeros of W': they only have to be finite
    if (e == cudaSuccess) e = cudaMemset(*dst[k], 0, sizeof(float) * len[k]);
    if (e != cudaSuccess) return e;
  }
  const uint64_t x[] = {(uint64_t)SC_W, (uint64_t)SC_W, (uint64_t)s->PPp, (uint64_t)s->PPp};
  const uint64_t rows[] = {(uint64_t)SC_W, (uint64_t)2 * R * SC_W, (uint64_t)SC_W, (uint64_t)SC_W};
  for (int k = 0; k < 8; ++k)
    if (!tc_encode_2d(s->tm[k], *dst[k], x[k / 2], rows[k / 2], 32, SC_W, true)) return cudaErrorInvalidValue;
  return cudaSuccess;
}

void s_core_free(SCore* s) {
  float** dst[] = {&s->zh, &s->zl, &s->th, &s->tl, &s->wh, &s->wl, &s->gh, &s->gl, &s->nc, &s->ax, &s->lin, &s->part};
  for (float** p : dst) {
    cudaFree(*p);
    *p = nullptr;
  }
}

cudaError_t s_core_flow(const SCore& s, const int32_t* rank, double* Z, double* acc, const double* Nnu,
                        const double* Axx, const float* Tp, const float* Wp, int PP, const Scheme& sc, double h,
                        uint32_t* status, cudaStream_t st) {
  static std::atomic<uint64_t> done_g{0}, done_w{0};
  cudaError_t e = set_smem_limit(s_core_g, SC_G_SMEM, done_g);
  if (e == cudaSuccess) e = set_smem_limit(s_core_wg, SC_WG_SMEM, done_w);
  if (e != cudaSuccess) return e;
  auto tm = [&](int k) -> const CUtensorMap& { return *reinterpret_cast<const CUtensorMap*>(s.tm[k]); };
  s_core_setup<<<608, 256, 0, st>>>(s.R, rank, s, PP, Tp, Wp, Nnu, Axx, Z);
  SGArgs a{};
  a.R = s.R;
  a.PPp = s.PPp;
  a.rank = rank;
  a.nc = s.nc;
  a.ax = s.ax;
  a.lin = s.lin;
  a.gh = s.gh;
  a.gl = s.gl;
  a.status = status;
  // From the second kernel on each starts its prologue and its loads of the
  // step's constants while the one before it drains (the first one's
  // constants are the setup's).
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  auto config = [&](int grid, size_t smem, bool dependent) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3(256);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &attr;
    c.numAttrs = dependent ? 1 : 0;
    return c;
  };
  static_assert(SC_NT == 256, "block size");
  bool first = true;
  for (int sub = 0; sub < sc.nsub; ++sub)
    for (int k = 0; k < sc.nstages; ++k) {
      const bool last = k + 1 == sc.nstages;
      cudaLaunchConfig_t c = config(2 * s.R, SC_G_SMEM, !first);
      if ((e = cudaLaunchKernelEx(&c, s_core_g, tm(0), tm(1), tm(2), tm(3), a)) != cudaSuccess) return e;
      c = config(SC_WG_CTAS, SC_WG_SMEM, true);
      e = cudaLaunchKernelEx(&c, s_core_wg, tm(4), tm(5), tm(6), tm(7), s.R, rank, s.part, status);
      if (e != cudaSuccess) return e;
      c = config(SC_W * SC_W / 256, 0, true);
      e = cudaLaunchKernelEx(&c, s_core_update, s.R, rank, (const float*)s.lin, (const float*)s.part, Z, acc, sc.b[k],
                             last ? 0.0 : h * sc.a[k + 1], h, (int)(k == 0), (int)last, s.zh, s.zl);
      if (e != cudaSuccess) return e;
      first = false;
    }
  return cudaGetLastError();
}

}  // namespace lri
