// engine_df.cu - double-float instantiation of the instance engine and the
// double <-> double-float conversion kernels used at the ABI boundary.
#include "engine_impl.cuh"

namespace lri {

template cudaError_t launch_step_occ<dfloat, 3>(const StepArgs<dfloat>&, int, cudaStream_t);
template size_t step_smem_bytes<dfloat>();

// The S step of a BUG step whose sides ran as sides_kernel (engine_sides.cu), one
// CTA per instance: basis swap of a first step, S~0 = M S0 N^T, the substep,
// the new projections (blocks B_RK, B_RL) made current.
static __global__ void __launch_bounds__(NT, 3) core_kernel(const __grid_constant__ StepArgs<dfloat> g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<dfloat>& sm = *reinterpret_cast<Smem<dfloat>*>(smem_raw);
  const int inst = g.order[blockIdx.x];
  const InstDesc d = g.inst[inst];
  const int r = g.rank[inst];
  if (r < 1 || r > d.rcap) return;  // reported by the sides
  Inst<dfloat> I;
  I.n = d.n; I.m = d.m; I.rcap = d.rcap; I.W = d.wcap; I.inst = inst;
  I.U = g.U + d.offU;
  I.S = g.S + d.offS;
  I.V = g.V + d.offV;
  I.small = g.small + d.offSmall;
  const int W = I.W;
  dfloat* GU = I.blk(B_GU);
  dfloat* GV = I.blk(B_GV);
  if (g.proj_valid[inst] == 0) {
    copy_mat<dfloat>(d.n, r, g.work + d.offWK, d.n, I.U, d.n);
    copy_mat<dfloat>(d.m, r, g.work + d.offWL, d.m, I.V, d.m);
    if (threadIdx.x == 0) g.proj_valid[inst] = 1;
  }
  copy_mat<dfloat>(r, r, I.blk(B_RK), W, GU + (int64_t)r * W, W);
  copy_mat<dfloat>(r, r, I.blk(B_RL), W, GV + (int64_t)r * W, W);
  dfloat* St = I.blk(B_ST);
  dfloat* T1 = I.blk(B_T1);
  small_gemm<dfloat>(r, r, r, dfloat(1), I.S, I.rcap, false, I.blk(B_N), W, true, dfloat(0), T1, W);
  small_gemm<dfloat>(r, r, r, dfloat(1), I.blk(B_M), W, false, T1, W, false, dfloat(0), St, W);
  substep_core<dfloat>(g, I, St, r, r, dfloat(1), GU, GV, I.U, I.V, g.sS, g.dt, sm);
  copy_mat<dfloat>(r, r, St, W, I.S, I.rcap);
  check_finite<dfloat>(g, I.S, r, I.rcap);
}

cudaError_t launch_core(const StepArgs<dfloat>& g, int count, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  cudaError_t e = set_smem_limit(core_kernel, (int)sizeof(Smem<dfloat>), done);
  if (e != cudaSuccess) return e;
  core_kernel<<<count, NT, sizeof(Smem<dfloat>), st>>>(g);
  return cudaGetLastError();
}

__global__ void f64_to_df_kernel(const double* __restrict__ in, dfloat* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = dfloat(in[i]);
}

__global__ void df_to_f64_kernel(const dfloat* __restrict__ in, double* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}

static int conv_grid(int64_t n) {
  int64_t g = (n + 255) / 256;
  if (g > 152 * 16) g = 152 * 16;
  return g < 1 ? 1 : (int)g;
}

// Bound by the launch for small factors (one launch for four copies with a gap
// after each) and by memory for large ones: the widest words that a part's
// ends and length allow.
template <class W>
__device__ void copy_words(const CopyParts& c, int p) {
  const size_t nt = (size_t)gridDim.x * blockDim.x, nw = c.bytes[p] / sizeof(W);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nw; i += nt)
    static_cast<W*>(c.dst[p])[i] = static_cast<const W*>(c.src[p])[i];
}

__global__ void __launch_bounds__(256) copy_parts_kernel(CopyParts c) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uintptr_t low = (uintptr_t)c.dst[p] | (uintptr_t)c.src[p] | c.bytes[p];
    if ((low & 15) == 0) copy_words<uint4>(c, p);
    else if ((low & 7) == 0) copy_words<uint2>(c, p);
    else copy_words<uint32_t>(c, p);
  }
}

cudaError_t copy_parts(const CopyParts& c, cudaStream_t stream) {
  size_t most = 0;
  for (size_t b : c.bytes) most = b > most ? b : most;
  const int64_t g = conv_grid((int64_t)(most / 16 + 1));
  copy_parts_kernel<<<(int)g, 256, 0, stream>>>(c);
  return cudaGetLastError();
}

cudaError_t convert_f64_to_df(const double* in, void* out, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  f64_to_df_kernel<<<conv_grid(n), 256, 0, stream>>>(in, static_cast<dfloat*>(out), n);
  return cudaGetLastError();
}

cudaError_t convert_df_to_f64(const void* in, double* out, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  df_to_f64_kernel<<<conv_grid(n), 256, 0, stream>>>(static_cast<const dfloat*>(in), out, n);
  return cudaGetLastError();
}

int local_flow_count() { return kLocalFlowCount; }

const char* local_flow_name(int id) {
  switch (id) {
#define LRI_FLOW_NAME(ID, TYPE, NAME) \
  case ID:                            \
    return NAME;
    LRI_LOCAL_FLOWS(LRI_FLOW_NAME)
#undef LRI_FLOW_NAME
    default:
      return nullptr;
  }
}

}  // namespace lri
