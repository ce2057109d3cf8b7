// burgers_panel.h - the K and L substep flows of the large Burgers engine at
// ranks 33 to 64 (FP32 panels): every RK stage of a flow in one or a few
// launches, the quadratic term on the tensor cores.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "engine_api.h"

namespace lri {

constexpr int PANEL_RMAX = 64;

// Operand copies of the two flow tensors (T'_V of the K flow, T'_L of the L flow).
struct PanelFlow {
  unsigned char* b[2] = {nullptr, nullptr};
};

cudaError_t panel_flow_init(PanelFlow* p);
void panel_flow_free(PanelFlow* p);

// operand copy k of the packed tensor Tp (ld PP, active columns *rank)
cudaError_t panel_flow_tensor(const PanelFlow& p, int k, int R, const int32_t* rank, const float* Tp, int PP,
                              cudaStream_t st);

// K flow  y' = (ih2 Dxx y) N_nu + alpha KR(Dx y, y) T' + beta Dx(KR(y, y) T'),
// Dx = ihx (shift - shift), over sc.nsub substeps of length h on the N x R
// panel `y` (ld N; active columns *rank, the others unchanged); `tmp`: a
// second N x R panel.  N_nu: FP64, ld R.  A bounded wait that gives up ORs
// ST_TIMEOUT into *status.
cudaError_t panel_k_flow(const PanelFlow& p, int N, int R, const int32_t* rank, float* y, float* tmp,
                         const double* Nnu, double ih2, double ihx, double alpha, double beta, const Scheme& sc,
                         double h, uint32_t* status, cudaStream_t st);

// L flow  y'_j = nu_j (y A_xx)_j + KR(y, y)_j T'  on the M x R panel `y`.
cudaError_t panel_l_flow(const PanelFlow& p, int M, int R, const int32_t* rank, float* y, const float* nu,
                         const double* Axx, const Scheme& sc, double h, uint32_t* status, cudaStream_t st);

}  // namespace lri
