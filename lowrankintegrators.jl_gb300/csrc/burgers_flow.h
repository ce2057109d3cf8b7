// burgers_flow.h - whole substep flows of the large Burgers engine in one or
// a few launches (active widths up to FLOW_KMAX).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "engine_api.h"

namespace lri {

// widest active panel of the flow kernels: K and L flows up to rank 32, the S
// flow up to rank 16 (2r columns)
constexpr int FLOW_KMAX = 32;

// K flow  y' = (ih2 Dxx y) N_nu + alpha KR(Dx y, y) T' + beta Dx(KR(y, y) T'),
// Dx = ihx (shift - shift), over sc.nsub substeps of length h on the N x R
// panel `y` (ld N; active columns *rank <= FLOW_KMAX, the others unchanged);
// `tmp` is a second N x R panel, kmax the caller's bound of the active width
// (16 or FLOW_KMAX: it sizes registers and shared memory; a wider device rank
// sets ST_BAD_SHAPE).  N_nu: FP64, ld R; T': packed pairs, ld PP.
template <typename T>
cudaError_t burgers_k_flow(int kmax, int N, int R, const int32_t* rank, T* y, T* tmp, const double* Nnu, const T* Tp, int PP,
                           double ih2, double ihx, double alpha, double beta, const Scheme& sc, double h, int sms,
                           uint32_t* status, cudaStream_t st);

// L flow  y'_j = nu_j (y A_xx)_j + KR(y, y)_j T'  on the M x R panel `y`.
template <typename T>
cudaError_t burgers_l_flow(int kmax, int M, int R, const int32_t* rank, T* y, const T* nu, const double* Axx, const T* Tp,
                           int PP, int nonlin, const Scheme& sc, double h, uint32_t* status, cudaStream_t st);

// S flow  Z' = A_xx Z N_nu + W : (Z T_c Z^T)_c  on the active block of the FP64
// core `Z` (ld 2R; active 2 *rank <= FLOW_KMAX): T' the packed tensor of
// Vhat, W' that of Uhat (nonlin = 0: both absent).  N_nu, A_xx: ld 2R.
template <typename T>
cudaError_t burgers_s_flow(int R, const int32_t* rank, double* Z, const double* Nnu, const double* Axx, const T* Tp,
                           const T* Wp, int PP, int nonlin, const Scheme& sc, double h, uint32_t* status,
                           cudaStream_t st);

}  // namespace lri
