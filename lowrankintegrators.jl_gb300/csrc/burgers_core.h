// burgers_core.h - the S flow of the large Burgers engine on the 2r x 2r core
// with tensor-core products (FP32 panels, ranks 17 to 64).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "engine_api.h"

namespace lri {

// Device buffers of one engine and their tensor maps (CUtensorMap storage).
struct SCore {
  int R = 0;
  int PPp = 0;                               // pair stride of W' and G (a multiple of 4)
  float* zh = nullptr; float* zl = nullptr;  // Z: 128 x 128 row-major, TF32 hi and lo
  float* th = nullptr; float* tl = nullptr;  // T_c: [c][a][b], TF32 hi and lo
  float* wh = nullptr; float* wl = nullptr;  // W': [d][pair]
  float* gh = nullptr; float* gl = nullptr;  // G = Z T_c Z^T: [c][pair]
  float* nc = nullptr;                       // N_nu: [c][k]
  float* ax = nullptr;                       // A_xx: [k][d]
  float* lin = nullptr;                      // A_xx Z N_nu: [c][d]
  float* part = nullptr;                     // partial sums of W' G: [cluster][c][d]
  alignas(64) unsigned char tm[8][128];      // zh, zl, th, tl, wh, wl, gh, gl
};

bool s_core_supported(int R);
cudaError_t s_core_init(SCore* s, int R);
void s_core_free(SCore* s);

// Z' = A_xx Z N_nu + W' : (Z T_c Z^T)_c over sc.nsub substeps of length h on the
// active block (2 *rank columns) of the FP64 core Z (ld 2R); acc: scratch of
// the same shape.  N_nu, A_xx: FP64, ld 2R; Tp, Wp: packed tensors of Vhat
// and Uhat, ld PP.  A bounded wait that gives up ORs ST_TIMEOUT into *status.
cudaError_t s_core_flow(const SCore& s, const int32_t* rank, double* Z, double* acc, const double* Nnu,
                        const double* Axx, const float* Tp, const float* Wp, int PP, const Scheme& sc, double h,
                        uint32_t* status, cudaStream_t st);

}  // namespace lri
