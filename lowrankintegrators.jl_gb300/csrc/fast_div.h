// fast_div.h - quotients by a fixed divisor from its FP32 reciprocal (host and
// device).
#pragma once

#ifdef __CUDACC__
#define LRI_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LRI_HOST_DEVICE inline
#endif

namespace lri {
namespace wide {

// e / d for 0 <= e < 2^31 and quotients up to 2^16, in a few instructions where
// the integer division takes tens.  Below e = 2^21 the rounding of (e + 1/2) / d
// stays under 1 / (2 d) and the estimate is the quotient; above, it is off by
// one at the ends of a column (first at 114 050 x 48), which the remainder
// shows.
struct FastDiv {
  int d;
  float inv;
  LRI_HOST_DEVICE explicit FastDiv(int d_) : d(d_), inv(1.0f / (float)(d_ > 1 ? d_ : 1)) {}
  LRI_HOST_DEVICE int div(int e) const {
    const int q = (int)(((float)e + 0.5f) * inv), rem = e - q * d;
    return q + (rem >= d) - (rem < 0);
  }
};

}  // namespace wide
}  // namespace lri
