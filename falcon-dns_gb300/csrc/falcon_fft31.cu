// The nonlinear pass for prime-factor FFT plans with a radix above 17 and
// for twiddled plans with a prime above 7 (falcon_fft.cuh): grids of exactly
// 3 Nm points, one instance.
#include "falcon_fft.cuh"

namespace falcon {

cudaError_t launch_nonlin_31(const NonlinArgs& a, cudaStream_t s) {
  return a.plan.pfa ? launch_nonlin_s<31, false, 4, 1, 1>(a, s) : launch_nonlin_s<31, true, 4, 1, 1>(a, s);
}

}  // namespace falcon
