// The nonlinear pass for prime-factor FFT plans whose largest radix is 11,
// 13 or 17 (falcon_fft.cuh): grids of exactly 3 Nm points, one instance.
#include "falcon_fft.cuh"

namespace falcon {

cudaError_t launch_nonlin_17(const NonlinArgs& a, cudaStream_t s) { return launch_nonlin_s<17, false, 4, 1, 1>(a, s); }

}  // namespace falcon
