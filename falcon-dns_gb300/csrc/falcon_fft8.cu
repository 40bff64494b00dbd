// The nonlinear pass for FFT plans of radices up to 8 (falcon_fft.cuh): the
// plans of make_line_plan, and grids of 3 Nm points with such factors.
#include "falcon_fft.cuh"

namespace falcon {

// Warps per half line and lines per block.  Few lines (up to two per SM) are
// a matter of latency: 8 warps a line.  With more, the shared memory of the
// lines (32 bytes a point) sets how many an SM holds, and S fills about 16
// warps with them: S = 1 up to 640 points, 2 up to 1152 (1024 points: 5 lines
// of 4 warps), 4 above (1536: 3 lines of 8).  Measured, us for Nr x B lines:
// 65 x 128 of 512 points 222 / 245 / 330 with S = 1 / 2 / 4; 97 x 16 of 1024
// points 157 / 132 / 134; 129 x 8 of 1536 points 200 / 165 / 144.
cudaError_t launch_nonlin_8(const NonlinArgs& a, cudaStream_t s) {
  if (a.plan.pfa) return launch_nonlin_s<8, false, 4, 1, 1>(a, s);
  if ((long)a.R * a.B <= 2 * sm_count() || a.plan.P > 1152) return launch_nonlin_s<8, true, 4, 1, 2>(a, s);
  if (a.plan.P > 640) return launch_nonlin_s<8, true, 2, 1, 4>(a, s);
  return launch_nonlin_s<8, true, 1, 2, 4>(a, s);
}

}  // namespace falcon
