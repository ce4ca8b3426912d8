// Register-staged IFFT -> potential step -> FFT passes, double fields, three components.
#include "launch.cuh"

int launch_pass2_d_nl3(atus_ctx *ctx, PassArgs &a, int axis) {
  return launch_pass2_n<double, 3, M2_NL, false>(ctx, a, axis);
}
