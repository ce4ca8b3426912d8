// Register-staged IFFT -> potential step -> FFT passes, float fields, three components.
#include "launch.cuh"

int launch_pass2_f_nl3(atus_ctx *ctx, PassArgs &a, int axis) {
  return launch_pass2_n<float, 3, M2_NL, false>(ctx, a, axis);
}
