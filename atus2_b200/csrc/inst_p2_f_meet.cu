// Register-staged IFFT -> potential step -> FFT passes, float fields, two
// components that meet in shared memory.
#include "launch.cuh"

int launch_pass2_f_meet(atus_ctx *ctx, PassArgs &a, int axis) {
  return launch_pass2_n<float, 2, M2_NL_MEET, false>(ctx, a, axis);
}
