// Register-staged passes at the ends of a Sobolev iteration, double fields.
#include "launch.cuh"

int launch_pass2_d_sob(atus_ctx *ctx, PassArgs &a, int axis, int mode) {
  if (mode == M2_FWD_SOB) return launch_pass2_n<double, 1, M2_FWD_SOB, false>(ctx, a, axis);
  if (mode == M2_INV_SOB) return launch_pass2_n<double, 1, M2_INV_SOB, false>(ctx, a, axis);
  return ATUS_E_UNSUPPORTED;
}
