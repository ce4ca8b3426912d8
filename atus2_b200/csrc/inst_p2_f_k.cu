// Register-staged FFT -> kinetic phase / Sobolev filter -> IFFT passes, float fields.
#include "launch.cuh"

int launch_pass2_f_k(atus_ctx *ctx, PassArgs &a, int axis) {
  if (a.op == OP_FILT) return ATUS_E_UNSUPPORTED;  // the descent runs in FP64
  return launch_pass2_n<float, 1, M2_KIN, true>(ctx, a, axis);
}
