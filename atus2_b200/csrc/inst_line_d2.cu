// 1D blocks of 256..16384 points on chip: double fields, two components.
#include "launch.cuh"

int launch_line_d2(atus_ctx *ctx, const LineArgs &a, bool bragg) {
  return bragg ? launch_line_n<double, 2, true>(ctx, a) : launch_line_n<double, 2, false>(ctx, a);
}
