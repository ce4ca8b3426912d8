// 1D blocks of 256..16384 points on chip: double fields, one component.
#include "launch.cuh"

int launch_line_d1(atus_ctx *ctx, const LineArgs &a) { return launch_line_n<double, 1, false>(ctx, a); }
