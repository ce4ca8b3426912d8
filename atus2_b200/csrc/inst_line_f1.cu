// 1D blocks of 256..16384 points on chip: float fields, one component.
#include "launch.cuh"

int launch_line_f1(atus_ctx *ctx, const LineArgs &a) { return launch_line_n<float, 1, false>(ctx, a); }
