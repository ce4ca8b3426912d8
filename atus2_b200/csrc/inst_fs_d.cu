// Four-step passes of long 1D axes, double fields.
#include "launch.cuh"

int launch_fs_d(atus_ctx *ctx, PassArgs &a, int mode, int tc) { return launch_fs<double>(ctx, a, mode, tc); }
