// Four-step passes of long 1D axes, float fields.
#include "launch.cuh"

int launch_fs_f(atus_ctx *ctx, PassArgs &a, int mode, int tc) { return launch_fs<float>(ctx, a, mode, tc); }
