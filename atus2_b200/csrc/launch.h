// launch.h -- exported launchers, one per precision and tile component count.
#pragma once
#include "ctx.h"
#include "line1d.cuh"
#include "pass2.cuh"

int launch_pass_d1(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass_d2(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass_d4(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass_f1(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass_f2(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass_f4(atus_ctx *ctx, PassArgs &a, int axis);
// A 1D block with the field on chip.  _line: 256..16384 points (bragg: two
// components, kind K_BRAGG; else pure phases); _block1d: 2..128 points.
// ATUS_E_UNSUPPORTED, nothing launched, where the field does not fit.
int launch_line_d1(atus_ctx *ctx, const LineArgs &a);
int launch_line_d2(atus_ctx *ctx, const LineArgs &a, bool bragg);
int launch_line_f1(atus_ctx *ctx, const LineArgs &a);
int launch_line_f2(atus_ctx *ctx, const LineArgs &a, bool bragg);
int launch_block1d_d1(atus_ctx *ctx, Block1DArgs &a);
int launch_block1d_d2(atus_ctx *ctx, Block1DArgs &a);
int launch_block1d_f1(atus_ctx *ctx, Block1DArgs &a);
int launch_block1d_f2(atus_ctx *ctx, Block1DArgs &a);
// Register-staged passes (pencils of 32..256 points).  _t: one transform
// (mode M2_FWD / M2_INV, strided or contiguous axis); _k: FFT, kinetic or
// Sobolev filter, IFFT along a strided axis; _nl: IFFT, potential step, FFT
// along the contiguous axis with tc components per tile (1 to 4; 3 and 4 in _nl3
// and _nl4).  All return
// ATUS_E_UNSUPPORTED, with the fields untouched, when they do not apply.
int launch_pass2_d_t(atus_ctx *ctx, PassArgs &a, int axis, int mode, bool strided);
int launch_pass2_f_t(atus_ctx *ctx, PassArgs &a, int axis, int mode, bool strided);
int launch_pass2_d_k(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_f_k(atus_ctx *ctx, PassArgs &a, int axis);
// _kr: the _k kinetic pass that also sums the Rabi balls (M2_KIN_RABI)
int launch_pass2_d_kr(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_f_kr(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_d_nl(atus_ctx *ctx, PassArgs &a, int axis, int tc);
int launch_pass2_f_nl(atus_ctx *ctx, PassArgs &a, int axis, int tc);
// _sob: first (M2_FWD_SOB) and last (M2_INV_SOB) pass of a Sobolev iteration,
// along the contiguous axis (32..256 points)
int launch_pass2_d_sob(atus_ctx *ctx, PassArgs &a, int axis, int mode);
// _fs: the passes of a long 1D axis seen as n1 x n2 points (M2_FS_*), axes of
// 128..4096 points; tc: components of M2_FS_NL (1 or 2)
int launch_fs_d(atus_ctx *ctx, PassArgs &a, int mode, int tc);
int launch_fs_f(atus_ctx *ctx, PassArgs &a, int mode, int tc);
int launch_pass2_d_nl3(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_d_nl4(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_f_nl3(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_f_nl4(atus_ctx *ctx, PassArgs &a, int axis);
// _meet: as _nl with two components, 32..2048 points, on dense grids (ctx.h)
int launch_pass2_d_meet(atus_ctx *ctx, PassArgs &a, int axis);
int launch_pass2_f_meet(atus_ctx *ctx, PassArgs &a, int axis);
