// ctx.h -- the engine context shared by the host translation units.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

#include <string>
#include <utility>

#include "../../include/atus_gpu.h"
#include "kernels.cuh"

using namespace atus;

struct atus_ctx {
  int dim = 0, ncomp = 0, prec = 0;
  int64_t n[3] = {1, 1, 1};
  int lg[3] = {0, 0, 0};
  int64_t npts = 0;
  double d[3] = {0, 0, 0}, dk[3] = {0, 0, 0};
  double ar = 0, ar_k = 0, t = 0, dt = 0.001;
  double alpha[MAXC][3] = {};
  double gs[MAXC * MAXC] = {};  // padded [i*MAXC + j]
  atus_laser laser = {};
  atus_laser laser2 = {};       // second species (two-species programs)
  double win_t0 = 0;            // pulse windows of the two-species bragg_ad:
  double win_dur[2] = {HUGE_VAL, HUGE_VAL};  // species s on while t1 - win_t0 <= win_dur[s]
  size_t csize = 16;            // bytes per complex value
  void *psi[MAXC] = {};
  double *V[MAXC] = {};
  void *scratch = nullptr;      // N complex128 (FP64 staging / spectra)
  void *tw = nullptr;           // twiddles in the field precision
  void *tw64 = nullptr;         // FP64 twiddles (spectra of the FP64 scratch buffer)
  double2 *kt[2][MAXC][3] = {}; // kinetic phase factors [half=0/full=1][comp][axis], FP64
  double *red_partial = nullptr;  // block sums of the reductions
  unsigned *red_count = nullptr;  // blocks done; zero between launches
  void *pinned = nullptr;         // host memory mapped into the device: h_red, h_sob, err_word
  double *h_red = nullptr;        // totals of a reduction, written by the device
  cudaStream_t own_stream = nullptr, stream = nullptr;
  int64_t launches = 0;
  int nsm = 0;                    // SMs of the device
  const void *prev_fn = nullptr;  // the last launch of launch_pdl
  int prev_resident = 0;
  bool use_pass2 = true;        // register-staged passes for pencils of 32..256 points
  // 2D and 3D grids of at most 8192 points with coupled components.  Boxes
  // this small hold so dense a field (dt g |psi|^2 of 0.5 and more) that a block
  // multiplies a rounding difference by up to 10^15, so their results are those
  // of one order of operations only; their potential passes, and their passes
  // over 4096 points, are the point-at-a-time ones (components meeting in
  // shared memory), which keep the order that these results have always had.
  // From 16384 points up FP64 rounding differences stay below 1e-10 over 200 steps.
  // What it costs, us a step: two components 64 x 64 12.1 (the warp-autonomous
  // pass 12.4), three 21.0 (register-staged 15.9), four 27.3 (18.2).
  bool dense = false;
  bool use_cluster1d = true;    // 1D blocks on a cluster of CTAs where that is faster
  bool use_tma = false;         // strided 256-point passes fed by TMA tile copies
  int *err_word = nullptr;      // error word of bounded waits (0: none)
  bool err_armed = false;       // a kernel that can set it ran since the last check
  long wait_limit = 1L << 22;   // TMA tile waits: try_wait rounds (atus_set_wait_limits)
  int drop_copies = 0;          // TMA passes issue no copies (error-path tests)
  int bragg_stable = 0;         // FP64 Bragg step in the eigenvalue-free form
  std::string err;
  // Sobolev state
  bool sob_ready = false;
  void *sob_lap[MAXC] = {}, *sob_psi[MAXC] = {}, *sob_grad[MAXC] = {};
  double sob_alpha[MAXC] = {};
  double stepsize = 0;
  void *sob_dev = nullptr;              // SobDev in device memory
  cudaGraphExec_t sob_graph = nullptr;  // a chunk of device-side iterations
  double sob_graph_step = 0;            // stepsize the graph was captured with
  void *h_sob = nullptr;                // pinned host copy of the SobDev
  // 1D fields longer than the longest pass (four-step transforms): the field
  // viewed as fs_n1 x fs_n2 (n = fs_n2 * n1 + n2), W_N^m for m < N, and a
  // second N-point FP64 buffer for reordering spectra into natural k order
  int64_t fs_n1 = 0, fs_n2 = 0;
  double2 *fs_tw = nullptr;
  void *fs_tmp = nullptr;
  double *blk_F = nullptr;              // pulse amplitudes of a 1D block (blk_F_n doubles)
  int blk_F_n = 0;
  // asynchronous output snapshots
  void *snap = nullptr;                 // ncomp x N complex128 staging copy
  cudaStream_t copy_stream = nullptr;   // its device->host copies
  cudaEvent_t snap_taken = nullptr;     // the staging copy is complete
  cudaEvent_t snap_read = nullptr;      // the last host copy from it is complete
};

// ------------------------------------------------------------------ errors
static inline int fail(atus_ctx *c, int code, const std::string &msg) {
  if (c) c->err = msg;
  return code;
}
static inline int cuda_check(atus_ctx *c, cudaError_t e, const char *what) {
  if (e == cudaSuccess) return ATUS_OK;
  return fail(c, ATUS_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
#define CK(call)                                           \
  do {                                                     \
    int _r = cuda_check(ctx, (call), #call);               \
    if (_r != ATUS_OK) return _r;                          \
  } while (0)
#define LAUNCHED(ctx)                                                     \
  do {                                                                    \
    (ctx)->launches++;                                                    \
    int _r = cuda_check((ctx), cudaGetLastError(), "kernel launch");      \
    if (_r != ATUS_OK) return _r;                                         \
  } while (0)


// Launch on the context's stream, allowed to overlap the end of the kernel
// before it (pdl_wait in kernels.cuh) where that is safe for its occupancy:
//  - the grid fills at most half of the places the device has for it
//    (resident CTAs on each of nsm SMs), or
//  - it or its predecessor takes one CTA per SM, or both are the same kernel.
// Elsewhere its first CTAs land between those of the predecessor still
// running, with another footprint, and when they are gone the holes left
// between do not hold the last ones: a persistent grid then runs in two waves
// (256^3 x 2 FP64 block 10.4 -> 11.8 ms, 128^3 descent 10.9 -> 12.0 ms with
// every launch overlapped).
template <typename... P, typename... A>
static inline cudaError_t launch_pdl(atus_ctx *ctx, void (*kernel)(P...), int nsm, int resident, unsigned grid,
                                     unsigned threads, size_t smem, A &&...args) {
  const void *fn = reinterpret_cast<const void *>(kernel);
  const bool overlap = 2 * (int64_t)grid <= (int64_t)nsm * resident || resident == 1 || ctx->prev_resident == 1 ||
                       ctx->prev_fn == fn;
  ctx->prev_fn = fn;
  ctx->prev_resident = resident;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

static inline Geo geo(const atus_ctx *ctx) {
  Geo g;
  for (int a = 0; a < 3; a++) g.lg[a] = ctx->lg[a];
  g.npts = ctx->npts;
  return g;
}

