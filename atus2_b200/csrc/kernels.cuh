// kernels.cuh -- split-step kernels of the ATUS-2 engine (sm_100a).
//
// Fields live in HBM as one contiguous array per component, row-major with x
// slowest (the .bin layout): complex128 in FP64 mode, complex64 in mixed mode.
//
// pass_kernel  one HBM read and one HBM write of a tile of pencils along one
//              axis: [transform] -> point-wise operator -> [transform].  Used
//              as  FFT_a -> kinetic phase -> IFFT_a   (k-space half-step) and
//              IFFT_a -> potential/Bragg step -> FFT_a (real-space half-step),
//              so each Strang step of a 2D grid is two passes over the fields.
// block1d_kernel  1D grids of 2..128 points: a whole Strang block (Nk steps) with
//              the field resident in shared memory (longer ones: line1d.cuh).
// nl_kernel    the potential step alone (Do_NL_Step / Do_Bragg_ad).
// reduce_*     deterministic two-level FP64 reductions.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "fft_device.cuh"

namespace atus {

constexpr int MAXC = 4;
constexpr int TWN = 16384;  // twiddle table length (largest supported pencil)

// Per-CTA tile budget in complex elements and threads per CTA.
template <typename R> struct Tile;
// MINB: CTAs per SM the register budget is sized for (two tiles resident per
// SM, so one CTA's loads overlap the other's transforms).
template <> struct Tile<double> { static constexpr int E = 2048; static constexpr int NT = 128; static constexpr int MINB = 3; };
template <> struct Tile<float> { static constexpr int E = 4096; static constexpr int NT = 256; static constexpr int MINB = 3; };

constexpr int BLOCK1D_NT = 256;  // threads of the resident 1D Strang-block kernel

enum { T_NONE = 0, T_FWD = -1, T_INV = 1 };
enum { OP_NONE = 0, OP_KIN = 1, OP_NL = 2, OP_FILT = 3 };
enum { FILT_SOBOLEV = 0, FILT_LAPLACE = 1 };
// step kinds: CRT_Base freeprop, CRT_Base_IF freeprop, bragg_ad, the
// three-level bragg_ad (double_bragg), CRT_Base_IF_2 freeprop (two species),
// the two-species bragg_ad (bragg_ds), and the numerical n-state "bragg" and
// three-state "raman" steps of CRT_Base_IF
enum { K_NL = 0, K_NL_IF = 1, K_BRAGG = 2, K_DBRAGG = 3, K_NL_IF2 = 4, K_BRAGG_DS = 5, K_NUM_BRAGG = 6, K_RAMAN = 7 };
// modes of the register-staged pass kernel (pass2.cuh)
// M2_KIN_RABI: M2_KIN that also sums |psi^(k)|^2 over the Rabi balls of the
// requested components while every axis is in k-space (the last kinetic pass
// of a block); a separate instantiation, so M2_KIN keeps its registers.
// M2_FWD_SOB, M2_INV_SOB: the first and the last pass of a Sobolev iteration
// (the transform of psi and W psi straight from psi; the inverse transform of
// S psi and S(W psi) with their products with psi).
// M2_FILT: FFT, Sobolev or Laplace filter, IFFT (apart from M2_KIN, whose
// complex64 x pass went from 160 to 170 us on 256^3 x 2 with both in one).
// M2_NL_MEET: M2_NL of two components that meet in shared memory, a point at a
// time (atus_ctx::dense).
// M2_FS_*: the passes of a long 1D axis seen as n1 x n2 points (four-step
// transforms), the twiddles W_N^{r c} applied in registers:
//   M2_FS_FWD  strided axis: FFT, twiddles
//   M2_FS_NL   strided axis: IFFT, potential step, FFT, twiddles
//   M2_FS_KIN  contiguous axis: FFT, kinetic factor, IFFT, conjugate twiddles
enum { M2_FWD = 0, M2_INV = 1, M2_KIN = 2, M2_NL = 3, M2_KIN_RABI = 4, M2_FWD_SOB = 5, M2_INV_SOB = 6,
       M2_FS_FWD = 7, M2_FS_NL = 8, M2_FS_KIN = 9, M2_FILT = 10, M2_NL_MEET = 11 };

struct LaserD {
  double beta0, DeltaL[MAXC], Amp0, laser_k0, laser_dk0, laser_domh0, phase0, chirp_rate0, chirp;
  double Amp1;  // second amplitude (Amp_1 entry 1), used by the numerical steps
};

// Potential-step parameters (by value).
struct NLArgs {
  int kind;                 // K_NL / K_NL_IF / K_BRAGG
  int ncomp;
  double mdt;               // -dt
  double dt;
  double gs[MAXC * MAXC];   // gs[i * MAXC + j] = g_ij (GS_(i+1) entry j)
  const double *V[MAXC];    // nullptr: no potential
  LaserD L;
  double t1;                // header t + dt/2
  double F;                 // pulse amplitude
  double dx0;               // grid step of axis 0
  int shift0;               // n0 / 2
  int stable;               // FP64 Bragg step in the eigenvalue-free form (1) or the reference's (0)
  // three-level Bragg step: beta . x over every axis (grid steps, centres and
  // log2 lengths of axes 1 and 2 to recover y and z from the grid index)
  double beta1, beta2, dx1, dx2;
  int shift1, shift2, lg1, lg2;
  // second species of the two-species programs (beta0, Amp0, laser_k0,
  // laser_dk0, laser_domh0, phase0, chirp_rate0 used) and its pulse factor
  LaserD L2;
  double F2;
  double th;  // header time at the potential step (the numerical "bragg" step's t1)
};

// Programmatic dependent launch: a pass may be launched before the kernel it
// depends on has ended, prepares its tables, and waits here until that
// kernel's writes are visible; then it lets its own successor be launched.
// (Without the launch attribute both are no-ops.)  Nothing that a kernel
// writes may be touched before.  Worth it where passes are short and a launch
// waits for the last CTAs of the one before: ten steps of 2^20 points 462 ->
// 410 us, twenty of 512 x 256 x 3 603 -> 502; none on 64^3 x 2 (391 -> 393),
// whose launches follow one another without a gap.
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct Geo {
  int lg[3];                // log2 of n0, n1, n2 (unused axes: 0)
  int64_t npts;
};

struct PassArgs {
  void *psi[MAXC];
  int nc;                   // components in the tile (NL) or 1 (per-component passes)
  int per_comp;             // 1: blockIdx.y selects the component
  int64_t sa;               // pencil stride in elements
  int64_t inner_tiles;      // strided: tiles per outer block; contiguous: unused
  int64_t npencils;         // contiguous: number of pencils
  int64_t ntiles;           // tiles per component
  int ncomp_grid;           // components walked by per-component passes
  int t1, op, t2;
  const double2 *kt[MAXC][3];  // kinetic phase factors per component and axis (FP64)
  double s_f, s_b;          // forward / backward transform scales (cft_*d::scale)
  const void *tw;           // twiddles exp(-2 pi i m / TWN)
  Geo g;
  NLArgs nl;
  int x_along;              // 1 when the pencil runs along axis 0 (x varies inside a pencil)
  int axis;                 // axis the pencils run along
  const double2 *fs_tw;     // M2_FS_*: W_N^{r c} at grid index r n2 + c
  // OP_FILT: real k-space filter of CSOB_Base (include/CSOB_Base.h:228-248):
  // 1/(1 + alpha k^2) or -alpha k^2, times the transform scale.
  int filt_mode;
  double filt_alpha, filt_scale;
  int filt_batch;  // 1 + alpha k^2 of four points multiplies without overflow
  double dk[3];
  int n[3];
  // M2_KIN_RABI: balls k0[c * rabi_n + m] (m < rabi_n) of component
  // rabi_comp[c] (c < rabi_ncomp), radius rabi_thr; sums of the unscaled
  // |psi^|^2 to rabi_out (red_finish with rabi_partial and rabi_count)
  int rabi_ncomp, rabi_n;
  int rabi_comp[2];
  double rabi_thr;
  double rabi_k0[8][3];
  double *rabi_partial, *rabi_out;
  unsigned *rabi_count;
  // M2_FWD_SOB / M2_INV_SOB: the components' fields, the one this pass works
  // for and its interaction row (potential: nl.V[0]); sums to rabi_out
  const double2 *sob_psi[MAXC];
  int sob_comp, sob_ncomp;
  double sob_gs[MAXC];
  int *err;  // error word, mapped host memory (a bounded wait that ran out sets it)
  long wait_limit;       // try_wait rounds before a TMA tile counts as lost
  int drop_copies;       // issue no tile copies, so every wait runs out (error-path tests; 0)
};

// kt[c][0] without an indexed copy of the parameter array.
__device__ __forceinline__ const double2 *pick_kt0(const PassArgs &a, int c) {
  const double2 *k = a.kt[0][0];
  #pragma unroll
  for (int i = 1; i < MAXC; i++)
    if (c == i) k = a.kt[i][0];
  return k;
}

__device__ __forceinline__ void idx3(const Geo &g, int64_t l, int &ix, int &iy, int &iz) {
  ix = (int)(l >> (g.lg[1] + g.lg[2]));
  iy = (int)((l >> g.lg[2]) & ((1 << g.lg[1]) - 1));
  iz = (int)(l & ((1 << g.lg[2]) - 1));
}

// ------------------------------------------------------------ phase helpers
// a - 2 pi rint(a / 2 pi), Cody-Waite with 2 pi = P1 + P2 (+P3), P1 with 32
// significant bits so q*P1 is exact for |q| < 2^20.
__device__ __forceinline__ double reduce_2pi(double a) {
  const double P1 = 6.2831853069365025, P2 = 2.430840202602477e-10, P3 = 1.40862394607328e-26;
  const double q = rint(a * 0.15915494309189535);
  double r = fma(-q, P1, a);
  r = fma(-q, P2, r);
  return fma(-q, P3, r);
}

// v with its sign bits flipped by mask sg (0 or 0x80000000).
__device__ __forceinline__ double flip1(double x, int sg) {
  return __hiloint2double(__double2hiint(x) ^ sg, __double2loint(x));
}
__device__ __forceinline__ float flip1(float x, int sg) { return __int_as_float(__float_as_int(x) ^ sg); }
template <typename C> __device__ __forceinline__ C flip(C v, int sg) {
  v.x = flip1(v.x, sg);
  v.y = flip1(v.y, sg);
  return v;
}

// e^{i x} for |x| < 2^17: x - q pi/2 by Cody and Waite's reduction (the parts
// of 2 pi above, over 4; q P1 is exact), then Taylor series on |r| <= pi/4 --
// sin to r^17, cos to r^16, truncation below 1e-19 and 2e-18 -- and the
// quadrant.  No branch, 30
// FP64 operations.
__device__ __forceinline__ double2 expi_cw(double x) {
  constexpr double P1 = 6.2831853069365025 / 4, P2 = 2.430840202602477e-10 / 4, P3 = 1.40862394607328e-26 / 4;
  const double q = rint(x * 0.63661977236758134308);
  const int n = __double2int_rn(q);
  double r = fma(-q, P1, x);
  r = fma(-q, P2, r);
  r = fma(-q, P3, r);
  const double r2 = r * r;
  double ps = fma(r2, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);
  ps = fma(ps, r2, 1.0 / 6227020800.0);
  ps = fma(ps, r2, -1.0 / 39916800.0);
  ps = fma(ps, r2, 1.0 / 362880.0);
  ps = fma(ps, r2, -1.0 / 5040.0);
  ps = fma(ps, r2, 1.0 / 120.0);
  ps = fma(ps, r2, -1.0 / 6.0);
  const double sn = fma(ps * r2, r, r);
  double pc = fma(r2, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
  pc = fma(pc, r2, 1.0 / 479001600.0);
  pc = fma(pc, r2, -1.0 / 3628800.0);
  pc = fma(pc, r2, 1.0 / 40320.0);
  pc = fma(pc, r2, -1.0 / 720.0);
  pc = fma(pc, r2, 1.0 / 24.0);
  pc = fma(pc, r2, -0.5);
  const double cs = fma(pc, r2, 1.0);
  const double c = (n & 1) ? sn : cs, s = (n & 1) ? cs : sn;
  return make_double2(flip1(c, ((n + 1) & 2) << 30), flip1(s, (n & 2) << 30));
}

// sincos() out of line: the step kernels call it from 8 or 16 places each, for
// arguments that a resolved time step rarely has, and its inlined copies cost
// the common path registers.
static __device__ __noinline__ double2 sincos_far(double x) {
  double s, c;
  sincos(x, &s, &c);
  return make_double2(c, s);
}

// sin and cos of an FP64 argument.  The phases of a time step are small
// (|dt V| << 1 in practice), so |x| <= 1/32 takes the series; larger
// arguments call sincos().
// (cos, sin) by Taylor series to x^8 (cos) and x^7 (sin): the first omitted
// terms, x^10/10! and x^9/9!, are below 2.5e-22 and 2.5e-18 x for |x| <= 1/32.
__device__ __forceinline__ double2 expi_series(double x) {
  const double x2 = x * x;
  double ps = fma(x2, -1.0 / 5040.0, 1.0 / 120.0);
  ps = fma(ps, x2, -1.0 / 6.0);
  double pc = fma(x2, 1.0 / 40320.0, -1.0 / 720.0);
  pc = fma(pc, x2, 1.0 / 24.0);
  pc = fma(pc, x2, -0.5);
  return make_double2(fma(pc, x2, 1.0), fma(ps * x2, x, x));
}
__device__ __forceinline__ void sincos_step(double x, double *s, double *c) {
  if (fabs(x) <= 0.03125) {
    // Taylor series to x^7 (sin) and x^8 (cos): the first omitted terms,
    // x^9/9! and x^10/10!, are below 2.5e-18 x and 2.5e-22 for |x| <= 1/32
    const double x2 = x * x;
    double ps = fma(x2, -1.0 / 5040.0, 1.0 / 120.0);
    ps = fma(ps, x2, -1.0 / 6.0);
    *s = fma(ps * x2, x, x);
    double pc = fma(x2, 1.0 / 40320.0, -1.0 / 720.0);
    pc = fma(pc, x2, 1.0 / 24.0);
    pc = fma(pc, x2, -0.5);
    *c = fma(pc, x2, 1.0);
  } else {
    sincos(x, s, c);
  }
}

// The same with its far arguments out of line (FAR), or not.
template <bool FAR> __device__ __forceinline__ void sincos_step_t(double x, double *s, double *c) {
  if constexpr (FAR) {
    const double2 e = fabs(x) <= 0.03125 ? expi_series(x) : sincos_far(x);
    *c = e.x;
    *s = e.y;
  } else {
    sincos_step(x, s, c);
  }
}

// Element of MAXC-entry arrays by a runtime index without local memory.
template <typename T> __device__ __forceinline__ T pick(const T (&a)[MAXC], int i) {
  T r = a[0];
  if (i == 1) r = a[1];
  if (i == 2) r = a[2];
  if (i == 3) r = a[3];
  return r;
}

template <typename R> __device__ __forceinline__ double2 to_d(cplx<R> v) { return make_double2((double)v.x, (double)v.y); }
template <typename R> __device__ __forceinline__ cplx<R> from_d(double2 v) { return mk<R>((R)v.x, (R)v.y); }

// Unit phase factor e^{i phi} in FP64.  Mixed precision: FP64 argument
// reduced modulo 2 pi, sincosf, then renormalised in FP64 so that |e| = 1 to
// FP64 accuracy (a fixed modulus error would drift the norm every step).
template <typename R> __device__ __forceinline__ double2 expi(double phi);
template <> __device__ __forceinline__ double2 expi<double>(double phi) {
  double s, c;
  sincos_step(phi, &s, &c);
  return make_double2(c, s);
}
template <> __device__ __forceinline__ double2 expi<float>(double phi) {
  if (fabs(phi) <= 0.03125) {  // the usual phase of one time step: FP64 Taylor, |e| = 1 to FP64
    double sd, cd;
    sincos_step(phi, &sd, &cd);
    return make_double2(cd, sd);
  }
  float s, c;
  sincosf((float)reduce_2pi(phi), &s, &c);
  const double cd = c, sd = s;
  const double inv = rsqrt(cd * cd + sd * sd);
  return make_double2(cd * inv, sd * inv);
}
// The same with its far arguments out of line.
static __device__ __noinline__ double2 expi_far_mixed(double phi) { return expi<float>(phi); }
template <typename R> __device__ __forceinline__ double2 expi_f(double phi) {
  if (fabs(phi) <= 0.03125) return expi_series(phi);
  if constexpr (sizeof(R) == 8) return sincos_far(phi);
  else return expi_far_mixed(phi);
}

// ------------------------------------------------------------ couplings
// What a step's coupling takes from x alone (and the step's time): the same
// for every point of a pencil that does not run along x, so the passes
// evaluate it once a pencil instead of once a point.
//   K_DBRAGG    Omega_+, Omega_-, cos, sin of -dk x / 2
//   K_BRAGG_DS  per species Omega_s, cos, sin of -(dk_s x + phase_s) / 2
//   K_RAMAN     cos, sin of k x
//   K_NUM_BRAGG per upper state cos, sin of (-domh + rate_i t) t + k_i x - phase / 2
constexpr int NCPL = 6;
__device__ __forceinline__ void coupling_x(const NLArgs &a, double x0, double *cp) {
  const double t1 = a.t1;
  if (a.kind == K_DBRAGG) {
    const double F = a.F < 0 ? 0.0 : a.F;
    double dw = a.L.laser_domh0 + a.L.chirp_rate0 * t1;
    cp[0] = F * a.L.Amp0 * cos(a.L.laser_k0 * x0 - dw * t1 - a.L.phase0 / 2);
    dw = a.L.laser_domh0 - a.L.chirp_rate0 * t1;
    cp[1] = F * a.L.Amp0 * cos(-a.L.laser_k0 * x0 - dw * t1 - a.L.phase0 / 2);
    sincos(-0.5 * a.L.laser_dk0 * x0, &cp[3], &cp[2]);
  } else if (a.kind == K_BRAGG_DS) {
    #pragma unroll
    for (int s = 0; s < 2; s++) {
      const LaserD &L = s ? a.L2 : a.L;
      cp[3 * s] = (s ? a.F2 : a.F) * L.Amp0 *
                  cos(L.laser_k0 * x0 - (L.laser_domh0 + L.chirp_rate0 * t1) * t1 + L.phase0 / 2);
      sincos(-0.5 * (L.laser_dk0 * x0 + L.phase0), &cp[3 * s + 2], &cp[3 * s + 1]);
    }
  } else if (a.kind == K_RAMAN) {
    sincos(a.L.laser_k0 * x0, &cp[1], &cp[0]);
  } else if (a.kind == K_NUM_BRAGG) {
    const double th = a.th;
    #pragma unroll
    for (int i = 0; i < 2; i++) {
      const double k = i == 0 ? a.L.laser_k0 : -a.L.laser_k0;
      const double rate = i == 0 ? a.L.chirp_rate0 : -a.L.chirp_rate0;
      sincos((-a.L.laser_domh0 + rate * th) * th + k * x0 - 0.5 * a.L.phase0, &cp[2 * i + 1], &cp[2 * i]);
    }
  }
}

// ------------------------------------------------------------ three-level Bragg step
// Bragg_double::Do_Double_Bragg_ad (source/interferometry/src/double_bragg.cpp:
// 123-256) at grid index l: state 1 (component 0) couples to states 2 and 3
// with Omega_+ = F Amp cos(k x - (domh + rate t1) t1 - phase/2) and Omega_- =
// F Amp cos(-k x - (domh - rate t1) t1 - phase/2); states 2 and 3 share V22;
// V includes beta . x over all axes.  The reference's operation order,
// including its O32 update that reads the already-updated O23 imaginary part
// (double_bragg.cpp:233).  FP64 arithmetic for both field precisions.
// CP: cp holds Omega_+, Omega_-, cos and sin of -dk x / 2 (coupling_x).
template <typename R, bool CP>
__device__ __forceinline__ void dbragg_point(const NLArgs &a, cplx<R> *v, int64_t l, double x0, const double *cp) {
  double bx = a.L.beta0 * x0;
  if (a.lg1 > 0) {
    const int iy = (int)((l >> a.lg2) & ((1 << a.lg1) - 1));
    bx += a.beta1 * ((double)(iy - a.shift1) * a.dx1);
  }
  if (a.lg2 > 0) {
    const int iz = (int)(l & ((1 << a.lg2) - 1));
    bx += a.beta2 * ((double)(iz - a.shift2) * a.dx2);
  }
  const double2 p1 = to_d<R>(v[0]), p2 = to_d<R>(v[1]), p3 = to_d<R>(v[2]);
  double tmp1 = p1.x * p1.x + p1.y * p1.y;
  double tmp2 = p2.x * p2.x + p2.y * p2.y;
  const double tmp3 = p3.x * p3.x + p3.y * p3.y;
  const double *gs = a.gs;  // padded rows: g_ij at i * MAXC + j
  const double V11 = gs[0] * tmp1 + gs[1] * tmp2 + gs[2] * tmp3 + bx;
  const double V22 = gs[MAXC] * tmp1 + gs[MAXC + 1] * tmp2 + gs[MAXC + 2] * tmp3 - a.L.DeltaL[1] + bx;
  const double t1 = a.t1, dt = a.dt;
  double Op, Om;
  if constexpr (CP) {
    Op = cp[0];
    Om = cp[1];
  } else {
    const double F = a.F < 0 ? 0.0 : a.F;
    double dw = a.L.laser_domh0 + a.L.chirp_rate0 * t1;
    Op = F * a.L.Amp0 * cos(a.L.laser_k0 * x0 - dw * t1 - a.L.phase0 / 2);
    dw = a.L.laser_domh0 - a.L.chirp_rate0 * t1;
    Om = F * a.L.Amp0 * cos(-a.L.laser_k0 * x0 - dw * t1 - a.L.phase0 / 2);
  }
  double re1, im1;
  if (Om == 0.0 && Op == 0.0) {
    sincos_step_t<CP>(-dt * V11, &im1, &re1);
    v[0] = from_d<R>(cmul(p1, make_double2(re1, im1)));
    sincos_step_t<CP>(-dt * V22, &im1, &re1);
    v[1] = from_d<R>(cmul(p2, make_double2(re1, im1)));
    v[2] = from_d<R>(cmul(p3, make_double2(re1, im1)));
    return;
  }
  double e0, e1;
  if constexpr (CP) {
    e0 = cp[2];
    e1 = cp[3];
  } else {
    sincos(-0.5 * a.L.laser_dk0 * x0, &e1, &e0);
  }
  const double OO = Op * Op + Om * Om;
  tmp1 = sqrt((V11 - V22) * (V11 - V22) + 4.0 * OO);
  const double E1 = 0.5 * (V11 + V22 + tmp1);
  const double E2 = 0.5 * (V11 + V22 - tmp1);
  double2 g1, g2, g3;
  sincos_step_t<CP>(-dt * E1, &im1, &re1);
  tmp1 = 1.0 / fabs((V22 - E1) * (V22 - E1) + Op * Op + Om * Om);
  g1 = make_double2(tmp1 * re1, tmp1 * im1);
  sincos_step_t<CP>(-dt * E2, &im1, &re1);
  tmp1 = 1.0 / fabs((V22 - E2) * (V22 - E2) + Op * Op + Om * Om);
  g2 = make_double2(tmp1 * re1, tmp1 * im1);
  sincos_step_t<CP>(-dt * V22, &im1, &re1);
  tmp1 = 1.0 / fabs(OO);
  g3 = make_double2(tmp1 * re1, tmp1 * im1);
  tmp1 = (V22 - E2) * (V22 - E2);
  tmp2 = (V22 - E1) * (V22 - E1);
  const double2 O11 = make_double2(tmp1 * g2.x + tmp2 * g1.x, tmp1 * g2.y + tmp2 * g1.y);
  tmp1 = (V22 - E2) * g2.x + (V22 - E1) * g1.x;
  tmp2 = (V22 - E2) * g2.y + (V22 - E1) * g1.y;
  const double2 A12 = make_double2(-Op * tmp1, -Op * tmp2);  // O12 = O21 before eta
  const double2 A13 = make_double2(-Om * tmp1, -Om * tmp2);  // O13 = O31 before eta
  const double2 O12 = make_double2(e0 * A12.x - e1 * A12.y, e1 * A12.x + e0 * A12.y);
  const double2 O21 = make_double2(e0 * A12.x + e1 * A12.y, e0 * A12.y - e1 * A12.x);
  const double2 O31 = make_double2(e0 * A13.x - e1 * A13.y, e1 * A13.x + e0 * A13.y);
  const double2 O13 = make_double2(e0 * A13.x + e1 * A13.y, e0 * A13.y - e1 * A13.x);
  tmp1 = Op * Op;
  tmp2 = Om * Om;
  const double2 O22 = make_double2(tmp1 * (g2.x + g1.x) + tmp2 * g3.x, tmp1 * (g2.y + g1.y) + tmp2 * g3.y);
  const double2 O33 = make_double2(tmp2 * (g2.x + g1.x) + tmp1 * g3.x, tmp2 * (g2.y + g1.y) + tmp1 * g3.y);
  tmp1 = Om * Op;
  const double2 A23 = make_double2(tmp1 * (g1.x + g2.x - g3.x), tmp1 * (g1.y + g2.y - g3.y));
  const double ep = e0 * e0 + e1 * e1, em = e0 * e0 - e1 * e1, e2 = 2 * e0 * e1;
  const double2 O23 = make_double2(ep * A23.x + e2 * A23.y, ep * A23.y - e2 * A23.x);
  const double2 O32 = make_double2(em * A23.x - e2 * A23.y, em * O23.y + e2 * A23.x);
  v[0] = from_d<R>(cadd(cadd(cmul(O11, p1), cmul(O12, p2)), cmul(O13, p3)));
  v[1] = from_d<R>(cadd(cadd(cmul(O21, p1), cmul(O22, p2)), cmul(O23, p3)));
  v[2] = from_d<R>(cadd(cadd(cmul(O31, p1), cmul(O32, p2)), cmul(O33, p3)));
}

// ------------------------------------------------------------ two-level exponential
// exp(-i dt [[V11, Omega eta], [Omega conj(eta), V22]]) applied to (p1, p2).
// FP64 and not `stable`: the reference's eigenvalue form (bragg.cpp:226-302,
// bragg_ds.cpp:215-248): E+- = (V11 + V22 +- sqrt((V11 - V22)^2 + 4 Omega^2))/2,
// gamma+- = e^{-i dt E+-} / |(V11 - E+-)^2 + Omega^2|, pure phases when
// Omega == 0.  Its error, about 2^-53 |V| / |Omega|, is part of what a caller
// of this form gets: on small dense grids (dt V of 1 and more) the nonlinear
// step multiplies a difference by 10 to 1000 a block, so that another form of
// the same map, however exact, ends elsewhere.  Otherwise the eigenvalue-free
// form
//   U = e^{-i dt m} [cos(r dt) I - i sin(r dt)/r [[d, W], [W, -d]]],
// m = (V11+V22)/2, d = (V11-V22)/2, W = Omega, r = sqrt(d^2 + W^2), built in
// FP64 from unit (cos, sin) pairs, so it is unitary to FP64 accuracy for every
// Omega (the eigenvalue form divides by (V11 - E)^2 + Omega^2, which loses
// unitarity once Omega is below the spacing of V and divides by zero once
// Omega^2 underflows).
template <bool FAR>
__device__ __forceinline__ void bragg_eigen(double dt, double V11, double V22, double Omega, double eta_c, double eta_s,
                                            double2 &q1, double2 &q2) {
  double re1, im1;
  if (Omega == 0.0) {
    sincos_step_t<FAR>(-dt * V11, &im1, &re1);
    q1 = cmul(q1, make_double2(re1, im1));
    sincos_step_t<FAR>(-dt * V22, &im1, &re1);
    q2 = cmul(q2, make_double2(re1, im1));
    return;
  }
  double tmp1 = sqrt((V11 - V22) * (V11 - V22) + 4.0 * Omega * Omega);
  const double Ep = 0.5 * (V11 + V22 + tmp1);
  const double Em = 0.5 * (V11 + V22 - tmp1);
  double2 gp, gm;
  // the reference's 1 / |(V11 - E+-)^2 + Omega^2| (sums of squares, so
  // |.| is the identity) from one division: 1/A = B/(AB), 1/B = A/(AB)
  const double Ap = (V11 - Ep) * (V11 - Ep) + Omega * Omega;
  const double Am = (V11 - Em) * (V11 - Em) + Omega * Omega;
  const double inv = 1.0 / (Ap * Am);
  sincos_step_t<FAR>(-dt * Ep, &im1, &re1);
  tmp1 = Am * inv;
  gp = make_double2(tmp1 * re1, tmp1 * im1);
  sincos_step_t<FAR>(-dt * Em, &im1, &re1);
  tmp1 = Ap * inv;
  gm = make_double2(tmp1 * re1, tmp1 * im1);
  const double O2 = Omega * Omega;
  const double2 O11 = make_double2(O2 * (gp.x + gm.x), O2 * (gp.y + gm.y));
  const double a1 = V11 - Ep, a2 = V11 - Em;
  const double2 O22 = make_double2(a1 * a1 * gp.x + a2 * a2 * gm.x, a1 * a1 * gp.y + a2 * a2 * gm.y);
  const double2 Os = make_double2(-Omega * (a1 * gp.x + a2 * gm.x), -Omega * (a1 * gp.y + a2 * gm.y));
  const double2 eta = make_double2(eta_c, eta_s);
  const double2 O12 = cmul(Os, eta);   // eta * O12
  const double2 O21 = cmulc(Os, eta);  // conj(eta) * O21
  const double2 p1 = q1, p2 = q2;
  q1 = cadd(cmul(O11, p1), cmul(O12, p2));
  q2 = cadd(cmul(O21, p1), cmul(O22, p2));
}

template <typename R>
__device__ __forceinline__ void bragg_pair(int stable, double dt, double V11, double V22, double Omega, double eta_c,
                                           double eta_s, cplx<R> &q1, cplx<R> &q2) {
  if constexpr (sizeof(R) == 8) {
    if (!stable) {
      bragg_eigen<false>(dt, V11, V22, Omega, eta_c, eta_s, q1, q2);
      return;
    }
  }
  const double m = 0.5 * (V11 + V22), d = 0.5 * (V11 - V22);
  const double r = sqrt(d * d + Omega * Omega);
  const double2 e = expi<R>(-dt * m);   // e^{-i dt m}
  const double2 rr = expi<R>(dt * r);   // (cos r dt, sin r dt)
  // sin(r dt) / r: Taylor series of sinc (truncation below 2^-72 for r dt <= 1/32)
  const double xr = dt * r;
  double sor;
  if (xr <= 0.03125) {
    const double x2 = xr * xr;
    double p = fma(x2, 1.0 / 362880.0, -1.0 / 5040.0);
    p = fma(p, x2, 1.0 / 120.0);
    p = fma(p, x2, -1.0 / 6.0);
    sor = dt * fma(p, x2, 1.0);
  } else {
    sor = rr.y / r;
  }
  const double fd = sor * d, fw = sor * Omega;
  // U11 = e(cos - i fd), U22 = e(cos + i fd), Uoff = e(-i fw)
  const double2 U11 = cmul(e, make_double2(rr.x, -fd));
  const double2 U22 = cmul(e, make_double2(rr.x, fd));
  const double2 Uo = cmul(e, make_double2(0.0, -fw));
  const double2 et = make_double2(eta_c, eta_s);
  const double2 U12 = cmul(Uo, et), U21 = cmulc(Uo, et);
  const double2 p1 = to_d<R>(q1), p2 = to_d<R>(q2);
  q1 = from_d<R>(cadd(cmul(U11, p1), cmul(U12, p2)));
  q2 = from_d<R>(cadd(cmul(U21, p1), cmul(U22, p2)));
}

template <typename R>
__device__ __noinline__ void bragg_stable_far(double dt, double V11, double V22, double Omega, double eta_c,
                                              double eta_s, double2 p1, double2 p2, double2 *o1, double2 *o2) {
  cplx<R> a = from_d<R>(p1), b = from_d<R>(p2);  // exact: they come from fields of this type
  bragg_pair<R>(1, dt, V11, V22, Omega, eta_c, eta_s, a, b);
  *o1 = to_d<R>(a);
  *o2 = to_d<R>(b);
}

// The eigenvalue-free form for x^2 = (r dt)^2 = x2 <= 2^-10, e = e^{-i dt m}:
// cos x and sin x / x are even in x, so they are short Taylor series in x^2
// and the step needs no square root and no division.  Truncation below 2.5e-22
// (cos, to x^8) and 2.6e-23 (sin x / x, to x^8).
template <typename R>
__device__ __forceinline__ void bragg_series(double dt, double x2, double d, double Omega, double2 e, double eta_c,
                                             double eta_s, cplx<R> &q1, cplx<R> &q2) {
  const double2 p1 = to_d<R>(q1), p2 = to_d<R>(q2);
  double ps = fma(x2, 1.0 / 362880.0, -1.0 / 5040.0);
  ps = fma(ps, x2, 1.0 / 120.0);
  ps = fma(ps, x2, -1.0 / 6.0);
  const double s = dt * fma(ps, x2, 1.0);  // sin(x) / r
  double pc = fma(x2, 1.0 / 40320.0, -1.0 / 720.0);
  pc = fma(pc, x2, 1.0 / 24.0);
  pc = fma(pc, x2, -0.5);
  const double c = fma(pc, x2, 1.0);
  const double fd = s * d, so = s * Omega;
  const double2 w = make_double2(so * eta_c, so * eta_s);
  // (c - i fd) p1 - i w p2 and (c + i fd) p2 - i conj(w) p1
  const double2 a = make_double2(c * p1.x + fd * p1.y + (w.x * p2.y + w.y * p2.x),
                                 c * p1.y - fd * p1.x - (w.x * p2.x - w.y * p2.y));
  const double2 b = make_double2(c * p2.x - fd * p2.y + (w.x * p1.y - w.y * p1.x),
                                 c * p2.y + fd * p2.x - (w.x * p1.x + w.y * p1.y));
  q1 = from_d<R>(cmul(e, a));
  q2 = from_d<R>(cmul(e, b));
}

// The same map for kernels that hold their fields in registers: the
// eigenvalue form with its far phases out of line; the eigenvalue-free form by
// series for a time step that resolves the coupling, and out of line beyond.
template <typename R>
__device__ __forceinline__ void bragg_pair_far(int stable, double dt, double V11, double V22, double Omega,
                                               double eta_c, double eta_s, cplx<R> &q1, cplx<R> &q2) {
  if constexpr (sizeof(R) == 8) {
    if (!stable) {
      bragg_eigen<true>(dt, V11, V22, Omega, eta_c, eta_s, q1, q2);
      return;
    }
  }
  const double m = 0.5 * (V11 + V22), d = 0.5 * (V11 - V22), O2 = Omega * Omega;
  const double x2 = (dt * dt) * (d * d + O2);
  if (x2 <= 0x1p-10) {
    bragg_series<R>(dt, x2, d, Omega, expi_f<R>(-dt * m), eta_c, eta_s, q1, q2);
    return;
  }
  double2 o1, o2;
  bragg_stable_far<R>(dt, V11, V22, Omega, eta_c, eta_s, to_d<R>(q1), to_d<R>(q2), &o1, &o2);
  q1 = from_d<R>(o1);
  q2 = from_d<R>(o2);
}

// ------------------------------------------------------------ two-species Bragg step
// Bragg_single::Do_Bragg_ad of the two-species program (source/interferometry/
// src/bragg_ds.cpp:111-322) at grid index l: components (0, 1) are species 1,
// (2, 3) species 2; V_i = sum_j g_ij |psi_j|^2 + (beta_s x - DeltaL_i) with
// beta_s of the component's species (x along axis 0 only); species s couples
// with Omega_s = F_s Amp_s cos(k_s x - (domh_s + rate_s t1) t1 + phase_s/2),
// eta_s = e^{-i (dk_s x + phase_s)/2}.  F_s is 0 outside the species' pulse
// window (bragg_ds.cpp:117-127), set on the host.
// CP: cp holds Omega_s, cos and sin of -(dk_s x + phase_s) / 2 per species
// (coupling_x).
template <typename R, bool CP>
__device__ __forceinline__ void bragg_ds_point(const NLArgs &a, cplx<R> *v, double x0, const double *cp) {
  double rho[MAXC];
  #pragma unroll
  for (int j = 0; j < MAXC; j++) rho[j] = (double)v[j].x * (double)v[j].x + (double)v[j].y * (double)v[j].y;
  double phi[MAXC];
  #pragma unroll
  for (int i = 0; i < MAXC; i++) {
    double p = a.gs[i * MAXC] * rho[0];
    #pragma unroll
    for (int j = 1; j < MAXC; j++) p += a.gs[i * MAXC + j] * rho[j];
    phi[i] = p + (((i < 2) ? a.L.beta0 : a.L2.beta0) * x0 - a.L.DeltaL[i]);
  }
  const double t1 = a.t1, dt = a.dt;
  #pragma unroll
  for (int s = 0; s < 2; s++) {
    if constexpr (CP) {
      bragg_pair_far<R>(a.stable, dt, phi[2 * s], phi[2 * s + 1], cp[3 * s], cp[3 * s + 1], cp[3 * s + 2], v[2 * s],
                        v[2 * s + 1]);
    } else {
      const LaserD &L = s ? a.L2 : a.L;
      const double Omega = (s ? a.F2 : a.F) * L.Amp0 *
                           cos(L.laser_k0 * x0 - (L.laser_domh0 + L.chirp_rate0 * t1) * t1 + L.phase0 / 2);
      double es, ec;
      sincos(-0.5 * (L.laser_dk0 * x0 + L.phase0), &es, &ec);
      bragg_pair<R>(a.stable, dt, phi[2 * s], phi[2 * s + 1], Omega, ec, es, v[2 * s], v[2 * s + 1]);
    }
  }
}

// ------------------------------------------------------------ numerical n-state steps
// psi <- exp(-i h A) psi for a Hermitian 3x3 matrix A (n = 2: the third row
// and column are zero and so is psi[2]).  The reference diagonalises A with
// GSL's gsl_eigen_hermv and forms V diag(e^{-i h lambda}) V^H psi
// (include/CRT_Base_IF.h:471-497, 581-607); here the same exponential comes
// from its Taylor series on the vector: the mean of the diagonal is taken out
// as a scalar phase, the rest is split into s substeps with
// h ||A||_inf / s <= 1/4 (||.||_inf bounded by |Re| + |Im| row sums), and each
// substep sums terms (-i h A / s)^k psi / k! until a term falls below 2^-60
// of the sum (k <= 18; the truncation error at k = 18 is below 1e-22).  No
// eigenvalues, so degenerate or nearly degenerate spectra need no care.
__device__ __forceinline__ void herm_expm_apply(double2 (&A)[3][3], int n, double h, double2 (&p)[3]) {
  double mu = 0.0;
  #pragma unroll
  for (int i = 0; i < 3; i++)
    if (i < n) mu += A[i][i].x;
  mu /= n;
  #pragma unroll
  for (int i = 0; i < 3; i++)
    if (i < n) A[i][i].x -= mu;
  double nu = 0.0;
  #pragma unroll
  for (int i = 0; i < 3; i++) {
    double r = 0.0;
    #pragma unroll
    for (int j = 0; j < 3; j++) r += fabs(A[i][j].x) + fabs(A[i][j].y);
    nu = fmax(nu, r);
  }
  nu *= h;
  int steps = 1;
  if (nu > 0.25) steps = (int)fmin(ceil(4.0 * nu), 1048576.0);
  const double hs = h / steps;
  // M = -i hs A
  double2 M[3][3];
  #pragma unroll
  for (int i = 0; i < 3; i++)
    #pragma unroll
    for (int j = 0; j < 3; j++) M[i][j] = make_double2(hs * A[i][j].y, -hs * A[i][j].x);
  constexpr double INVK[19] = {0.0,      1.0,       1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,
                               1.0 / 7,  1.0 / 8,   1.0 / 9,  1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13,
                               1.0 / 14, 1.0 / 15,  1.0 / 16, 1.0 / 17, 1.0 / 18};
  for (int st = 0; st < steps; st++) {
    double2 y[3] = {p[0], p[1], p[2]}, t[3] = {p[0], p[1], p[2]};
    #pragma unroll 1
    for (int k = 1; k <= 18; k++) {
      double2 u[3];
      #pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 acc = cmul(M[i][0], t[0]);
        acc = cadd(acc, cmul(M[i][1], t[1]));
        acc = cadd(acc, cmul(M[i][2], t[2]));
        u[i] = make_double2(acc.x * INVK[k], acc.y * INVK[k]);
      }
      double tn = 0.0, yn = 0.0;
      #pragma unroll
      for (int i = 0; i < 3; i++) {
        t[i] = u[i];
        y[i] = cadd(y[i], u[i]);
        tn += fabs(u[i].x) + fabs(u[i].y);
        yn += fabs(y[i].x) + fabs(y[i].y);
      }
      if (tn <= 0x1p-60 * yn) break;
    }
    p[0] = y[0];
    p[1] = y[1];
    p[2] = y[2];
  }
  double sn, cs;
  sincos_step(-h * mu, &sn, &cs);
  const double2 e = make_double2(cs, sn);
  #pragma unroll
  for (int i = 0; i < 3; i++) p[i] = cmul(p[i], e);
}

// beta . x over every axis at grid index l (x0 given; y and z from the index).
__device__ __forceinline__ double beta_dot_x(const NLArgs &a, int64_t l, double x0) {
  double bx = a.L.beta0 * x0;
  if (a.lg1 > 0) {
    const int iy = (int)((l >> a.lg2) & ((1 << a.lg1) - 1));
    bx += a.beta1 * ((double)(iy - a.shift1) * a.dx1);
  }
  if (a.lg2 > 0) {
    const int iz = (int)(l & ((1 << a.lg2) - 1));
    bx += a.beta2 * ((double)(iz - a.shift2) * a.dx2);
  }
  return bx;
}

// The numerical steps of CRT_Base_IF at grid index l (n = ncomp components):
// diagonal V_i = sum_j g_ij |psi_j|^2 + (beta . x - DeltaL_i);
//  "bragg" (Numerical_Bragg, include/CRT_Base_IF.h:426-526): state 0 couples
//   to state i+1 with eta_i = (Amp0 + Amp1)/2 cos(a_i) + i (Amp0 - Amp1)/2
//   sin(a_i), a_i = (-domh + rate_i t) t + k_i x - phase/2, k_1 = -k_0,
//   rate_1 = -rate_0, t the header time;
//  "raman" (Numerical_Raman, :533-632): V_2 + domh, A_02 = Amp0/2 e^{i k x},
//   A_12 = Amp1/2 e^{-i k x}.
// Then psi <- exp(-i dt A) psi in FP64 for both field precisions.
// Not inlined: the pass kernels that carry it keep their register budget for
// the common steps.
template <typename R, int TC, bool CP = false>
__device__ __noinline__ void num_point(const NLArgs &a, cplx<R> *v, int64_t l, double x0, const double *cp = nullptr) {
  constexpr int NC = TC < 3 ? TC : 3;
  const int n = a.ncomp;
  const double bx = beta_dot_x(a, l, x0);
  double2 p[3];
  double rho[3];
  #pragma unroll
  for (int j = 0; j < 3; j++) {
    p[j] = (j < NC && j < n) ? to_d<R>(v[j]) : make_double2(0.0, 0.0);
    rho[j] = p[j].x * p[j].x + p[j].y * p[j].y;
  }
  double2 A[3][3];
  #pragma unroll
  for (int i = 0; i < 3; i++)
    #pragma unroll
    for (int j = 0; j < 3; j++) A[i][j] = make_double2(0.0, 0.0);
  #pragma unroll
  for (int i = 0; i < NC; i++) {
    if (i >= n) break;
    double phi = 0.0;
    #pragma unroll
    for (int j = 0; j < NC; j++)
      if (j < n) phi += a.gs[i * MAXC + j] * rho[j];
    A[i][i].x = phi + (bx - a.L.DeltaL[i]);
  }
  if (a.kind == K_RAMAN) {
    if constexpr (NC >= 3) {
      A[2][2].x += a.L.laser_domh0;
      double sn, cs;
      if constexpr (CP) {
        cs = cp[0];
        sn = cp[1];
      } else {
        sincos(a.L.laser_k0 * x0, &sn, &cs);
      }
      const double h0 = a.L.Amp0 / 2, h1 = a.L.Amp1 / 2;
      A[0][2] = make_double2(h0 * cs, h0 * sn);
      A[2][0] = make_double2(h0 * cs, -h0 * sn);
      A[1][2] = make_double2(h1 * cs, -h1 * sn);
      A[2][1] = make_double2(h1 * cs, h1 * sn);
    }
  } else {
    const double t1 = a.th;
    #pragma unroll
    for (int i = 0; i + 1 < NC; i++) {
      if (i + 1 >= n) break;
      double sn, cs;
      if constexpr (CP) {
        cs = cp[2 * i];
        sn = cp[2 * i + 1];
      } else {
        const double k = i == 0 ? a.L.laser_k0 : -a.L.laser_k0;
        const double rate = i == 0 ? a.L.chirp_rate0 : -a.L.chirp_rate0;
        sincos((-a.L.laser_domh0 + rate * t1) * t1 + k * x0 - 0.5 * a.L.phase0, &sn, &cs);
      }
      const double er = a.L.Amp0 * cs / 2 + a.L.Amp1 * cs / 2, ei = a.L.Amp0 * sn / 2 - a.L.Amp1 * sn / 2;
      A[i + 1][0] = make_double2(er, ei);
      A[0][i + 1] = make_double2(er, -ei);
    }
  }
  herm_expm_apply(A, n, a.dt, p);
  #pragma unroll
  for (int j = 0; j < NC; j++)
    if (j < n) v[j] = from_d<R>(p[j]);
}


template <typename C> __device__ __forceinline__ C shfl_xor_c(C v, int mask) {
  v.x = __shfl_xor_sync(0xffffffffu, v.x, mask);
  v.y = __shfl_xor_sync(0xffffffffu, v.y, mask);
  return v;
}

// The Bragg step of a point whose component c the thread holds as own, the
// other as oth, in the order of the components whichever thread does it.
template <typename R>
__device__ __forceinline__ void bragg_pair_at(const NLArgs &a, int stable, int c, double x0, double om, double ec,
                                              double es, cplx<R> &own, cplx<R> &oth) {
  using C = cplx<R>;
  C p1 = c ? oth : own, p2 = c ? own : oth;
  const double r1 = (double)p1.x * (double)p1.x + (double)p1.y * (double)p1.y;
  const double r2 = (double)p2.x * (double)p2.x + (double)p2.y * (double)p2.y;
  const double V11 = fma(a.L.beta0, x0, a.gs[0] * r1 + a.gs[1] * r2);
  const double V22 = fma(a.L.beta0, x0, a.gs[MAXC] * r1 + a.gs[MAXC + 1] * r2 - a.L.DeltaL[1]);
  bragg_pair_far<R>(stable, a.dt, V11, V22, om, ec, es, p1, p2);
  own = c ? p2 : p1;
  oth = c ? p1 : p2;
}

// Potential step of two components on 16 points a thread, the components of a
// point in two lanes of a warp (partner = lane ^ mask).  Thread c (0 or 1)
// holds its component's points in the order m ^ 8c, m < 16, so registers
// m < 8 are the points it steps for both components, and registers m + 8
// those its partner does: one shuffle brings the partner's value of a point,
// one returns the result, with no shared memory, no barrier and no register
// selection.  Point of register m: grid index l0 + dl (m ^ 8c).  x0, om, ec, es
// belong to the pencil; live: it is inside the grid.
//
// nl_pair16_any takes every step kind and size of phase, on a copy in local
// memory: with its calls inlined eight or sixteen times the common path lost
// its registers to spills (z pass of 256^3 FP64: 0.35 ms).
template <typename R>
__device__ __noinline__ void nl_pair16_any(const NLArgs &a, cplx<R> *v, int c, int mask, bool live, double x0,
                                           double om, double ec, double es, int64_t l0, int dl) {
  using C = cplx<R>;
  if (a.kind == K_BRAGG || a.kind == K_NUM_BRAGG) {
    double cp[NCPL];
    if (a.kind == K_NUM_BRAGG) coupling_x(a, x0, cp);
    #pragma unroll 1
    for (int m = 0; m < 8; m++) {
      C own = v[m], oth = shfl_xor_c(v[m + 8], mask);
      if (a.kind == K_BRAGG) {
        bragg_pair_at<R>(a, a.stable, c, x0, om, ec, es, own, oth);
      } else {
        C w[2] = {c ? oth : own, c ? own : oth};
        num_point<R, 2, true>(a, w, l0 + (int64_t)dl * (m ^ (8 * c)), x0, cp);
        own = c ? w[1] : w[0];
        oth = c ? w[0] : w[1];
      }
      v[m] = own;
      v[m + 8] = shfl_xor_c(oth, mask);
    }
    return;
  }
  // pure phases: a point needs only the partner's density
  const double *const Vp = (a.kind == K_NL && live) ? (c ? a.V[1] : a.V[0]) : nullptr;
  const double b = (a.kind == K_NL_IF2 && c) ? a.L2.beta0 : a.L.beta0;
  const double off = (a.kind == K_NL) ? 0.0 : b * x0 - (c ? a.L.DeltaL[1] : a.L.DeltaL[0]);
  #pragma unroll 2
  for (int m = 0; m < 8; m++) {  // registers m and m + 8 together: their densities cross over
    const C v0 = v[m], v1 = v[m + 8];
    const double w0 = Vp ? __ldg(&Vp[l0 + (int64_t)dl * (m ^ (8 * c))]) : 0.0;
    const double w1 = Vp ? __ldg(&Vp[l0 + (int64_t)dl * ((m + 8) ^ (8 * c))]) : 0.0;
    const double r0 = (double)v0.x * (double)v0.x + (double)v0.y * (double)v0.y;
    const double r1 = (double)v1.x * (double)v1.x + (double)v1.y * (double)v1.y;
    const double t0 = __shfl_xor_sync(0xffffffffu, r1, mask), t1 = __shfl_xor_sync(0xffffffffu, r0, mask);
    const double g_oo = a.gs[c * (MAXC + 1)], g_ot = a.gs[c ? MAXC : 1];
    v[m] = from_d<R>(cmul(to_d<R>(v0), expi_f<R>((w0 + (g_oo * r0 + g_ot * t0 + off)) * a.mdt)));
    v[m + 8] = from_d<R>(cmul(to_d<R>(v1), expi_f<R>((w1 + (g_oo * r1 + g_ot * t1 + off)) * a.mdt)));
  }
}

// A double above every finite one whose high word (less the sign) is at most
// h: the next high word, or NaN, which no bound holds, for infinity and NaN.
__device__ __forceinline__ double above(int h) { return __hiloint2double(min(h, 0x7ff00000) + 1, 0); }

// Largest |re| or |im| of v[0..16), rounded up; NaN if one is not finite.
__device__ __forceinline__ double abs_bound(const double2 *v) {
  int h = 0;
  #pragma unroll
  for (int m = 0; m < 16; m++)
    h = max(h, max(__double2hiint(v[m].x) & 0x7fffffff, __double2hiint(v[m].y) & 0x7fffffff));
  return above(h);
}
__device__ __forceinline__ double abs_bound(const float2 *v) {
  int h = 0;
  #pragma unroll
  for (int m = 0; m < 16; m++)
    h = max(h, max(__float_as_int(v[m].x) & 0x7fffffff, __float_as_int(v[m].y) & 0x7fffffff));
  return h < 0x7f800000 ? (double)__int_as_float(h) : above(0x7ff00000);
}

// The step's form; apart, each keeps its registers (z pass of 256^3 FP64 with
// both forms of the Bragg step in one kernel 336 us, the eigenvalue form alone
// 309, the other 276).
enum { PAIR_PHASE = 0, PAIR_FREE = 1, PAIR_EIGEN = 2 };  // not K_BRAGG; K_BRAGG eigenvalue-free; its eigenvalue form
template <typename R>
__device__ __host__ __forceinline__ int pair_form(const NLArgs &a) {
  return a.kind != K_BRAGG ? PAIR_PHASE : (sizeof(R) == 8 && !a.stable) ? PAIR_EIGEN : PAIR_FREE;
}
template <typename R, int FORM>
__device__ __forceinline__ void nl_pair16(const NLArgs &a, cplx<R> *v, int c, int mask, bool live, double x0, double om,
                                          double ec, double es, int64_t l0, int dl) {
  using C = cplx<R>;
  if constexpr (FORM == PAIR_EIGEN) {
    // the reference's form, bound by its FP64 operations (a square root, a
    // division, two phases): two points at a time from v[0], v[1] and their
    // partners, then the registers move up by two.  z pass of 256^3: two at a
    // time 309 us, one 315, four 321.
    #pragma unroll 1
    for (int it = 0; it < 4; it++) {
      #pragma unroll
      for (int u = 0; u < 2; u++) {
        C own = v[u], oth = shfl_xor_c(v[8 + u], mask);
        bragg_pair_at<R>(a, 0, c, x0, om, ec, es, own, oth);
        v[u] = own;
        v[8 + u] = shfl_xor_c(oth, mask);
      }
      #pragma unroll
      for (int h = 0; h < 16; h += 8) {
        const C v0 = v[h], v1 = v[h + 1];
        #pragma unroll
        for (int m = 0; m < 6; m++) v[h + m] = v[h + m + 2];
        v[h + 6] = v0;
        v[h + 7] = v1;
      }
    }
    return;
  }
  // The series serve every point of the warp if they do for the largest
  // potential that its points allow: |V| <= G rho + |off| + max |V_c|, with
  // rho <= 2 max(|re|, |im|)^2 over the pencil and G the larger row sum of |g|.
  const double bx = a.L.beta0 * x0, bd = bx - a.L.DeltaL[1];
  const double m1 = abs_bound(v), m2 = __shfl_xor_sync(0xffffffffu, m1, mask);
  const double mx = m1 >= m2 ? m1 : m2 >= m1 ? m2 : m1 + m2;  // NaN where one is (fmax would drop it)
  const double G = fmax(fabs(a.gs[0]) + fabs(a.gs[1]), fabs(a.gs[MAXC]) + fabs(a.gs[MAXC + 1]));
  const double Vrho = 2.0 * G * (mx * mx);
  const double *const Vp = (a.kind == K_NL && live) ? (c ? a.V[1] : a.V[0]) : nullptr;
  // pure phases: the constant part of the component's potential
  const double off = (a.kind == K_NL) ? 0.0
                                      : ((a.kind == K_NL_IF2 && c) ? a.L2.beta0 : a.L.beta0) * x0 -
                                            (c ? a.L.DeltaL[1] : a.L.DeltaL[0]);
  bool small = false;
  if constexpr (FORM == PAIR_FREE) {
    const double V = Vrho + fmax(fabs(bx), fabs(bd)), O2 = om * om;
    small = fabs(a.dt) * V <= 0.03125 && (a.dt * a.dt) * (V * V + O2) <= 0x1p-10;
  } else if (a.kind != K_NUM_BRAGG) {
    int h = 0;
    if (Vp) {
      #pragma unroll
      for (int m = 0; m < 16; m++) h = max(h, __double2hiint(__ldg(&Vp[l0 + (int64_t)dl * m])) & 0x7fffffff);
    }
    small = fabs(a.dt) * (Vrho + fabs(off) + (Vp ? above(h) : 0.0)) <= 0.03125;
  }
  if (!__all_sync(0xffffffffu, small)) {
    C w[16];
    #pragma unroll
    for (int m = 0; m < 16; m++) w[m] = v[m];
    nl_pair16_any<R>(a, w, c, mask, live, x0, om, ec, es, l0, dl);
    #pragma unroll
    for (int m = 0; m < 16; m++) v[m] = w[m];
    return;
  }
  if constexpr (FORM == PAIR_PHASE) {  // a point needs only the partner's density
    const double s_oo = a.gs[c * (MAXC + 1)], s_ot = a.gs[c ? MAXC : 1];
    #pragma unroll
    for (int m = 0; m < 8; m++) {  // registers m and m + 8 together: their densities cross over
      const C v0 = v[m], v1 = v[m + 8];
      const double w0 = Vp ? __ldg(&Vp[l0 + (int64_t)dl * (m ^ (8 * c))]) : 0.0;
      const double w1 = Vp ? __ldg(&Vp[l0 + (int64_t)dl * ((m + 8) ^ (8 * c))]) : 0.0;
      const double r0 = (double)v0.x * (double)v0.x + (double)v0.y * (double)v0.y;
      const double r1 = (double)v1.x * (double)v1.x + (double)v1.y * (double)v1.y;
      const double t0 = __shfl_xor_sync(0xffffffffu, r1, mask), t1 = __shfl_xor_sync(0xffffffffu, r0, mask);
      v[m] = from_d<R>(cmul(to_d<R>(v0), expi_series((w0 + (s_oo * r0 + s_ot * t0 + off)) * a.mdt)));
      v[m + 8] = from_d<R>(cmul(to_d<R>(v1), expi_series((w1 + (s_oo * r1 + s_ot * t1 + off)) * a.mdt)));
    }
    return;
  }
  const double g_oo = a.gs[c * (MAXC + 1)], g_ot = a.gs[c ? MAXC : 1];
  const double g_to = a.gs[c ? 1 : MAXC], g_tt = a.gs[c ? 0 : MAXC + 1];
  const double off_o = c ? bd : bx, off_t = c ? bx : bd, se = c ? -es : es, dt2 = a.dt * a.dt, O2 = om * om;
  #pragma unroll
  for (int m = 0; m < 8; m++) {
    C own = v[m], oth = shfl_xor_c(v[m + 8], mask);
    const double ro = (double)own.x * (double)own.x + (double)own.y * (double)own.y;
    const double rt = (double)oth.x * (double)oth.x + (double)oth.y * (double)oth.y;
    const double Vo = g_oo * ro + g_ot * rt + off_o, Vt = g_to * ro + g_tt * rt + off_t;
    const double d = 0.5 * (Vo - Vt);
    bragg_series<R>(a.dt, dt2 * (d * d + O2), d, om, expi_series(a.mdt * (0.5 * (Vo + Vt))), ec, se, own, oth);
    v[m] = own;
    v[m + 8] = shfl_xor_c(oth, mask);
  }
}

// Potential step of one component on 16 points a thread: register m is grid
// index l0 + dl m; XP: x varies along the pencil (x0 + dx m), else it is x0.
// Eight points at a time: their potential is loaded together, and where every
// phase of the warp is small (or below 2^17) they take the series (or the
// reduced series) without a branch a point
// (16 sites with a call each for larger phases cost the loop its overlap).
// One component with a potential, FP64: z pass of 256^3 178 -> 138 us, y pass of
// 2048^2 60 -> 53.
template <typename R> __device__ __noinline__ void phase8_any(cplx<R> *v, const double *ph) {
  #pragma unroll 2
  for (int m = 0; m < 8; m++) v[m] = from_d<R>(cmul(to_d<R>(v[m]), expi_f<R>(ph[m])));
}
template <typename R, bool XP>
__device__ __forceinline__ void nl_single16(const NLArgs &a, cplx<R> *v, bool live, double x0, double dx, int64_t l0,
                                            int64_t dl) {
  using C = cplx<R>;
  const double *const Vp = (a.kind == K_NL && live) ? a.V[0] : nullptr;
  const double beta = a.kind == K_NL ? 0.0 : a.L.beta0, shift = a.kind == K_NL ? 0.0 : a.L.DeltaL[0], g = a.gs[0];
  #pragma unroll
  for (int h = 0; h < 16; h += 8) {
    double ph[8];
    #pragma unroll
    for (int m = 0; m < 8; m++) ph[m] = Vp ? __ldg(&Vp[l0 + dl * (h + m)]) : 0.0;
    bool small = true, mid = true;
    #pragma unroll
    for (int m = 0; m < 8; m++) {
      const double rho = (double)v[h + m].x * (double)v[h + m].x + (double)v[h + m].y * (double)v[h + m].y;
      const double x = XP ? x0 + dx * (h + m) : x0;
      ph[m] = (a.kind == K_NL ? ph[m] + g * rho : g * rho + (beta * x - shift)) * a.mdt;
      small = small && fabs(ph[m]) <= 0.03125;
      mid = mid && fabs(ph[m]) < 131072.0;
    }
    if (__all_sync(0xffffffffu, small)) {
      #pragma unroll
      for (int m = 0; m < 8; m++) v[h + m] = from_d<R>(cmul(to_d<R>(v[h + m]), expi_series(ph[m])));
    } else if (sizeof(R) == 8 && __all_sync(0xffffffffu, mid)) {  // complex64: expi<float>, as everywhere
      #pragma unroll
      for (int m = 0; m < 8; m++) v[h + m] = from_d<R>(cmul(to_d<R>(v[h + m]), expi_cw(ph[m])));
    } else {  // on copies in local memory: calls from here would take the common path's registers
      C w[8];
      double q[8];
      #pragma unroll
      for (int m = 0; m < 8; m++) {
        w[m] = v[h + m];
        q[m] = ph[m];
      }
      phase8_any<R>(w, q);
      #pragma unroll
      for (int m = 0; m < 8; m++) v[h + m] = w[m];
    }
  }
}

// ------------------------------------------------------------ potential step
// Point-wise potential step on the ncomp values v[] at grid index l.
// FP64: the reference's formulas (include/CRT_Base.h:410-439,
// CRT_Base_IF.h:392-418, bragg.cpp:210-302).  Mixed: FP64 phase arguments,
// FP32 field arithmetic, and the eigenvalue-free form of the 2x2 exponential.
// TC: the number of components the calling kernel holds (ncomp <= TC); step
// kinds that need more components are compiled out.  CP: the caller has the
// pencil's couplings of three- and four-component steps (coupling_x).  FAR: as
// in bragg_pair_far.
template <typename R, int TC = MAXC, bool CP = false, bool FAR = false>
__device__ __forceinline__ void nl_point(const NLArgs &a, cplx<R> *v, int64_t l, double x0, double Omega,
                                         double eta_c, double eta_s, const double *cp = nullptr) {
  if constexpr (TC >= 3) {
    if (a.kind == K_DBRAGG) {
      dbragg_point<R, CP>(a, v, l, x0, cp);
      return;
    }
  }
  if constexpr (TC >= 4) {
    if (a.kind == K_BRAGG_DS) {
      bragg_ds_point<R, CP>(a, v, x0, cp);
      return;
    }
  }
  if constexpr (TC >= 2) {
    if (a.kind == K_NUM_BRAGG || a.kind == K_RAMAN) {
      // the out-of-line step gets a copy: were the caller's array handed to
      // it, its address would escape and the array would live in local
      // memory on every path
      cplx<R> w[TC];
      #pragma unroll
      for (int c = 0; c < TC; c++) w[c] = v[c];
      num_point<R, TC, CP>(a, w, l, x0, cp);
      #pragma unroll
      for (int c = 0; c < TC; c++) v[c] = w[c];
      return;
    }
  }
  const int n = a.ncomp;
  double rho[TC];
  #pragma unroll
  for (int j = 0; j < TC; j++)
    if (j < n) rho[j] = (double)v[j].x * (double)v[j].x + (double)v[j].y * (double)v[j].y;
  if (TC < 2 || a.kind != K_BRAGG) {
    #pragma unroll
    for (int i = 0; i < TC; i++) {
      if (i >= n) break;
      double phi;
      if (a.kind == K_NL) {
        phi = a.V[i] ? a.V[i][l] : 0.0;
        #pragma unroll
        for (int j = 0; j < TC; j++)
          if (j < n) phi += a.gs[i * MAXC + j] * rho[j];
      } else {
        phi = 0.0;
        #pragma unroll
        for (int j = 0; j < TC; j++)
          if (j < n) phi += a.gs[i * MAXC + j] * rho[j];
        // CRT_Base_IF_2 (two species): beta of the component's species
        const double b = (a.kind == K_NL_IF2 && 2 * i >= n) ? a.L2.beta0 : a.L.beta0;
        phi += b * x0 - a.L.DeltaL[i];
      }
      phi *= a.mdt;
      const double2 e = expi<R>(phi);
      v[i] = from_d<R>(cmul(to_d<R>(v[i]), e));
    }
    return;
  }
  if constexpr (TC >= 2) {
    // Bragg 2x2 (components 0 and 1)
    const double V11 = a.gs[0] * rho[0] + a.gs[1] * rho[1] + a.L.beta0 * x0;
    const double V22 = a.gs[MAXC] * rho[0] + a.gs[MAXC + 1] * rho[1] - a.L.DeltaL[1] + a.L.beta0 * x0;
    if constexpr (FAR) bragg_pair_far<R>(a.stable, a.dt, V11, V22, Omega, eta_c, eta_s, v[0], v[1]);
    else bragg_pair<R>(a.stable, a.dt, V11, V22, Omega, eta_c, eta_s, v[0], v[1]);
  }
}

// Omega(x0) and eta(x0) of the Bragg step (bragg.cpp:224, 243).
__device__ __forceinline__ void bragg_coupling(const NLArgs &a, double x0, double &Omega, double &ec, double &es) {
  const double t1 = a.t1;
  Omega = a.F * a.L.Amp0 *
          cos(a.L.laser_k0 * x0 - (a.L.laser_domh0 + a.L.chirp * t1 + a.L.chirp_rate0 * t1) * t1 + a.L.phase0 / 2);
  sincos(-0.5 * (a.L.laser_dk0 * x0), &es, &ec);
}

// v times a twiddle (DIR > 0: its conjugate), in FP64 for both precisions.
template <typename R, int DIR> __device__ __forceinline__ cplx<R> fs_mul(cplx<R> v, double2 w) {
  return from_d<R>(DIR < 0 ? cmul(to_d<R>(v), w) : cmulc(to_d<R>(v), w));
}

// psi^ <- ((psi^ s_f) K) s_b in FP64.
template <typename R> __device__ __forceinline__ cplx<R> kin_mul(cplx<R> v, double2 K, double s_f, double s_b) {
  double2 u = to_d<R>(v);
  u.x *= s_f;
  u.y *= s_f;
  u = cmul(u, K);
  u.x *= s_b;
  u.y *= s_b;
  return from_d<R>(u);
}

// ------------------------------------------------------------ kinetic step
template <typename C>
__device__ __forceinline__ C kin_phase(const C *kx, const C *ky, const C *kz, int ix, int iy, int iz) {
  return cmul(cmul(__ldg(&kx[ix]), __ldg(&ky[iy])), __ldg(&kz[iz]));
}

// ------------------------------------------------------------ pass kernel
// Asynchronous global -> shared copies (cp.async): a tile's loads are issued
// without registers and complete while the previous tile is transformed.
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, double2) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, float2) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::); }

template <typename R, int N, int TC>
struct PassCfg {
  static constexpr int NT = Tile<R>::NT;
  static constexpr int B0 = Tile<R>::E / (N * TC);
  static constexpr int B1 = B0 > 0 ? B0 : 1;
  static constexpr int B = B1 < 256 ? B1 : 256;  // pencils per tile
  static constexpr int NP = Pad<N>::NP;
  static constexpr int TILE = TC * B * NP;       // complex values per buffer
  // two buffers (prefetch of the next work item) when they fit, else one
  static constexpr int NBUF = (2 * sizeof(cplx<R>) * (size_t)TILE + 3 * 8 * B <= 227 * 1024) ? 2 : 1;
  static constexpr size_t smem = NBUF * sizeof(cplx<R>) * (size_t)TILE;
};

struct TileGeo {
  int64_t base0;    // grid index of element 0 of pencil 0
  int64_t pstride;  // distance between the tile's pencils
  int nb;           // pencils of the tile inside the grid
  int comp0;        // first component
};

template <int B, int N>
__device__ __forceinline__ TileGeo tile_geo(const PassArgs &a, int64_t w) {
  TileGeo g;
  int64_t t = w;
  g.comp0 = 0;
  if (a.per_comp) {
    g.comp0 = (int)(w / a.ntiles);
    t = w % a.ntiles;
  }
  if (a.sa > 1) {
    const int64_t o = t / a.inner_tiles;
    const int64_t r0 = (t % a.inner_tiles) * B;
    g.base0 = o * (int64_t)N * a.sa + r0;
    g.pstride = 1;
    g.nb = (int)((a.sa - r0) < B ? (a.sa - r0) : B);
  } else {
    const int64_t p0 = t * B;
    g.base0 = p0 * N;
    g.pstride = N;
    g.nb = (int)((a.npencils - p0) < B ? (a.npencils - p0) : B);
  }
  return g;
}

// Persistent pass kernel: each CTA walks work items (tile, component) with a
// stride of the grid size, double buffered -- the cp.async loads of item w+1
// fly while item w is transformed and stored.
template <typename R, int N, int TC>
__global__ void __launch_bounds__(Tile<R>::NT, Tile<R>::MINB) pass_kernel(PassArgs a) {
  using C = cplx<R>;
  using Cfg = PassCfg<R, N, TC>;
  constexpr int B = Cfg::B, NT = Cfg::NT, NP = Cfg::NP, TILE = Cfg::TILE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *const sbase = reinterpret_cast<C *>(smem_raw);
  __shared__ double s_om[B], s_ec[B], s_es[B];
  static_assert((B * N) % NT == 0, "tile must be a multiple of the CTA size");
  constexpr int LPT = B * N / NT;
  const int64_t W = a.per_comp ? a.ntiles * a.ncomp_grid : a.ntiles;
  const typename TwTab<R>::type *tw = (const typename TwTab<R>::type *)a.tw;

  auto issue = [&](int64_t w, C *s) {
    const TileGeo g = tile_geo<B, N>(a, w);
    const int nc = a.per_comp ? 1 : a.nc;
    #pragma unroll
    for (int c = 0; c < TC; c++) {
      const C *src = (const C *)pick(a.psi, g.comp0 + c);
      #pragma unroll
      for (int k = 0; k < LPT; k++) {
        const int r = threadIdx.x + k * NT;
        int b, i;
        if (a.sa > 1) { b = r % B; i = r / B; } else { i = r % N; b = r / N; }
        C *dst = &s[c * B * NP + Pad<N>::idx(b, i)];
        if (c < nc && b < g.nb) cp_async(dst, &src[g.base0 + b * g.pstride + (int64_t)i * a.sa], C{});
        else *dst = mk<R>(0, 0);
      }
    }
  };

  pdl_wait();
  int64_t w = blockIdx.x;
  int buf = 0;
  if (Cfg::NBUF == 2) {
    if (w < W) issue(w, sbase);
    cp_commit();
  }
  for (; w < W; w += gridDim.x) {
    C *s = sbase + buf * TILE;
    if (Cfg::NBUF == 2) {
      const int64_t wn = w + gridDim.x;
      if (wn < W) issue(wn, sbase + (buf ^ 1) * TILE);
      cp_commit();
      cp_wait_prev();
    } else {
      issue(w, s);
      cp_commit();
      asm volatile("cp.async.wait_all;\n" ::);
    }
    __syncthreads();

    const TileGeo g = tile_geo<B, N>(a, w);
    const int nc = a.per_comp ? 1 : a.nc;
    const int64_t base0 = g.base0, pstride = g.pstride;
    const int nb = g.nb, comp0 = g.comp0;
    if (a.t1 == T_FWD) fft_tile<R, N, TC * B, NT, -1, TWN>(s, tw);
    else if (a.t1 == T_INV) fft_tile<R, N, TC * B, NT, +1, TWN>(s, tw);

    if (a.op == OP_KIN) {
      // psi^ <- ((psi^ s_f) K) s_b with K = Kx Ky Kz in FP64: the two scales of
      // the reference's ft(-1) / ft(+1) as separate products (no folded,
      // once-rounded constant that would bias every step the same way)
      const double2 *kx = a.kt[0][0], *ky = a.kt[0][1], *kz = a.kt[0][2];
      #pragma unroll
      for (int c = 1; c < MAXC; c++)
        if (comp0 == c) { kx = a.kt[c][0]; ky = a.kt[c][1]; kz = a.kt[c][2]; }
      #pragma unroll 4
      for (int e = threadIdx.x; e < B * N; e += NT) {
        const int b = e / N, i = e % N;
        if (b < nb) {
          const int64_t l = base0 + b * pstride + (int64_t)i * a.sa;
          int ix, iy, iz;
          idx3(a.g, l, ix, iy, iz);
          const double2 k = kin_phase(kx, ky, kz, ix, iy, iz);
          const int si = Pad<N>::idx(b, i);
          double2 v = to_d<R>(s[si]);
          v.x *= a.s_f;
          v.y *= a.s_f;
          v = cmul(v, k);
          v.x *= a.s_b;
          v.y *= a.s_b;
          s[si] = from_d<R>(v);
        }
      }
      __syncthreads();
    } else if (a.op == OP_FILT) {
      for (int e = threadIdx.x; e < B * N; e += NT) {
        const int b = e / N, i = e % N;
        if (b < nb) {
          const int64_t l = base0 + b * pstride + (int64_t)i * a.sa;
          int ijk[3];
          idx3(a.g, l, ijk[0], ijk[1], ijk[2]);
          double phi = 0;
          #pragma unroll
          for (int ax = 0; ax < 3; ax++) {
            const int t = (ijk[ax] + a.n[ax] / 2) % a.n[ax];
            const double k = a.dk[ax] * (double)(t - a.n[ax] / 2);
            phi += (k * a.filt_alpha) * k;
          }
          const double f = (a.filt_mode == FILT_SOBOLEV ? 1.0 / (1.0 + phi) : -phi) * a.filt_scale;
          const int si = Pad<N>::idx(b, i);
          C v = s[si];
          v.x = (R)((double)v.x * f);
          v.y = (R)((double)v.y * f);
          s[si] = v;
        }
      }
      __syncthreads();
    } else if (a.op == OP_NL) {
      const bool bragg = (a.nl.kind == K_BRAGG);
      if (bragg && !a.x_along) {
        for (int b = threadIdx.x; b < B; b += NT) {
          double om = 0, ec = 1, es = 0;
          if (b < nb) {
            int ix, iy, iz;
            idx3(a.g, base0 + b * pstride, ix, iy, iz);
            bragg_coupling(a.nl, (double)(ix - a.nl.shift0) * a.nl.dx0, om, ec, es);
          }
          s_om[b] = om; s_ec[b] = ec; s_es[b] = es;
        }
        __syncthreads();
      }
      #pragma unroll 2
      for (int e = threadIdx.x; e < B * N; e += NT) {
        const int b = e / N, i = e % N;
        if (b < nb) {
          const int64_t l = base0 + b * pstride + (int64_t)i * a.sa;
          int ix, iy, iz;
          idx3(a.g, l, ix, iy, iz);
          const double x0 = (double)(ix - a.nl.shift0) * a.nl.dx0;
          double om = 0, ec = 1, es = 0;
          if (bragg) {
            if (a.x_along) bragg_coupling(a.nl, x0, om, ec, es);
            else { om = s_om[b]; ec = s_ec[b]; es = s_es[b]; }
          }
          C v[MAXC];
          #pragma unroll
          for (int c = 0; c < TC; c++) v[c] = s[c * B * NP + Pad<N>::idx(b, i)];
          nl_point<R, TC>(a.nl, v, l, x0, om, ec, es);
          #pragma unroll
          for (int c = 0; c < TC; c++) s[c * B * NP + Pad<N>::idx(b, i)] = v[c];
        }
      }
      __syncthreads();
    }

    if (a.t2 == T_FWD) fft_tile<R, N, TC * B, NT, -1, TWN>(s, tw);
    else if (a.t2 == T_INV) fft_tile<R, N, TC * B, NT, +1, TWN>(s, tw);

    #pragma unroll
    for (int c = 0; c < TC; c++) {
      if (c < nc) {
        C *dst = (C *)pick(a.psi, comp0 + c);
        #pragma unroll
        for (int k = 0; k < LPT; k++) {
          const int r = threadIdx.x + k * NT;
          int b, i;
          if (a.sa > 1) { b = r % B; i = r / B; } else { i = r % N; b = r / N; }
          if (b < nb) dst[base0 + b * pstride + (int64_t)i * a.sa] = s[c * B * NP + Pad<N>::idx(b, i)];
        }
      }
    }
    __syncthreads();  // the buffer is refilled two items later
    if (Cfg::NBUF == 2) buf ^= 1;
  }
  asm volatile("cp.async.wait_all;\n" ::);
}

// ------------------------------------------------------------ 1D Strang block
struct Block1DArgs {
  void *psi[MAXC];
  const double2 *kh[MAXC], *kf[MAXC];  // half / full kinetic phase factors (FP64)
  double s_f, s_b;                     // forward / backward transform scales
  const void *tw;
  NLArgs nl;
  int nk;
  double t0;                        // header time at block start
  const double *F;                  // per potential step, or nullptr
};

template <typename R, int N, int TC>
__device__ __forceinline__ void kin_1d(cplx<R> *s, const double2 *const (&tab)[TC], int nc, double s_f, double s_b) {
  constexpr int NT = BLOCK1D_NT, NP = Pad<N>::NP;
  #pragma unroll
  for (int c = 0; c < TC; c++) {
    if (c < nc) {
      for (int i = threadIdx.x; i < N; i += NT) {
        const int si = c * NP + Pad<N>::idx(0, i);
        double2 v = to_d<R>(s[si]);
        v.x *= s_f;
        v.y *= s_f;
        v = cmul(v, __ldg(&tab[c][i]));
        v.x *= s_b;
        v.y *= s_b;
        s[si] = from_d<R>(v);
      }
    }
  }
  __syncthreads();
}

template <typename R, int N, int TC>
__global__ void __launch_bounds__(BLOCK1D_NT) block1d_kernel(Block1DArgs a) {
  using C = cplx<R>;
  constexpr int NT = BLOCK1D_NT, NP = Pad<N>::NP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int nc = a.nl.ncomp;
  const typename TwTab<R>::type *tw = (const typename TwTab<R>::type *)a.tw;
  C *fld[TC];
  const double2 *kh[TC], *kf[TC];
  #pragma unroll
  for (int c = 0; c < TC; c++) {
    fld[c] = (C *)a.psi[c];
    kh[c] = a.kh[c];
    kf[c] = a.kf[c];
  }
  #pragma unroll
  for (int c = 0; c < TC; c++)
    for (int i = threadIdx.x; i < N; i += NT) s[c * NP + Pad<N>::idx(0, i)] = (c < nc) ? fld[c][i] : mk<R>(0, 0);
  __syncthreads();
  double t = a.t0;
  const double dt = a.nl.dt;
  // half kinetic step
  fft_tile<R, N, TC, NT, -1, TWN>(s, tw);
  kin_1d<R, N, TC>(s, kh, nc, a.s_f, a.s_b);
  fft_tile<R, N, TC, NT, +1, TWN>(s, tw);
  t += 0.5 * dt;
  // the step parameters in shared memory (thread 0 sets the step's time and
  // pulse amplitude): a per-thread copy of the ~0.5 KB block sat in local memory
  __shared__ NLArgs s_nl;
  const NLArgs &nl = s_nl;
  if (threadIdx.x == 0) s_nl = a.nl;
  for (int j = 0; j < a.nk; j++) {
    if (threadIdx.x == 0) {
      s_nl.t1 = t + 0.5 * dt;
      s_nl.F = a.F ? a.F[j] : 1.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += NT) {
      const double x0 = (double)(i - nl.shift0) * nl.dx0;
      double om = 0, ec = 1, es = 0;
      if (nl.kind == K_BRAGG) bragg_coupling(nl, x0, om, ec, es);
      C v[MAXC];
      #pragma unroll
      for (int c = 0; c < TC; c++) v[c] = s[c * NP + Pad<N>::idx(0, i)];
      nl_point<R, TC>(nl, v, i, x0, om, ec, es);
      #pragma unroll
      for (int c = 0; c < TC; c++) s[c * NP + Pad<N>::idx(0, i)] = v[c];
    }
    __syncthreads();
    const bool last = (j == a.nk - 1);
    fft_tile<R, N, TC, NT, -1, TWN>(s, tw);
    if (last) kin_1d<R, N, TC>(s, kh, nc, a.s_f, a.s_b);
    else kin_1d<R, N, TC>(s, kf, nc, a.s_f, a.s_b);
    fft_tile<R, N, TC, NT, +1, TWN>(s, tw);
    t += last ? 0.5 * dt : dt;
  }
  #pragma unroll
  for (int c = 0; c < TC; c++)
    if (c < nc)
      for (int i = threadIdx.x; i < N; i += NT) fld[c][i] = s[c * NP + Pad<N>::idx(0, i)];
}

// ------------------------------------------------------------ point-wise kernels
struct NLKArgs {
  void *psi[MAXC];
  NLArgs nl;
  Geo g;
};

template <typename R>
__global__ void nl_kernel(NLKArgs a) {
  using C = cplx<R>;
  const int n = a.nl.ncomp;
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < a.g.npts;
       l += (int64_t)gridDim.x * blockDim.x) {
    int ix, iy, iz;
    idx3(a.g, l, ix, iy, iz);
    const double x0 = (double)(ix - a.nl.shift0) * a.nl.dx0;
    double om = 0, ec = 1, es = 0;
    if (a.nl.kind == K_BRAGG) bragg_coupling(a.nl, x0, om, ec, es);
    C v[MAXC];
    #pragma unroll
    for (int c = 0; c < MAXC; c++)
      if (c < n) v[c] = ((C *)a.psi[c])[l];
    nl_point<R>(a.nl, v, l, x0, om, ec, es);
    #pragma unroll
    for (int c = 0; c < MAXC; c++)
      if (c < n) ((C *)a.psi[c])[l] = v[c];
  }
}

// psi *= e^{i p.x}  (Setup_Momentum)
template <typename R>
__global__ void momentum_kernel(void *psi, Geo g, double p0, double p1, double p2, double dx0, double dx1,
                                double dx2, int s0, int s1, int s2) {
  using C = cplx<R>;
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < g.npts; l += (int64_t)gridDim.x * blockDim.x) {
    int ix, iy, iz;
    idx3(g, l, ix, iy, iz);
    const double dot = p0 * ((double)(ix - s0) * dx0) + p1 * ((double)(iy - s1) * dx1) + p2 * ((double)(iz - s2) * dx2);
    C *P = (C *)psi;
    P[l] = from_d<R>(cmul(to_d<R>(P[l]), expi<R>(dot)));
  }
}

// FP64 <-> field precision conversions (mixed mode upload / download).
template <typename R>
__global__ void convert_in_kernel(void *dst, const double2 *src, int64_t n) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < n; l += (int64_t)gridDim.x * blockDim.x)
    ((cplx<R> *)dst)[l] = mk<R>((R)src[l].x, (R)src[l].y);
}
template <typename R>
__global__ void convert_out_kernel(double2 *dst, const void *src, int64_t n) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < n; l += (int64_t)gridDim.x * blockDim.x) {
    const cplx<R> v = ((const cplx<R> *)src)[l];
    dst[l] = make_double2((double)v.x, (double)v.y);
  }
}

// ------------------------------------------------------------ Sobolev helpers
// G = -Lap psi_i + (V_i + sum_j g_ij |psi_j|^2) psi_i   (CSOB_Base.h:317-326)
struct SobArgs {
  const double2 *psi[MAXC];
  const double2 *lap;
  const double *V;
  double2 *grad;
  double2 *copy;  // when set, also receives psi[comp]
  int comp, ncomp;
  double gs[MAXC * MAXC];
  int64_t npts;
};

// ------------------------------------------------------------ reductions
// Quantities per mode (all FP64 accumulations, fixed order per thread, fixed
// tree per block, block sums in a fixed order).
enum { RED_NORM = 0, RED_POS = 1, RED_MOM = 2, RED_RABI = 3, RED_DOT2 = 4, RED_MU = 5 };
constexpr int RED_MAXQ = 8;
constexpr int RED_PER_SM = 4;
constexpr int RED_BLOCKS = RED_PER_SM * 148;  // fixed: the order of the sums does not follow the device
constexpr int RED_ROWS = 1184;   // rows of block sums (the passes that sum run up to 8 CTAs per SM)
constexpr int RED_THREADS = 256;

struct RedArgs {
  int mode;
  int nq;
  const void *a, *b, *c;   // field operands
  const double *V;
  Geo g;
  double d[3], dk[3];
  int n[3], shift[3];
  double k0[8][3];         // Rabi centres
  double thr;
  // mu
  const void *psi_all[MAXC];
  int ncomp, comp;
  double gs[MAXC * MAXC];
};

// |psi^|^2 = den at wavenumber k into the Rabi bins, with the bin rule of
// compute_rabi_integrals (include/CRT_Base_IF.h:231-257): a point inside a
// ball adds to the current bin and the bin index does not advance for it.
// Inside is sqrt(|k0 - k|^2) < thr; the root is only taken within a few
// roundings of the surface, elsewhere the squares decide.
template <int ND>
__device__ __forceinline__ void red_balls(const double (*k0)[3], int n, double thr, const double *k, double den,
                                          double *q) {
  const double t2 = thr * thr, lo = thr > 0 ? t2 * (1 - 1e-14) : -1.0, hi = thr > 0 ? t2 * (1 + 1e-14) : -1.0;
  int j = 0;
  #pragma unroll
  for (int m = 0; m < RED_MAXQ; m++) {
    if (m >= n) break;
    double dd = 0;
    #pragma unroll
    for (int ax = 0; ax < ND; ax++) {
      const double d = k0[m][ax] - k[ax];
      dd += d * d;
    }
    if (dd < lo || (!(dd > hi) && sqrt(dd) < thr)) {
      #pragma unroll
      for (int i = 0; i <= m; i++) q[i] += (i == j) ? den : 0.0;
      continue;
    }
    j++;
  }
}

// The operands of one point, loaded before any is used, so that a thread's
// loads of several points are in flight together.
template <typename R, int MODE> struct RedIn {
  cplx<R> v, b, c;
  double pot;
};

template <typename R, int MODE>
__device__ __forceinline__ void red_fetch(const RedArgs &a, int64_t l, RedIn<R, MODE> &in) {
  using C = cplx<R>;
  in.v = ((const C *)a.a)[l];
  if constexpr (MODE == RED_DOT2 || MODE == RED_MU) in.b = ((const C *)a.b)[l];
  if constexpr (MODE == RED_DOT2) in.c = a.c ? ((const C *)a.c)[l] : mk<R>(0, 0);
  if constexpr (MODE == RED_MU) in.pot = a.V ? a.V[l] : 0.0;
}

template <typename R, int MODE>
__device__ __forceinline__ void red_point(const RedArgs &a, int64_t l, const RedIn<R, MODE> &in, double *q) {
  using C = cplx<R>;
  const C v = in.v;
  const double den = (double)v.x * (double)v.x + (double)v.y * (double)v.y;
  if constexpr (MODE == RED_NORM) q[0] += den;
  if constexpr (MODE == RED_POS || MODE == RED_MOM || MODE == RED_RABI) {
    int ijk[3];
    idx3(a.g, l, ijk[0], ijk[1], ijk[2]);
    double x[3];
    #pragma unroll
    for (int ax = 0; ax < 3; ax++) {  // axis lengths are powers of two (unused axes: one point)
      const int t = (MODE == RED_POS) ? ijk[ax] : ((ijk[ax] + a.shift[ax]) & (a.n[ax] - 1));
      x[ax] = (double)(t - a.shift[ax]) * ((MODE == RED_POS) ? a.d[ax] : a.dk[ax]);
    }
    if constexpr (MODE != RED_RABI) {
      #pragma unroll
      for (int ax = 0; ax < 3; ax++) q[ax] += x[ax] * den;
    } else {
      red_balls<3>(a.k0, a.nq, a.thr, x, den, q);
    }
  }
  if constexpr (MODE == RED_DOT2) {  // Re<a,b>, Re<a,c>, <a,a>
    q[0] += (double)v.x * (double)in.b.x + (double)v.y * (double)in.b.y;
    q[1] += (double)v.x * (double)in.c.x + (double)v.y * (double)in.c.y;
    q[2] += den;
  }
  if constexpr (MODE == RED_MU) {  // a = psi_i, b = Lap psi_i
    double nl = 0;
    #pragma unroll
    for (int j = 0; j < MAXC; j++) {
      if (j < a.ncomp) {
        const C pj = ((const C *)a.psi_all[j])[l];
        nl += a.gs[a.comp * MAXC + j] * ((double)pj.x * (double)pj.x + (double)pj.y * (double)pj.y);
      }
    }
    q[0] += -((double)v.x * (double)in.b.x + (double)v.y * (double)in.b.y) + (in.pot + nl) * den;
  }
}

// Block sums of q[0..nq) over NT threads, then -- in the block that finishes
// last -- the sums over all blocks, in a fixed order whichever block that is.
// partial: gridDim.x rows of RED_MAXQ; count: zero before the launch and left
// at zero; out: nq totals (device memory or mapped host memory).
// Measured against a second launch whose one thread per quantity added 592
// rows: that launch took 25-29 us by itself, of 50 us for a reduction over
// 2^21 points.
// Returns true in every thread of that last block.
template <int NT>
__device__ __forceinline__ bool red_finish(double *q, int nq, double *partial, unsigned *count, double *out) {
  static_assert(NT % 32 == 0 && NT >= 4 * RED_MAXQ, "whole warps, several rows per quantity");
  constexpr int NW = NT / 32, ROWS = NT / RED_MAXQ;
  __shared__ double sh[NT];
  __shared__ int last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();
  #pragma unroll
  for (int i = 0; i < RED_MAXQ; i++) {
    if (i < nq) {
      double v = q[i];
      #pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sh[warp * RED_MAXQ + i] = v;
    }
  }
  __syncthreads();
  if (tid < nq) {
    double v = sh[tid];
    #pragma unroll
    for (int w = 1; w < NW; w++) v += sh[w * RED_MAXQ + tid];
    partial[(int64_t)blockIdx.x * RED_MAXQ + tid] = v;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = (atomicAdd(count, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int i = tid % RED_MAXQ, r0 = tid / RED_MAXQ;
  double v = 0;
  if (i < nq) {
    #pragma unroll 8
    for (int r = r0; r < (int)gridDim.x; r += ROWS) v += __ldcg(&partial[(int64_t)r * RED_MAXQ + i]);
  }
  sh[tid] = v;
  __syncthreads();
  if (tid < nq) {
    v = sh[tid];
    for (int r = 1; r < ROWS; r++) v += sh[r * RED_MAXQ + tid];
    out[tid] = v;
  }
  if (tid == 0) *count = 0;
  return true;
}

// Points a thread loads before it uses the first: with 32 warps on an SM
// four 16-byte loads each keep 64 KB in flight, more than the ~45 KB that
// HBM's latency times its rate asks of an SM.
constexpr int RED_AHEAD = 4;

template <typename R, int MODE>
__global__ void __launch_bounds__(RED_THREADS) reduce_kernel(RedArgs a, double *partial, unsigned *count, double *out) {
  double q[RED_MAXQ];
  #pragma unroll
  for (int i = 0; i < RED_MAXQ; i++) q[i] = 0;
  pdl_wait();
  const int64_t stride = (int64_t)gridDim.x * RED_THREADS;
  for (int64_t l0 = blockIdx.x * (int64_t)RED_THREADS + threadIdx.x; l0 < a.g.npts; l0 += RED_AHEAD * stride) {
    RedIn<R, MODE> in[RED_AHEAD];
    #pragma unroll
    for (int u = 0; u < RED_AHEAD; u++)
      if (l0 + u * stride < a.g.npts) red_fetch<R, MODE>(a, l0 + u * stride, in[u]);
    #pragma unroll
    for (int u = 0; u < RED_AHEAD; u++)
      if (l0 + u * stride < a.g.npts) red_point<R, MODE>(a, l0 + u * stride, in[u], q);
  }
  red_finish<RED_THREADS>(q, a.nq, partial, count, out);
}


}  // namespace atus
