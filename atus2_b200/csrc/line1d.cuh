// line1d.cuh -- a whole 1D Strang block with the field on chip: one CTA, or a
// thread-block cluster of C CTAs that exchange through distributed shared
// memory.  Single contexts (line1d_kernel) and the batched sweep's 1D classes
// (line1d_batch_kernel) share it.
//
// N = 8 P points of one or two components, 8 values per thread in registers
// from the first load to the last store.  With n = p + P r (r < 8) and
// k = k1 + 8 k2 (k1 < 8):
//
//   X[k1 + 8 k2] = sum_p W_P^{p k2} W_N^{p k1} sum_r x[p + P r] W_8^{r k1}.
//
// Home layout: a thread holds column p, points p + P r: the radix-8 DFT over r
// and the potential step are in registers.  Bin layout: the 8 pencils y[.][k1]
// of P points are dealt out to the C CTAs (8 / C each), M = P / 8 threads a
// pencil, thread t holding points t + M m: a Stockham transform (first radix
// 2, 4 or 8, then 8 throughout) starts and ends in that layout, so the kinetic
// factor is applied in registers too.  A kinetic step is: radix 8 and twiddles
// W_N^{p k1}, exchange home -> bin, P-point transform, factor, inverse
// transform, exchange bin -> home, conjugate twiddles, radix 8.  The two
// exchanges are the only ones that leave a warp (P <= 256), a CTA (C = 1) or
// cross the cluster (remote stores, then one cluster barrier each); they have
// a buffer each, so the barrier of one covers the reuse of the other.
//
// Why 8 values: a block advances one step after another, so what counts is the
// latency of a step.  16 values a thread leave 4096 points to 256 threads, and
// the radix-16 butterflies of the shared-memory transform this replaces ran in
// 16 threads of each CTA; 8 values put two to four times the warps on the same
// butterflies, and no stage but an exchange touches shared memory.
//
// Held per block, not recomputed per step: W_N^{p k1}; the constant part of a
// point's phase, e^{-i dt V}; cos and sin of k x for the Bragg coupling
// (cos(k x + theta_j) by the addition theorem, theta_j of 64 steps at a time by
// 64 threads); eta.  The kinetic factors of the full step are in shared memory.
// In FP64 throughout for these, whatever the field type.
#pragma once
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace atus {

// Gaussian pulse envelope exp(-(t - tc)^2 / (2 sigma^2)); two_sigma2 <= 0: 1.
struct Pulse {
  double tc, two_sigma2;
};
__device__ __forceinline__ double pulse_at(const Pulse &p, double t) {
  if (p.two_sigma2 <= 0.0) return 1.0;
  const double u = t - p.tc;
  return exp(-(u * u) / p.two_sigma2);
}

// One run: fields, tables, parameters.
struct LineInst {
  void *psi[2];
  const double2 *kh[2], *kf[2];  // half / full kinetic factors (FP64, N entries)
  double s_f, s_b;               // transform scales
  Pulse pulse;                   // used where no amplitudes are given
  NLArgs nl;
  int fs_lg1, fs_lg2;            // kinetic tables in four-step order (logs of the view), or 0
};
constexpr int LINE_F_INLINE = 32;  // pulse amplitudes that travel with the launch
struct LineArgs {
  LineInst in;
  const void *tw;
  int nk, nf;                    // nf: amplitudes in f[] (then F is not read)
  double t0;
  const double *F;               // nk amplitudes in device memory, or nullptr: in.pulse
  double f[LINE_F_INLINE];
};

constexpr int LINE_CHUNK = 64;   // steps whose couplings are prepared together

// Exchanges of a P-point transform (first radix r0, then 8).
__host__ __device__ constexpr int n_line(int P, int r0) { return r0 >= P ? 0 : 1 + n_line(P, r0 * 8); }

template <typename R, int N, int TC, int C>
struct LineCfg {
  using V = cplx<R>;
  static constexpr int P = N / 8, M = P / 8;
  static constexpr int COLS = P / C;           // columns (threads per component) of a CTA
  static constexpr int PB = 8 / C;             // pencils of a CTA
  static constexpr int NT = COLS * TC;
  static constexpr int LG = lg2c(P) % 3;       // first radix of the P-point transform
  static constexpr int R0 = P == 1 ? 1 : LG == 0 ? 8 : LG == 1 ? 2 : 4;
  static constexpr int PS = P + P / 8 + (M < 8 ? 4 : 0);  // pencil pitch, one pad per 8 elements
  // component pitch: = half a 128-byte wavefront, so that the two components'
  // lanes (alternating) do not meet in a bank
  static constexpr int HALF = 64 / (int)sizeof(V);
  static constexpr int CS = (PB * PS + 2 * HALF - 1) / (2 * HALF) * (2 * HALF) + HALF;
  static constexpr size_t buf = sizeof(V) * TC * CS;      // one exchange buffer
  static constexpr int TWL = P;                           // local twiddles: sum of 7 Ns < P
  static constexpr size_t smem_tw = sizeof(typename TwTab<R>::type) * TWL;
  static constexpr size_t smem_k = sizeof(double2) * TC * PB * P;
  static constexpr size_t smem = 3 * buf + smem_tw + smem_k;
  // the field fits, with whole warps and at most 128 registers a thread to ask for
  static constexpr bool fits = N >= 256 && C <= 8 && NT >= 32 && NT <= 512 && M >= 1 && smem + 8192 <= 227 * 1024;
};

// CTAs of a single context's block: as many as shorten a step.  Measured, us a
// step (one component with a potential / two components bragg_ad, FP64 in the
// eigenvalue form; last column: the FP64 kernels these replace, one CTA up to
// 1024 points, 16 CTAs up to 8192, four-step passes beyond):
//   points      1 CTA        2            4            8          before
//   FP64
//     256    1.6 / 2.6    -- / 3.1     --           --          2.8 / 4.2
//     512    1.4 / 2.9   1.9 / 3.2    -- / 3.2     --           4.3 / 6.6
//    1024    2.1 / 4.8   2.3 / 4.0   2.2 / 3.8    -- / 3.7      5.6 / 10.7
//    2048    3.3 / --    2.8 / 6.2   2.5 / 4.8   2.5 / 4.2      4.9 / 6.4
//    4096       --       4.9 / --    3.4 / 6.7   2.9 / 5.0      6.7 / 8.7
//    8192       --          --       6.1 / --    4.2 / 8.2      9.4 / 12.5
//   16384       --          --          --       6.8 / --      42.1 / 55.6
//   complex64
//     256    1.4 / 1.8    -- / 2.2     --           --
//     512    1.4 / 1.9   1.8 / 2.3    -- / 2.3     --
//    1024    1.8 / 3.2   2.1 / 2.7   2.1 / 2.6    -- / 2.6
//    2048    3.0 / 5.8   2.5 / 4.0   2.3 / 3.0   2.3 / 2.8
//    4096    5.5 / --    3.9 / 6.9   2.7 / 4.3   2.4 / 3.4
//    8192       --       7.9 / --    4.9 / 8.5   3.4 / 5.1
//   16384       --          --       8.9 / --    5.4 / 9.2
// (-- : does not fit, or leaves a CTA less than a warp.)  The counts taken are
// within 3 % of the fastest at every length, precision and component count.
template <typename R, int N, int TC> constexpr int line_ctas = N <= 512 ? 1 : N == 1024 ? (TC == 1 ? 1 : 4) : 8;

// dft8 with 1/sqrt 2 as hi + lo in FP64 too (FP32 always: kmul).  The constant
// is 6.8e-17 (relative) too large as a double; a quarter of the values take it
// in each of eight stages a step, so the norm grows by 1e-16 a step and with
// it the nonlinear phase: 20000 steps of the trap run on 4096 points ended
// 9.1e-11 from the reference's arithmetic with the plain constant (numpy's FFT:
// 6.2e-11).
__device__ __forceinline__ float line_s2(float x) { return kmul(x, SQRT1_2); }
__device__ __forceinline__ double line_s2(double x) { return fma(x, SQRT1_2, x * -4.833646656726456726e-17); }
template <int DIR, typename V> __device__ __forceinline__ void line_dft8(V *v) {
  V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  V o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<DIR>(e0, e1, e2, e3);
  dft4<DIR>(o0, o1, o2, o3);
  V a1, a3;  // o1 e^{DIR i pi/4}, o3 e^{DIR 3 i pi/4}
  if (DIR < 0) {
    a1.x = line_s2(o1.x + o1.y); a1.y = line_s2(o1.y - o1.x);
    a3.x = line_s2(o3.y - o3.x); a3.y = -line_s2(o3.x + o3.y);
  } else {
    a1.x = line_s2(o1.x - o1.y); a1.y = line_s2(o1.x + o1.y);
    a3.x = -line_s2(o3.x + o3.y); a3.y = line_s2(o3.x - o3.y);
  }
  o2 = mul_i<DIR>(o2);
  v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
  v[1] = cadd(e1, a1); v[5] = csub(e1, a1);
  v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
  v[3] = cadd(e3, a3); v[7] = csub(e3, a3);
}
template <int R_, int DIR, typename V> __device__ __forceinline__ void line_dft(V *v) {
  if constexpr (R_ == 8) line_dft8<DIR>(v);
  else dftR<R_, DIR>(v);
}

__device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }

// Barrier of the threads that share a pencil.
template <bool WARP> __device__ __forceinline__ void line_sync() {
  if constexpr (WARP) __syncwarp();
  else __syncthreads();
}

// Stages of the P-point transform after the first: NS elements are already
// transformed.  bufs alternate; tw: this stage's 7 NS twiddles (row r, k).
template <typename R, int P, int DIR, int NS, bool WARP>
__device__ __forceinline__ void line_stages(cplx<R> *v, cplx<R> *b0, cplx<R> *b1, const typename TwTab<R>::type *tw,
                                            int t) {
  if constexpr (NS < P) {
    using TW = typename TwTab<R>::type;
    constexpr int M = P / 8;
    const int k = t & (NS - 1);
    TW w[8];
    #pragma unroll
    for (int r = 1; r < 8; r++) w[r] = tw[(r - 1) * NS + k];
    line_sync<WARP>();
    #pragma unroll
    for (int r = 0; r < 8; r++) v[r] = b0[pad8(t + M * r)];
    #pragma unroll
    for (int r = 1; r < 8; r++) v[r] = twmul<DIR>(v[r], w[r]);
    line_dft8<DIR>(v);
    if constexpr (NS * 8 < P) {
      const int o = (t / NS) * NS * 8 + k;
      #pragma unroll
      for (int r = 0; r < 8; r++) b1[pad8(o + r * NS)] = v[r];
      line_stages<R, P, DIR, NS * 8, WARP>(v, b1, b0, tw + 7 * NS, t);
    }
  }
}

// P-point transform of the thread's values (points t + M m in and out).  b0 is
// written first; the caller's last reads of b1 lie before the first barrier.
template <typename R, int P, int R0, int DIR, bool WARP>
__device__ __forceinline__ void line_fft(cplx<R> *v, cplx<R> *b0, cplx<R> *b1, const typename TwTab<R>::type *tw, int t) {
  using V = cplx<R>;
  constexpr int M = P / 8, T0 = 8 / R0;
  #pragma unroll
  for (int u = 0; u < T0; u++) {
    V x[R0];
    #pragma unroll
    for (int r = 0; r < R0; r++) x[r] = v[u + T0 * r];
    line_dft<R0, DIR>(x);
    if constexpr (R0 == P) {
      #pragma unroll
      for (int r = 0; r < R0; r++) v[u + T0 * r] = x[r];
    } else {
      #pragma unroll
      for (int r = 0; r < R0; r++) b0[pad8((t + M * u) * R0 + r)] = x[r];
    }
  }
  line_stages<R, P, DIR, R0, WARP>(v, b0, b1, tw, t);
}

// All of a run's steps; see the head of the file.  tid-mapping: component c =
// tid % TC, column / bin thread tau = tid / TC.
// BRAGG: nl.kind is K_BRAGG (two components); else pure phases.
template <typename R, int N, int TC, int C, bool BRAGG>
__device__ __forceinline__ void line_run(const LineInst &in, const NLArgs &nl, const double *F, int nf, int nk, double t0,
                                         const void *twv, unsigned char *smem, double2 *s_th, double *s_t) {
  using V = cplx<R>;
  using TW = typename TwTab<R>::type;
  using Cfg = LineCfg<R, N, TC, C>;
  constexpr int P = Cfg::P, M = Cfg::M, COLS = Cfg::COLS, PB = Cfg::PB, NT = Cfg::NT, PS = Cfg::PS, CS = Cfg::CS;
  constexpr bool WARP = M * TC <= 32;  // a pencil's threads are lanes of one warp
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int q = C > 1 ? (int)cl.block_rank() : 0;
  V *const XA = reinterpret_cast<V *>(smem);                  // home -> bin
  V *const HB = reinterpret_cast<V *>(smem + Cfg::buf);       // bin -> home
  V *const L = reinterpret_cast<V *>(smem + 2 * Cfg::buf);    // local
  TW *const twl = reinterpret_cast<TW *>(smem + 3 * Cfg::buf);
  double2 *const ks = reinterpret_cast<double2 *>(smem + 3 * Cfg::buf + Cfg::smem_tw);
  const int tid = threadIdx.x, c = tid % TC, tau = tid / TC;
  const int p = q * COLS + tau;               // home: column
  const int b = tau / M, t = tau % M;         // bin: local pencil, thread of it
  const int k1 = q * PB + b;
  const int sw = TC == 2 ? 4 * c : 0;         // register r holds point p + P (r ^ sw)
  const int sg = (TC == 2 && c) ? (int)0x80000000 : 0;
  const TW *const tw = static_cast<const TW *>(twv);
  const double dt = nl.dt;
  // wavenumber index -> entry of the kinetic tables
  auto kat = [&](int k) { return in.fs_lg1 ? ((k & ((1 << in.fs_lg1) - 1)) << in.fs_lg2) + (k >> in.fs_lg1) : k; };

  // tables: local twiddles (stage by stage, row r then k), kinetic factors
  {
    int base = 0;
    #pragma unroll
    for (int NS = Cfg::R0; NS < P; NS *= 8) {
      for (int e = tid; e < 7 * NS; e += NT) {
        const int r = e / NS + 1, k = e % NS;
        twl[base + e] = tw[(r * k) * (TWN / (8 * NS))];
      }
      base += 7 * NS;
    }
    for (int e = tid; e < TC * PB * P; e += NT) {
      const int cc = e / (PB * P), bb = (e / P) % PB, k2 = e % P;
      const double2 *kf = TC == 2 && cc ? in.kf[1] : in.kf[0];
      ks[e] = kf[kat(q * PB + bb + 8 * k2)];
    }
  }
  TW wn[8];
  #pragma unroll
  for (int r = 1; r < 8; r++) wn[r] = tw[(p * r) * (TWN / N)];

  V *const fld = static_cast<V *>(TC == 2 && c ? in.psi[1] : in.psi[0]);
  V v[8];
  #pragma unroll
  for (int r = 0; r < 8; r++) v[r] = fld[p + P * (r ^ sw)];

  // what a point's phase and coupling keep over the steps
  static_assert(!BRAGG || TC == 2, "the Bragg step couples two components");
  constexpr int NS_ = TC == 2 ? 4 : 1;  // points a thread steps for both components
  double2 kx[NS_], eta[NS_];
  double2 es[8];
  if constexpr (BRAGG) {
    #pragma unroll
    for (int m = 0; m < NS_; m++) {
      const double x0 = (double)(p + P * (m ^ sw) - nl.shift0) * nl.dx0;
      sincos(nl.L.laser_k0 * x0, &kx[m].y, &kx[m].x);
      eta[m] = make_double2(1.0, 0.0);
      if (nl.L.laser_dk0 != 0.0) sincos(-0.5 * (nl.L.laser_dk0 * x0), &eta[m].y, &eta[m].x);
    }
  } else {
    const double *const Vp = nl.kind == K_NL ? (TC == 2 && c ? nl.V[1] : nl.V[0]) : nullptr;
    const double beta = (nl.kind == K_NL_IF2 && TC == 2 && c) ? nl.L2.beta0 : nl.L.beta0;
    const double dl = TC == 2 && c ? nl.L.DeltaL[1] : nl.L.DeltaL[0];
    #pragma unroll
    for (int r = 0; r < 8; r++) {
      const int i = p + P * (r ^ sw);
      double ph = 0.0;
      if (nl.kind == K_NL) { if (Vp) ph = Vp[i]; }
      else ph = beta * ((double)(i - nl.shift0) * nl.dx0) - dl;
      sincos(ph * nl.mdt, &es[r].y, &es[r].x);
    }
  }
  const double g_oo = TC == 2 && c ? nl.gs[MAXC + 1] : nl.gs[0], g_ot = TC == 2 ? (c ? nl.gs[MAXC] : nl.gs[1]) : 0.0;

  auto cross_sync = [&]() {
    if constexpr (C > 1) cl.sync();
    else __syncthreads();
  };
  cross_sync();  // tables written; every CTA of the cluster is there
  // one kinetic step; half: factors from global memory (twice a block)
  auto kinetic = [&](bool half) {
    line_dft8<-1>(v);
    if constexpr (TC == 2) {  // inputs rotated by 4 negate the odd outputs
      #pragma unroll
      for (int r = 1; r < 8; r += 2) v[r] = flip(v[r], sg);
    }
    #pragma unroll
    for (int r = 0; r < 8; r++) {
      if (r) v[r] = twmul<-1>(v[r], wn[r]);
      V *dst = XA;
      if constexpr (C > 1) dst = cl.map_shared_rank(XA, r / PB);
      dst[c * CS + (r % PB) * PS + p] = v[r];
    }
    cross_sync();
    V *const my = XA + c * CS + b * PS, *const loc = L + c * CS + b * PS;
    #pragma unroll
    for (int m = 0; m < 8; m++) v[m] = my[t + M * m];
    // exchanges alternate between L and XA; the inverse transform goes on
    // where the forward one stopped (one exchange when P is 16..64)
    constexpr bool ODD = (n_line(P, Cfg::R0) & 1) != 0;
    line_fft<R, P, Cfg::R0, -1, WARP>(v, loc, my, twl, t);
    if (half) {
      const double2 *kh = TC == 2 && c ? in.kh[1] : in.kh[0];
      #pragma unroll
      for (int m = 0; m < 8; m++) v[m] = kin_mul<R>(v[m], __ldg(&kh[kat(k1 + 8 * (t + M * m))]), in.s_f, in.s_b);
    } else {
      const double2 *kf = ks + (c * PB + b) * P + t;
      #pragma unroll
      for (int m = 0; m < 8; m++) v[m] = kin_mul<R>(v[m], kf[M * m], in.s_f, in.s_b);
    }
    line_fft<R, P, Cfg::R0, +1, WARP>(v, ODD ? my : loc, ODD ? loc : my, twl, t);
    #pragma unroll
    for (int m = 0; m < 8; m++) {
      // point t + M m of pencil k1 belongs to column t + M m: CTA and thread of it
      const int col = t + M * m;
      V *dst = HB;
      if constexpr (C > 1) dst = cl.map_shared_rank(HB, col / COLS);
      dst[c * CS + k1 * COLS + col % COLS] = v[m];
    }
    cross_sync();
    #pragma unroll
    for (int r = 0; r < 8; r++) {
      v[r] = HB[c * CS + r * COLS + tau];
      if (r) v[r] = twmul<+1>(v[r], wn[r]);
    }
    if constexpr (TC == 2) {  // outputs come out rotated by 4
      #pragma unroll
      for (int r = 1; r < 8; r += 2) v[r] = flip(v[r], sg);
    }
    line_dft8<+1>(v);
  };

  kinetic(true);
  double th = t0 + 0.5 * dt;  // header time, added up as the reference does
  for (int j = 0; j < nk; j++) {
    if (BRAGG && j % LINE_CHUNK == 0) {
      // pulse amplitude and phase of the next steps: Omega = A cos(k x + theta)
      __syncthreads();
      if (tid == 0) {
        for (int s = 0; s < LINE_CHUNK && j + s < nk; s++) {
          s_t[s] = th + 0.5 * dt;
          th += dt;
        }
      }
      __syncthreads();
      for (int s = tid; s < LINE_CHUNK && j + s < nk; s += NT) {
        const double t1 = s_t[s];
        const double A = (nf ? F[j + s] : pulse_at(in.pulse, t1)) * nl.L.Amp0;
        const double ph = nl.L.phase0 / 2 - (nl.L.laser_domh0 + nl.L.chirp * t1 + nl.L.chirp_rate0 * t1) * t1;
        double sn, cs;
        sincos(ph, &sn, &cs);
        s_th[s] = make_double2(A * cs, A * sn);
      }
      __syncthreads();
    }
    if constexpr (BRAGG) {
      {
        const double2 a = s_th[j % LINE_CHUNK];
        #pragma unroll
        for (int m = 0; m < 4; m++) {
          V own = v[m], oth = shfl_xor_c(v[m + 4], 1);
          bragg_pair_at<R>(nl, nl.stable, c, (double)(p + P * (m ^ sw) - nl.shift0) * nl.dx0,
                           kx[m].x * a.x - kx[m].y * a.y, eta[m].x, eta[m].y, own, oth);
          v[m] = own;
          v[m + 4] = shfl_xor_c(oth, 1);
        }
      }
    } else {
      #pragma unroll
      for (int r = 0; r < 8 / TC; r++) {
        const double a0 = (double)v[r].x * (double)v[r].x + (double)v[r].y * (double)v[r].y;
        if constexpr (TC == 2) {  // registers r and r + 4 together: their densities cross over
          const double a1 = (double)v[r + 4].x * (double)v[r + 4].x + (double)v[r + 4].y * (double)v[r + 4].y;
          const double f0 = g_oo * a0 + g_ot * __shfl_xor_sync(0xffffffffu, a1, 1);
          const double f1 = g_oo * a1 + g_ot * __shfl_xor_sync(0xffffffffu, a0, 1);
          v[r] = from_d<R>(cmul(to_d<R>(v[r]), cmul(es[r], expi_f<double>(f0 * nl.mdt))));
          v[r + 4] = from_d<R>(cmul(to_d<R>(v[r + 4]), cmul(es[r + 4], expi_f<double>(f1 * nl.mdt))));
        } else {
          v[r] = from_d<R>(cmul(to_d<R>(v[r]), cmul(es[r], expi_f<double>(g_oo * a0 * nl.mdt))));
        }
      }
    }
    kinetic(j == nk - 1);
  }
  #pragma unroll
  for (int r = 0; r < 8; r++) fld[p + P * (r ^ sw)] = v[r];
}

template <typename R, int N, int TC, int C, bool BRAGG>
__global__ void __launch_bounds__(LineCfg<R, N, TC, C>::NT, 1) line1d_kernel(const __grid_constant__ LineArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ double2 s_th[LINE_CHUNK];
  __shared__ double s_t[LINE_CHUNK];
  line_run<R, N, TC, C, BRAGG>(a.in, a.in.nl, a.nf ? a.f : a.F, a.nf || a.F, a.nk, a.t0, a.tw, smem_raw, s_th, s_t);
}

// Runs order[0..ninst) of insts (t0 indexed alike), cluster by cluster.
template <typename R, int N, int C>
__global__ void __launch_bounds__(LineCfg<R, N, 2, C>::NT, 1)
    line1d_batch_kernel(const LineInst *__restrict__ insts, const int *__restrict__ order, const double *__restrict__ t0,
                        int ninst, int nk, const void *tw) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ double2 s_th[LINE_CHUNK];
  __shared__ double s_t[LINE_CHUNK];
  // the run's parameters in shared memory (~0.6 KB: a per-thread copy would
  // sit in local memory)
  __shared__ LineInst in;
  for (int k = blockIdx.x / C; k < ninst; k += gridDim.x / C) {
    const int id = order[k];
    static_assert(sizeof(LineInst) % 8 == 0, "copied in 8-byte words");
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&insts[id]);
    for (int e = threadIdx.x; e < (int)(sizeof(LineInst) / 8); e += blockDim.x)
      reinterpret_cast<unsigned long long *>(&in)[e] = src[e];
    __syncthreads();
    line_run<R, N, 2, C, true>(in, in.nl, nullptr, 0, nk, t0[id], tw, smem_raw, s_th, s_t);
    if constexpr (C > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();  // shared memory is reused by the next run
  }
}

}  // namespace atus
