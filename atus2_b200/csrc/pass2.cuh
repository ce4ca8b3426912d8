// pass2.cuh -- register-staged pass kernel for pencils of 32..256 points.
//
// A pencil of N = 16 R2 points is transformed in the two Stockham stages of
// fft_tile (radix 16 over inputs j + R2 r, then radix R2 with twiddles
// exp(-+2 pi i r k / N)), with the same arithmetic in the same order.  What
// differs is where the data lives between the stages:
//
//   HBM -> registers (stage-1 inputs)  -> stage 1 -> shared exchange ->
//   stage 2 -> registers (outputs j + R2 m, m < 16) -> HBM
//
// The thread that reads inputs j + R2 r (r < 16) of stage 1 ends up with the
// outputs j + R2 m of stage 2, which are again the inputs of a stage 1.  So
// FFT -> point-wise operator -> IFFT runs in registers with one shared-memory
// exchange per transform, where the tile kernel (pass_kernel) makes six sweeps
// through shared memory per transform plus the tile load and store.  Twiddles
// come from a padded per-pencil-length table in shared memory.
//
// Thread layout: along a strided axis consecutive threads take consecutive
// pencils (the inner grid index), so one warp-wide load covers whole 128-byte
// rows; along the contiguous axis consecutive threads take consecutive points.
#pragma once
#include <type_traits>

#include "kernels.cuh"

namespace atus {

// Tile budget (complex values) and threads; one thread owns 16 values.
template <typename R> struct Tile2;
template <> struct Tile2<double> { static constexpr int E = 2048, NT = 128, MINB = 5; };
template <> struct Tile2<float> { static constexpr int E = 4096, NT = 256, MINB = 3; };

// CTAs per SM the register budget is sized for: the passes at the ends of a
// Sobolev iteration, the potential passes and the four-step passes hold
// potential values or twiddles beside a thread's 16 points (256^3, one
// component, z pass: 5 CTAs with spills 207 us, 4 without 178 us).
template <typename R, int MODE, int TC = 1>
constexpr int p2_minb =
    TC >= 3 ? (TC == 3 ? 3 : sizeof(R) == 8 ? 4 : 2) :
    (((MODE >= M2_FWD_SOB && MODE < M2_FILT) || MODE == M2_NL) && sizeof(R) == 8) ? 4 : Tile2<R>::MINB;

// Passes whose two components meet inside a warp (the batched passes; a
// single grid's run in pass2_pair.cuh).
template <int TC, int MODE, bool STRIDED> constexpr bool p2_pair = (MODE == M2_NL && TC == 2 && !STRIDED);

template <typename R, int N, int TC>
struct P2Cfg {
  static constexpr int R2 = N / 16;        // stage-2 radix
  static constexpr int T2 = 16 / R2;       // stage-2 butterflies per thread
  // threads: a power of two of pencil-components, or, for three components
  // (no quarter of the threads idle), three times one
  static constexpr int NT = TC == 3 ? 192 : Tile2<R>::NT;
  static constexpr int B = NT / (R2 * TC); // pencils per tile
  static constexpr int NPC = B * TC;       // pencil-components per tile
  static constexpr int PB = 17 * R2 + 1;   // exchange pitch: R2 rows of 16 + 1 pad, odd
  static constexpr int TP = R2 + 1;        // twiddle row pitch (odd)
  static constexpr int TWP = 16 * TP;      // twiddle table: row k holds W_N^{r k}, r < R2
  static constexpr size_t smem_ex = (sizeof(cplx<R>) * NPC * PB + 15) / 16 * 16;  // 16-byte twiddles follow
  static constexpr size_t smem_tw = sizeof(typename TwTab<R>::type) * TWP;
  static constexpr size_t smem = smem_ex + smem_tw;
  // k-space passes also keep the along-axis kinetic factors of up to two
  // components in shared memory (FP64)
  static constexpr size_t smem_kin = smem + 2 * N * sizeof(double2);
  // the kinetic factors go to shared memory only if that keeps MINB CTAs per SM
  static constexpr bool kin_smem = (smem_kin + 1024) * Tile2<R>::MINB <= 228 * 1024;
};

// Exchange layout of one pencil-component: row-major R2 x 16 with row pitch
// 17.  Stage-1 butterfly j writes row j (its 16 outputs, Stockham index
// 16 j + q); stage-2 butterfly k reads column k.  Point i of the natural order
// sits at row i / 16, column i % 16.
__device__ __forceinline__ int ex_at(int row, int col) { return 17 * row + col; }

// Stage 2 of a transform: butterflies k = j + R2 t (t < T2) of the pencil whose
// exchange rows start at ex; o[t + T2 r] = output k + 16 r = point j + R2 (t + T2 r).
// Twiddle W_N^{r k} is entry r of row k (pitch R2 + 1, odd): the eight threads
// of a quarter warp, which hold eight different k on the contiguous axis, hit
// eight different bank groups.
// sg (0 or the sign bit): with the odd inputs of every radix-R2 DFT negated its
// outputs come out rotated by R2 / 2, so o[m] is point j + R2 (m ^ 8).
template <typename R, int N, int DIR, bool FLIP = false>
__device__ __forceinline__ void p2_stage2(const cplx<R> *ex, const typename TwTab<R>::type *twS, int j, cplx<R> *o,
                                          int sg = 0) {
  using C = cplx<R>;
  constexpr int R2 = N / 16, T2 = 16 / R2;
  #pragma unroll
  for (int t = 0; t < T2; t++) {
    const int k = j + R2 * t;
    C u[R2];
    #pragma unroll
    for (int r = 0; r < R2; r++) u[r] = ex[ex_at(r, k)];
    #pragma unroll
    for (int r = 1; r < R2; r++) u[r] = twmul<DIR>(u[r], twS[k * (R2 + 1) + r]);
    if constexpr (FLIP) {
      #pragma unroll
      for (int r = 1; r < R2; r += 2) u[r] = flip(u[r], sg);
    }
    dftR<R2, DIR>(u);
    #pragma unroll
    for (int r = 0; r < R2; r++) o[t + T2 * r] = u[r];
  }
}

// One transform of the thread's 16 values v (stage-1 inputs j + R2 r on entry,
// points j + R2 m on return).  The leading barrier protects the exchange rows
// that other threads may still be reading from the previous use.  WARP: the
// R2 threads of each pencil are consecutive lanes of one warp (the contiguous
// mapping), so the exchange needs only a warp barrier; the strided mapping
// spreads a pencil over the CTA's warps and needs the CTA barrier.  FLIP (in
// or out: 1 or 2) with sg set: the 16 values come in, or go out, in the order
// m ^ 8 (inputs rotated by 8 negate the odd outputs of a 16-point DFT).
template <typename R, int N, int DIR, bool WARP = false, int FLIP = 0>
__device__ __forceinline__ void p2_transform(cplx<R> *v, cplx<R> *ex, const typename TwTab<R>::type *twS, int j,
                                             int sg = 0) {
  dft16<DIR>(v);
  if constexpr (FLIP == 1) {
    #pragma unroll
    for (int q = 1; q < 16; q += 2) v[q] = flip(v[q], sg);
  }
  if constexpr (WARP) __syncwarp(); else __syncthreads();
  #pragma unroll
  for (int q = 0; q < 16; q++) ex[ex_at(j, q)] = v[q];
  if constexpr (WARP) __syncwarp(); else __syncthreads();
  p2_stage2<R, N, DIR, FLIP == 2>(ex, twS, j, v, sg);
}

// Shared-memory set-up of a CTA, once per launch: the twiddle rows and, for
// k-space passes, the along-axis kinetic factors of components 0 and 1.
// Returns whether those factors are in shared memory.
template <typename R, int N, int TC, int MODE>
__device__ __forceinline__ bool p2_setup(const PassArgs &a, unsigned char *smem_raw) {
  using TW = typename TwTab<R>::type;
  using Cfg = P2Cfg<R, N, TC>;
  constexpr int R2 = Cfg::R2, NT = Cfg::NT;
  const int tid = threadIdx.x;
  TW *const twS = reinterpret_cast<TW *>(smem_raw + Cfg::smem_ex);
  {  // W_N^{r k} = exp(-2 pi i r k / N) from the TWN-point table
    const TW *tw = (const TW *)a.tw;
    for (int e = tid; e < 16 * R2; e += NT) {
      const int k = e / R2, r = e % R2;
      twS[k * Cfg::TP + r] = tw[(r * k) * (TWN / N)];
    }
  }
  // k-space passes: along-axis kinetic factors of components 0 and 1
  double2 *const s_kt = reinterpret_cast<double2 *>(smem_raw + Cfg::smem);
  const bool kt_shared = (MODE == M2_KIN || MODE == M2_KIN_RABI) && Cfg::kin_smem && a.ncomp_grid <= 2;
  if (kt_shared) {
    for (int e = tid; e < a.ncomp_grid * N; e += NT) {
      const int cc = e / N, i = e % N;
      const double2 *t0 = (a.axis == 0) ? a.kt[0][0] : (a.axis == 1) ? a.kt[0][1] : a.kt[0][2];
      const double2 *t1 = (a.axis == 0) ? a.kt[1][0] : (a.axis == 1) ? a.kt[1][1] : a.kt[1][2];
      s_kt[e] = (cc == 0) ? t0[i] : t1[i];
    }
  }
  return kt_shared;
}

// Rabi sums of one thread's 16 values (k-space points j + R2 m of the pencil
// whose point 0 has axis indices p0) into rq, with the ball rule of
// compute_rabi_integrals (include/CRT_Base_IF.h:231-257): a point inside a
// ball adds to the current bin and the bin index does not advance for it.
template <typename R, int N>
__device__ __forceinline__ void p2_rabi(const PassArgs &a, int ci, const int *p0, int j, const cplx<R> *v, double *rq) {
  constexpr int R2 = N / 16;
  #pragma unroll 1
  for (int m = 0; m < 16; m++) {
    const int i = j + R2 * m;
    const double den = (double)v[m].x * (double)v[m].x + (double)v[m].y * (double)v[m].y;
    double k[3];
    #pragma unroll
    for (int ax = 0; ax < 3; ax++) {
      const int idx = (ax == a.axis) ? i : p0[ax];
      const int sh = a.n[ax] / 2;
      const int t = (idx + sh) % a.n[ax];
      k[ax] = a.dk[ax] * (double)(t - sh);
    }
    red_balls<3>(&a.rabi_k0[ci * a.rabi_n], a.rabi_n, a.rabi_thr, k, den, &rq[ci * a.rabi_n]);
  }
}

// sum_j g_j |psi_j|^2 at grid index l (several components).
__device__ __forceinline__ double sob_interaction(const PassArgs &a, int64_t l) {
  double nl = 0;
  #pragma unroll
  for (int c = 0; c < MAXC; c++) {
    if (c < a.sob_ncomp) {
      const double2 p = a.sob_psi[c][l];
      nl += a.sob_gs[c] * (p.x * p.x + p.y * p.y);
    }
  }
  return nl;
}

// Bragg coupling of pencil b of tile g (contiguous axis).
__device__ __forceinline__ void p2_coupling(const PassArgs &a, const TileGeo &g, int b, double &om, double &ec,
                                            double &es) {
  om = 0;
  ec = 1;
  es = 0;
  if (b < g.nb) {
    int ix, iy, iz;
    idx3(a.g, g.base0 + b * g.pstride, ix, iy, iz);
    bragg_coupling(a.nl, (double)(ix - a.nl.shift0) * a.nl.dx0, om, ec, es);
  }
}

// After-load hook of p2_item (the TMA kernel refills the tile buffer there).
struct P2NoHook {
  __device__ __forceinline__ void operator()() const {}
};

// Tile of a strided pass as a TMA box writes it: row i (point i of the B
// pencils) is B values.  Rows of 128 bytes come with the 128-byte swizzle
// (16-byte chunk c at position c ^ (i & 7)); longer rows unswizzled (the
// threads of a quarter warp read consecutive pencils of one row).  Value of
// pencil b at point i.
template <typename R, int B>
__device__ __forceinline__ cplx<R> p2_tile_at(const unsigned char *tile, int i, int b) {
  constexpr int ROW = B * (int)sizeof(cplx<R>);
  if constexpr (ROW != 128)
    return *reinterpret_cast<const cplx<R> *>(tile + i * ROW + b * (int)sizeof(cplx<R>));
  else if constexpr (sizeof(R) == 8)
    return *reinterpret_cast<const cplx<R> *>(tile + i * 128 + ((b ^ (i & 7)) << 4));
  else
    return *reinterpret_cast<const cplx<R> *>(tile + i * 128 + (((b >> 1) ^ (i & 7)) << 4) + ((b & 1) << 3));
}

// One work item.  SMEM_TILE (strided passes): the tile's inputs come from
// `tile` (swizzled, see p2_tile_at) instead of global memory, and hook()
// runs once every thread has taken its values.
template <typename R, int N, int TC, int MODE, bool STRIDED, bool SMEM_TILE = false, typename Hook = P2NoHook>
__device__ __forceinline__ void p2_item(const PassArgs &a, const TileGeo &g, unsigned char *smem_raw, bool kt_shared,
                                        double *s_om, double *s_ec, double *s_es, double *rq = nullptr,
                                        const unsigned char *tile = nullptr, Hook hook = Hook()) {
  using C = cplx<R>;
  using TW = typename TwTab<R>::type;
  using Cfg = P2Cfg<R, N, TC>;
  constexpr int R2 = Cfg::R2, B = Cfg::B, NT = Cfg::NT, PB = Cfg::PB;
  static_assert(N >= 32 && N <= 256, "two-stage pencils only");
  static_assert(Cfg::NPC * R2 == NT, "one thread per stage-1 butterfly");
  C *const ex = reinterpret_cast<C *>(smem_raw);
  const TW *const twS = reinterpret_cast<const TW *>(smem_raw + Cfg::smem_ex);
  const double2 *const s_kt = reinterpret_cast<const double2 *>(smem_raw + Cfg::smem);
  const int tid = threadIdx.x;
  // PAIR: the two components of a pencil in one warp, so that the potential
  // step meets through shuffles (nl_pair16); exchange rows (b, c) at a pitch
  // of 17 R2, which spreads the lanes of a bank group over the banks
  constexpr bool PAIR = p2_pair<TC, MODE, STRIDED>;
  int b, j, c;
  if (STRIDED) { b = tid % B; j = (tid / B) % R2; c = tid / (B * R2); }
  else if (PAIR) { j = tid % R2; c = (tid / R2) & 1; b = tid / (2 * R2); }
  else { j = tid % R2; b = (tid / R2) % B; c = tid / (R2 * B); }
  C *const my = PAIR ? ex + (2 * b + c) * (17 * R2) : ex + (c * B + b) * PB;
  const int nc = a.per_comp ? 1 : a.nc;
  const bool live = (b < g.nb) && (c < nc);
  C *const f = (C *)pick(a.psi, g.comp0 + c);
  const int64_t lb = g.base0 + b * g.pstride;  // grid index of the pencil's point 0
  const int64_t step = (int64_t)R2 * a.sa;     // distance of points j + R2 m and j + R2 (m+1)
  const C *src = live ? f + lb + (int64_t)j * a.sa : nullptr;

  if constexpr (MODE == M2_NL && TC > 2) {
    // coupling of each pencil (x is constant along it); read after the
    // barriers of the first transform
    for (int p = tid; p < B; p += NT)
      if (p < g.nb) {
        int ix, iy, iz;
        idx3(a.g, g.base0 + p * g.pstride, ix, iy, iz);
        coupling_x(a.nl, (double)(ix - a.nl.shift0) * a.nl.dx0, s_om + NCPL * p);
      }
  }
  if constexpr (MODE == M2_NL_MEET) {
    if (a.nl.kind == K_BRAGG)
    for (int p = tid; p < B; p += NT) {
      double om = 0, ec = 1, es = 0;
      if (p < g.nb) {
        int ix, iy, iz;
        idx3(a.g, g.base0 + p * g.pstride, ix, iy, iz);
        bragg_coupling(a.nl, (double)(ix - a.nl.shift0) * a.nl.dx0, om, ec, es);
      }
      s_om[p] = om; s_ec[p] = ec; s_es[p] = es;
    }
  }

  C v[16];
  if constexpr (SMEM_TILE) {
    static_assert(STRIDED, "shared-memory tiles of strided passes only");
    #pragma unroll
    for (int r = 0; r < 16; r++) v[r] = p2_tile_at<R, B>(tile, j + R2 * r, b);
    hook();
  } else if constexpr (MODE == M2_FWD_SOB) {
    // item component 0: psi, 1: W psi, W = V + sum_j g_j |psi_j|^2
    const double2 *const own = pick(a.sob_psi, a.sob_comp) + lb + (int64_t)j * a.sa;
    const double *const Vp = a.nl.V[0];
    #pragma unroll
    for (int r = 0; r < 16; r++) v[r] = live ? own[r * step] : mk<R>(0, 0);
    if (live && g.comp0 == 1) {
      #pragma unroll
      for (int r = 0; r < 16; r++) {
        const int64_t l = lb + (int64_t)(j + R2 * r) * a.sa;
        double W = Vp ? __ldg(&Vp[l]) : 0.0;
        W += a.sob_ncomp == 1 ? a.sob_gs[0] * (v[r].x * v[r].x + v[r].y * v[r].y) : sob_interaction(a, l);
        v[r].x *= W;
        v[r].y *= W;
      }
    }
  } else {
    #pragma unroll
    for (int r = 0; r < 16; r++) v[r] = live ? src[r * step] : mk<R>(0, 0);
  }

  // outputs times W_N^{r c} or its conjugate (four-step passes)
  auto fs_twiddle = [&](auto dir) {
    constexpr int DIR = decltype(dir)::value;
    const double2 *const T = a.fs_tw + lb + (int64_t)j * a.sa;
    if (live) {
      #pragma unroll
      for (int m = 0; m < 16; m++) v[m] = fs_mul<R, DIR>(v[m], __ldg(&T[m * step]));
    }
  };

  if constexpr (MODE == M2_FS_FWD) {
    p2_transform<R, N, -1, !STRIDED>(v, my, twS, j);
    fs_twiddle(std::integral_constant<int, -1>());
  } else if constexpr (MODE == M2_FS_KIN) {
    p2_transform<R, N, -1, !STRIDED>(v, my, twS, j);
    const double2 *const K = pick_kt0(a, g.comp0) + lb + j;
    #pragma unroll
    for (int m = 0; m < 16; m++) v[m] = kin_mul<R>(v[m], __ldg(&K[R2 * m]), a.s_f, a.s_b);
    p2_transform<R, N, +1, !STRIDED>(v, my, twS, j);
    fs_twiddle(std::integral_constant<int, 1>());
  } else if constexpr (MODE == M2_FWD || MODE == M2_FWD_SOB) {
    p2_transform<R, N, -1, !STRIDED>(v, my, twS, j);
  } else if constexpr (MODE == M2_INV) {
    p2_transform<R, N, +1, !STRIDED>(v, my, twS, j);
  } else if constexpr (MODE == M2_INV_SOB) {
    p2_transform<R, N, +1, !STRIDED>(v, my, twS, j);
    // Item component 0 (v = S psi) takes every product of the iteration:
    // rq = <S psi, W psi> (= <psi, S(W psi)>, S being self-adjoint),
    // <psi, S psi>, <psi, psi>.  psi arrives in the pencil's exchange rows by
    // cp.async, all 16 points of a thread in flight without registers (two
    // 128^3 fields: 43 us; loads into registers, four at a time, 52 us; the
    // plain inverse pass and a reduction over three fields 19 + 22 us plus a
    // launch, and a sweep that forms the gradient).
    if (g.comp0 == 0) {
      const double2 *const own = pick(a.sob_psi, a.sob_comp) + lb + (int64_t)j * a.sa;
      const double *const Vp = a.nl.V[0];
      __syncwarp();  // the pencil's stage-2 reads are done
      #pragma unroll
      for (int m = 0; m < 16; m++)
        if (live) cp_async(&my[ex_at(j, m)], own + m * step, double2{});
      cp_commit();
      double W[16];
      #pragma unroll
      for (int m = 0; m < 16; m++) W[m] = (live && Vp) ? __ldg(&Vp[lb + (int64_t)(j + R2 * m) * a.sa]) : 0.0;
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      if (live) {
        #pragma unroll
        for (int m = 0; m < 16; m++) {
          const double2 p = my[ex_at(j, m)];
          const double pv = p.x * v[m].x + p.y * v[m].y, pp = p.x * p.x + p.y * p.y;
          const double w = W[m] + (a.sob_ncomp == 1
                                       ? a.sob_gs[0] * pp
                                       : sob_interaction(a, lb + (int64_t)(j + R2 * m) * a.sa));
          rq[0] += w * pv;
          rq[1] += pv;
          rq[2] += pp;
        }
      }
    }
  } else if constexpr (MODE == M2_KIN || MODE == M2_KIN_RABI || MODE == M2_FILT) {
    p2_transform<R, N, -1, !STRIDED>(v, my, twS, j);
    int p0[3];
    idx3(a.g, lb, p0[0], p0[1], p0[2]);
    if constexpr (MODE == M2_KIN_RABI) {
      int ci = -1;
      for (int c = 0; c < a.rabi_ncomp; c++)
        if (a.rabi_comp[c] == g.comp0) ci = c;
      if (live && ci >= 0) p2_rabi<R, N>(a, ci, p0, j, v, rq);
    }
    if constexpr (MODE != M2_FILT) {
      if (a.op == OP_KIN) {  // always: a branch keeps the factors' loads out of the transform above
        // psi^ <- ((psi^ s_f) K) s_b in FP64, K = K_along (product of the other
        // two axis factors, x before y before z); complex64 fields take the
        // scales folded into K
        const double2 *kx = a.kt[0][0], *ky = a.kt[0][1], *kz = a.kt[0][2];
        #pragma unroll
        for (int cc = 1; cc < MAXC; cc++)
          if (g.comp0 == cc) { kx = a.kt[cc][0]; ky = a.kt[cc][1]; kz = a.kt[cc][2]; }
        const double2 KX = __ldg(&kx[p0[0]]), KY = __ldg(&ky[p0[1]]), KZ = __ldg(&kz[p0[2]]);
        double2 Kp = (a.axis == 0) ? cmul(KY, KZ) : (a.axis == 1) ? cmul(KX, KZ) : cmul(KX, KY);
        const double2 *along = (a.axis == 0) ? kx : (a.axis == 1) ? ky : kz;
        const double2 *sk = s_kt + (g.comp0 == 1 ? N : 0);
        if (sizeof(R) == 4) {
          const double sc = a.s_f * a.s_b;
          Kp.x *= sc;
          Kp.y *= sc;
        }
        #pragma unroll
        for (int m = 0; m < 16; m++) {
          const int i = j + R2 * m;
          const double2 K = cmul(kt_shared ? sk[i] : __ldg(&along[i]), Kp);
          double2 u = to_d<R>(v[m]);
          if (sizeof(R) == 8) {
            u.x *= a.s_f;
            u.y *= a.s_f;
          }
          u = cmul(u, K);
          if (sizeof(R) == 8) {
            u.x *= a.s_b;
            u.y *= a.s_b;
          }
          v[m] = from_d<R>(u);
        }
      }
    } else {
      // alpha k^2 of the pencil's two fixed axes, and of the point's own
      auto ak2 = [&](int ax, int ii) {
        const int sh = a.n[ax] >> 1;  // lengths are powers of two
        const double k = a.dk[ax] * (double)(((ii + sh) & (a.n[ax] - 1)) - sh);
        return (k * a.filt_alpha) * k;
      };
      double rest = 0;
      #pragma unroll
      for (int ax = 0; ax < 3; ax++)
        if (ax != a.axis) rest += ak2(ax, p0[ax]);
      if (a.filt_mode == FILT_SOBOLEV && a.filt_batch) {
        // 1 / (1 + alpha k^2) of four points from one division (with the
        // axis indices wrapped by masks instead of integer division: 46 ->
        // 29 us for two 128^3 fields)
        #pragma unroll
        for (int m0 = 0; m0 < 16; m0 += 4) {
          double d[4];
          #pragma unroll
          for (int u = 0; u < 4; u++) d[u] = 1.0 + (ak2(a.axis, j + R2 * (m0 + u)) + rest);
          const double d01 = d[0] * d[1], d23 = d[2] * d[3];
          const double inv = a.filt_scale / (d01 * d23);
          const double i01 = inv * d23, i23 = inv * d01;
          const double f[4] = {i01 * d[1], i01 * d[0], i23 * d[3], i23 * d[2]};
          #pragma unroll
          for (int u = 0; u < 4; u++) {
            v[m0 + u].x = (R)((double)v[m0 + u].x * f[u]);
            v[m0 + u].y = (R)((double)v[m0 + u].y * f[u]);
          }
        }
      } else {
        #pragma unroll
        for (int m = 0; m < 16; m++) {
          const double phi = ak2(a.axis, j + R2 * m) + rest;
          const double fk = (a.filt_mode == FILT_SOBOLEV ? 1.0 / (1.0 + phi) : -phi) * a.filt_scale;
          v[m].x = (R)((double)v[m].x * fk);
          v[m].y = (R)((double)v[m].y * fk);
        }
      }
    }
    p2_transform<R, N, +1, !STRIDED>(v, my, twS, j);
  } else {  // M2_NL, M2_NL_MEET, M2_FS_NL: IFFT -> potential step -> FFT
    constexpr bool FS = (MODE == M2_FS_NL);  // axis 0 is the whole grid index
    const int sg = (PAIR && c) ? (int)0x80000000 : 0;
    p2_transform<R, N, +1, !STRIDED, PAIR ? 2 : 0>(v, my, twS, j, sg);
    if constexpr (PAIR) {
      int p0[3];
      idx3(a.g, lb, p0[0], p0[1], p0[2]);
      const double x0 = (double)(p0[0] - a.nl.shift0) * a.nl.dx0;
      const int form = pair_form<R>(a.nl);
      if (sizeof(R) == 8 && form == PAIR_EIGEN)
        nl_pair16<R, PAIR_EIGEN>(a.nl, v, c, R2, live, x0, s_om[b], s_ec[b], s_es[b], lb + j, R2);
      else if (form == PAIR_FREE)
        nl_pair16<R, PAIR_FREE>(a.nl, v, c, R2, live, x0, s_om[b], s_ec[b], s_es[b], lb + j, R2);
      else
        nl_pair16<R, PAIR_PHASE>(a.nl, v, c, R2, live, x0, 0.0, 1.0, 0.0, lb + j, R2);
    } else if constexpr (TC == 1) {
      int p0[3];
      idx3(a.g, lb, p0[0], p0[1], p0[2]);
      const int64_t l0 = lb + (int64_t)j * a.sa;
      if (FS || a.axis == 0) {
        const int i0 = FS ? (int)l0 : j;
        nl_single16<R, true>(a.nl, v, live, (double)(i0 - a.nl.shift0) * a.nl.dx0,
                             (double)(FS ? step : R2) * a.nl.dx0, l0, step);
      } else {
        nl_single16<R, false>(a.nl, v, live, (double)(p0[0] - a.nl.shift0) * a.nl.dx0, 0.0, l0, step);
      }
    } else {
      // all components of a point meet in shared memory (natural order)
      __syncthreads();
      #pragma unroll
      for (int m = 0; m < 16; m++) {
        const int i = j + R2 * m;
        my[ex_at(i >> 4, i & 15)] = v[m];
      }
      __syncthreads();
      const bool bragg = TC == 2 && (a.nl.kind == K_BRAGG);
      #pragma unroll 1  // measured fastest: unrolling 2/4/8 points was 4-50 % slower
      for (int p = tid; p < B * N; p += NT) {
        int pb, i;
        if (STRIDED) { pb = p % B; i = p / B; } else { i = p % N; pb = p / N; }
        if (pb < g.nb) {
          const int64_t l = g.base0 + pb * g.pstride + (int64_t)i * a.sa;
          int ix, iy, iz;
          idx3(a.g, l, ix, iy, iz);
          const double x0 = (double)((FS ? (int)l : ix) - a.nl.shift0) * a.nl.dx0;
          double om = 0, ec = 1, es = 0;
          if (bragg) {
            if constexpr (FS) bragg_coupling(a.nl, x0, om, ec, es);
            else { om = s_om[pb]; ec = s_ec[pb]; es = s_es[pb]; }
          }
          const double *const cp = (MODE == M2_NL && TC > 2) ? s_om + NCPL * pb : nullptr;
          C u[MAXC];
          #pragma unroll
          for (int cc = 0; cc < TC; cc++) u[cc] = ex[(cc * B + pb) * PB + ex_at(i >> 4, i & 15)];
          nl_point<R, TC, (MODE == M2_NL && TC > 2), MODE != M2_NL_MEET>(a.nl, u, l, x0, om, ec, es, cp);
          #pragma unroll
          for (int cc = 0; cc < TC; cc++) ex[(cc * B + pb) * PB + ex_at(i >> 4, i & 15)] = u[cc];
        }
      }
      __syncthreads();
      #pragma unroll
      for (int r = 0; r < 16; r++) {
        const int i = j + R2 * r;
        v[r] = my[ex_at(i >> 4, i & 15)];
      }
    }
    p2_transform<R, N, -1, !STRIDED, PAIR ? 1 : 0>(v, my, twS, j, sg);
    if constexpr (FS) fs_twiddle(std::integral_constant<int, -1>());
  }

  if (live) {
    C *dst = f + lb + (int64_t)j * a.sa;
    #pragma unroll
    for (int m = 0; m < 16; m++) dst[m * step] = v[m];
  }
}

// Strided tiles: asks L2 for the CTA's next tile (one prefetch per 128-byte
// line; the B pencils of a row are adjacent, the N rows sa apart) while this
// one is transformed, so that its loads wait on L2 rather than HBM.  (The
// same for contiguous tiles measured slower.)
template <typename R, int N, int TC>
__device__ __forceinline__ void p2_prefetch_l2(const PassArgs &a, const TileGeo &g) {
  using Cfg = P2Cfg<R, N, TC>;
  constexpr int LINE = 128 / (int)sizeof(cplx<R>);  // complex values per 128-byte line
  constexpr int SEG = (Cfg::B + LINE - 1) / LINE;
  const int nc = a.per_comp ? 1 : a.nc;
  for (int e = threadIdx.x; e < nc * N * SEG; e += Cfg::NT) {
    const int c = e / (N * SEG), rem = e % (N * SEG);
    const int i = rem / SEG, seg = rem % SEG;
    if (seg * LINE >= g.nb) continue;
    const cplx<R> *f = (const cplx<R> *)pick(a.psi, g.comp0 + c);
    const cplx<R> *p = f + g.base0 + (int64_t)(seg * LINE) * g.pstride + (int64_t)i * a.sa;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  }
}

template <typename R, int N, int TC, int MODE, bool STRIDED>
__global__ void __launch_bounds__(P2Cfg<R, N, TC>::NT, p2_minb<R, MODE, TC>) pass2_kernel(PassArgs a) {
  using Cfg = P2Cfg<R, N, TC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_om[TC > 2 ? NCPL * Cfg::B : Cfg::B], s_ec[Cfg::B], s_es[Cfg::B];  // couplings of the pencils
  const bool kt_shared = p2_setup<R, N, TC, MODE>(a, smem_raw);
  pdl_wait();
  __syncthreads();  // twiddle rows and kinetic factors visible to every warp
  const int64_t W = a.per_comp ? a.ntiles * a.ncomp_grid : a.ntiles;
  constexpr bool SUMS = (MODE == M2_KIN_RABI || MODE == M2_INV_SOB);
  double rq[SUMS ? RED_MAXQ : 1];
  #pragma unroll
  for (int q = 0; q < (SUMS ? RED_MAXQ : 1); q++) rq[q] = 0.0;
  for (int64_t w = blockIdx.x; w < W; w += gridDim.x) {
    if (STRIDED && w + gridDim.x < W) p2_prefetch_l2<R, N, TC>(a, tile_geo<Cfg::B, N>(a, w + gridDim.x));
    p2_item<R, N, TC, MODE, STRIDED>(a, tile_geo<Cfg::B, N>(a, w), smem_raw, kt_shared, s_om, s_ec, s_es, rq);
  }
  if constexpr (SUMS) {
    // the tiles of a CTA are fixed by the grid size, so the result does not
    // depend on scheduling
    red_finish<Cfg::NT>(rq, MODE == M2_INV_SOB ? 3 : a.rabi_ncomp * a.rabi_n, a.rabi_partial, a.rabi_count,
                        a.rabi_out);
  }
}

}  // namespace atus
