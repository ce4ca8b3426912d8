// pass2_pair.cuh -- IFFT -> potential step -> FFT along the contiguous axis
// (pencils of 32..256 points) for two components, one warp at a time.
//
// A warp holds PW = 32 / (2 R2) pencils of both components: lane = j + R2 (c +
// 2 p), 16 values each, transformed as in pass2.cuh (radix 16, one exchange,
// radix R2 = N / 16).  Everything a pencil needs is inside its warp: the
// exchange takes warp barriers, and the components of a point meet through
// shuffles (nl_pair16).  So warps run through their items on their own, with
// no CTA barrier between a load, a transform and a store.
//
// What bounded the CTA-wide form was the exposed latency of its loads (35 % of
// the stall cycles at 16-20 warps per SM, issue slots 27 % used): here the
// next item's values are on their way into shared memory (cp.async, 16 per
// lane into the lane's own slots, read back without conflicts) while this
// item is transformed.  To make room for them FP64 values cross the exchange
// as real parts, then imaginary parts, in half the space.  16 warps per SM at
// 128 registers.  z pass of 256^3, two components, against the CTA-wide form
// with the components meeting in shared memory: bragg_ad FP64 0.368 -> 0.309
// ms (eigenvalue form; eigenvalue-free 0.337 -> 0.276), complex64 0.279 ->
// 0.227; freeprop (NL_IF) FP64 0.321 -> 0.219, complex64 0.252 -> 0.217.
// Shuffles alone, loads not ahead: 0.349-0.361 (FP64, eigenvalue-free).  The
// two forms of the Bragg step and the pure phases are three instantiations: with
// the phases in one, the Bragg step lost 0.026 ms to spills.
#pragma once
#include "pass2.cuh"

namespace atus {

template <typename R, int N>
struct PairCfg {
  using C = cplx<R>;
  static constexpr int R2 = N / 16;
  static constexpr int PW = 16 / R2;            // pencils of a warp
  static constexpr int WPC = 4;                 // warps of a CTA
  static constexpr int NT = 32 * WPC;
  static constexpr int MINB = sizeof(R) == 8 ? 4 : 5;
  static constexpr int TP = R2 + 1, TWP = 16 * TP;
  static constexpr int EX = 32 * 17;            // 8-byte units a warp exchanges at a time
  static constexpr size_t smem_tw = (sizeof(typename TwTab<R>::type) * TWP + 15) / 16 * 16;
  static constexpr size_t smem_warp = EX * 8 + 512 * sizeof(C);
  static constexpr size_t smem = smem_tw + WPC * smem_warp;
};

// The exchange of a transform: butterfly j's outputs q to row j, column q;
// back come the inputs (r, k = j + R2 t) at v[t R2 + r].  my: the
// pencil-component's R2 rows at pitch 17.
template <int R2>
__device__ __forceinline__ void pair_exchange(double2 *v, double *my, int j) {
  __syncwarp();
  #pragma unroll
  for (int q = 0; q < 16; q++) my[17 * j + q] = v[q].x;
  __syncwarp();
  #pragma unroll
  for (int t = 0; t < 16 / R2; t++)
    #pragma unroll
    for (int r = 0; r < R2; r++) v[t * R2 + r].x = my[17 * r + j + R2 * t];
  __syncwarp();
  #pragma unroll
  for (int q = 0; q < 16; q++) my[17 * j + q] = v[q].y;
  __syncwarp();
  #pragma unroll
  for (int t = 0; t < 16 / R2; t++)
    #pragma unroll
    for (int r = 0; r < R2; r++) v[t * R2 + r].y = my[17 * r + j + R2 * t];
}
template <int R2>
__device__ __forceinline__ void pair_exchange(float2 *v, double *my_, int j) {
  float2 *const my = reinterpret_cast<float2 *>(my_);
  __syncwarp();
  #pragma unroll
  for (int q = 0; q < 16; q++) my[17 * j + q] = v[q];
  __syncwarp();
  #pragma unroll
  for (int t = 0; t < 16 / R2; t++)
    #pragma unroll
    for (int r = 0; r < R2; r++) v[t * R2 + r] = my[17 * r + j + R2 * t];
}

// The second stage on the exchanged values; FLIP as in p2_stage2.
template <typename R, int N, int DIR, bool FLIP>
__device__ __forceinline__ void pair_stage2(cplx<R> *v, const typename TwTab<R>::type *twS, int j, int sg) {
  using C = cplx<R>;
  constexpr int R2 = N / 16, T2 = 16 / R2;
  C o[16];
  #pragma unroll
  for (int t = 0; t < T2; t++) {
    C u[R2];
    #pragma unroll
    for (int r = 0; r < R2; r++) u[r] = v[t * R2 + r];
    #pragma unroll
    for (int r = 1; r < R2; r++) u[r] = twmul<DIR>(u[r], twS[(j + R2 * t) * (R2 + 1) + r]);
    if constexpr (FLIP) {
      #pragma unroll
      for (int r = 1; r < R2; r += 2) u[r] = flip(u[r], sg);
    }
    dftR<R2, DIR>(u);
    #pragma unroll
    for (int r = 0; r < R2; r++) o[t + T2 * r] = u[r];
  }
  #pragma unroll
  for (int m = 0; m < 16; m++) v[m] = o[m];
}

template <typename R, int N, int FORM>
__global__ void __launch_bounds__(PairCfg<R, N>::NT, PairCfg<R, N>::MINB) pass2_pair_kernel(PassArgs a) {
  constexpr bool BRAGG = FORM != PAIR_PHASE;
  using C = cplx<R>;
  using TW = typename TwTab<R>::type;
  using Cfg = PairCfg<R, N>;
  constexpr int R2 = Cfg::R2, PW = Cfg::PW, CPI = 32 / PW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TW *const twS = reinterpret_cast<TW *>(smem_raw);
  {  // W_N^{r k} = exp(-2 pi i r k / N) from the TWN-point table
    const TW *tw = (const TW *)a.tw;
    for (int e = threadIdx.x; e < 16 * R2; e += Cfg::NT) twS[(e / R2) * Cfg::TP + e % R2] = tw[((e % R2) * (e / R2)) * (TWN / N)];
  }
  pdl_wait();
  __syncthreads();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int j = lane % R2, c = (lane / R2) & 1, p = lane / (2 * R2);
  unsigned char *const mem = smem_raw + Cfg::smem_tw + warp * Cfg::smem_warp;
  C *const next = reinterpret_cast<C *>(mem) + lane;  // slot r of this lane at next[32 r]
  double *const my = reinterpret_cast<double *>(mem + 512 * sizeof(C)) + (2 * p + c) * (17 * R2);
  C *const f = (C *)(c ? a.psi[1] : a.psi[0]);
  const int sg = c ? (int)0x80000000 : 0;
  const int64_t items = (a.npencils + PW - 1) / PW, nwarps = (int64_t)gridDim.x * Cfg::WPC;
  auto fetch = [&](int64_t w) {
    const int64_t pen = w * PW + p;
    if (w < items && pen < a.npencils) {
      const C *src = f + pen * N + j;
      #pragma unroll
      for (int r = 0; r < 16; r++) cp_async(&next[32 * r], src + R2 * r, C{});
    }
    cp_commit();
  };
  int64_t w = blockIdx.x * (int64_t)Cfg::WPC + warp;
  fetch(w);
  double om_l = 0, ec_l = 1, es_l = 0;
  int it = 0;
  for (; w < items; w += nwarps, it = (it + 1) % CPI) {
    const int64_t pen = w * PW + p, lb = pen * N;
    const bool live = pen < a.npencils;
    if (BRAGG && it == 0) {
      // couplings (x is constant along a pencil) of the warp's next CPI items:
      // one evaluation, a lane for each pencil
      const int64_t pa = (w + (lane / PW) * nwarps) * PW + lane % PW;
      if (pa < a.npencils) {
        int ix, iy, iz;
        idx3(a.g, pa * N, ix, iy, iz);
        bragg_coupling(a.nl, (double)(ix - a.nl.shift0) * a.nl.dx0, om_l, ec_l, es_l);
      }
    }
    const double om = __shfl_sync(0xffffffffu, om_l, it * PW + p), ec = __shfl_sync(0xffffffffu, ec_l, it * PW + p),
                 es = __shfl_sync(0xffffffffu, es_l, it * PW + p);
    C v[16];
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    #pragma unroll
    for (int r = 0; r < 16; r++) v[r] = live ? next[32 * r] : mk<R>(0, 0);
    dft16<+1>(v);
    pair_exchange<R2>(v, my, j);
    fetch(w + nwarps);  // the slots have been read: their values went through the exchange
    pair_stage2<R, N, +1, true>(v, twS, j, sg);
    int ix, iy, iz;
    idx3(a.g, lb, ix, iy, iz);
    nl_pair16<R, FORM>(a.nl, v, c, R2, live, (double)(ix - a.nl.shift0) * a.nl.dx0, om, ec, es,
                 lb + j, R2);
    dft16<-1>(v);
    #pragma unroll
    for (int q = 1; q < 16; q += 2) v[q] = flip(v[q], sg);
    pair_exchange<R2>(v, my, j);
    pair_stage2<R, N, -1, false>(v, twS, j, 0);
    if (live) {
      C *dst = f + lb + j;
      #pragma unroll
      for (int m = 0; m < 16; m++) dst[R2 * m] = v[m];
    }
  }
}

}  // namespace atus
