// pass3_pipe.cuh -- strided FP64 passes over pencils of 1024..4096 points whose
// next tile arrives while this one is transformed.
//
// The tile of pass3_kernel (8192 values: 8 to 2 adjacent pencils, 512 threads of
// 16 values, one CTA per SM) loads, transforms and stores in turn, with nothing
// else on the SM to run meanwhile.  Here values cross the exchange as real
// parts, then imaginary parts, in half the space, and the shared memory that
// frees holds most of the next tile: PF of a thread's 16 values by cp.async
// (its own slots, read back without conflicts), the others in registers,
// asked for before this tile's stores.  Eight barriers a transform instead of
// four.  For grids of more than one tile per SM; below that there is nothing
// to overlap.  Measured, FP64 x pass: 2048 x 2048 63.6 -> 54.9 us, 4096 x 2048
// 157 -> 139, 2048 x 4096 132 -> 105, 1024 x 4096 x 2 124 -> 95.
#pragma once
#include "pass3.cuh"

namespace atus {

template <int N>
struct P3PipeCfg {
  static constexpr int M = N / 16, R3 = M / 16, T3 = 16 / R3;
  static constexpr int NT = 512, B = 8192 / N;
  // pencil pitch in doubles: the B pencils x 16 / B rows of a half warp on
  // sixteen distinct 8-byte banks
  static constexpr int PB = 17 * M + 16 / B;
  static constexpr size_t smem_ex = 8 * (size_t)B * PB;
  static constexpr size_t smem_tw = 16 * (size_t)(16 * M + 16 * R3);
  static constexpr size_t left = (227 * 1024 - 2048 - smem_ex - smem_tw) / (16 * NT);
  static constexpr int PF = left < 16 ? (int)left : 16;
  static constexpr size_t smem = smem_ex + smem_tw + 16 * (size_t)NT * PF;
  static_assert(smem_ex % 16 == 0 && N >= 1024 && N <= 4096, "");
};

// As p3_transform, in halves; hook() runs once every value has left its slot.
template <int N, int DIR, typename Hook>
__device__ __forceinline__ void p3p_transform(double2 *v, double *ex, const double2 *twN, const double2 *twM, int t,
                                              Hook hook) {
  constexpr int M = N / 16, R3 = M / 16, T3 = 16 / R3;
  const int qa = t & 15, j2 = t >> 4;
  dft16<DIR>(v);
  #pragma unroll
  for (int q = 1; q < 16; q++) v[q] = twmul<DIR>(v[q], twN[q * M + t]);
  __syncthreads();
  #pragma unroll
  for (int q = 0; q < 16; q++) ex[17 * t + q] = v[q].x;
  __syncthreads();
  hook();
  #pragma unroll
  for (int r = 0; r < 16; r++) v[r].x = ex[17 * (j2 + R3 * r) + qa];
  __syncthreads();
  #pragma unroll
  for (int q = 0; q < 16; q++) ex[17 * t + q] = v[q].y;
  __syncthreads();
  #pragma unroll
  for (int r = 0; r < 16; r++) v[r].y = ex[17 * (j2 + R3 * r) + qa];
  dft16<DIR>(v);
  #pragma unroll
  for (int q2 = 1; q2 < 16; q2++) v[q2] = twmul<DIR>(v[q2], twM[q2 * R3 + j2]);
  // stage 3 input jj of butterfly s at v[s R3 + jj] (j2 is also its q2')
  __syncthreads();
  #pragma unroll
  for (int q2 = 0; q2 < 16; q2++) ex[qa + 16 * (j2 + R3 * q2)] = v[q2].x;
  __syncthreads();
  #pragma unroll
  for (int s = 0; s < T3; s++)
    #pragma unroll
    for (int jj = 0; jj < R3; jj++) v[s * R3 + jj].x = ex[qa + 16 * (jj + R3 * (j2 + R3 * s))];
  __syncthreads();
  #pragma unroll
  for (int q2 = 0; q2 < 16; q2++) ex[qa + 16 * (j2 + R3 * q2)] = v[q2].y;
  __syncthreads();
  #pragma unroll
  for (int s = 0; s < T3; s++)
    #pragma unroll
    for (int jj = 0; jj < R3; jj++) v[s * R3 + jj].y = ex[qa + 16 * (jj + R3 * (j2 + R3 * s))];
  double2 o[16];
  #pragma unroll
  for (int s = 0; s < T3; s++) {
    dftR<R3, DIR>(v + s * R3);
    #pragma unroll
    for (int k3 = 0; k3 < R3; k3++) o[s + T3 * k3] = v[s * R3 + k3];
  }
  #pragma unroll
  for (int m = 0; m < 16; m++) v[m] = o[m];
}

template <int N, int MODE>
__global__ void __launch_bounds__(512, 1) pass3_pipe_kernel(PassArgs a) {
  using Cfg = P3PipeCfg<N>;
  constexpr int M = Cfg::M, R3 = Cfg::R3, B = Cfg::B, NT = Cfg::NT, PF = Cfg::PF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *const twN = reinterpret_cast<double2 *>(smem_raw + Cfg::smem_ex), *const twM = twN + 16 * M;
  const int tid = threadIdx.x, b = tid % B, t = tid / B;
  double *const my = reinterpret_cast<double *>(smem_raw) + b * Cfg::PB;
  double2 *const slot = reinterpret_cast<double2 *>(smem_raw + Cfg::smem_ex + Cfg::smem_tw) + tid;  // value r: slot[NT r]
  {
    const double2 *tw = (const double2 *)a.tw;
    for (int e = tid; e < 16 * M; e += NT) twN[e] = tw[((e % M) * (e / M)) * (TWN / N)];
    for (int e = tid; e < 16 * R3; e += NT) twM[e] = tw[((e % R3) * (e / R3)) * (TWN / M)];
  }
  pdl_wait();
  __syncthreads();
  const int64_t W = a.ntiles * a.ncomp_grid, step = (int64_t)M * a.sa;
  double2 nx[PF < 16 ? 16 - PF : 1];
  // this thread's point t of the item's pencil b, or nullptr
  auto source = [&](int64_t w) -> double2 * {
    if (w >= W) return nullptr;
    const TileGeo g = tile_geo<B, N>(a, w);
    return b < g.nb ? (double2 *)pick(a.psi, g.comp0) + g.base0 + b + (int64_t)t * a.sa : nullptr;
  };
  auto fetch = [&](const double2 *src) {
    if (src) {
      #pragma unroll
      for (int r = 0; r < PF; r++) cp_async(&slot[NT * r], src + r * step, double2{});
    }
    cp_commit();
  };
  auto fetch_rest = [&](const double2 *src) {
    #pragma unroll
    for (int r = PF; r < 16; r++) nx[r - PF] = src ? src[r * step] : make_double2(0, 0);
  };
  int64_t w = blockIdx.x;
  double2 *cur = source(w);
  fetch(cur);
  fetch_rest(cur);
  for (; w < W; w += gridDim.x) {
    const double2 *const nextp = source(w + gridDim.x);
    double2 v[16];
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    #pragma unroll
    for (int r = 0; r < PF; r++) v[r] = cur ? slot[NT * r] : make_double2(0, 0);
    #pragma unroll
    for (int r = PF; r < 16; r++) v[r] = nx[r - PF];
    auto refill = [&]() { fetch(nextp); };
    auto none = []() {};
    if constexpr (MODE == M2_INV) {
      p3p_transform<N, +1>(v, my, twN, twM, t, refill);
    } else {
      p3p_transform<N, -1>(v, my, twN, twM, t, refill);
    }
    if constexpr (MODE == M2_KIN) {
      if (a.op == OP_KIN) {  // always: keeps the factors' loads out of the transform above
        const TileGeo g = tile_geo<B, N>(a, w);
        int p0[3];
        idx3(a.g, cur ? g.base0 + b : 0, p0[0], p0[1], p0[2]);
        const double2 *kx = a.kt[0][0], *ky = a.kt[0][1], *kz = a.kt[0][2];
        #pragma unroll
        for (int cc = 1; cc < MAXC; cc++)
          if (g.comp0 == cc) { kx = a.kt[cc][0]; ky = a.kt[cc][1]; kz = a.kt[cc][2]; }
        const double2 KX = __ldg(&kx[p0[0]]), KY = __ldg(&ky[p0[1]]), KZ = __ldg(&kz[p0[2]]);
        const double2 Kp = (a.axis == 0) ? cmul(KY, KZ) : (a.axis == 1) ? cmul(KX, KZ) : cmul(KX, KY);
        const double2 *const along = ((a.axis == 0) ? kx : (a.axis == 1) ? ky : kz) + t;
        #pragma unroll
        for (int m = 0; m < 16; m++) v[m] = kin_mul<double>(v[m], cmul(__ldg(&along[M * m]), Kp), a.s_f, a.s_b);
      }
      p3p_transform<N, +1>(v, my, twN, twM, t, none);
    }
    fetch_rest(nextp);
    if (cur) {
      #pragma unroll
      for (int m = 0; m < 16; m++) cur[m * step] = v[m];
    }
    cur = const_cast<double2 *>(nextp);
  }
}

}  // namespace atus
