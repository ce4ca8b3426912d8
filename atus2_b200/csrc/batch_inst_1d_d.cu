// Batched 1D Strang-block kernels, double fields: every (length, CTAs a run)
// combination the autotuner may pick.
#include "batch.cuh"

using namespace atus;

template <int N, int C>
static bool k1(BKernel *k) {
  using Cfg = LineCfg<double, N, 2, C>;
  if constexpr (Cfg::fits) {
    k->fn = (const void *)line1d_batch_kernel<double, N, C>;
    k->nt = Cfg::NT;
    k->smem = Cfg::smem;
    k->B = 0;
    k->cluster = C;
    return true;
  } else {
    return false;
  }
}
template <int N>
static bool k1c(int C, BKernel *k) {
  switch (C) {
    case 1: return k1<N, 1>(k);
    case 2: return k1<N, 2>(k);
    case 4: return k1<N, 4>(k);
    case 8: return k1<N, 8>(k);
    default: return false;
  }
}

// One CTA a run, one component in shared memory (lengths without a one-CTA
// line1d_batch_kernel).
template <int N>
static bool kcta(BKernel *k) {
  k->fn = (const void *)batch1d_cta_kernel<double, N>;
  k->cluster = 1;
  k->nt = BCTA_NT;
  k->smem = sizeof(cplx<double>) * Pad<N>::NP;
  k->B = 0;
  return true;
}
bool batch1d_cta_info_d(int N, BKernel *k) {
  switch (N) {
    case 2048: return kcta<2048>(k);
    case 4096: return kcta<4096>(k);
    case 8192: return kcta<8192>(k);
    default: return false;
  }
}

bool batch1d_info_d(int N, int C, BKernel *k) {
  switch (N) {
    case 1024: return k1c<1024>(C, k);
    case 2048: return k1c<2048>(C, k);
    case 4096: return k1c<4096>(C, k);
    case 8192: return k1c<8192>(C, k);
    case 16384: return k1c<16384>(C, k);
    default: return false;
  }
}
