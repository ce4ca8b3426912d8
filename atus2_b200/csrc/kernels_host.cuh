// kernels_host.cuh -- non-template kernels, compiled once (in capi.cu).
#pragma once
#include "kernels.cuh"

namespace atus {

__global__ void sob_assemble_kernel(SobArgs a) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < a.npts; l += (int64_t)gridDim.x * blockDim.x) {
    double nl = 0;
    #pragma unroll
    for (int j = 0; j < MAXC; j++) {
      if (j < a.ncomp) {
        const double2 p = a.psi[j][l];
        nl += a.gs[a.comp * MAXC + j] * (p.x * p.x + p.y * p.y);
      }
    }
    const double pot = a.V ? a.V[l] : 0.0;
    const double2 p = a.psi[a.comp][l];
    if (a.copy) a.copy[l] = p;
    if (a.lap) {
      const double2 L = a.lap[l];
      a.grad[l] = make_double2(-L.x + (pot + nl) * p.x, -L.y + (pot + nl) * p.y);
    } else {  // the potential term alone (W psi)
      a.grad[l] = make_double2((pot + nl) * p.x, (pot + nl) * p.y);
    }
  }
}

// y -= f * x
__global__ void axpy_kernel(double2 *y, const double2 *x, double f, int64_t n) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < n; l += (int64_t)gridDim.x * blockDim.x) {
    double2 v = y[l];
    const double2 u = x[l];
    v.x -= f * u.x;
    v.y -= f * u.y;
    y[l] = v;
  }
}

__global__ void scale_kernel(double2 *y, double f, int64_t n) {
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < n; l += (int64_t)gridDim.x * blockDim.x) {
    double2 v = y[l];
    v.x *= f;
    v.y *= f;
    y[l] = v;
  }
}

// ------------------------------------------------------------ Sobolev run on the device
// Scalars of the descent kept in device memory, so that a chunk of iterations
// runs (as a CUDA graph) without host round trips.
struct SobDev {
  double q[MAXC][3];    // Re<psi, S(W psi)>, Re<psi, S psi>, <psi, psi> per component
  double g2[MAXC];      // sum |G|^2 of the projected gradient
  double res;           // residual of the last active iteration
  double N[MAXC];       // particle numbers of the last active iteration
  double eps;
  int max_iter;
  int iters;            // iterations done
  int done;             // no further iteration updates psi
};

// The point-wise end of an iteration for component comp, in one pass:
//   G = S(W psi) + psi - S psi - (q0 / q1) S psi   (the projected gradient),
//   psi <- psi * scale - stepsize G,  g2 = sum |G|^2,
// q0 = Re<psi, S(W psi) + psi - S psi>, q1 = Re<psi, S psi>, scale = 1/sqrt(N)
// of every component when some |N - 1| > 1e-5 (Renormalize_All_Psi), else 1.
// All of these are known before the pass, so the projection, its norm and the
// update need not be three sweeps.  Only an active iteration (not yet
// converged, below max_iter) does anything.  After the last component
// (finish != 0) the block that ends last takes the residual (Compute_res),
// counts the iteration and decides whether it was the converging one.
// Bound by L2 and HBM latency (three fields read, one written: 134 MB at 128^3
// in 23 us); projection, scalars, update and commit as launches of their own
// took 36 us.
__global__ void __launch_bounds__(RED_THREADS) sob_step_kernel(double2 *psi, const double2 *sw, const double2 *ps,
                                                               double step, SobDev *d, int comp, int ncomp, int finish,
                                                               double ar, int64_t n, double *partial, unsigned *count) {
  pdl_wait();
  const bool active = !d->done && d->iters < d->max_iter;
  if (!active) return;
  bool renorm = false;
  for (int i = 0; i < ncomp; i++)
    if (fabs(ar * d->q[i][2] - 1) > 1e-5) renorm = true;
  const double f = renorm ? 1.0 / sqrt(ar * d->q[comp][2]) : 1.0;
  const double fak = (d->q[comp][0] + d->q[comp][2] - d->q[comp][1]) / d->q[comp][1];
  double q[RED_MAXQ] = {};
  const int64_t stride = (int64_t)gridDim.x * RED_THREADS;
  for (int64_t l0 = blockIdx.x * (int64_t)RED_THREADS + threadIdx.x; l0 < n; l0 += RED_AHEAD * stride) {
    double2 p[RED_AHEAD], g[RED_AHEAD], s[RED_AHEAD];
    #pragma unroll
    for (int u = 0; u < RED_AHEAD; u++) {
      const int64_t l = l0 + u * stride;
      if (l < n) {
        p[u] = psi[l];
        g[u] = sw[l];
        s[u] = ps[l];
      }
    }
    #pragma unroll
    for (int u = 0; u < RED_AHEAD; u++) {
      const int64_t l = l0 + u * stride;
      if (l < n) {
        double2 v = g[u];
        v.x += p[u].x - s[u].x;
        v.y += p[u].y - s[u].y;
        v.x -= fak * s[u].x;
        v.y -= fak * s[u].y;
        q[0] += v.x * v.x + v.y * v.y;
        psi[l] = make_double2(p[u].x * f - step * v.x, p[u].y * f - step * v.y);
      }
    }
  }
  const bool last = red_finish<RED_THREADS>(q, 1, partial, count, &d->g2[comp]);
  if (last && finish && threadIdx.x == 0) {
    double res = 0;
    for (int i = 0; i < ncomp; i++) {
      const double r = d->g2[i] * ar;
      res += r * r;
      d->N[i] = ar * d->q[i][2];
    }
    res = sqrt(res);
    d->res = res;
    d->iters++;
    if (!(res > d->eps)) d->done = 1;
  }
}

}  // namespace atus
