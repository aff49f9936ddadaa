// r3d_reduce.cuh -- what one iteration decides from its sums: RMS, converged
// / diverged / maxstep (iterate.cu:48-59, cal_rms.cu:14-26) and the AN2
// coefficients (anderson.cu:54-130).  Used by k_reduce (a launch of its own)
// and by the last CTA of k_rt_inv.
#pragma once

#include "r3d_common.cuh"

namespace r3d {

// leg (anderson.cu:105-130): 2x2 Gaussian elimination, no pivoting.
__device__ __forceinline__ void leg2(double *a, double *x, double *bb) {
  double p = a[0];
  a[1] /= p;
  double r = bb[0] /= p;
  double q = a[2];
  a[3] -= q * a[1];
  bb[1] -= q * r;
  x[1] = bb[1] / a[3];
  x[0] = bb[0] - a[1] * x[1];
}

// One thread: sums[0] = sum R^2, sums[1 + 5 v + k] the theta dots of site v.
// mode 0: an iteration's decisions; 1: mix regardless of convergence (the
// explicit anderson() call); 2: record the rms only (calculate()).
__device__ __forceinline__ void reduce_finish(const Desc &d, const double *sums, int mode) {
  Ctl *c = d.ctl;
  if (mode == 2) {
    c->ss = sums[0];
    c->rms = sqrt(sums[0] / ((double)d.N * d.n));
    c->step += 1;
    return;
  }
  if (mode == 0) {
    c->ss = sums[0];
    c->rms = sqrt(sums[0] / ((double)d.N * d.n));
    c->step += 1;
    if (c->step <= c->maxstep) d.rmslog[c->step - 1] = c->rms;
    if (!isfinite(c->rms) || c->err) {  // err: a kernel's bounded wait ran out
      c->status = DIVERGED;
      c->mix_flag = 0;
      return;
    }
    if (c->rms <= c->tol) {
      c->status = CONVERGED;
      c->mix_flag = 0;
      return;
    }
    // The last allowed evaluation ends the solve without a mix: t stays the
    // t of that evaluation, whose g and h the results are computed from.
    if (c->step >= c->maxstep) {
      c->status = MAXSTEP;
      c->mix_flag = 0;
      return;
    }
  }
  c->mix_flag = 1;
  if (d.mixer == MIX_AN2) {
    if (c->count_left > 0) {  // newdt0 (Picard) step
      c->count_left -= 1;
      c->coef[0] = 0;
      c->coef[1] = 0;
      c->coef[2] = -1.0;  // marker: Picard
      c->coef[3] = (double)c->binary;
    } else {
      double a[4], cc[2], x[2];
      cc[0] = cc[1] = a[0] = a[1] = a[3] = 0.0;
      for (int v = 0; v < d.n; ++v) {  // cal_theta, anderson.cu:81-102
        cc[0] += sums[1 + 5 * v + 0] * d.irho[v];
        cc[1] += sums[1 + 5 * v + 1] * d.irho[v];
        a[0] += sums[1 + 5 * v + 2] * d.irho[v];
        a[1] += sums[1 + 5 * v + 3] * d.irho[v];
        a[3] += sums[1 + 5 * v + 4] * d.irho[v];
      }
      a[2] = a[1];
      leg2(a, x, cc);
      c->coef[0] = x[0] + d.mp * ((c->binary == 0) ? 0 : 1);
      c->coef[1] = x[1] + d.mp * ((c->binary == 0) ? 1 : 0);
      c->coef[2] = 1.0;
      c->coef[3] = (double)c->binary;
    }
    c->binary = (c->binary == 0) ? 1 : 0;
  }
}

// The whole CTA: sums of k_rt_inv's partials ([site][6][rt_icps]: sum R^2 and
// the five dots of each CTA), one warp per sum (its lanes stride over the
// CTAs, then a butterfly: an order that depends on nothing but the launch
// geometry), then reduce_finish in one thread.
template <int NT>
__device__ __forceinline__ void rt_reduce(const Desc &d, int mode, bool dots) {
  __shared__ double sums[kPartials], ssv[kMaxSites];
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, nc = d.rt_icps, nk = 6 * d.n;
  for (int k = threadIdx.x >> 5; k < nk; k += NW) {
    const int v = k / 6, j = k - 6 * v;
    if (j > 0 && !dots) continue;
    const double *p = d.partials + (size_t)k * nc;
    double s = 0;
    for (int i = lane; i < nc; i += 32) s += __ldcg(p + i);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      if (j == 0)
        ssv[v] = s;
      else
        sums[5 * v + j] = s;
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double ss = 0;
  for (int v = 0; v < d.n; ++v) ss += ssv[v];
  sums[0] = ss;
  reduce_finish(d, sums, mode);
}

}  // namespace r3d
