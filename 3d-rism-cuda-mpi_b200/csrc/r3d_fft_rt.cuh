// r3d_fft_rt.cuh -- in-place register-pass FFT for any length, planned at run time.
//
// A length L = R_0 R_1 ... R_{P-1} (radices 2..13 and 16) is transformed in P
// passes over a tile in shared memory.  The forward transform is decimation
// in frequency: pass s cuts blocks of L_b = R_s M_s elements (M_s the product
// of the later radices); a task (block, k) reads the R_s elements k + j M_s,
// takes their DFT in registers, multiplies output u by W_{L_b}^{u k} and
// writes it to k + u M_s -- the elements it read, so a pass needs one barrier
// and no second buffer.  The output is left digit-reversed.  The inverse
// transform runs the passes backwards (decimation in time with conjugate
// twiddles) and takes digit-reversed input to natural output, so a forward
// and an inverse transform with a pointwise step between them never permute.
// The position of an index under digit reversal comes from a table
// (RtPlan's, built by the host), and the position of L - 1 - k is L - 1 minus
// the position of k (every digit complemented).
//
// Only the radix of a pass is a template constant.  Lengths, strides and
// twiddle steps are run-time values (divisions by multiply-high), which lets
// one kernel serve every grid; tasks run along the tile's contiguous or
// odd-stride direction, so shared-memory accesses are free of bank conflicts
// and a warp's twiddle reads are (nearly) uniform.
#pragma once

#include "r3d_fft.cuh"
#include "r3d_fft_sr.cuh"
#include "r3d_internal.h"

namespace r3d {

// x / d for x * d < 2^32, magic = ceil(2^32 / d) (d = 1: magic 0)
__device__ __forceinline__ int rt_div(int x, uint32_t magic) {
  return magic ? (int)__umulhi((uint32_t)x, magic) : x;
}

// cos and sin of 2 pi e / R for the prime radices 7, 11 and 13
template <int R>
__device__ __forceinline__ constexpr double rt_cos(int e) {
  constexpr double c7[7] = {1.0, 0.62348980185873353053, -0.22252093395631440429,
                            -0.90096886790241912624, -0.90096886790241912624,
                            -0.22252093395631440429, 0.62348980185873353053};
  constexpr double c11[11] = {1.0, 0.84125353283118116886, 0.41541501300188642553,
                              -0.14231483827328514044, -0.65486073394528506406,
                              -0.95949297361449738989, -0.95949297361449738989,
                              -0.65486073394528506406, -0.14231483827328514044,
                              0.41541501300188642553, 0.84125353283118116886};
  constexpr double c13[13] = {1.0, 0.88545602565320989590, 0.56806474673115580251,
                              0.12053668025532305335, -0.35460488704253562597,
                              -0.74851074817110109863, -0.97094181742605202716,
                              -0.97094181742605202716, -0.74851074817110109863,
                              -0.35460488704253562597, 0.12053668025532305335,
                              0.56806474673115580251, 0.88545602565320989590};
  return R == 7 ? c7[e % 7] : R == 11 ? c11[e % 11] : c13[e % 13];
}
template <int R>
__device__ __forceinline__ constexpr double rt_sin(int e) {
  constexpr double s7[7] = {0.0, 0.78183148246802980871, 0.97492791218182360702,
                            0.43388373911755812048, -0.43388373911755812048,
                            -0.97492791218182360702, -0.78183148246802980871};
  constexpr double s11[11] = {0.0, 0.54064081745559758211, 0.90963199535451837141,
                              0.98982144188093273238, 0.75574957435425828377,
                              0.28173255684142969771, -0.28173255684142969771,
                              -0.75574957435425828377, -0.98982144188093273238,
                              -0.90963199535451837141, -0.54064081745559758211};
  constexpr double s13[13] = {0.0, 0.46472317204376854566, 0.82298386589365639458,
                              0.99270887409805399280, 0.93501624268541482344,
                              0.66312265824079520238, 0.23931566428755776715,
                              -0.23931566428755776715, -0.66312265824079520238,
                              -0.93501624268541482344, -0.99270887409805399280,
                              -0.82298386589365639458, -0.46472317204376854566};
  return R == 7 ? s7[e % 7] : R == 11 ? s11[e % 11] : s13[e % 13];
}

// R-point DFT for an odd prime R from the sums and differences of the pairs
// (a_m, a_{R-m})
template <int R, int DIR, typename C>
__device__ __forceinline__ void rt_dft_prime(C *a) {
  using Rt = decltype(a[0].x);
  constexpr int H = (R - 1) / 2;
  C p[H], q[H];
  C s0 = a[0];
#pragma unroll
  for (int m = 1; m <= H; ++m) {
    p[m - 1] = cadd(a[m], a[R - m]);
    q[m - 1] = csub(a[m], a[R - m]);
    s0 = cadd(s0, p[m - 1]);
  }
  const C x0 = a[0];
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    C u = x0, w = C{0, 0};
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      const Rt c = (Rt)rt_cos<R>((k * m) % R), s = (Rt)rt_sin<R>((k * m) % R);
      u.x += c * p[m - 1].x;
      u.y += c * p[m - 1].y;
      w.x += s * q[m - 1].x;
      w.y += s * q[m - 1].y;
    }
    const C v = cmuli<DIR>(w);
    a[k] = cadd(u, v);
    a[R - k] = csub(u, v);
  }
  a[0] = s0;
}
template <int R, int DIR, typename C>
__device__ __forceinline__ void rt_dft(C *a) {
  if constexpr (R == 7 || R == 11 || R == 13)
    rt_dft_prime<R, DIR>(a);
  else
    sr_dft<R, DIR>(a);
}

// Radices of a length: the fewest passes (at most four), then the smallest
// largest radix, in descending order.  rm, the largest radix: 16 (FP32), 13
// (FP64, where radix 16 would fill the register file) or 10 (kernels of
// run-time sizes, whose registers are those of their largest radix).  n = 0:
// no plan (a larger prime factor, or too long).  The same function plans
// run-time lengths on the host and compile-time ones in the kernels.
__host__ __device__ constexpr bool rt_is_radix(int r, int rm) {
  return r >= 2 && r <= rm && (r <= 13 || r == 16);
}
__host__ __device__ constexpr RtPlan rt_plan_of(int L, int rm) {
  RtPlan p{};
  int b[4] = {0, 0, 0, 0}, n = 0;
  for (int r0 = 2; r0 <= 16 && !n; ++r0)
    if (r0 == L && rt_is_radix(r0, rm)) b[0] = r0, n = 1;
  for (int r0 = 2; r0 <= 16 && !n; ++r0) {
    if (!rt_is_radix(r0, rm) || L % r0) continue;
    const int r1 = L / r0;
    if (r1 <= r0 && rt_is_radix(r1, rm)) b[0] = r0, b[1] = r1, n = 2;
  }
  for (int r0 = 2; r0 <= 16 && !n; ++r0) {
    if (!rt_is_radix(r0, rm) || L % r0) continue;
    for (int r1 = r0; r1 >= 2 && !n; --r1) {
      if (!rt_is_radix(r1, rm) || (L / r0) % r1) continue;
      const int r2 = L / r0 / r1;
      if (r2 <= r1 && rt_is_radix(r2, rm)) b[0] = r0, b[1] = r1, b[2] = r2, n = 3;
    }
  }
  for (int r0 = 2; r0 <= 16 && !n; ++r0) {
    if (!rt_is_radix(r0, rm) || L % r0) continue;
    for (int r1 = r0; r1 >= 2 && !n; --r1) {
      if (!rt_is_radix(r1, rm) || (L / r0) % r1) continue;
      for (int r2 = r1; r2 >= 2 && !n; --r2) {
        if (!rt_is_radix(r2, rm) || (L / r0 / r1) % r2) continue;
        const int r3 = L / r0 / r1 / r2;
        if (r3 <= r2 && rt_is_radix(r3, rm)) b[0] = r0, b[1] = r1, b[2] = r2, b[3] = r3, n = 4;
      }
    }
  }
  p.L = L;
  p.n = n;
  int m = L;
  for (int s = 0; s < n; ++s) {
    m /= b[s];
    p.r[s] = b[s];
    p.m[s] = m;
    p.tws[s] = L / (b[s] * m);
    p.mg[s] = m > 1 ? 0xffffffffu / (uint32_t)m + 1 : 0;
  }
  return p;
}
__host__ __device__ constexpr int rt_max_radix(int L, int rm) { return rt_plan_of(L, rm).r[0]; }
__host__ __device__ constexpr uint32_t rt_magic(int v) {
  return v > 1 ? 0xffffffffu / (uint32_t)v + 1 : 0;
}

// One pass: lanes run over W "columns" (lane index c fastest), then over the
// L / R tasks of a column.  ld(c, i) and st(c, i, value) access element i of
// column c.  M, mgM: the pass's M_s and its division magic; tws = L / L_b.
// DIR -1: DFT, then twiddles; DIR +1: conjugate twiddles, then the DFT.
template <int R, int DIR, int NT, typename C, typename Ld, typename St>
__device__ __forceinline__ void rt_pass(int W, uint32_t mgW, int L, int M, uint32_t mgM, int tws,
                                        const C *tw, Ld ld, St st) {
  const int ntask = W * (L / R);
#pragma unroll 1
  for (int task = threadIdx.x; task < ntask; task += NT) {
    const int q = rt_div(task, mgW), c = task - q * W;
    const int blk = rt_div(q, mgM), k = q - blk * M;
    const int base = blk * (R * M) + k;
    C a[R];
#pragma unroll
    for (int j = 0; j < R; ++j) a[j] = ld(c, base + j * M);
    if constexpr (DIR > 0) {
      if (M > 1) {
        const int e = k * tws;
#pragma unroll
        for (int j = 1; j < R; ++j) a[j] = cmul(a[j], cconj(tw[j * e]));
      }
    }
    rt_dft<R, DIR>(a);
    if constexpr (DIR < 0) {
      if (M > 1) {
        const int e = k * tws;
#pragma unroll
        for (int j = 1; j < R; ++j) a[j] = cmul(a[j], tw[j * e]);
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) st(c, base + j * M, a[j]);
  }
}

// Pass s of a length.  LS > 0: the length is a template constant and s an
// integral_constant, so that the plan, every stride and every division fold;
// LS = 0: plan p (RtPlan's members, of any length), s an int.
template <int LS, int DIR, int NT, int RM, typename PL, typename S, typename C, typename Ld,
          typename St>
__device__ __forceinline__ void rt_pass_s(const PL &p, S sc, int W, uint32_t mgW, const C *tw,
                                          Ld ld, St st) {
  if constexpr (LS > 0) {
    constexpr RtPlan pl = rt_plan_of(LS, RM);
    constexpr int s = S::value;
    rt_pass<pl.r[s], DIR, NT>(W, mgW, LS, pl.m[s], pl.mg[s], pl.tws[s], tw, ld, st);
  } else {
    const int s = sc;
    const int M = p.m[s], tws = p.tws[s];
    const uint32_t mg = p.mg[s];
    switch (p.r[s]) {
#define R3D_RT_CASE(RR)                                                            \
  case RR:                                                                         \
    if constexpr (RR <= RM) rt_pass<RR, DIR, NT>(W, mgW, p.L, M, mg, tws, tw, ld, st); \
    break;
      R3D_RT_CASE(2)
      R3D_RT_CASE(3)
      R3D_RT_CASE(4)
      R3D_RT_CASE(5)
      R3D_RT_CASE(6)
      R3D_RT_CASE(7)
      R3D_RT_CASE(8)
      R3D_RT_CASE(9)
      R3D_RT_CASE(10)
      R3D_RT_CASE(11)
      R3D_RT_CASE(12)
      R3D_RT_CASE(13)
      R3D_RT_CASE(16)
      default: break;
#undef R3D_RT_CASE
    }
  }
}

template <int S>
struct rt_int {  // a pass number as a template constant
  static constexpr int value = S;
  __device__ constexpr operator int() const { return S; }
};
// body(s) for every pass, first to last (REV: last to first)
template <int LS, int RM, bool REV, int K = 0, typename F>
__device__ __forceinline__ void rt_each(int n, F body) {
  if constexpr (LS > 0) {
    constexpr int N = rt_plan_of(LS, RM).n;
    if constexpr (K < N) {
      body(rt_int<(REV ? N - 1 - K : K)>{});
      rt_each<LS, RM, REV, K + 1>(n, body);
    }
  } else {
    for (int k = 0; k < n; ++k) body(REV ? n - 1 - k : k);
  }
}
// the pass at the spectrum's side (the forward's last, the inverse's first)
// with one body, the others with another
template <int LS, int RM, typename S, typename FA, typename FB>
__device__ __forceinline__ void rt_edge(int n, S s, FA edge, FB inner) {
  if constexpr (LS > 0) {
    if constexpr (S::value == rt_plan_of(LS, RM).n - 1)
      edge();
    else
      inner();
  } else {
    if ((int)s == n - 1)
      edge();
    else
      inner();
  }
}

}  // namespace r3d
