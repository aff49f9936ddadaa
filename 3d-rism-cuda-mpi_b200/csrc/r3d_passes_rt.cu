// r3d_passes_rt.cu -- the iteration in three launches, for any grid: x and y
// transforms of a whole z-plane in one CTA.
//
//   k_rt_fwd   AN2 mix of the previous iteration (when requested), closure,
//              c_s and packing, x transform; in plane mode also the y
//              transform: the half spectrum is written once
//   k_rt_y     the y transform alone, where a plane does not fit one CTA
//   k_rt_zoz   z transform, Ornstein-Zernike, inverse z transform
//   k_rt_inv   (plane mode: inverse y,) inverse x transform, residual, sum
//              R^2 and AN2 dots; the solve's last CTA reduces them and takes
//              the iteration's decisions (the reduce kernel of the other paths)
//
// The passes compute what those of r3d_kernels.cu compute (which names the
// reference lines) on the in-place engine of r3d_fft_rt.cuh.  The spectrum is
// left digit-reversed in k_x and k_y (nothing between the forward and the
// inverse transform needs an order, only each point's |k| shell, which comes
// through the position tables in d.rtrev).
//
// Against one kernel per axis this moves the half spectrum through memory
// four times less per iteration (16 of 116 bytes per voxel and site, mixed),
// and small grids, whose arrays sit in L2 and whose kernels last a few
// microseconds, save three launches.  Inputs come straight from global memory
// in vectors (every load of a thread's voxels issued before the first use),
// not through shared-memory staging: the tile then leaves room for more CTAs
// per SM, whose phases (loads, transforms, stores) overlap.
//
// Debug builds check the indexes of the real grids, the spectrum, the shell index
// and the partials (R3D_IN); the position tables are indexed by a tile's own
// positions, the chi table of a non-cubic cell by the shell index as it is stored.
#include "r3d_common.cuh"
#include "r3d_fft_rt.cuh"
#include "r3d_reduce.cuh"

#ifndef R3D_CT_FP64
#define R3D_CT_FP64 1
#endif
// Compiled in three parts per precision (build time): 0 the forward kernels,
// 1 the inverse ones, 2 the y and z ones
#ifndef R3D_RT_PART
#define R3D_RT_PART 0
#endif

// element i of the kernel's part of the spectrum (w), checked in debug builds
#define R3D_W(i) R3D_IN(d, w - (const S *)d.w + (i), d.n * d.Nhs)

namespace r3d {

// the arithmetic of a set of kernels: FP64, FP32, or FP64 on FP32 grids
enum RtKind { RT_FP64 = 0, RT_FP32 = 1, RT_MIXED = 2 };
bool rt_static_x(int kind, int nx, int ny, bool plane);
bool rt_static_y(int kind, int ny);
bool rt_static_z(int kind, int nz, int n);

#if R3D_CT_FP64 == 1
using PRT = P64;
#elif R3D_CT_FP64 == 2
using PRT = PMixD;
#else
using PRT = PMix;
#endif

// largest radix of the compile-time-sized kernels, and of the run-time-sized
// ones unless a length needs more (see rt_plan_of)
template <typename P>
constexpr int rt_rm() {
  return sizeof(typename P::A) == 4 ? 16 : 13;
}
constexpr int kRtLean = 10;

// between the spectrum's storage type and the arithmetic's
template <typename O, typename I>
__device__ __forceinline__ O rt_cvt(I a) {
  return O{(decltype(O::x))a.x, (decltype(O::x))a.y};
}
// FP64 or grid-type table `k` (twx, pwx, twy, pwy, twz, pwz) for the arithmetic
template <typename P>
__device__ __forceinline__ const typename Cx<typename P::A>::T *rt_table(const Desc &d, int k) {
  using C = typename Cx<typename P::A>::T;
  if constexpr (sizeof(typename P::A) > sizeof(typename P::R)) {
    const int len[6] = {d.hx, d.hx, d.ny, d.ny, d.nz, d.nz};
    int off = 0;
    for (int i = 0; i < k; ++i) off += len[i];
    return (const C *)d.tw64 + off;
  } else {
    const void *const t[6] = {d.twx, d.pwx, d.twy, d.pwy, d.twz, d.pwz};
    return (const C *)t[k];
  }
}

// V consecutive elements from p, aligned to V elements
template <int V, typename X>
__device__ __forceinline__ void ldv(X (&o)[V], const X *p) {
  if constexpr (V == 1) {
    o[0] = *p;
  } else if constexpr (sizeof(X) == 4 && V == 2) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    o[0] = v.x, o[1] = v.y;
  } else {
    static_assert(V == 2 && sizeof(X) == 8, "vector width");
    const double2 v = *reinterpret_cast<const double2 *>(p);
    o[0] = v.x, o[1] = v.y;
  }
}
template <int V, typename X>
__device__ __forceinline__ void stv(X *p, const X (&o)[V]) {
  if constexpr (V == 1) {
    *p = o[0];
  } else if constexpr (sizeof(X) == 4 && V == 2) {
    *reinterpret_cast<float2 *>(p) = make_float2(o[0], o[1]);
  } else {
    static_assert(V == 2 && sizeof(X) == 8, "vector width");
    *reinterpret_cast<double2 *>(p) = make_double2(o[0], o[1]);
  }
}

// The half-sample twiddles of the y and z transforms, e^{-i pi y / ny} and
// e^{-i pi z / nz}, are constants of a row of the x tile, so the x passes
// apply them (conjugated on the way back) and the y and z passes, which are
// bound by their instructions, carry none: row[r] = their product for row
// row0 + r.
template <typename P, int NT, typename C>
__device__ __forceinline__ void rt_row_factors(C *row, const Desc &d, int row0, int nrow, int ny) {
  const C *pwy = rt_table<P>(d, 3), *pwz = rt_table<P>(d, 5);
  for (int r = threadIdx.x; r < nrow; r += NT) {
    const int z = (row0 + r) / ny, y = row0 + r - z * ny;
    row[r] = cmul(pwy[y], pwz[z]);
  }
}

// use(in, e) for e = threadIdx.x, + NT, ... below n, with the loads of the
// next D - 1 elements in flight (D sets of registers)
template <int D, int NT, typename In, typename Load, typename Use>
__device__ __forceinline__ void rt_stream(int n, Load load, Use use) {
  In in[D];
  int e = threadIdx.x;
#pragma unroll
  for (int k = 0; k < D - 1; ++k)
    if (e + k * NT < n) load(in[k], e + k * NT);
  // without guards while the whole CTA has every element of a round (a
  // branch around a load would end the scheduling block it should overlap)
  const int rounds = max(0, (n / NT - (D - 1)) / D);
#pragma unroll 1
  for (int it = 0; it < rounds; ++it, e += D * NT)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      load(in[(k + D - 1) % D], e + (k + D - 1) * NT);
      use(in[k], e + k * NT);
    }
#pragma unroll 1
  for (; e < n; e += D * NT)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (e + (k + D - 1) * NT < n) load(in[(k + D - 1) % D], e + (k + D - 1) * NT);
      if (e + k * NT < n) use(in[k], e + k * NT);
    }
}

// shared-memory row stride of an x tile (odd: lanes along rows then fall on
// different banks)
__host__ __device__ inline int rt_ldx(int hx) { return hx | 1; }

// --------------------------------------------------------------- forward
// Sizes: HX > 0 and NY > 0: planes of compile-time size; HX > 0, NY = 0: row
// tiles of compile-time length; HX = 0: run-time sizes, either form.
//
// A thread takes V elements of each half of a row and has the next ones'
// loads (72 to 144 bytes per thread and array set) in flight while it works
// on these: with one set in flight the kernel waited for memory two thirds of
// its time (16 warps per SM; 144^3, four sites, mixed: 235 us).
template <typename P, int V>
struct FwdIn {
  typename P::T t[2][V];
  typename P::R u[2][V], c[2][V], r[2][V], a0[2][V], a1[2][V], b0[2][V], b1[2][V];
};

template <typename P, int HX, int NY, int V, int NT, int MINB, int RM = rt_rm<P>()>
__global__ void __launch_bounds__(NT, MINB) k_rt_fwd(Batch b, int allow_mix) {
  using R = typename P::R;
  using T = typename P::T;
  using C = typename Cx<typename P::A>::T;  // arithmetic
  using S = typename Cx<R>::T;              // spectrum
  constexpr bool MIXP = sizeof(R) < sizeof(T);  // mixed precision: FP32 t differences, c_ref
  extern __shared__ __align__(16) char smem[];
  const int si = find_solve(b, blockIdx.x);
  const Desc &d = b.d[si];
  const Ctl *ctl = d.ctl;
  if (ctl->status != RUNNING) return;
  const int hx = HX ? HX : d.hx, nx = 2 * hx, ny = NY ? NY : d.ny, LDX = rt_ldx(hx);
  const bool plane = HX ? NY != 0 : d.rt_plane != 0;
  const int cta = blockIdx.x - b.prefix[si];
  const int v = cta / d.rt_tps, tile = cta - v * d.rt_tps;
  const int pr = NY ? NY : d.rt_pr;
  const int row0 = tile * pr, nrow = NY ? NY : min(pr, ny * d.nz - row0);
  C *buf = (C *)smem, *row = buf + pr * LDX, *twx = row + pr, *pw = twx + hx, *twy = pw + hx;
  for (int e = threadIdx.x; e < hx; e += NT) {
    twx[e] = rt_table<P>(d, 0)[e];
    pw[e] = rt_table<P>(d, 1)[e];
  }
  if (plane)
    for (int e = threadIdx.x; e < ny; e += NT) twy[e] = rt_table<P>(d, 2)[e];
  rt_row_factors<P, NT>(row, d, row0, nrow, ny);
  __syncthreads();

  const long long niv = (long long)d.n * d.Ns;
  const long long gbase = (long long)v * d.Ns + (long long)row0 * nx;
  // the mix that the last iteration requested: 0 none, 1 Picard, 2 AN2
  const int mixing = !(allow_mix && d.mixer == MIX_AN2 && ctl->mix_flag != 0) ? 0
                     : ctl->coef[2] < 0                                       ? 1
                                                                              : 2;
  const long long boff = (long long)ctl->coef[3] * niv, noff = niv - boff;
  const double s1 = ctl->coef[0], s2 = ctl->coef[1], mm = d.m;
  const bool old0 = boff == 0;  // slot 0 holds the older entry
  const bool has_cref = MIXP && d.cref != nullptr;
  T *t = (T *)d.t + gbase, *gq = (T *)d.gq + gbase;
  const R *u = (const R *)d.u + gbase, *cref = (const R *)d.cref + (has_cref ? gbase : 0);
  const R *res = (const R *)d.res + gbase, *rp0 = (const R *)d.hist_b + gbase, *rp1 = rp0 + niv;
  // mixed: the t slots hold differences of successive t (newest, then the
  // other); FP64: copies of t in slot order
  const R *ha0 = (const R *)d.hist_a + (MIXP ? noff : 0) + gbase;
  const R *ha1 = (const R *)d.hist_a + (MIXP ? boff : niv) + gbase;
  R *hao = (R *)d.hist_a + boff + gbase, *hbo = (R *)d.hist_b + boff + gbase;
  const int clos = d.clos, pse_n = d.pse_n;
  const int hv = hx / V, nel = nrow * hv;
  const int y0 = row0 % ny, par0 = (y0 + row0 / ny) & 1;
  const uint32_t mghv = HX ? rt_magic(HX / V) : d.rt_mghv;
  auto work = [&](auto mode) {
    constexpr int MODE = decltype(mode)::value;
    auto load = [&](FwdIn<P, V> &in, int e) {
      const int r = rt_div(e, mghv), i0 = r * nx + (e - r * hv) * V;
      if (!R3D_IN(d, gbase + i0 + hx + V - 1, niv)) return;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + h * hx;
        ldv<V>(in.t[h], t + i);
        ldv<V>(in.u[h], u + i);
        if (MIXP && has_cref) ldv<V>(in.c[h], cref + i);
        if constexpr (MODE > 0) ldv<V>(in.r[h], res + i);
        if constexpr (MODE == 2) {
          ldv<V>(in.a0[h], ha0 + i);
          ldv<V>(in.a1[h], ha1 + i);
          ldv<V>(in.b0[h], rp0 + i);
          ldv<V>(in.b1[h], rp1 + i);
        }
      }
    };
    auto use = [&](FwdIn<P, V> &in, int e) {
      const int r = rt_div(e, mghv), m = (e - r * hv) * V, i0 = r * nx + m;
      if (!R3D_IN(d, gbase + i0 + hx + V - 1, niv)) return;
      const int par = (par0 + r + (plane ? 0 : ((y0 + r) / ny) * (1 - ny))) & 1;
      using Ar = typename P::A;
      Ar f[2][V];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + h * hx;
        if constexpr (MODE > 0) {
          R dn[V];
          T tn[V];
#pragma unroll
          for (int q = 0; q < V; ++q) {
            const double tt = in.t[h][q], rr = in.r[h][q];
            double x;
            if constexpr (MODE == 1) {  // newdt0: t_{k+1} = t_k + R_k
              x = tt + rr;
            } else {  // newdt
              const double p0 = in.b0[h][q], p1 = in.b1[h][q];
              double uu, vv;
              if constexpr (MIXP) {
                const double dnew = in.a0[h][q], dold = (double)in.a1[h][q] + dnew;
                const double e0 = old0 ? dold : dnew, e1 = old0 ? dnew : dold;  // t_slot - t_k
                uu = tt + s1 * e0 + s2 * e1;
                vv = tt + rr + s1 * (e0 + p0 - rr) + s2 * (e1 + p1 - rr);
              } else {
                const double tp0 = in.a0[h][q], tp1 = in.a1[h][q];
                uu = tt + s1 * (tp0 - tt) + s2 * (tp1 - tt);
                vv = tt + rr + s1 * (tp0 + p0 - tt - rr) + s2 * (tp1 + p1 - tt - rr);
              }
              x = uu + mm * (vv - uu);
            }
            dn[q] = MIXP ? (R)(tt - x) : (R)tt;
            tn[q] = (T)x;
          }
          stv<V>(hao + i, dn);
          stv<V>(hbo + i, in.r[h]);
          stv<V>(t + i, tn);
#pragma unroll
          for (int q = 0; q < V; ++q) in.t[h][q] = tn[q];
        }
        // trm1mt on the short-range parts (calculate_cuda.cu:18-24)
        T gv[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const double tt = in.t[h][q];
          const double g = closure_g<double>(clos, pse_n, -(double)in.u[h][q] + tt);
          gv[q] = g;
          double c = g - 1.0 - tt;
          if (MIXP && has_cref) c -= (double)in.c[h][q];
          const Ar fc = (Ar)c;
          f[h][q] = ((m + q + h * hx + par) & 1) ? -fc : fc;
        }
        stv<V>(gq + i, gv);
      }
      const C rf = row[r];
#pragma unroll
      for (int q = 0; q < V; ++q)
        buf[r * LDX + m + q] = cmul(cmul(C{f[0][q], -f[1][q]}, pw[m + q]), rf);
    };
    rt_stream<2, NT, FwdIn<P, V>>(nel, load, use);
  };
  if (mixing == 2)
    work(rt_int<2>{});
  else if (mixing == 1)
    work(rt_int<1>{});
  else
    work(rt_int<0>{});
  __syncthreads();
  // x transform of the rows, lanes along rows
  const uint32_t mgr = NY ? rt_magic(NY) : nrow == pr ? d.rt_mgpr : rt_magic(nrow);
  const uint32_t mghx = HX ? rt_magic(HX) : d.rt_mghx;
  rt_each<HX, RM, false>(HX ? 0 : d.rtx.n, [&](auto s) {
    auto ld = [&](int r, int i) { return buf[r * LDX + i]; };
    auto st = [&](int r, int i, C a) { buf[r * LDX + i] = a; };
    rt_pass_s<HX, -1, NT, RM>(d.rtx, s, nrow, mgr, twx, ld, st);
    __syncthreads();
  });
  S *w = (S *)d.w + (long long)v * d.Nhs + (long long)row0 * hx;
  if (!plane) {
    for (int e = threadIdx.x; e < nrow * hx; e += NT) {
      const int r = rt_div(e, mghx), p = e - r * hx;
      if (R3D_W(e)) w[e] = rt_cvt<S>(buf[r * LDX + p]);
    }
    return;
  }
  // y transform of the columns, lanes along k_x, the last pass straight to
  // the spectrum
  rt_each<NY, RM, false>(NY ? 0 : d.rty.n, [&](auto s) {
    auto ld = [&](int p, int y) { return buf[y * LDX + p]; };
    rt_edge<NY, RM>(
        NY ? 0 : d.rty.n, s,
        [&] {
          auto st = [&](int p, int y, C a) {
            if (R3D_W(y * hx + p)) w[y * hx + p] = rt_cvt<S>(a);
          };
          rt_pass_s<NY, -1, NT, RM>(d.rty, s, hx, mghx, twy, ld, st);
        },
        [&] {
          auto st = [&](int p, int y, C a) { buf[y * LDX + p] = a; };
          rt_pass_s<NY, -1, NT, RM>(d.rty, s, hx, mghx, twy, ld, st);
          __syncthreads();
        });
  });
}

// --------------------------------------------------------------- y pass
// A tile is rt_pcy x-columns of one (site, z) plane; global -> registers in
// the first pass, registers -> global in the last.
template <typename P, int NY, int DIR, int NT, int MINB, int RM = rt_rm<P>()>
__global__ void __launch_bounds__(NT, MINB) k_rt_y(Batch b) {
  using C = typename Cx<typename P::A>::T;  // arithmetic
  using S = typename Cx<typename P::R>::T;  // spectrum
  constexpr int PC = sizeof(typename P::R) == 4 ? 16 : 8;
  extern __shared__ __align__(16) char smem[];
  const int si = find_solve(b, blockIdx.x);
  const Desc &d = b.d[si];
  if (d.ctl->status != RUNNING) return;
  const int hx = d.hx, ny = NY ? NY : d.ny, pt = (hx + PC - 1) / PC;
  int tile = blockIdx.x - b.prefix[si];
  const int p0 = (tile % pt) * PC, zv = tile / pt;
  const int z = zv % d.nz, v = zv / d.nz, pc = min(PC, hx - p0);
  C *buf = (C *)smem, *tw = buf + ny * PC;
  for (int e = threadIdx.x; e < ny; e += NT) tw[e] = rt_table<P>(d, 2)[e];
  S *w = (S *)d.w + (long long)v * d.Nhs + (long long)z * ny * hx + p0;
  __syncthreads();
  // lanes along the columns (those past the last column idle)
  constexpr uint32_t mg = rt_magic(PC);
  const int n = NY ? 0 : d.rty.n;
  rt_each<NY, RM, (DIR > 0)>(n, [&](auto s) {
    const bool first = (int)s == (DIR < 0 ? 0 : (NY ? rt_plan_of(NY, RM).n : n) - 1);
    const bool last = (int)s == (DIR < 0 ? (NY ? rt_plan_of(NY, RM).n : n) - 1 : 0);
    auto ld = [&](int p, int y) {
      if (!first) return buf[y * PC + p];
      return p < pc && R3D_W(y * hx + p) ? rt_cvt<C>(w[y * hx + p]) : C{0, 0};
    };
    auto st = [&](int p, int y, C a) {
      if (!last)
        buf[y * PC + p] = a;
      else if (p < pc && R3D_W(y * hx + p))
        w[y * hx + p] = rt_cvt<S>(a);
    };
    rt_pass_s<NY, DIR, NT, RM>(d.rty, s, PC, mg, tw, ld, st);
    if (!last) __syncthreads();
  });
}

// --------------------------------------------------------------- z pass
// A tile is PC x-columns of one k_y row, all NS sites and all z; forward z
// transform, OZ, inverse z transform.
// Lanes run along columns, then sites (the site stride is an odd multiple of
// PC, so the lanes of a shared-memory access fall on different banks).
__host__ __device__ inline int rt_zstride(int nz, int pc) { return (nz | 1) * pc; }

template <typename P, int NZ, int NS, int PC, int NT, int MINB, int RM = rt_rm<P>()>
__global__ void __launch_bounds__(NT, MINB) k_rt_zoz(Batch b) {
  using R = typename P::R;
  using C = typename Cx<typename P::A>::T;  // arithmetic
  using S = typename Cx<R>::T;              // spectrum
  extern __shared__ __align__(16) char smem[];
  const int si = find_solve(b, blockIdx.x);
  const Desc &d = b.d[si];
  if (d.ctl->status != RUNNING) return;
  const int hx = d.hx, ny = d.ny, nz = NZ ? NZ : d.nz, pt = (hx + PC - 1) / PC;
  const int tile = blockIdx.x - b.prefix[si];
  const int yp = tile / pt, p0 = (tile - yp * pt) * PC, pc = min(PC, hx - p0);
  const int SV = rt_zstride(nz, PC);
  C *buf = (C *)smem, *tw = buf + NS * SV;
  for (int e = threadIdx.x; e < nz; e += NT) tw[e] = rt_table<P>(d, 4)[e];
  const long long zs = (long long)ny * hx, Nhs = d.Nhs;
  S *w = (S *)d.w + (long long)yp * hx + p0;
  const int n = NZ ? 0 : d.rtz.n;
  __syncthreads();
  constexpr int W = NS * PC;
  constexpr uint32_t mgW = rt_magic(W);
  // lane c of a pass: column c % PC of site c / PC
  auto lds = [&](int c, int z) { return buf[(c / PC) * SV + z * PC + c % PC]; };
  auto sts = [&](int c, int z, C a) { buf[(c / PC) * SV + z * PC + c % PC] = a; };
  rt_each<NZ, RM, false>(n, [&](auto s) {
    const bool first = (int)s == 0;
    auto ld = [&](int c, int z) {
      if (!first) return lds(c, z);
      const int p = c % PC, v = c / PC;
      return p < pc && R3D_W(v * Nhs + z * zs + p) ? rt_cvt<C>(w[v * Nhs + z * zs + p]) : C{0, 0};
    };
    rt_pass_s<NZ, -1, NT, RM>(d.rtz, s, W, mgW, tw, ld, sts);
    __syncthreads();
  });
  // OZ, in place.  Positions s and nz - 1 - s hold k_z and nz - 1 - k_z, the
  // same |k| shell, and share one chi block.  Q lanes of a warp take one pair
  // of points, NS / Q output sites each: a lane reads its sites' rows of the
  // shell's chi matrix (the lanes of a pair read one contiguous block), every
  // site's inputs and, once the pair's lanes have read, writes its outputs.
  // A lane keeps its column, so that a pair's shell is one table read, an
  // add and a shift.
  {
    constexpr int Q = NS == 4 ? 2 : NS, OS = NS / Q;    // lanes per pair, sites per lane
    constexpr int G = 32 / Q, SPI = G / PC, NW = NT / 32;  // pairs a warp takes: SPI rows of PC
    static_assert(SPI >= 1, "a warp takes whole rows of columns");
    constexpr int U = 4;  // pairs whose chi rows are in flight together
    const int *xrev = d.rtrev, *yrev = xrev + hx, *zrev = yrev + ny;
    const int lane = threadIdx.x & 31, q0 = (lane % Q) * OS, grp = lane / Q;
    const int p = grp % PC, sub = grp / PC;
    const bool lane_on = grp < SPI * PC && p < pc;
    const int kx = lane_on ? xrev[p0 + p] : 0, ky = yrev[yp];
    using X = typename P::A;
    const X *chi = (const X *)(sizeof(X) > sizeof(R) ? d.chi64 : d.chi) + q0 * NS;
    const bool cubic = d.cubic != 0;
    const int chis = d.chis, half = nz / 2;
    const int ax = 4 * kx - d.nx + 1, ay = 2 * ky - ny + 1, axy = ax * ax + ay * ay - 3;
    const uint32_t *kidx = d.kidx + (long long)ky * hx + kx;
    for (int s0 = (threadIdx.x >> 5) * SPI; s0 < half; s0 += U * NW * SPI) {
      X x[U][OS][NS];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int s = s0 + k * NW * SPI + sub;
        if (!lane_on || s >= half) continue;
        const int kz = zrev[s], az = 2 * kz - nz + 1;
        // cubic cells: shell (ax^2 + ay^2 + az^2 - 3) / 8, below 2^31 up to
        // 2048 points a side
        if (!cubic && !R3D_IN(d, ((long long)kz * ny + ky) * hx + kx, d.Nh)) continue;
        const uint32_t shell = cubic ? (uint32_t)(axy + az * az) >> 3 : kidx[kz * zs];
        if (cubic && !R3D_IN(d, shell, (3LL * (nz - 1) * (nz - 1) - 3) / 8 + 1)) continue;
        const X *ch = chi + (size_t)shell * chis;
#pragma unroll
        for (int o = 0; o < OS; ++o) {
          if constexpr (NS == 4 && sizeof(X) == 4) {
            const float4 v4 = *reinterpret_cast<const float4 *>(ch + o * NS);
            x[k][o][0] = v4.x, x[k][o][1] = v4.y, x[k][o][2] = v4.z, x[k][o][3] = v4.w;
          } else if constexpr (NS == 4 || NS == 2) {
#pragma unroll
            for (int j = 0; j < NS; j += 2) {
              X two[2];
              ldv<2>(two, ch + o * NS + j);
              x[k][o][j] = two[0], x[k][o][j + 1] = two[1];
            }
          } else {
#pragma unroll
            for (int j = 0; j < NS; ++j) x[k][o][j] = ch[o * NS + j];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int s = s0 + k * NW * SPI + sub;
        const bool on = lane_on && s < half;
        C *c1 = buf + s * PC + p, *c2 = buf + (nz - 1 - s) * PC + p;
        C h1[OS], h2[OS];
        if (on) {
          C a[NS], e[NS];
#pragma unroll
          for (int j = 0; j < NS; ++j) a[j] = c1[j * SV], e[j] = c2[j * SV];
#pragma unroll
          for (int o = 0; o < OS; ++o) {
            h1[o] = h2[o] = C{0, 0};
#pragma unroll
            for (int j = 0; j < NS; ++j) {
              const X xj = x[k][o][j];
              h1[o].x += a[j].x * xj;
              h1[o].y += a[j].y * xj;
              h2[o].x += e[j].x * xj;
              h2[o].y += e[j].y * xj;
            }
          }
        }
        __syncwarp();
        if (on) {
#pragma unroll
          for (int o = 0; o < OS; ++o) c1[(q0 + o) * SV] = h1[o], c2[(q0 + o) * SV] = h2[o];
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  rt_each<NZ, RM, true>(n, [&](auto s) {
    const bool last = (int)s == 0;
    auto st = [&](int c, int z, C a) {
      if (!last) {
        sts(c, z, a);
      } else {
        const int p = c % PC, v = c / PC;
        if (p < pc && R3D_W(v * Nhs + z * zs + p))
          w[v * Nhs + z * zs + p] = rt_cvt<S>(a);
      }
    };
    rt_pass_s<NZ, 1, NT, RM>(d.rtz, s, W, mgW, tw, lds, st);
    if (!last) __syncthreads();
  });
}

// --------------------------------------------------------------- inverse
// CTA c of a solve takes up to rt_iper consecutive tiles of one site.
// mode: what the solve's last CTA does with the sums (reduce_finish).
template <typename P, int V>
struct InvIn {
  typename P::T g[2][V];
  typename P::R l[2][V], p0[2][V], p1[2][V];
};

template <typename P, int HX, int NY, int V, int NT, int MINB, int RM = rt_rm<P>()>
__global__ void __launch_bounds__(NT, MINB) k_rt_inv(Batch b, int mode) {
  using R = typename P::R;
  using T = typename P::T;
  using C = typename Cx<typename P::A>::T;  // arithmetic
  using S = typename Cx<R>::T;              // spectrum
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) char smem[];
  __shared__ double red[6][NW];
  __shared__ int last_cta;
  const int si = find_solve(b, blockIdx.x);
  const Desc &d = b.d[si];
  if (d.ctl->status != RUNNING) return;
  const int hx = HX ? HX : d.hx, nx = 2 * hx, ny = NY ? NY : d.ny, LDX = rt_ldx(hx);
  const bool plane = HX ? NY != 0 : d.rt_plane != 0;
  const int cta = blockIdx.x - b.prefix[si];
  const int v = cta / d.rt_icps, part = cta - v * d.rt_icps;
  const bool dots = d.mixer == MIX_AN2 && d.ctl->count_left <= 0;
  const int pr = NY ? NY : d.rt_pr;
  C *buf = (C *)smem, *row = buf + pr * LDX, *twx = row + pr, *pw = twx + hx, *twy = pw + hx;
  for (int e = threadIdx.x; e < hx; e += NT) {
    twx[e] = rt_table<P>(d, 0)[e];
    pw[e] = rt_table<P>(d, 1)[e];
  }
  if (plane)
    for (int e = threadIdx.x; e < ny; e += NT) twy[e] = rt_table<P>(d, 2)[e];
  const long long niv = (long long)d.n * d.Ns;
  const int hv = hx / V;
  const uint32_t mghx = HX ? rt_magic(HX) : d.rt_mghx, mghv = HX ? rt_magic(HX / V) : d.rt_mghv;
  double q[6] = {0, 0, 0, 0, 0, 0};
  const int tile1 = min(d.rt_tps, (part + 1) * d.rt_iper);
  for (int tile = part * d.rt_iper; tile < tile1; ++tile) {
    const int row0 = tile * pr, nrow = NY ? NY : min(pr, ny * d.nz - row0);
    const S *w = (const S *)d.w + (long long)v * d.Nhs + (long long)row0 * hx;
    const long long gbase = (long long)v * d.Ns + (long long)row0 * nx;
    rt_row_factors<P, NT>(row, d, row0, nrow, ny);
    __syncthreads();
    if (plane) {  // inverse y transform, first pass straight from the spectrum
      rt_each<NY, RM, true>(NY ? 0 : d.rty.n, [&](auto s) {
        auto st = [&](int p, int y, C a) { buf[y * LDX + p] = a; };
        rt_edge<NY, RM>(
            NY ? 0 : d.rty.n, s,
            [&] {
              auto ld = [&](int p, int y) {
                return R3D_W(y * hx + p) ? rt_cvt<C>(w[y * hx + p]) : C{0, 0};
              };
              rt_pass_s<NY, 1, NT, RM>(d.rty, s, hx, mghx, twy, ld, st);
            },
            [&] {
              auto ld = [&](int p, int y) { return buf[y * LDX + p]; };
              rt_pass_s<NY, 1, NT, RM>(d.rty, s, hx, mghx, twy, ld, st);
            });
        __syncthreads();
      });
    } else {
      // (128 bytes of loads per thread in flight)
      constexpr int U = 128 / (int)sizeof(S);
      for (int e0 = threadIdx.x; e0 < nrow * hx; e0 += U * NT) {
        S a[U];
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (e0 + k * NT < nrow * hx && R3D_W(e0 + k * NT))
            a[k] = w[e0 + k * NT];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int e = e0 + k * NT, r = rt_div(e, mghx), p = e - r * hx;
          if (e < nrow * hx) buf[r * LDX + p] = rt_cvt<C>(a[k]);
        }
      }
      __syncthreads();
    }
    const uint32_t mgr = NY ? rt_magic(NY) : nrow == pr ? d.rt_mgpr : rt_magic(nrow);
    rt_each<HX, RM, true>(HX ? 0 : d.rtx.n, [&](auto s) {
      auto ld = [&](int r, int i) { return buf[r * LDX + i]; };
      auto st = [&](int r, int i, C a) { buf[r * LDX + i] = a; };
      rt_pass_s<HX, 1, NT, RM>(d.rtx, s, nrow, mgr, twx, ld, st);
      __syncthreads();
    });
    // unpacking, residual R = h + 1 - g (calculate_cuda.cu:54-60), sum R^2
    // (cal_rms.cu:14-26) and the five theta dots (anderson_cuda.cu:25-67);
    // the next elements' loads are in flight while these are worked on
    const T *gq = (const T *)d.gq + gbase;
    const R *lr = (const R *)d.lr + gbase;
    const R *rp0 = (const R *)d.hist_b + gbase, *rp1 = rp0 + niv;
    R *res = (R *)d.res + gbase;
    const int y0 = row0 % ny, par0 = (y0 + row0 / ny) & 1, nel = nrow * hv;
    auto work = [&](auto with_dots) {
    constexpr bool DOTS = decltype(with_dots)::value != 0;
    auto load = [&](InvIn<P, V> &in, int e) {
      const int r = rt_div(e, mghv), i0 = r * nx + (e - r * hv) * V;
      if (!R3D_IN(d, gbase + i0 + hx + V - 1, niv)) return;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + h * hx;
        ldv<V>(in.g[h], gq + i);
        ldv<V>(in.l[h], lr + i);
        if constexpr (DOTS) {
          ldv<V>(in.p0[h], rp0 + i);
          ldv<V>(in.p1[h], rp1 + i);
        }
      }
    };
    auto use = [&](const InvIn<P, V> &in, int e) {
      const int r = rt_div(e, mghv), m = (e - r * hv) * V, i0 = r * nx + m;
      if (!R3D_IN(d, gbase + i0 + hx + V - 1, niv)) return;
      const C rf = cconj(row[r]);
      const int par = (par0 + r + (plane ? 0 : ((y0 + r) / ny) * (1 - ny))) & 1;
      R ro[2][V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const C z = cmul(cmul(buf[r * LDX + m + k], rf), cconj(pw[m + k]));
        const double h0 = ((m + k + par) & 1) ? -z.x : z.x;
        const double h1 = ((m + k + hx + par) & 1) ? z.y : -z.y;
        ro[0][k] = (R)(h0 + (double)in.l[0][k] - (double)in.g[0][k]);
        ro[1][k] = (R)(h1 + (double)in.l[1][k] - (double)in.g[1][k]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        stv<V>(res + i0 + h * hx, ro[h]);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const double rr = ro[h][k];
          q[0] += rr * rr;
          if constexpr (DOTS) {
            const double t1 = rr - (double)in.p0[h][k], t2 = rr - (double)in.p1[h][k];
            q[1] += rr * t1;
            q[2] += rr * t2;
            q[3] += t1 * t1;
            q[4] += t1 * t2;
            q[5] += t2 * t2;
          }
        }
      }
    };
    rt_stream<2, NT, InvIn<P, V>>(nel, load, use);
    };
    if (dots)
      work(rt_int<1>{});
    else
      work(rt_int<0>{});
    if (tile + 1 < tile1) __syncthreads();  // buf is free again
  }
  // this CTA's sums, in a fixed order: butterflies, then the warps in order
#pragma unroll
  for (int k = 0; k < 6; ++k)
    for (int o = 16; o > 0; o >>= 1) q[k] += __shfl_xor_sync(0xffffffffu, q[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < 6; ++k) red[k][threadIdx.x >> 5] = q[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) s += red[threadIdx.x][i];
    if (R3D_IN(d, (v * 6 + threadIdx.x) * d.rt_icps + part, 6 * d.n * d.rt_icps))
      d.partials[((size_t)v * 6 + threadIdx.x) * d.rt_icps + part] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0)
    last_cta = atomicAdd(&d.ctl->done, 1u) == (unsigned)(d.n * d.rt_icps) - 1;
  __syncthreads();
  if (!last_cta) return;
  __threadfence();
  rt_reduce<NT>(d, mode, dots);
  if (threadIdx.x == 0) d.ctl->done = 0;
}

#if R3D_CT_FP64 == 1 && R3D_RT_PART == 1
// the reduce alone (anderson(): mode 1), one CTA per solve
__global__ void __launch_bounds__(kThreads) k_rt_reduce(const Desc *descs, int mode) {
  const Desc &d = descs[blockIdx.x];
  rt_reduce<kThreads>(d, mode, d.mixer == MIX_AN2 && d.ctl->count_left <= 0);
}
#endif

// ------------------------------------------------------------ launchers
// Compile-time sizes, of the configurations' cubic grids: n^2 planes (CUBES),
// rows of n in tiles and columns of n (LONG), z columns (Z) -- of each, those
// that a kind's rule can choose (plan_rt, rt_double): FP64 planes up to 96^2
// fit two to an SM, FP32 arithmetic serves the larger grids only.  Every other
// grid runs the run-time-sized kernels.
#define R3D_RT_CUBES(X) X(48) X(64) X(80) X(96) X(128) X(144)
#define R3D_RT_LONG(X) X(96) X(128) X(144) X(160) X(192) X(256) X(512)
#define R3D_RT_Z(X) X(48) X(64) X(80) X(96) X(128) X(144) X(160) X(192) X(256) X(512)
constexpr bool rt_has_cube(int kind, int n) { return kind == RT_FP32 ? n >= 128 : n <= 96; }
constexpr bool rt_has_long(int kind, int n) {
  return kind == RT_MIXED ? n == 96 || n == 144 : true;
}
constexpr bool rt_has_z(int kind, int n) {
  return kind == RT_FP64 || (kind == RT_FP32 ? n >= 96 : n <= 96 || n == 144);
}
template <typename P>
constexpr int rt_kind() {
  return sizeof(typename P::R) == 8 ? RT_FP64 : sizeof(typename P::A) == 8 ? RT_MIXED : RT_FP32;
}

// the run-time-sized x kernels with small radices serve these plans
static bool rt_lean(const Desc &d) {
  return d.rtx.r[0] <= kRtLean && (!d.rt_plane || d.rty.r[0] <= kRtLean);
}

template <typename P>
constexpr int rt_pcz() {  // 64-byte rows of spectrum columns
  return sizeof(typename P::R) == 4 ? 8 : 4;
}
// vector width of the x passes: pairs where both halves of a row start on an
// even element (FP64: single elements, two sets of which fill the registers)
template <typename P>
constexpr int rt_vec() {
  return sizeof(typename P::R) == 4 ? 2 : 1;
}

// f(kernel) for the kernel of this geometry; nt: its threads
template <typename P, typename F>
static void rt_fwd_kernel(const Desc &d, int nt, F f) {
  constexpr int V = rt_vec<P>(), RM = rt_rm<P>();
#define R3D_RT_F(N)                                                                  \
  if constexpr (rt_has_cube(rt_kind<P>(), N))                                        \
    if (d.rt_plane && d.nx == N && d.ny == N) {                                      \
      if constexpr (N <= 64)                                                         \
        if (nt == 512) return f(k_rt_fwd<P, N / 2, N, V, 512, 1>);                   \
      return f(k_rt_fwd<P, N / 2, N, V, 256, 2>);                                    \
    }
  R3D_RT_CUBES(R3D_RT_F)
#undef R3D_RT_F
#define R3D_RT_F(N)                           \
  if constexpr (rt_has_long(rt_kind<P>(), N)) \
    if (!d.rt_plane && d.nx == N) return f(k_rt_fwd<P, N / 2, 0, V, 256, 2>);
  R3D_RT_LONG(R3D_RT_F)
#undef R3D_RT_F
  const bool pairs = V == 2 && d.hx % 2 == 0;
  if (rt_lean(d)) {
    if constexpr (rt_kind<P>() != RT_FP32)
      if (nt == 512)
        return pairs ? f(k_rt_fwd<P, 0, 0, V, 512, 1, kRtLean>) : f(k_rt_fwd<P, 0, 0, 1, 512, 1, kRtLean>);
    return pairs ? f(k_rt_fwd<P, 0, 0, V, 256, 2, kRtLean>) : f(k_rt_fwd<P, 0, 0, 1, 256, 2, kRtLean>);
  }
  return pairs ? f(k_rt_fwd<P, 0, 0, V, 256, 2, RM>) : f(k_rt_fwd<P, 0, 0, 1, 256, 2, RM>);
}
// (tiles: single elements in mixed precision too, whose fewer registers let
// the scheduler keep the loads early: 256^3, 415 us against 446)
template <typename P, typename F>
static void rt_inv_kernel(const Desc &d, int nt, F f) {
  constexpr int V = rt_vec<P>(), RM = rt_rm<P>();
#define R3D_RT_F(N)                                                                  \
  if constexpr (rt_has_cube(rt_kind<P>(), N))                                        \
    if (d.rt_plane && d.nx == N && d.ny == N) {                                      \
      if constexpr (N <= 64)                                                         \
        if (nt == 512) return f(k_rt_inv<P, N / 2, N, V, 512, 1>);                   \
      return f(k_rt_inv<P, N / 2, N, V, 256, 2>);                                    \
    }
  R3D_RT_CUBES(R3D_RT_F)
#undef R3D_RT_F
#define R3D_RT_F(N)                           \
  if constexpr (rt_has_long(rt_kind<P>(), N)) \
    if (!d.rt_plane && d.nx == N) return f(k_rt_inv<P, N / 2, 0, 1, 256, 2>);
  R3D_RT_LONG(R3D_RT_F)
#undef R3D_RT_F
  const bool pairs = V == 2 && d.hx % 2 == 0;
  if (rt_lean(d)) {
    if constexpr (rt_kind<P>() != RT_FP32)
      if (nt == 512)
        return pairs ? f(k_rt_inv<P, 0, 0, V, 512, 1, kRtLean>) : f(k_rt_inv<P, 0, 0, 1, 512, 1, kRtLean>);
    return pairs ? f(k_rt_inv<P, 0, 0, V, 256, 2, kRtLean>) : f(k_rt_inv<P, 0, 0, 1, 256, 2, kRtLean>);
  }
  return pairs ? f(k_rt_inv<P, 0, 0, V, 256, 2, RM>) : f(k_rt_inv<P, 0, 0, 1, 256, 2, RM>);
}
template <typename P, typename F>
static void rt_y_kernel(const Desc &d, int dir, F f) {
  constexpr int MB = sizeof(typename P::A) == 4 ? 3 : 2, RM = rt_rm<P>();
#define R3D_RT_F(N)                                          \
  if constexpr (rt_has_long(rt_kind<P>(), N))                \
    if (d.ny == N) {                                         \
      if (dir < 0) return f(k_rt_y<P, N, -1, kThreads, MB>); \
      return f(k_rt_y<P, N, 1, kThreads, MB>);               \
    }
  R3D_RT_LONG(R3D_RT_F)
#undef R3D_RT_F
  if (d.rty.r[0] <= kRtLean)
    return dir < 0 ? f(k_rt_y<P, 0, -1, kThreads, MB, kRtLean>) : f(k_rt_y<P, 0, 1, kThreads, MB, kRtLean>);
  dir < 0 ? f(k_rt_y<P, 0, -1, kThreads, 2, RM>) : f(k_rt_y<P, 0, 1, kThreads, 2, RM>);
}
// resident CTAs the z pass' registers are held to.  Short columns: four, so
// that a small grid's tiles are all resident (96^3, two sites, mixed: 8.3 us
// against 10.4 with two or three; 64^3 FP64: 7.1 against 8.3).  Long ones need
// their radices' registers (144^3, four sites, mixed: 37 us with three, 44 with
// two; 256^3: 221 us with two, 244 and 262 with three and four; FP64 461, 516,
// 532).
template <typename P>
constexpr int rt_z_ctas(int nz) {
  return nz <= 96 ? 4 : sizeof(typename P::A) == 4 && nz <= 192 ? 3 : 2;
}
template <typename P, int NS, typename F>
static void rt_zoz_kernel_ns(const Desc &d, F f) {
  constexpr int PC = rt_pcz<P>();
  if constexpr (NS == 2 || NS == 4) {
#define R3D_RT_F(N)                        \
  if constexpr (rt_has_z(rt_kind<P>(), N)) \
    if (d.nz == N) return f(k_rt_zoz<P, N, NS, PC, kThreads, rt_z_ctas<P>(N)>);
    R3D_RT_Z(R3D_RT_F)
#undef R3D_RT_F
  }
  constexpr int MB = sizeof(typename P::A) == 4 ? 3 : 2;
  if (d.rtz.r[0] <= kRtLean)
    f(k_rt_zoz<P, 0, NS, PC, kThreads, MB, kRtLean>);
  else
    f(k_rt_zoz<P, 0, NS, PC, kThreads, 2, rt_rm<P>()>);
}
template <typename P, typename F>
static void rt_zoz_kernel(const Desc &d, F f) {
  switch (d.n) {
    case 1: rt_zoz_kernel_ns<P, 1>(d, f); break;
    case 2: rt_zoz_kernel_ns<P, 2>(d, f); break;
    case 3: rt_zoz_kernel_ns<P, 3>(d, f); break;
    default: rt_zoz_kernel_ns<P, 4>(d, f); break;
  }
}

static auto rt_allow = [](auto k) {
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
};

// The launches, and per kernel family the opt-in into large shared memory for
// a geometry (before any capture; the inverse's returns its resident CTAs per
// SM).
#if R3D_RT_PART == 0
template <typename P>
void rt_launch_fwd(const Desc &d, Batch b, int grid, int nt, size_t smem, cudaStream_t s,
                   int allow_mix) {
  rt_fwd_kernel<P>(d, nt, [&](auto k) { k<<<grid, nt, smem, s>>>(b, allow_mix); });
}
template <typename P>
void rt_allow_fwd(const Desc &d, int nt) {
  rt_fwd_kernel<P>(d, nt, rt_allow);
}
template void rt_launch_fwd<PRT>(const Desc &, Batch, int, int, size_t, cudaStream_t, int);
template void rt_allow_fwd<PRT>(const Desc &, int);
#elif R3D_RT_PART == 1
template <typename P>
void rt_launch_inv(const Desc &d, Batch b, int grid, int nt, size_t smem, cudaStream_t s, int mode) {
  rt_inv_kernel<P>(d, nt, [&](auto k) { k<<<grid, nt, smem, s>>>(b, mode); });
}
template <typename P>
int rt_allow_inv(const Desc &d, int nt, size_t smem) {
  int nb = 0;
  rt_inv_kernel<P>(d, nt, [&](auto k) {
    rt_allow(k);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, nt, smem);
  });
  return nb;
}
template void rt_launch_inv<PRT>(const Desc &, Batch, int, int, size_t, cudaStream_t, int);
template int rt_allow_inv<PRT>(const Desc &, int, size_t);
#else
template <typename P>
void rt_launch_y(const Desc &d, int dir, Batch b, int grid, size_t smem, cudaStream_t s) {
  rt_y_kernel<P>(d, dir, [&](auto k) { k<<<grid, kThreads, smem, s>>>(b); });
}
template <typename P>
void rt_launch_zoz(const Desc &d, Batch b, int grid, size_t smem, cudaStream_t s) {
  rt_zoz_kernel<P>(d, [&](auto k) { k<<<grid, kThreads, smem, s>>>(b); });
}
template <typename P>
void rt_allow_yz(const Desc &d) {
  if (!d.rt_plane) {
    rt_y_kernel<P>(d, -1, rt_allow);
    rt_y_kernel<P>(d, 1, rt_allow);
  }
  rt_zoz_kernel<P>(d, rt_allow);
}
template void rt_launch_y<PRT>(const Desc &, int, Batch, int, size_t, cudaStream_t);
template void rt_launch_zoz<PRT>(const Desc &, Batch, int, size_t, cudaStream_t);
template void rt_allow_yz<PRT>(const Desc &);
#endif

#if R3D_CT_FP64 == 1 && R3D_RT_PART == 1
void launch_rt_reduce(const Desc *d, int ns, int mode, cudaStream_t s) {
  k_rt_reduce<<<ns, kThreads, 0, s>>>(d, mode);
}
size_t rt_smem_x(int hx, int ny, int pr, bool plane, size_t csz) {
  return csz * ((size_t)pr * (rt_ldx(hx) + 1) + 2 * (size_t)hx + (plane ? ny : 0));
}
size_t rt_smem_y(int ny, int pc, size_t csz) { return csz * ((size_t)ny * pc + (size_t)ny); }
size_t rt_smem_z(int nz, int n, int pc, size_t csz) {
  return csz * ((size_t)n * rt_zstride(nz, pc) + (size_t)nz);
}

// Plans a geometry's axes (d.rt_plane set): a compile-time-sized kernel's
// radices where one serves the axis, else the run-time-sized kernels' small
// ones unless they cost a pass more.  Returns false where a length has no plan.
bool rt_plan_axes(Desc &d, int kind) {
  const int rm = kind == RT_FP32 ? 16 : 13;
  auto any = [&](int L) {
    const RtPlan full = rt_plan_of(L, rm), lean = rt_plan_of(L, kRtLean);
    return lean.n && lean.n <= full.n ? lean : full;
  };
  const bool sx = rt_static_x(kind, d.nx, d.ny, d.rt_plane != 0),
             sy = d.rt_plane ? sx : rt_static_y(kind, d.ny), sz = rt_static_z(kind, d.nz, d.n);
  d.rtx = sx ? rt_plan_of(d.hx, rm) : any(d.hx);
  d.rty = sy ? rt_plan_of(d.ny, rm) : any(d.ny);
  d.rtz = sz ? rt_plan_of(d.nz, rm) : any(d.nz);
  return d.rtx.n && d.rty.n && d.rtz.n;
}
// threads of a plane's x kernels: 512 where the planes do not fill the SMs
// and a kernel of 512 serves them (64^3, two sites, FP64: 31 us an iteration
// against 34)
int rt_threads(const Desc &d, int kind, int nsm) {
  if (!d.rt_plane || d.n * d.rt_tps > nsm || kind == RT_FP32) return 256;
  if (rt_static_x(kind, d.nx, d.ny, true)) return d.nx <= 64 ? 512 : 256;
  return rt_lean(d) ? 512 : 256;
}
int rt_passes(int L, bool dbl) { return rt_plan_of(L, dbl ? 13 : 16).n; }
// whether a length is among the compile-time ones, whatever the kind
bool rt_listed(int n) {
#define R3D_RT_F(N) \
  if (n == N) return true;
  R3D_RT_Z(R3D_RT_F)
#undef R3D_RT_F
  return false;
}
// whether compile-time-sized kernels serve an x (and, of a plane, y) axis, a
// y axis of its own, a z axis of n sites
bool rt_static_x(int kind, int nx, int ny, bool plane) {
#define R3D_RT_F(N) \
  if (plane && nx == N && ny == N) return rt_has_cube(kind, N);
  R3D_RT_CUBES(R3D_RT_F)
#undef R3D_RT_F
#define R3D_RT_F(N) \
  if (!plane && nx == N) return rt_has_long(kind, N);
  R3D_RT_LONG(R3D_RT_F)
#undef R3D_RT_F
  return false;
}
bool rt_static_y(int kind, int ny) {
#define R3D_RT_F(N) \
  if (ny == N) return rt_has_long(kind, N);
  R3D_RT_LONG(R3D_RT_F)
#undef R3D_RT_F
  return false;
}
bool rt_static_z(int kind, int nz, int n) {
#define R3D_RT_F(N) \
  if (nz == N) return (n == 2 || n == 4) && rt_has_z(kind, N);
  R3D_RT_Z(R3D_RT_F)
#undef R3D_RT_F
  return false;
}
#endif

}  // namespace r3d
