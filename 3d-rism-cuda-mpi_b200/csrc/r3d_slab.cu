// r3d_slab.cu -- the stages of the shifted 3D transform on one rank's slab
// of a grid split over several GPUs (r3d_slab_transform).
//
// The reference distributes its transform over MPI ranks as 1D cuFFT passes
// and Alltoall transposes of pencils (fft3d.cu:81-163, the decomposition of
// cell.cc:30-48).  Here a grid split over P GPUs is cut in z-slabs (rank r
// owns z-planes [r nz/P, (r+1) nz/P)) for the x and y passes and in y-slabs
// for the z pass; one all-to-all per direction moves the half spectrum
// between the two (slabs.py drives it with NCCL).  This file runs one
// rank's stages on its own device buffers:
//   stage 0  z-slab real grid [nzl][ny][nx] -> packed x and y transforms ->
//            half spectrum [nzl][ny][nx/2]          (d_real in, d_spec out)
//   stage 1  y-slab half spectrum [nz][nyl][nx/2] -> z transform (in place)
//   stage 2  y-slab inverse z transform (in place)
//   stage 3  z-slab half spectrum -> inverse y and x transforms -> real grid
//            (d_spec in, destroyed; d_real out)
// in the transform units of the iteration's passes: unnormalised, the
// checkerboard and half-sample factors inside, the constant phase dv C(k)
// outside (the full-grid seam r3d_fft3d applies it).  The checkerboard sign
// (-1)^(x+y+z) uses the slab's local z, which equals the global z's parity
// when every slab starts on an even plane (the caller's partition).
//
// The kernels are the run-time-planned engine's (r3d_fft_rt.cuh) on natural
// order: a tile's rows or columns are permuted on their way out of (or into)
// shared memory.  They take their arguments by value and make their twiddles
// in shared memory, once per resident CTA (each walks many tiles), so a call
// uploads nothing and keeps nothing.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "../../include/rism3d_b200.h"
#include "r3d_common.cuh"
#include "r3d_fft_rt.cuh"

namespace r3d {
size_t smem_x(int hx, int n, int S, size_t csz);
size_t smem_y(int ny, int P, size_t csz);
size_t smem_z(int nz, int n, int P, size_t csz);
void set_last_error(const std::string &m);

namespace {
// A plan of up to eight passes: RtPlan's where there is one, else (5^5, 7 5^4)
// the largest radices first.
struct SlabPlan {
  int L, n;
  int r[8], m[8], tws[8];
  uint32_t mg[8];
};
SlabPlan slab_plan(int L) {
  SlabPlan p{};
  p.L = L;
  const RtPlan q = rt_plan_of(L, 13);
  int m = L;
  auto add = [&](int r) {
    m /= r;
    p.r[p.n] = r;
    p.m[p.n] = m;
    p.tws[p.n] = L / (r * m);
    p.mg[p.n] = rt_magic(m);
    ++p.n;
  };
  for (int s = 0; s < q.n; ++s) add(q.r[s]);
  for (int r = 13; r >= 2; --r)
    while (m % r == 0 && p.n < 8) add(r);
  if (m > 1) p.n = 0;
  return p;
}

// tables of one length in shared memory: W_L^e, the half-sample twiddles
// e^{-i pi a / n} (n = L, or 2 L for the packed x transform) and the position
// of each index under the engine's digit reversal
struct SlabTab {
  double2 *tw, *pw;
  uint16_t *pos, *rev;  // position of an index, index at a position (one of the two)
  __device__ int idx(int P) const { return rev[P]; }
};
template <bool POS>
__device__ __forceinline__ SlabTab slab_tables(char *sm, const SlabPlan &p, int n) {
  SlabTab t;
  t.tw = (double2 *)sm;
  t.pw = t.tw + p.L;
  t.pos = t.rev = (uint16_t *)(t.pw + p.L);
  for (int e = threadIdx.x; e < p.L; e += blockDim.x) {
    double s, c;
    sincospi(-2.0 * (double)e / (double)p.L, &s, &c);
    t.tw[e] = make_double2(c, s);
    sincospi(-(double)e / (double)n, &s, &c);
    t.pw[e] = make_double2(c, s);
    int K = 0, P = e, scale = 1;
    for (int k = 0; k < p.n; ++k) {
      const int u = P / p.m[k];
      P -= u * p.m[k];
      K += u * scale;
      scale *= p.r[k];
    }
    if (POS)
      t.pos[K] = (uint16_t)e;
    else
      t.rev[e] = (uint16_t)K;
  }
  return t;
}
__host__ __device__ inline size_t slab_tab_bytes(int L) {
  return ((size_t)L * 34 + 15) / 16 * 16;
}

// The packed x transform of pr rows a tile: DIR -1 real rows -> half spectrum
// (natural k_x), +1 back.  Rows run over sites, z and y.
template <int DIR>
__global__ void __launch_bounds__(kThreads, 2)
    k_slab_x(SlabPlan px, int ny, int nz, long long rows, int pr, double *real, double2 *spec) {
  extern __shared__ __align__(16) char smem[];
  const int hx = px.L, nx = 2 * hx, LDX = hx | 1;
  const SlabTab t = slab_tables<true>(smem, px, nx);
  double2 *buf = (double2 *)(smem + slab_tab_bytes(hx));
  const uint32_t mghx = rt_magic(hx);
  const long long tiles = (rows + pr - 1) / pr;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long row0 = tile * pr;
    const int nrow = (int)min((long long)pr, rows - row0), nel = nrow * hx;
    const uint32_t mgr = rt_magic(nrow);
    double *f = real + row0 * nx;
    double2 *w = spec + row0 * hx;
    // checkerboard sign of a row's first element: (y + z) & 1
    auto parity = [&](int r) {
      const long long rs = (row0 + r) % ((long long)ny * nz);
      return (int)((rs % ny + rs / ny) & 1);
    };
    __syncthreads();  // the tables; the last tile's buf is free
    if constexpr (DIR < 0) {
      constexpr int U = 4;  // loads of eight values in flight
      for (int e0 = threadIdx.x; e0 < nel; e0 += U * kThreads) {
        double a[U], b[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int e = e0 + k * kThreads, r = rt_div(e, mghx), m = e - r * hx;
          if (e < nel) a[k] = f[r * nx + m], b[k] = f[r * nx + m + hx];
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int e = e0 + k * kThreads, r = rt_div(e, mghx), m = e - r * hx;
          if (e >= nel) continue;
          const int par = parity(r);
          const double f0 = ((m + par) & 1) ? -a[k] : a[k];
          const double f1 = ((m + hx + par) & 1) ? -b[k] : b[k];
          buf[r * LDX + m] = cmul(make_double2(f0, -f1), t.pw[m]);
        }
      }
    } else {
      constexpr int U = 4;
      for (int e0 = threadIdx.x; e0 < nel; e0 += U * kThreads) {
        double2 a[U];
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (e0 + k * kThreads < nel) a[k] = w[e0 + k * kThreads];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int e = e0 + k * kThreads, r = rt_div(e, mghx), p = e - r * hx;
          if (e < nel) buf[r * LDX + t.pos[p]] = a[k];
        }
      }
    }
    __syncthreads();
    auto ld = [&](int r, int i) { return buf[r * LDX + i]; };
    auto st = [&](int r, int i, double2 a) { buf[r * LDX + i] = a; };
    for (int k = 0; k < px.n; ++k) {
      rt_pass_s<0, DIR, kThreads, 13>(px, DIR < 0 ? k : px.n - 1 - k, nrow, mgr, t.tw, ld, st);
      __syncthreads();
    }
    for (int e = threadIdx.x; e < nel; e += kThreads) {
      const int r = rt_div(e, mghx), m = e - r * hx;
      if constexpr (DIR < 0) {
        w[e] = buf[r * LDX + t.pos[m]];
      } else {
        const double2 z = cmul(buf[r * LDX + m], cconj(t.pw[m]));
        const int par = parity(r);
        f[r * nx + m] = ((m + par) & 1) ? -z.x : z.x;
        f[r * nx + m + hx] = ((m + hx + par) & 1) ? z.y : -z.y;
      }
    }
  }
}

// A y or z transform in place: columns of py.L elements `stride` apart, ncol
// adjacent columns in each of nb blocks `bstride` apart, PC columns a tile;
// natural order in and out.
template <int DIR, int PC>
__global__ void __launch_bounds__(kThreads, 2)
    k_slab_col(SlabPlan py, long long stride, long long ncol, long long nb, long long bstride,
               double2 *spec) {
  extern __shared__ __align__(16) char smem[];
  const int L = py.L;
  const SlabTab t = slab_tables<false>(smem, py, L);
  double2 *buf = (double2 *)(smem + slab_tab_bytes(L));
  const long long ct = (ncol + PC - 1) / PC, tiles = ct * nb;
  constexpr uint32_t mg = rt_magic(PC);
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long p0 = (tile % ct) * PC;
    const int pc = (int)min((long long)PC, ncol - p0);
    double2 *w = spec + (tile / ct) * bstride + p0;
    __syncthreads();  // the tables; the last tile's buf is free
    for (int k = 0; k < py.n; ++k) {
      const bool first = k == 0, last = k == py.n - 1;
      auto ld = [&](int p, int y) {
        if (!first) return buf[y * PC + p];
        if (p >= pc) return make_double2(0.0, 0.0);
        if (DIR < 0) return cmul(w[y * stride + p], t.pw[y]);
        return w[t.idx(y) * stride + p];
      };
      auto st = [&](int p, int y, double2 a) {
        if (!last)
          buf[y * PC + p] = a;
        else if (p < pc)
          w[(DIR < 0 ? t.idx(y) : y) * stride + p] = DIR < 0 ? a : cmul(a, cconj(t.pw[y]));
      };
      rt_pass_s<0, DIR, kThreads, 13>(py, DIR < 0 ? k : py.n - 1 - k, PC, mg, t.tw, ld, st);
      if (!last) __syncthreads();
    }
  }
}

int slab_fail(int code, const std::string &m) {
  set_last_error("r3d_slab_transform: " + m);
  return code;
}

// one wave of CTAs over `tiles`
template <typename K>
int slab_grid(K k, size_t smem, long long tiles) {
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 221 * 1024);
  int nb = 0, dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kThreads, smem);
  return (int)std::min<long long>(tiles, (long long)nsm * std::max(nb, 1));
}
template <int DIR>
void slab_x(const SlabPlan &px, int ny, int nz, int n, double *real, double2 *spec, cudaStream_t s) {
  const int hx = px.L;
  const long long rows = (long long)n * ny * nz;
  int pr = 32;
  while (pr > 1 && slab_tab_bytes(hx) + (size_t)pr * (hx | 1) * 16 > 100 * 1024) pr /= 2;
  const size_t sm = slab_tab_bytes(hx) + (size_t)pr * (hx | 1) * 16;
  const int grid = slab_grid(k_slab_x<DIR>, sm, (rows + pr - 1) / pr);
  k_slab_x<DIR><<<grid, kThreads, sm, s>>>(px, ny, nz, rows, pr, real, spec);
}
template <int DIR>
void slab_col(const SlabPlan &py, long long stride, long long ncol, long long nb, long long bstride,
              double2 *spec, cudaStream_t s) {
  auto go = [&](auto kern, int pc) {
    const size_t sm = slab_tab_bytes(py.L) + (size_t)py.L * pc * 16;
    const int grid = slab_grid(kern, sm, ((ncol + pc - 1) / pc) * nb);
    kern<<<grid, kThreads, sm, s>>>(py, stride, ncol, nb, bstride, spec);
  };
  // 128-byte rows of columns, fewer where a long column would not fit
  if (slab_tab_bytes(py.L) + (size_t)py.L * 8 * 16 <= 100 * 1024)
    go(k_slab_col<DIR, 8>, 8);
  else if (slab_tab_bytes(py.L) + (size_t)py.L * 2 * 16 <= 221 * 1024)
    go(k_slab_col<DIR, 2>, 2);
  else
    go(k_slab_col<DIR, 1>, 1);
}
}  // namespace
}  // namespace r3d

using namespace r3d;

extern "C" int r3d_slab_transform_sites(int device, int stage, int nsites, int nx, int ny,
                                        int nz, double *d_spec, double *d_real, void *stream) {
  if (stage < 0 || stage > 3 || !d_spec || ((stage == 0 || stage == 3) && !d_real) ||
      nsites < 1 || nsites > kMaxSites)
    return slab_fail(R3D_EINVAL, "bad arguments");
  if (nx < 4 || (nx & 1) || ny < 1 || nz < 1 || device < 0 || device >= 64)
    return slab_fail(R3D_EINVAL, "nx must be even and >= 4, ny and nz >= 1");
  const int hx = nx / 2;
  int8_t rad[kMaxRadices];
  if (factor_length(hx, rad) < 0 || factor_length(ny, rad) < 0 || factor_length(nz, rad) < 0)
    return slab_fail(R3D_EINVAL, "grid sizes must factor into primes <= 13");
  // the sizes the call takes: those whose tiles of every site (rows, z
  // columns) or of one site (y columns) fit one CTA's shared memory
  const size_t cs = sizeof(double2), budget = 100 * 1024;
  int S = 16;
  while (S > 1 && (((long long)ny * nz) % S || smem_x(hx, nsites, S, cs) > budget)) S >>= 1;
  int Py = 8;
  while (Py > 1 && (hx % Py || smem_y(ny, Py, cs) > budget)) Py >>= 1;
  int Pz = 4;
  while (Pz > 1 && (hx % Pz || smem_z(nz, nsites, Pz, cs) > budget)) Pz >>= 1;
  const size_t limit = 220 * 1024;
  if (smem_x(hx, nsites, S, cs) > limit || smem_y(ny, Py, cs) > limit ||
      smem_z(nz, nsites, Pz, cs) > limit)
    return slab_fail(R3D_EINVAL, "slab too large for one CTA's shared memory");
  const SlabPlan px = slab_plan(hx), py = slab_plan(ny), pz = slab_plan(nz);
  if ((hx > 1 && !px.n) || (ny > 1 && !py.n) || (nz > 1 && !pz.n))
    return slab_fail(R3D_EINVAL, "a grid size has too many factors");

  int caller = -1;
  cudaError_t e = cudaGetDevice(&caller);
  if (e != cudaSuccess) return slab_fail(R3D_ECUDA, cudaGetErrorString(e));
  struct Restore {
    int dev;
    ~Restore() { cudaSetDevice(dev); }
  } restore{caller};
  if ((e = cudaSetDevice(device)) != cudaSuccess) return slab_fail(R3D_ECUDA, cudaGetErrorString(e));
  cudaStream_t s = (cudaStream_t)stream;
  double2 *w = (double2 *)d_spec;
  const long long plane = (long long)ny * hx;
  // (a transform of length 1 is the identity)
  switch (stage) {
    case 0:
      slab_x<-1>(px, ny, nz, nsites, d_real, w, s);
      if (ny > 1) slab_col<-1>(py, hx, hx, (long long)nsites * nz, plane, w, s);
      break;
    case 1:
      if (nz > 1) slab_col<-1>(pz, plane, plane, nsites, plane * nz, w, s);
      break;
    case 2:
      if (nz > 1) slab_col<1>(pz, plane, plane, nsites, plane * nz, w, s);
      break;
    default:
      if (ny > 1) slab_col<1>(py, hx, hx, (long long)nsites * nz, plane, w, s);
      slab_x<1>(px, ny, nz, nsites, d_real, w, s);
      break;
  }
  if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return slab_fail(R3D_ECUDA, cudaGetErrorString(e));
  return R3D_OK;
}

extern "C" int r3d_slab_transform(int device, int stage, int nx, int ny, int nz, double *d_spec,
                                  double *d_real, void *stream) {
  return r3d_slab_transform_sites(device, stage, 1, nx, ny, nz, d_spec, d_real, stream);
}
