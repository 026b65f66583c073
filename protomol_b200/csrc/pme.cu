// Ewald Coulomb delivered as smooth PME (Essmann et al., J. Chem. Phys.
// 103, 8577 (1995)) plus the two O(exclusions) / O(1) terms of ProtoMol's
// NonbondedFullEwaldSystemForce:
//   * spread: cardinal B-spline (order p) charge spreading into an int64
//     fixed-point grid (order independent, bit reproducible);
//   * 3-D real-to-complex FFT, convolution with the influence function
//     exp(-pi^2 m^2/alpha^2)/(pi V m^2) |b(m)|^2 with the energy and virial
//     reduced on the way, complex-to-real FFT: three kernels (fft.cuh), or
//     cuFFT and two kernels for grids those do not take;
//   * gather: forces from the B-spline derivatives;
//   * correctionTerm (NonbondedFullEwaldSystemForce.h:1092-1131) in FP64.
// The reciprocal energy matches the reference's convention
// E = (4 pi / V) sum_{half space k} exp(-k^2/4a^2)/k^2 |S(k)|^2 (:1013-1054).
#include <algorithm>
#include <cmath>
#include <vector>

#include "pm_device.cuh"

namespace pmgpu {

constexpr int kMaxOrder = 8;
constexpr double kGridScale = 4294967296.0;  // 2^32 per (scaled) charge

struct PmeArgs {
  Box box;
  int n;
  int K[3];
  int order;
  double inv_L[3];
  const double *pos, *charge;
  long long *grid_fixed;  // spread target (int64 fixed point)
  const float *phi;       // potential grid the gather reads
  long long *force;
};

// B-spline weights M_p(fr + k), k = 0..p-1, and their derivatives with
// respect to u, by the Cox-de Boor recursion of the cardinal B-spline
// (fully unrolled for a compile-time order, so the weights stay in
// registers).
template <int P>
__device__ __forceinline__ void bspline(float fr, float *th, float *dth) {
  float m[P];
  m[0] = fr;
  m[1] = 1.f - fr;
#pragma unroll
  for (int k = 2; k < P; k++) m[k] = 0.f;
#pragma unroll
  for (int n = 3; n <= P; n++) {
    if (n == P) {
      // derivative of M_p from M_{p-1}
      dth[0] = m[0];
#pragma unroll
      for (int k = 1; k < P; k++) dth[k] = m[k] - m[k - 1];
    }
    // 1 / (n - 1) as an FP32 pair: the rounding of 1/3 alone would scale every
    // charge on the grid by 3e-8 per axis and the energy by 1.8e-7
    const float div = 1.f / (float)(n - 1);
    const float div_lo = (float)(1.0 / (double)(n - 1) - (double)div);
    float prev = 0.f;
#pragma unroll
    for (int k = 0; k < n; k++) {
      float cur = k < n - 1 ? m[k] : 0.f;
      float x = fr + (float)k;
      const float v = x * cur + ((float)n - x) * prev;
      m[k] = div_lo != 0.f ? fmaf(v, div, v * div_lo) : div * v;
      prev = cur;
    }
  }
  if (P == 2) {
    dth[0] = 1.f;
    dth[1] = -1.f;
  }
#pragma unroll
  for (int k = 0; k < P; k++) th[k] = m[k];
}

// Grid coordinate of one atom along one axis: u = K * (frac), with frac
// taken from the minimal-image position so it lies in [0, 1].
__device__ __forceinline__ void grid_coord(const PmeArgs &a, int axis, double w,
                                           int &iu, float &fr) {
  double f = (w - a.box.min[axis] + a.box.origin[axis]) * a.inv_L[axis];
  f -= floor(f);
  double u = f * a.K[axis];
  double fl = floor(u);
  iu = (int)fl;
  fr = (float)(u - fl);
  if (iu >= a.K[axis]) iu -= a.K[axis];
}

// Spread: L lanes per atom (L = order rounded up to a power of two); lane
// kx < P adds the P^2 points of its x plane.
template <int P, int L>
__device__ __forceinline__ void spread_body(const PmeArgs &a, Blk b) {
  const double *__restrict__ pos = a.pos;
  const double *__restrict__ charge = a.charge;
  long long *__restrict__ grid = a.grid_fixed;
  const int gt = b.x * blockDim.x + threadIdx.x;
  const int t = gt / L, kx = gt & (L - 1);
  if (t >= a.n || kx >= P) return;
  const int i = t;
  double wx, wy, wz;
  box_minpos(a.box, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], wx, wy, wz);
  int iu[3];
  float fr[3];
  grid_coord(a, 0, wx, iu[0], fr[0]);
  grid_coord(a, 1, wy, iu[1], fr[1]);
  grid_coord(a, 2, wz, iu[2], fr[2]);
  float thx[P], thy[P], thz[P], d[P];
  bspline<P>(fr[0], thx, d);
  bspline<P>(fr[1], thy, d);
  bspline<P>(fr[2], thz, d);
  // this lane's x weight without a dynamically indexed array
  float tx = thx[0];
#pragma unroll
  for (int k = 1; k < P; k++)
    if (kx == k) tx = thx[k];
  int gx = iu[0] - kx;
  if (gx < 0) gx += a.K[0];
  const double qx = charge[i] * (double)tx;
#pragma unroll
  for (int ky = 0; ky < P; ky++) {
    int gy = iu[1] - ky;
    if (gy < 0) gy += a.K[1];
    const double qxy = qx * (double)thy[ky];
    long long *row = grid + ((size_t)gx * a.K[1] + gy) * a.K[2];
#pragma unroll
    for (int kz = 0; kz < P; kz++) {
      int gz = iu[2] - kz;
      if (gz < 0) gz += a.K[2];
      red_add(&row[gz], to_fixed(qxy * (double)thz[kz], kGridScale));
    }
  }
}

template <int P, int L>
__global__ void __launch_bounds__(128) k_pme_spread(PmeArgs a) {
  spread_body<P, L>(a, own_blk());
}
template <int P, int L>
__global__ void __launch_bounds__(128)
k_pme_spread_batch(const PmeArgs *__restrict__ tab, const int *__restrict__ first, int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  spread_body<P, L>(tab[m], batch_blk(first, m));
}

// Converts the fixed-point charge grid to FP32 and clears it for the next
// spread (the grid is zero at allocation and after every conversion, so no
// separate clearing pass is needed).
struct GridConvArgs {
  int total;
  long long *g;
  float *out;
};
__device__ __forceinline__ void fixed_to_float_body(const GridConvArgs &a, Blk b) {
  int i = b.x * blockDim.x + threadIdx.x;
  if (i < a.total) {
    a.out[i] = (float)((double)a.g[i] * (1.0 / kGridScale));
    a.g[i] = 0;
  }
}
__global__ void k_pme_fixed_to_float(GridConvArgs a) { fixed_to_float_body(a, own_blk()); }
__global__ void k_pme_fixed_to_float_batch(const GridConvArgs *__restrict__ tab,
                                           const int *__restrict__ first, int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  fixed_to_float_body(tab[m], batch_blk(first, m));
}

// Multiply by the influence function (precomputed for the box:
// exp(-pi^2 m^2/alpha^2)/(pi V m^2) |b(m)|^2, zero at m = 0); with em >= 1
// reduce the energy, with em == 2 also the virial.
// m index convention: m in [0, K/2] -> m, (K/2, K) -> m - K.
struct ConvolveArgs {
  int K0, K1, K2;
  double L0, L1, L2, alpha;
  const float *infl;
  float2 *c;
  long long *acc;
  int em;
};
// Mode idx's share of the reciprocal energy (em >= 1) and virial (em 2): g
// its influence, f its amplitude before the convolution.
__device__ __forceinline__ void mode_energy(const ConvolveArgs &A, int idx, float g, float2 f,
                                            double &e, double (&v)[6]) {
  const int Kh = A.K2 / 2 + 1;
  const int mz = idx % Kh;
  const double w = (mz == 0 || (A.K2 % 2 == 0 && mz == A.K2 / 2)) ? 1.0 : 2.0;
  const double f2 = (double)f.x * f.x + (double)f.y * f.y;
  const double emode = 0.5 * w * (double)g * f2;
  e += emode;
  if (A.em == 2 && g != 0.f) {
    const int my_ = (idx / Kh) % A.K1, mx_ = idx / (Kh * A.K1);
    const int mx = mx_ <= A.K0 / 2 ? mx_ : mx_ - A.K0;
    const int my = my_ <= A.K1 / 2 ? my_ : my_ - A.K1;
    const double hx = mx / A.L0, hy = my / A.L1, hz = mz / A.L2;
    const double h2 = hx * hx + hy * hy + hz * hz;
    const double pa = M_PI * M_PI / (A.alpha * A.alpha);
    const double cc = 2.0 * (1.0 / h2 + pa);
    v[0] += emode * (1.0 - cc * hx * hx);
    v[1] -= emode * cc * hx * hy;
    v[2] -= emode * cc * hx * hz;
    v[3] += emode * (1.0 - cc * hy * hy);
    v[4] -= emode * cc * hy * hz;
    v[5] += emode * (1.0 - cc * hz * hz);
  }
}
__device__ __forceinline__ void mode_reduce(const ConvolveArgs &A, double e, double (&v)[6]) {
  if (!A.em) return;
  e = warp_sum(e);
  if (A.em == 2)
    for (int q = 0; q < 6; q++) v[q] = warp_sum(v[q]);
  if ((threadIdx.x & 31) == 0) {
    red_add(&A.acc[ACC_COULOMB], to_fixed(e, kEnergyScale));
    if (A.em == 2) {
      const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
      for (int q = 0; q < 9; q++)
        red_add(&A.acc[ACC_VIRIAL + q], to_fixed(v[map[q]], kEnergyScale));
    }
  }
}
__device__ __forceinline__ void convolve_body(const ConvolveArgs &A, Blk b) {
  const int total = A.K0 * A.K1 * (A.K2 / 2 + 1);
  const int idx = b.x * blockDim.x + threadIdx.x;
  double e = 0, v[6] = {0, 0, 0, 0, 0, 0};
  if (idx < total) {
    const float g = A.infl[idx];
    const float2 f = A.c[idx];
    A.c[idx] = make_float2(g * f.x, g * f.y);
    if (A.em) mode_energy(A, idx, g, f, e, v);
  }
  mode_reduce(A, e, v);
}
__global__ void k_pme_convolve(ConvolveArgs a) { convolve_body(a, own_blk()); }
__global__ void k_pme_convolve_batch(const ConvolveArgs *__restrict__ tab,
                                     const int *__restrict__ first, int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  convolve_body(tab[m], batch_blk(first, m));
}

// ---------------------------------------------------------- own FFT
// The transforms and the convolution of a grid (fft.cuh).  Ten dependent
// launches of spread, conversion, six cuFFT kernels, convolution and gather
// become five, and an ensemble's launches no longer grow with the number of
// its grid sizes: a launch's plane or column blocks come from every member.
// Bound by latency (trips to memory, then five to seven short synchronised
// passes): at 64^3 the three kernels take 8.0, 7.3 and 7.3 us against 28 us
// for the eight they replace, at 40^3 6.8, 5.9 and 6.2 against 23 us (caches
// warm); with the first version of them a 5,001-atom MD step 52.7 against 55.2 us, 24 boxes of nine grid
// sizes 259 against 338 us a step.  Launching the chain as programmatic
// dependents was slower (5,776 against 5,048 us for 50 steps of 23,550
// atoms: waiting blocks hold room the pair kernel needs).
struct FftArgs {
  FftGrid g;
  long long *fixed;  // fixed-point charges (read and cleared)
  float *grid;       // potential
  ConvolveArgs cv;   // c: the half-complex grid between the kernels
};
constexpr int kFftXThreads = 128;  // also fixes the energy's partial sums

extern __shared__ float2 fft_smem[];

// Elements 0..n-1 dealt to the block's threads, load(k) of kFftLoads of them
// in flight before the first store(k, value): one trip to memory per
// kFftLoads elements of a thread instead of one per element.
constexpr int kFftLoads = 8;
template <typename T, typename L, typename S>
__device__ __forceinline__ void fft_stream(int n, L load, S store) {
  for (int k0 = threadIdx.x; k0 < n; k0 += kFftLoads * blockDim.x) {
    T v[kFftLoads];
#pragma unroll
    for (int u = 0; u < kFftLoads; u++) {
      const int k = k0 + u * blockDim.x;
      if (k < n) v[u] = load(k);
    }
#pragma unroll
    for (int u = 0; u < kFftLoads; u++) {
      const int k = k0 + u * blockDim.x;
      if (k < n) store(k, v[u]);
    }
  }
}

// The block's n twiddles into dst.  A thread's first one is loaded before
// the data (fft_first) and stored after it, so the block waits for memory
// once, not twice; k_fft_x has the influence function on its way as well.
// Langevin runs of 50 steps by themselves (no copies to or from the host):
// 5,001 atoms 1942 -> 1909 us, 750 1685 -> 1654, 23,550 3614 -> 3598.
__device__ __forceinline__ float2 fft_first(const float2 *tw, int n) {
  return (int)threadIdx.x < n ? __ldg(tw + threadIdx.x) : make_float2(0.f, 0.f);
}
__device__ __forceinline__ void fft_twiddles(float2 *dst, const float2 *tw, int n, float2 first) {
  if ((int)threadIdx.x < n) dst[threadIdx.x] = first;
  for (int k = threadIdx.x + blockDim.x; k < n; k += blockDim.x) dst[k] = __ldg(tw + k);
}

__device__ __forceinline__ void fft_yz_body(const FftArgs &A, Blk b) {
  const FftGrid &g = A.g;
  float2 *sm = fft_smem;
  const int t0 = threadIdx.x, nt = blockDim.x, buf = fft_plane_buf(g);
  const int ty = 2 * buf, tz = ty + g.K1, nz = g.K2, np = g.K1 * g.K2;
  // a plane's charges: element (row, z) is the real part of pair row / 2 for
  // an even row, the imaginary part for an odd one
  long long *plane = A.fixed + (size_t)b.x * np;
  const float iz = 1.0f / (float)nz;
  float *sf = reinterpret_cast<float *>(sm);
  const float2 tw0 = fft_first(g.tw + g.K0, g.K1 + g.K2);
  fft_stream<long long>(np, [&](int k) { return plane[k]; },
                        [&](int k, long long q) {
                          const int row = fft_div(k, iz), z = k - row * nz;
                          // the same rounding as through FP64: scaling by 2^-32 is exact
                          sf[2 * (z * g.ldz + (row >> 1)) + (row & 1)] =
                              __ll2float_rn(q) * (float)(1.0 / kGridScale);
                        });
  fft_twiddles(sm + ty, g.tw + g.K0, g.K1 + g.K2, tw0);
  if (g.K1 & 1)
    for (int z = t0; z < nz; z += nt) sf[2 * (z * g.ldz + g.P - 1) + 1] = 0.f;
  for (int k = t0; k < np; k += nt) plane[k] = 0;  // ready for the next spread
  __syncthreads();
  int r = fft_lines(g.d[2], sm, 0, buf, g.P, g.ldz, tz, t0, nt);
  fft_unpack_rows(g, sm, r, buf - r, t0, nt);
  __syncthreads();
  r = fft_lines(g.d[1], sm, buf - r, r, g.Kh, g.Kh, ty, t0, nt);
  float2 *c = A.cv.c + (size_t)b.x * g.K1 * g.Kh;
  for (int k = t0; k < g.K1 * g.Kh; k += nt) c[k] = sm[r + k];
}

__device__ __forceinline__ void fft_x_body(const FftArgs &A, Blk b) {
  const FftGrid &g = A.g;
  float2 *sm = fft_smem;
  const int t0 = threadIdx.x, nt = blockDim.x, C = g.cols, ncol = g.K1 * g.Kh;
  const int lc = C == 16 ? 4 : 3, c0 = b.x * C, buf = g.K0 * C, tx = 2 * buf;
  const float2 tw0 = fft_first(g.tw, g.K0);
  auto influence = [&](int k) {
    const int col = c0 + (k & (C - 1));
    return k < buf && col < ncol ? __ldg(A.cv.infl + (k >> lc) * ncol + col) : 0.f;
  };
  // the influence function of a thread's first elements, on its way with the
  // data
  float w[kFftLoads];
#pragma unroll
  for (int u = 0; u < kFftLoads; u++) w[u] = influence(t0 + u * nt);
  fft_stream<float2>(buf,
                     [&](int k) {
                       const int col = c0 + (k & (C - 1));
                       return col < ncol ? A.cv.c[(size_t)(k >> lc) * ncol + col]
                                         : make_float2(0.f, 0.f);
                     },
                     [&](int k, float2 v) { sm[k] = v; });
  fft_twiddles(sm + tx, g.tw, g.K0, tw0);
  __syncthreads();
  int r = 0;
#pragma unroll 1
  for (int inverse = 0; inverse < 2; inverse++) {
    r = fft_lines(g.d[0], sm, r, buf - r, C, C, tx, t0, nt);
    if (inverse) break;
    double e = 0, v[6] = {0, 0, 0, 0, 0, 0};
    for (int k0 = t0; k0 < buf; k0 += kFftLoads * nt) {
      if (k0 != t0)
#pragma unroll
        for (int u = 0; u < kFftLoads; u++) w[u] = influence(k0 + u * nt);
#pragma unroll
      for (int u = 0; u < kFftLoads; u++) {
        const int k = k0 + u * nt, col = c0 + (k & (C - 1));
        if (k >= buf) break;
        const float2 f = sm[r + k];
        // swapped: the next transform is the inverse
        sm[r + k] = make_float2(w[u] * f.y, w[u] * f.x);
        if (A.cv.em && col < ncol) mode_energy(A.cv, (k >> lc) * ncol + col, w[u], f, e, v);
      }
    }
    mode_reduce(A.cv, e, v);
    __syncthreads();
  }
  for (int k = t0; k < buf; k += nt) {
    const int col = c0 + (k & (C - 1));
    if (col < ncol) A.cv.c[(size_t)(k >> lc) * ncol + col] = sm[r + k];
  }
}

__device__ __forceinline__ void fft_zy_body(const FftArgs &A, Blk b) {
  const FftGrid &g = A.g;
  float2 *sm = fft_smem;
  const int t0 = threadIdx.x, nt = blockDim.x, buf = fft_plane_buf(g);
  const int ty = 2 * buf, tz = ty + g.K1, nz = g.K2, np = g.K1 * g.K2;
  const float2 *c = A.cv.c + (size_t)b.x * g.K1 * g.Kh;
  const float2 tw0 = fft_first(g.tw + g.K0, g.K1 + g.K2);
  fft_stream<float2>(g.K1 * g.Kh, [&](int k) { return c[k]; },
                     [&](int k, float2 v) { sm[k] = v; });
  fft_twiddles(sm + ty, g.tw + g.K0, g.K1 + g.K2, tw0);
  __syncthreads();
  int r = fft_lines(g.d[1], sm, 0, buf, g.Kh, g.Kh, ty, t0, nt);
  fft_pack_rows(g, sm, r, buf - r, t0, nt);
  __syncthreads();
  r = fft_lines(g.d[2], sm, buf - r, r, g.P, g.ldz, tz, t0, nt);
  // swapped: row 2p in the imaginary part, row 2p + 1 in the real part
  float *plane = A.grid + (size_t)b.x * np;
  const float iz = 1.0f / (float)nz;
  const float *sf = reinterpret_cast<const float *>(sm + r);
  for (int k = t0; k < np; k += nt) {
    const int row = fft_div(k, iz), z = k - row * nz;
    plane[k] = sf[2 * (z * g.ldz + (row >> 1)) + 1 - (row & 1)];
  }
}

__global__ void __launch_bounds__(512) k_fft_yz(FftArgs a) {
  fft_yz_body(a, own_blk());
}
__global__ void __launch_bounds__(kFftXThreads) k_fft_x(FftArgs a) {
  fft_x_body(a, own_blk());
}
__global__ void __launch_bounds__(512) k_fft_zy(FftArgs a) {
  fft_zy_body(a, own_blk());
}
__global__ void __launch_bounds__(512)
k_fft_yz_batch(const FftArgs *__restrict__ tab, const int *__restrict__ first, int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(FftArgs)];
  const int m = batch_member(first, nm, blockIdx.x);
  fft_yz_body(batch_args_shared(tab, m, raw), batch_blk(first, m));
}
__global__ void __launch_bounds__(kFftXThreads)
k_fft_x_batch(const FftArgs *__restrict__ tab, const int *__restrict__ first, int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(FftArgs)];
  const int m = batch_member(first, nm, blockIdx.x);
  fft_x_body(batch_args_shared(tab, m, raw), batch_blk(first, m));
}
__global__ void __launch_bounds__(512)
k_fft_zy_batch(const FftArgs *__restrict__ tab, const int *__restrict__ first, int nm) {
  __shared__ __align__(16) unsigned char raw[sizeof(FftArgs)];
  const int m = batch_member(first, nm, blockIdx.x);
  fft_zy_body(batch_args_shared(tab, m, raw), batch_blk(first, m));
}

// Gather: L lanes per atom, lane kx < P sums its x plane; the partial
// forces are reduced over the lanes with shuffles.
template <int P, int L>
__device__ __forceinline__ void gather_body(const PmeArgs &a, Blk b) {
  const double *__restrict__ pos = a.pos;
  const double *__restrict__ charge = a.charge;
  const float *__restrict__ phi = a.phi;
  long long *__restrict__ force = a.force;
  const int gt = b.x * blockDim.x + threadIdx.x;
  const int t = gt / L, kx = gt & (L - 1);
  const int i = t;
  const bool valid = t < a.n;
  float sx = 0.f, sy = 0.f, sz = 0.f;
  if (valid) {
    double wx, wy, wz;
    box_minpos(a.box, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], wx, wy, wz);
    int iu[3];
    float fr[3];
    grid_coord(a, 0, wx, iu[0], fr[0]);
    grid_coord(a, 1, wy, iu[1], fr[1]);
    grid_coord(a, 2, wz, iu[2], fr[2]);
    float thx[P], dthx[P], thy[P], dthy[P], thz[P], dthz[P];
    bspline<P>(fr[0], thx, dthx);
    bspline<P>(fr[1], thy, dthy);
    bspline<P>(fr[2], thz, dthz);
    if (kx < P) {
      float tx = thx[0], dtx = dthx[0];
#pragma unroll
      for (int k = 1; k < P; k++)
        if (kx == k) {
          tx = thx[k];
          dtx = dthx[k];
        }
      int gx = iu[0] - kx;
      if (gx < 0) gx += a.K[0];
#pragma unroll
      for (int ky = 0; ky < P; ky++) {
        int gy = iu[1] - ky;
        if (gy < 0) gy += a.K[1];
        const float *row = phi + ((size_t)gx * a.K[1] + gy) * a.K[2];
        const float txy = tx * thy[ky];
        const float dxy = dtx * thy[ky];
        const float txdy = tx * dthy[ky];
#pragma unroll
        for (int kz = 0; kz < P; kz++) {
          int gz = iu[2] - kz;
          if (gz < 0) gz += a.K[2];
          const float v = __ldg(&row[gz]);
          sx += dxy * thz[kz] * v;
          sy += txdy * thz[kz] * v;
          sz += txy * dthz[kz] * v;
        }
      }
    }
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
    sz += __shfl_xor_sync(0xffffffffu, sz, o);
  }
  if (valid && kx == 0) {
    const double q = charge[i];
    red_add(&force[i], to_fixed(-q * (double)sx * a.K[0] * a.inv_L[0], kForceScale));
    red_add(&force[a.n + i], to_fixed(-q * (double)sy * a.K[1] * a.inv_L[1], kForceScale));
    red_add(&force[2 * a.n + i], to_fixed(-q * (double)sz * a.K[2] * a.inv_L[2], kForceScale));
  }
}

template <int P, int L>
__global__ void __launch_bounds__(128) k_pme_gather(PmeArgs a) {
  gather_body<P, L>(a, own_blk());
}
template <int P, int L>
__global__ void __launch_bounds__(128)
k_pme_gather_batch(const PmeArgs *__restrict__ tab, const int *__restrict__ first, int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  gather_body<P, L>(tab[m], batch_blk(first, m));
}

// correctionTerm, NonbondedFullEwaldSystemForce.h:1092-1131, FP64.
struct CorrectionArgs {
  Box box;
  int nexcl;
  const int *ex;
  const double *pos, *charge;
  double alpha, csf;
  int n;
  long long *force, *acc;
  int em;
};
__device__ __forceinline__ void correction_body(const CorrectionArgs &A, Blk b) {
  const Box &box = A.box;
  const int nexcl = A.nexcl, n = A.n, em = A.em;
  const double alpha = A.alpha, csf = A.csf;
  const int *__restrict__ ex = A.ex;
  const double *__restrict__ pos = A.pos;
  const double *__restrict__ charge = A.charge;
  long long *__restrict__ force = A.force;
  long long *__restrict__ acc = A.acc;
  int k = b.x * blockDim.x + threadIdx.x;
  double e = 0, v[6] = {0, 0, 0, 0, 0, 0};
  if (k < nexcl) {
    int a1 = ex[3 * k], a2 = ex[3 * k + 1], cl = ex[3 * k + 2];
    double dx, dy, dz;
    double r2 = box_mindiff(box, pos[3 * a1], pos[3 * a1 + 1], pos[3 * a1 + 2],
                            pos[3 * a2], pos[3 * a2 + 1], pos[3 * a2 + 2], dx, dy, dz);
    double qq = charge[a1] * charge[a2];
    if (cl == PMGPU_EXCL_MODIFIED) qq *= 1 - csf;
    double r = sqrt(r2);
    double rr = 1 / r;
    // the reference's erf() here is the C library's (bit-exact against it)
    double ee = erf(alpha * r) * rr;
    e = -qq * ee;
    double a2pi = 2.0 * alpha / sqrt(M_PI);
    double g = qq * (a2pi * exp(-(alpha * alpha) * r2) - ee) * rr * rr;
    double fx = dx * g, fy = dy * g, fz = dz * g;
    red_add(&force[a1], to_fixed(-fx, kForceScale));
    red_add(&force[n + a1], to_fixed(-fy, kForceScale));
    red_add(&force[2 * n + a1], to_fixed(-fz, kForceScale));
    red_add(&force[a2], to_fixed(fx, kForceScale));
    red_add(&force[n + a2], to_fixed(fy, kForceScale));
    red_add(&force[2 * n + a2], to_fixed(fz, kForceScale));
    if (em == 2) {
      v[0] = fx * dx; v[1] = fx * dy; v[2] = fx * dz;
      v[3] = fy * dy; v[4] = fy * dz; v[5] = fz * dz;
    }
  }
  if (!em) return;
  e = warp_sum(e);
  if (em == 2)
    for (int q = 0; q < 6; q++) v[q] = warp_sum(v[q]);
  if ((threadIdx.x & 31) == 0) {
    red_add(&acc[ACC_COULOMB], to_fixed(e, kEnergyScale));
    if (em == 2) {
      const int map[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
      for (int q = 0; q < 9; q++) red_add(&acc[ACC_VIRIAL + q], to_fixed(v[map[q]], kEnergyScale));
    }
  }
}

__global__ void k_ewald_correction(CorrectionArgs a) { correction_body(a, own_blk()); }
__global__ void k_ewald_correction_batch(const CorrectionArgs *__restrict__ tab,
                                         const int *__restrict__ first, int nm) {
  const int m = batch_member(first, nm, blockIdx.x);
  correction_body(tab[m], batch_blk(first, m));
}

// ------------------------------------------------------------ host side
// |b(m)|^2 = 1 / |sum_{k=0}^{p-2} M_p(k+1) exp(2 pi i m k / K)|^2
// (Essmann et al. eq. 4.4), with the usual fix for the zero of the
// denominator at odd orders (average of the neighbours).
static void bspline_moduli(int K, int p, std::vector<float> &out) {
  std::vector<double> M(p + 1, 0.0);
  // M_p at integer points 1..p-1 by the recursion on a unit fractional part
  std::vector<double> m(p, 0.0);
  m[0] = 0.0;  // fr = 0
  m[1] = 1.0;
  for (int n = 3; n <= p; n++) {
    double prev = 0.0;
    for (int k = 0; k < n; k++) {
      double cur = k < n - 1 ? m[k] : 0.0;
      double x = (double)k;
      m[k] = (x * cur + ((double)n - x) * prev) / (double)(n - 1);
      prev = cur;
    }
  }
  // m[k] = M_p(k) for k = 0..p-1
  std::vector<double> mod(K);
  for (int i = 0; i < K; i++) {
    double sr = 0, si = 0;
    for (int k = 0; k < p - 1; k++) {
      double arg = 2.0 * M_PI * i * k / K;
      sr += m[k + 1] * cos(arg);
      si += m[k + 1] * sin(arg);
    }
    mod[i] = sr * sr + si * si;
  }
  for (int i = 0; i < K; i++)
    if (mod[i] < 1e-7) mod[i] = 0.5 * (mod[(i - 1 + K) % K] + mod[(i + 1) % K]);
  out.resize(K);
  for (int i = 0; i < K; i++) out[i] = (float)(1.0 / mod[i]);
}

// Planes above 48 KB need the kernels' dynamic shared memory raised.
static int fft_set_smem() {
  const int most = (int)kFftSmem;
  const void *k[] = {(const void *)k_fft_yz,       (const void *)k_fft_x,
                     (const void *)k_fft_zy,       (const void *)k_fft_yz_batch,
                     (const void *)k_fft_x_batch,  (const void *)k_fft_zy_batch};
  for (const void *q : k)
    PM_CUDA(cudaFuncSetAttribute(q, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  return PMGPU_OK;
}

// Threads of a plane block: eight points of the plane each (one trip to
// memory, about one butterfly a pass).
static int fft_plane_threads(const FftGrid &g) {
  return std::min(512, std::max(128, ((g.K1 * g.K2 / 8 + 31) / 32) * 32));
}
static int fft_x_blocks(const FftGrid &g) { return (g.K1 * g.Kh + g.cols - 1) / g.cols; }

// Whether the three kernels are the faster form of a grid they take.  Not
// where a plane kernel's blocks come in a second wave (more planes than are
// resident at once, one an SM from about 118 x 118 points on), where few
// planes are large, or where a column block's 128 threads have more than 32
// elements each.  Reciprocal term of a small box, cuFFT and the kernels, us:
//   128^3 69 and 67, 144^3 80 and 74, 160^3 113 and 135;
//   144 x 128 x 128 70 and 68, 160 x 128 x 128 78 and 97, 200 x 100 x 100
//   (two planes an SM) 78 and 69;
//   48 x 128 x 128 58 and 58, 32 x 128 x 128 51 and 59, 32 x 108 x 108 51 and
//   52, 32 x 144 x 144 52 and 63;
//   256 x 64 x 64 61 and 53, 512 x 64 x 64 74 and 80; 512 x 16 x 16 51 and 45,
//   1024 x 16 x 16 58 and 67.
constexpr int kFftSms = 148;
constexpr size_t kSmSmem = 228 * 1024;  // shared memory of an SM; a block takes 1 KB more
static bool fft_pays(const FftGrid &g) {
  const int per_sm = std::min((int)(kSmSmem / (fft_plane_smem(g) + 1024)),
                              2048 / fft_plane_threads(g));
  return g.K0 <= kFftSms * per_sm && (g.K0 >= 48 || g.K1 * g.K2 < 128 * 128) &&
         g.K0 * g.cols <= 32 * kFftXThreads;
}

static FftArgs fft_args(const System *s, const Force *f, int em) {
  return FftArgs{f->fft, f->d_grid_fixed, f->d_grid,
                 ConvolveArgs{f->grid[0], f->grid[1], f->grid[2], s->box.e[0], s->box.e[1],
                              s->box.e[2], f->alpha, f->d_influence, f->d_cgrid, s->d_acc, em}};
}

int pme_init(System *s, Force *f) {
  if (!s->box.periodic) return fail(PMGPU_ERR_UNSUPPORTED, "PME needs a periodic box");
  if (f->order < 2 || f->order > kMaxOrder)
    return fail(PMGPU_ERR_ARG, "PME order must be in [2, 8]");
  for (int a = 0; a < 3; a++)
    if (f->grid[a] < f->order || f->grid[a] > 1024)
      return fail(PMGPU_ERR_ARG, "PME grid dimension out of range");
  if (!(f->ewald_flags & PMGPU_EWALD_RECIPROCAL)) return PMGPU_OK;
  int K0 = f->grid[0], K1 = f->grid[1], K2 = f->grid[2];
  size_t nreal = (size_t)K0 * K1 * K2;
  size_t ncplx = (size_t)K0 * K1 * (K2 / 2 + 1);
  PM_CHECK(dev_alloc(s, &f->d_grid, sizeof(float) * nreal));
  PM_CHECK(dev_alloc(s, &f->d_grid_fixed, sizeof(long long) * nreal));
  PM_CUDA(cudaMemsetAsync(f->d_grid_fixed, 0, sizeof(long long) * nreal, s->stream));
  PM_CHECK(dev_alloc(s, &f->d_cgrid, sizeof(float2) * ncplx));
  {
    // influence function of the box (fixed for the life of the system)
    std::vector<float> bm[3];
    for (int a = 0; a < 3; a++) bspline_moduli(f->grid[a], f->order, bm[a]);
    const int Kh = K2 / 2 + 1;
    const double L0 = s->box.e[0], L1 = s->box.e[1], L2 = s->box.e[2], V = s->box.V;
    const double pa = M_PI * M_PI / (f->alpha * f->alpha);
    std::vector<float> g(ncplx);
    for (int mx_ = 0; mx_ < K0; mx_++)
      for (int my_ = 0; my_ < K1; my_++)
        for (int mz = 0; mz < Kh; mz++) {
          const int mx = mx_ <= K0 / 2 ? mx_ : mx_ - K0;
          const int my = my_ <= K1 / 2 ? my_ : my_ - K1;
          const size_t idx = ((size_t)mx_ * K1 + my_) * Kh + mz;
          if (mx == 0 && my == 0 && mz == 0) {
            g[idx] = 0.f;
            continue;
          }
          const double hx = mx / L0, hy = my / L1, hz = mz / L2;
          const double h2 = hx * hx + hy * hy + hz * hz;
          g[idx] = (float)(std::exp(-pa * h2) / (M_PI * V * h2) * (double)bm[0][mx_] *
                           (double)bm[1][my_] * (double)bm[2][mz]);
        }
    PM_CHECK(dev_alloc(s, &f->d_influence, sizeof(float) * ncplx));
    PM_CUDA(cudaMemcpyAsync(f->d_influence, g.data(), sizeof(float) * ncplx,
                            cudaMemcpyHostToDevice, s->stream));
    PM_CUDA(cudaStreamSynchronize(s->stream));
  }
  if (fft_plan(K0, K1, K2, &f->fft) && fft_pays(f->fft)) {
    std::vector<float2> tw;
    for (int a = 0; a < 3; a++)
      for (int m = 0; m < f->grid[a]; m++) {
        const double x = 2.0 * M_PI * m / f->grid[a];
        tw.push_back(make_float2((float)std::cos(x), (float)-std::sin(x)));
      }
    PM_CHECK(dev_alloc(s, &f->d_twiddle, sizeof(float2) * tw.size()));
    PM_CUDA(cudaMemcpyAsync(f->d_twiddle, tw.data(), sizeof(float2) * tw.size(),
                            cudaMemcpyHostToDevice, s->stream));
    PM_CUDA(cudaStreamSynchronize(s->stream));
    f->fft.tw = f->d_twiddle;
    PM_CHECK(fft_set_smem());
    f->own_fft = 1;
    return PMGPU_OK;
  }
  // other grids: cuFFT plans without their own work area: one stream-ordered
  // work area serves both (they run back to back on the system's stream).  A
  // pair left by an ended system of the same grid is taken from the context
  // first.
  size_t ws_r2c = 0, ws_c2r = 0;
  bool reused = false;
  {
    std::lock_guard<std::mutex> lock(s->ctx->fft_mu);
    auto &pool = s->ctx->fft_free;
    for (size_t k = 0; k < pool.size(); k++)
      if (pool[k].dims[0] == K0 && pool[k].dims[1] == K1 && pool[k].dims[2] == K2) {
        f->plan_r2c = pool[k].r2c;
        f->plan_c2r = pool[k].c2r;
        ws_r2c = ws_c2r = pool[k].work;
        pool.erase(pool.begin() + k);
        reused = true;
        break;
      }
  }
  if (!reused &&
      (cufftCreate(&f->plan_r2c) != CUFFT_SUCCESS || cufftCreate(&f->plan_c2r) != CUFFT_SUCCESS ||
       cufftSetAutoAllocation(f->plan_r2c, 0) != CUFFT_SUCCESS ||
       cufftSetAutoAllocation(f->plan_c2r, 0) != CUFFT_SUCCESS ||
       cufftMakePlan3d(f->plan_r2c, K0, K1, K2, CUFFT_R2C, &ws_r2c) != CUFFT_SUCCESS ||
       cufftMakePlan3d(f->plan_c2r, K0, K1, K2, CUFFT_C2R, &ws_c2r) != CUFFT_SUCCESS))
    return fail(PMGPU_ERR_CUDA, "cuFFT plan creation failed");
  f->fft_work_bytes = std::max(ws_r2c, ws_c2r);
  PM_CHECK(dev_alloc(s, &f->d_fft_work, f->fft_work_bytes));
  if (cufftSetWorkArea(f->plan_r2c, f->d_fft_work) != CUFFT_SUCCESS ||
      cufftSetWorkArea(f->plan_c2r, f->d_fft_work) != CUFFT_SUCCESS ||
      cufftSetStream(f->plan_r2c, s->stream) != CUFFT_SUCCESS ||
      cufftSetStream(f->plan_c2r, s->stream) != CUFFT_SUCCESS)
    return fail(PMGPU_ERR_CUDA, "cuFFT work area / stream set-up failed");
  return PMGPU_OK;
}

int pme_free(System *s, Force *f) {
  if (f->plan_r2c && f->plan_c2r && s->ctx) {
    // back to the context for the next system of this grid (its next user
    // sets the work area and the stream again)
    std::lock_guard<std::mutex> lock(s->ctx->fft_mu);
    s->ctx->fft_free.push_back(
        {{f->grid[0], f->grid[1], f->grid[2]}, f->plan_r2c, f->plan_c2r, f->fft_work_bytes});
  } else {
    if (f->plan_r2c) cufftDestroy(f->plan_r2c);
    if (f->plan_c2r) cufftDestroy(f->plan_c2r);
  }
  f->plan_r2c = f->plan_c2r = 0;
  void *ptrs[] = {f->d_grid, f->d_grid_fixed, f->d_cgrid, f->d_influence, f->d_fft_work,
                  f->d_ewtab, f->d_twiddle};
  for (void *p : ptrs) dev_free(s, p);
  f->d_grid = nullptr; f->d_grid_fixed = nullptr; f->d_cgrid = nullptr;
  f->d_influence = nullptr;
  f->d_ewtab = nullptr;
  f->d_twiddle = nullptr;
  f->own_fft = 0;
  f->terms.ewtab = nullptr;
  f->d_fft_work = nullptr;
  return PMGPU_OK;
}

template <int P>
static void launch_spread_gather(const PmeArgs &a, System *s, Force *f,
                                 int gather) {
  constexpr int L = P <= 4 ? 4 : 8;
  const int nb = (int)(((long long)a.n * L + 127) / 128);
  if (!gather)
    k_pme_spread<P, L><<<nb, 128, 0, s->stream>>>(a);
  else
    k_pme_gather<P, L><<<nb, 128, 0, s->stream>>>(a);
}

static void spread_gather(const PmeArgs &a, System *s, Force *f,
                          int gather) {
  switch (f->order) {
    case 2: launch_spread_gather<2>(a, s, f, gather); break;
    case 3: launch_spread_gather<3>(a, s, f, gather); break;
    case 4: launch_spread_gather<4>(a, s, f, gather); break;
    case 5: launch_spread_gather<5>(a, s, f, gather); break;
    case 6: launch_spread_gather<6>(a, s, f, gather); break;
    case 7: launch_spread_gather<7>(a, s, f, gather); break;
    default: launch_spread_gather<8>(a, s, f, gather); break;
  }
}

// em: 0 forces only, 1 + energy, 2 + energy and virial.
int pme_reciprocal(System *s, Force *f, int em, long long *launched) {
  int n = s->n;
  if (n == 0) return PMGPU_OK;
  PmeArgs a;
  a.box = s->box;
  a.n = n;
  for (int d = 0; d < 3; d++) {
    a.K[d] = f->grid[d];
    a.inv_L[d] = 1.0 / s->box.e[d];
  }
  a.order = f->order;
  a.pos = s->d_pos;
  a.charge = s->d_charge;
  a.grid_fixed = f->d_grid_fixed;
  a.phi = f->d_grid;
  a.force = s->d_force;
  int K0 = f->grid[0], K1 = f->grid[1], K2 = f->grid[2];
  // Atoms are spread and gathered in their own order: PME does not wait for
  // the pair list's sort, so it runs beside the list work of a step.
  spread_gather(a, s, f, 0);
  if (f->own_fft) {
    const FftArgs fa = fft_args(s, f, em);
    const int T = fft_plane_threads(fa.g);
    const size_t plane = fft_plane_smem(fa.g);
    k_fft_yz<<<K0, T, plane, s->stream>>>(fa);
    k_fft_x<<<fft_x_blocks(fa.g), kFftXThreads, fft_x_smem(fa.g), s->stream>>>(fa);
    k_fft_zy<<<K0, T, plane, s->stream>>>(fa);
    *launched += 5;
  } else {
    // the plans run on whichever stream this evaluation uses
    if (cufftSetStream(f->plan_r2c, s->stream) != CUFFT_SUCCESS ||
        cufftSetStream(f->plan_c2r, s->stream) != CUFFT_SUCCESS)
      return fail(PMGPU_ERR_CUDA, "cufftSetStream failed");
    const size_t nreal = (size_t)K0 * K1 * K2, ncplx = (size_t)K0 * K1 * (K2 / 2 + 1);
    k_pme_fixed_to_float<<<(int)((nreal + 255) / 256), 256, 0, s->stream>>>(
        GridConvArgs{(int)nreal, f->d_grid_fixed, f->d_grid});
    if (cufftExecR2C(f->plan_r2c, f->d_grid, (cufftComplex *)f->d_cgrid) != CUFFT_SUCCESS)
      return fail(PMGPU_ERR_CUDA, "cufftExecR2C failed");
    k_pme_convolve<<<(int)((ncplx + 255) / 256), 256, 0, s->stream>>>(
        ConvolveArgs{K0, K1, K2, s->box.e[0], s->box.e[1], s->box.e[2], f->alpha,
                     f->d_influence, f->d_cgrid, s->d_acc, em});
    if (cufftExecC2R(f->plan_c2r, (cufftComplex *)f->d_cgrid, f->d_grid) != CUFFT_SUCCESS)
      return fail(PMGPU_ERR_CUDA, "cufftExecC2R failed");
    *launched += 4;  // spread, conversion, convolution, gather (+ cuFFT's)
  }
  spread_gather(a, s, f, 1);
  PM_CUDA(cudaGetLastError());
  return PMGPU_OK;
}

int ewald_correction(System *s, Force *f, int em) {
  if (s->n_excl == 0) return PMGPU_OK;
  k_ewald_correction<<<(s->n_excl + 127) / 128, 128, 0, s->stream>>>(
      CorrectionArgs{s->box, s->n_excl, s->d_excl_pairs, s->d_pos, s->d_charge, f->alpha,
                     s->coulomb_scaling, s->n, s->d_force, s->d_acc, em});
  PM_CUDA(cudaGetLastError());
  return PMGPU_OK;
}

// ---------------------------------------------------------------- batches
// The PME chain and the Ewald correction of an ensemble's members as
// batched launches: the members' own FFTs share one launch per kernel.
// Members whose grids need cuFFT form a bucket per grid size: their real
// and complex grids are slices of one buffer, and one batched cuFFT plan
// pair transforms the bucket at once.
struct PmeBucket {
  int K[3];
  std::vector<int> members;
  cufftHandle r2c = 0, c2r = 0;
  float *grid = nullptr;
  float2 *cgrid = nullptr;
};
struct PmeBatch {
  int order = 4;
  BatchTable<PmeArgs> atoms;  // spread and gather
  BatchTable<FftArgs> yz, fx[2], zy;  // members with the own FFT
  int plane_threads = 128;
  size_t plane_smem = 0, x_smem = 0;
  int sizes = 0;                      // distinct grid dimensions
  BatchTable<GridConvArgs> conv;      // members with cuFFT
  BatchTable<ConvolveArgs> convolve[2];
  BatchTable<CorrectionArgs> corr[2];
  std::vector<PmeBucket> buckets;
  std::vector<System *> sys;
  std::vector<Force *> forces;
};

PmeBatch *pme_batch_new() { return new PmeBatch(); }

// Gives every member its own grids again and frees the buckets.
void pme_batch_free(PmeBatch *b) {
  if (!b) return;
  for (auto &bk : b->buckets) {
    for (int k : bk.members) {
      System *s = b->sys[k];
      Force *f = b->forces[k];
      const size_t nreal = (size_t)f->grid[0] * f->grid[1] * f->grid[2];
      const size_t ncplx = (size_t)f->grid[0] * f->grid[1] * (f->grid[2] / 2 + 1);
      f->d_grid = nullptr;
      f->d_cgrid = nullptr;
      dev_alloc(s, &f->d_grid, sizeof(float) * nreal);
      dev_alloc(s, &f->d_cgrid, sizeof(float2) * ncplx);
      s->graph_version++;  // graphs captured with the bucket's grids
    }
    if (bk.r2c) cufftDestroy(bk.r2c);
    if (bk.c2r) cufftDestroy(bk.c2r);
    if (bk.grid) cudaFree(bk.grid);
    if (bk.cgrid) cudaFree(bk.cgrid);
  }
  b->atoms.release();
  b->conv.release();
  b->yz.release();
  b->zy.release();
  for (int e = 0; e < 2; e++) {
    b->fx[e].release();
    b->convolve[e].release();
    b->corr[e].release();
  }
  delete b;
}

int pme_batch_build(PmeBatch *b, System *const *m, int n, Force *const *fs) {
  b->sys.assign(m, m + n);
  b->forces.assign(fs, fs + n);
  b->order = fs[0]->order;
  // buckets by grid dimensions
  std::vector<const Force *> seen;
  for (int k = 0; k < n; k++) {
    const Force *f = fs[k];
    if (f->order != b->order || !(f->ewald_flags & PMGPU_EWALD_RECIPROCAL))
      return fail(PMGPU_ERR_UNSUPPORTED, "ensemble members need one PME order");
    const bool known = std::any_of(seen.begin(), seen.end(), [f](const Force *o) {
      return o->grid[0] == f->grid[0] && o->grid[1] == f->grid[1] && o->grid[2] == f->grid[2];
    });
    if (!known) seen.push_back(f);
    if (f->own_fft) continue;
    int found = -1;
    for (size_t q = 0; q < b->buckets.size(); q++)
      if (b->buckets[q].K[0] == f->grid[0] && b->buckets[q].K[1] == f->grid[1] &&
          b->buckets[q].K[2] == f->grid[2])
        found = (int)q;
    if (found < 0) {
      b->buckets.push_back(PmeBucket());
      found = (int)b->buckets.size() - 1;
      for (int a = 0; a < 3; a++) b->buckets[found].K[a] = f->grid[a];
    }
    b->buckets[found].members.push_back(k);
  }
  b->sizes = (int)seen.size();
  for (auto &bk : b->buckets) {
    const int B = (int)bk.members.size();
    // slices of an even number of floats: a member's own plan transforms its
    // slice too, and cuFFT refuses a real grid that is not 8-byte aligned
    const size_t G = ((size_t)bk.K[0] * bk.K[1] * bk.K[2] + 1) / 2 * 2;
    const size_t Gc = (size_t)bk.K[0] * bk.K[1] * (bk.K[2] / 2 + 1);
    PM_CUDA(cudaMalloc(&bk.grid, sizeof(float) * G * B));
    PM_CUDA(cudaMalloc(&bk.cgrid, sizeof(float2) * Gc * B));
    // (without the embedding arrays cuFFT takes the slices as packed)
    int dims[3] = {bk.K[0], bk.K[1], bk.K[2]}, half[3] = {bk.K[0], bk.K[1], bk.K[2] / 2 + 1};
    if (cufftPlanMany(&bk.r2c, 3, dims, dims, 1, (int)G, half, 1, (int)Gc, CUFFT_R2C, B) !=
            CUFFT_SUCCESS ||
        cufftPlanMany(&bk.c2r, 3, dims, half, 1, (int)Gc, dims, 1, (int)G, CUFFT_C2R, B) !=
            CUFFT_SUCCESS)
      return fail(PMGPU_ERR_CUDA, "batched cuFFT plan creation failed");
    for (int q = 0; q < B; q++) {
      System *s = m[bk.members[q]];
      Force *f = fs[bk.members[q]];
      PM_CUDA(cudaStreamSynchronize(s->stream));
      dev_free(s, f->d_grid);
      dev_free(s, f->d_cgrid);
      f->d_grid = bk.grid + G * q;
      f->d_cgrid = bk.cgrid + Gc * q;
      s->graph_version++;  // graphs captured with the member's own grids
    }
  }
  // argument tables in member order
  b->atoms.clear();
  b->conv.clear();
  b->yz.clear();
  b->zy.clear();
  for (int e = 0; e < 2; e++) {
    b->fx[e].clear();
    b->convolve[e].clear();
    b->corr[e].clear();
  }
  int L = b->order <= 4 ? 4 : 8;
  for (int k = 0; k < n; k++) {
    System *s = m[k];
    Force *f = fs[k];
    PmeArgs a;
    a.box = s->box;
    a.n = s->n;
    for (int d = 0; d < 3; d++) {
      a.K[d] = f->grid[d];
      a.inv_L[d] = 1.0 / s->box.e[d];
    }
    a.order = f->order;
    a.pos = s->d_pos;
    a.charge = s->d_charge;
    a.grid_fixed = f->d_grid_fixed;
    a.phi = f->d_grid;
    a.force = s->d_force;
    b->atoms.add(a, (int)(((long long)s->n * L + 127) / 128));
    if (f->own_fft) {
      const FftArgs fa = fft_args(s, f, 0);
      b->yz.add(fa, f->grid[0]);
      b->zy.add(fa, f->grid[0]);
      for (int e = 0; e < 2; e++) b->fx[e].add(fft_args(s, f, e), fft_x_blocks(fa.g));
      b->plane_threads = std::max(b->plane_threads, fft_plane_threads(fa.g));
      b->plane_smem = std::max(b->plane_smem, fft_plane_smem(fa.g));
      b->x_smem = std::max(b->x_smem, fft_x_smem(fa.g));
    } else {
      const size_t nreal = (size_t)f->grid[0] * f->grid[1] * f->grid[2];
      const size_t ncplx = (size_t)f->grid[0] * f->grid[1] * (f->grid[2] / 2 + 1);
      b->conv.add(GridConvArgs{(int)nreal, f->d_grid_fixed, f->d_grid},
                  (int)((nreal + 255) / 256));
      for (int e = 0; e < 2; e++)
        b->convolve[e].add(ConvolveArgs{f->grid[0], f->grid[1], f->grid[2], s->box.e[0],
                                        s->box.e[1], s->box.e[2], f->alpha, f->d_influence,
                                        f->d_cgrid, s->d_acc, e},
                           (int)((ncplx + 255) / 256));
    }
    for (int e = 0; e < 2; e++) {
      b->corr[e].add(CorrectionArgs{s->box, s->n_excl, s->d_excl_pairs, s->d_pos, s->d_charge,
                                    f->alpha, s->coulomb_scaling, s->n, s->d_force, s->d_acc, e},
                     (s->n_excl + 127) / 128);
    }
  }
  PM_CUDA(b->atoms.upload());
  PM_CUDA(b->conv.upload());
  PM_CUDA(b->yz.upload());
  PM_CUDA(b->zy.upload());
  for (int e = 0; e < 2; e++) {
    PM_CUDA(b->fx[e].upload());
    PM_CUDA(b->convolve[e].upload());
    PM_CUDA(b->corr[e].upload());
  }
  return PMGPU_OK;
}

template <int P>
static void pme_batch_atoms(PmeBatch *b, int gather, cudaStream_t st) {
  constexpr int L = P <= 4 ? 4 : 8;
  BatchTable<PmeArgs> &t = b->atoms;
  if (!t.total()) return;
  if (!gather)
    k_pme_spread_batch<P, L><<<t.total(), 128, 0, st>>>(t.d, t.d_first, t.members());
  else
    k_pme_gather_batch<P, L><<<t.total(), 128, 0, st>>>(t.d, t.d_first, t.members());
}

static void pme_batch_sg(PmeBatch *b, int gather, cudaStream_t st) {
  switch (b->order) {
    case 2: pme_batch_atoms<2>(b, gather, st); break;
    case 3: pme_batch_atoms<3>(b, gather, st); break;
    case 4: pme_batch_atoms<4>(b, gather, st); break;
    case 5: pme_batch_atoms<5>(b, gather, st); break;
    case 6: pme_batch_atoms<6>(b, gather, st); break;
    case 7: pme_batch_atoms<7>(b, gather, st); break;
    default: pme_batch_atoms<8>(b, gather, st); break;
  }
}

// The reciprocal term of every member (pme_reciprocal of each), em as
// there.
int pme_batch_reciprocal(PmeBatch *b, int em, cudaStream_t st, long long *launched) {
  const int nm = b->atoms.members();
  if (!nm) return PMGPU_OK;
  *launched += 2;  // spread, gather
  pme_batch_sg(b, 0, st);
  if (b->yz.members()) {
    BatchTable<FftArgs> &fx = b->fx[em ? 1 : 0];
    k_fft_yz_batch<<<b->yz.total(), b->plane_threads, b->plane_smem, st>>>(b->yz.d, b->yz.d_first,
                                                                           b->yz.members());
    k_fft_x_batch<<<fx.total(), kFftXThreads, b->x_smem, st>>>(fx.d, fx.d_first, fx.members());
    k_fft_zy_batch<<<b->zy.total(), b->plane_threads, b->plane_smem, st>>>(b->zy.d, b->zy.d_first,
                                                                           b->zy.members());
    *launched += 3;
  }
  if (b->conv.members()) {
    const int nc = b->conv.members();
    k_pme_fixed_to_float_batch<<<b->conv.total(), 256, 0, st>>>(b->conv.d, b->conv.d_first, nc);
    for (auto &bk : b->buckets) {
      if (cufftSetStream(bk.r2c, st) != CUFFT_SUCCESS ||
          cufftExecR2C(bk.r2c, bk.grid, (cufftComplex *)bk.cgrid) != CUFFT_SUCCESS)
        return fail(PMGPU_ERR_CUDA, "batched cufftExecR2C failed");
    }
    BatchTable<ConvolveArgs> &cv = b->convolve[em ? 1 : 0];
    k_pme_convolve_batch<<<cv.total(), 256, 0, st>>>(cv.d, cv.d_first, nc);
    for (auto &bk : b->buckets) {
      if (cufftSetStream(bk.c2r, st) != CUFFT_SUCCESS ||
          cufftExecC2R(bk.c2r, (cufftComplex *)bk.cgrid, bk.grid) != CUFFT_SUCCESS)
        return fail(PMGPU_ERR_CUDA, "batched cufftExecC2R failed");
    }
    *launched += 2;  // conversion, convolution (+ cuFFT's)
  }
  pme_batch_sg(b, 1, st);
  PM_CUDA(cudaGetLastError());
  return PMGPU_OK;
}

int pme_batch_buckets(const PmeBatch *b) { return b->sizes; }

int pme_batch_correction(PmeBatch *b, int em, cudaStream_t st, long long *launched) {
  BatchTable<CorrectionArgs> &t = b->corr[em ? 1 : 0];
  if (!t.members() || !t.total()) return PMGPU_OK;
  *launched += 1;
  k_ewald_correction_batch<<<t.total(), 128, 0, st>>>(t.d, t.d_first, t.members());
  PM_CUDA(cudaGetLastError());
  return PMGPU_OK;
}

}  // namespace pmgpu
