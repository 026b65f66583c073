// The PME grids' own 3-D FFT: real-to-complex, the convolution and
// complex-to-real in three kernels (pme.cu), each of which transforms whole
// lines in shared memory:
//   * k_fft_yz: one x plane per block; reads the fixed-point charge plane
//     (and clears it), transforms z (two real rows as one complex line) and
//     then y, writes the half-complex plane;
//   * k_fft_x: columns of the x direction; transforms x, multiplies by the
//     influence function (reducing the energy on the way) and transforms
//     back;
//   * k_fft_zy: one x plane per block; transforms y and z back, writes the
//     potential plane.
// A line of length N = R1 R2 ... is transformed by one Stockham pass per
// factor (autosort, two shared-memory buffers), each thread holding one
// radix-R butterfly in registers.  Buffers are laid out [element][line], so
// the threads of a warp work on neighbouring lines without bank conflicts.
// The inverse is the forward transform of the real/imaginary-swapped data
// (swap, transform, swap), so only forward butterflies exist.
//
// Sizes: every dimension a product of 2, 3 and 5 whose plane fits the
// shared memory (fft_plan) and where the kernels are the faster form
// (fft_pays, pme.cu); others keep cuFFT (pme.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

namespace pmgpu {

constexpr int kFftMaxStages = 6;
constexpr int kFftMaxRadix = 10;

// One dimension: length and the radices of its passes.
struct FftDim {
  int n, ns;
  int radix[kFftMaxStages];
};

struct FftGrid {
  int K0, K1, K2, Kh;  // Kh = K2 / 2 + 1
  int P;               // pairs of z rows: (K1 + 1) / 2
  int ldz;             // line stride of the z passes (odd, >= P)
  int cols;            // columns a block of k_fft_x takes (power of two)
  FftDim d[3];
  const float2 *tw;    // exp(-2 pi i m / K) of K0, K1 and K2, one after another
};

// Floats2 per shared-memory buffer of the plane kernels and of k_fft_x.
__host__ __device__ inline int fft_plane_buf(const FftGrid &g) {
  const int a = g.K2 * g.ldz, b = g.K1 * g.Kh;
  return a > b ? a : b;
}
__host__ __device__ inline size_t fft_plane_smem(const FftGrid &g) {
  return sizeof(float2) * (2 * (size_t)fft_plane_buf(g) + g.K1 + g.K2);
}
__host__ __device__ inline size_t fft_x_smem(const FftGrid &g) {
  return sizeof(float2) * (2 * (size_t)g.K0 * g.cols + g.K0);
}

// Fewest passes over n with radices up to kFftMaxRadix (no 7), the largest
// radix as small as possible among those; false when n has another prime.
inline bool fft_radices(int n, FftDim *d) {
  static const int R[] = {10, 9, 8, 6, 5, 4, 3, 2};
  FftDim best{n, 0, {0}}, cur{n, 0, {0}};
  int best_max = 99;
  struct Rec {
    static void go(int left, int from, FftDim &cur, FftDim &best, int &best_max) {
      if (left == 1) {
        int m = 0;
        for (int k = 0; k < cur.ns; k++) m = std::max(m, cur.radix[k]);
        if (best.ns == 0 || cur.ns < best.ns || (cur.ns == best.ns && m < best_max)) {
          best = cur;
          best_max = m;
        }
        return;
      }
      if (cur.ns == kFftMaxStages) return;
      for (int q = from; q < 8; q++)
        if (left % R[q] == 0) {
          cur.radix[cur.ns++] = R[q];
          go(left / R[q], q, cur, best, best_max);
          cur.ns--;
        }
    }
  };
  if (n > 1) Rec::go(n, 0, cur, best, best_max);
  *d = best;
  return best.ns > 0;
}

// Plans a grid; false when the kernels do not take its dimensions.
// A block has up to 227 KB of shared memory: planes up to 162 x 162 fit.
constexpr size_t kFftSmem = 216 * 1024;
inline bool fft_plan(int K0, int K1, int K2, FftGrid *g) {
  g->K0 = K0; g->K1 = K1; g->K2 = K2;
  g->Kh = K2 / 2 + 1;
  g->P = (K1 + 1) / 2;
  g->ldz = g->P | 1;
  // enough blocks for the SMs before wider reads: a 16-column block reads
  // 128-byte segments, an 8-column one 64-byte segments
  g->cols = K1 * g->Kh >= 16 * 120 ? 16 : 8;
  const int K[3] = {K0, K1, K2};
  for (int a = 0; a < 3; a++)
    if (!fft_radices(K[a], &g->d[a])) return false;
  g->tw = nullptr;
  return fft_plane_smem(*g) <= kFftSmem && fft_x_smem(*g) <= kFftSmem;
}

// a / b for 0 <= a < 2^20 from inv = 1.0f / b.
__device__ __forceinline__ int fft_div(int a, float inv) {
  return (int)(((float)a + 0.5f) * inv);
}

__device__ __forceinline__ float2 c_add(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ float2 c_mul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a - i b and a + i b
__device__ __forceinline__ float2 c_sub_i(float2 a, float2 b) {
  return make_float2(a.x + b.y, a.y - b.x);
}
__device__ __forceinline__ float2 c_add_i(float2 a, float2 b) {
  return make_float2(a.x - b.y, a.y + b.x);
}

// exp(-2 pi i m / R) of the composite butterflies (folded: m is a constant
// after unrolling).
template <int R>
__device__ __forceinline__ float2 fft_root(int m) {
  if (R == 6) {
    constexpr float c[6] = {1.f, 0.5f, -0.5f, -1.f, -0.5f, 0.5f};
    constexpr float s[6] = {0.f, -0.86602540378443865f, -0.86602540378443865f, 0.f,
                            0.86602540378443865f, 0.86602540378443865f};
    return make_float2(c[m], s[m]);
  }
  if (R == 8) {
    constexpr float h = 0.70710678118654752f;
    constexpr float c[8] = {1.f, h, 0.f, -h, -1.f, -h, 0.f, h};
    constexpr float s[8] = {0.f, -h, -1.f, -h, 0.f, h, 1.f, h};
    return make_float2(c[m], s[m]);
  }
  if (R == 9) {
    constexpr float c[5] = {1.f, 0.76604444311897804f, 0.17364817766693035f, -0.5f,
                            -0.93969262078590838f};
    constexpr float s[5] = {0.f, -0.64278760968653933f, -0.98480775301220806f,
                            -0.86602540378443865f, -0.34202014332566873f};
    return make_float2(c[m], s[m]);  // m <= 4: products of the 3 x 3 split
  }
  constexpr float c[5] = {1.f, 0.80901699437494742f, 0.30901699437494742f,
                          -0.30901699437494742f, -0.80901699437494742f};
  constexpr float s[5] = {0.f, -0.58778525229247313f, -0.95105651629515357f,
                          -0.95105651629515357f, -0.58778525229247313f};
  return make_float2(c[m], s[m]);  // R == 10, m <= 4: products of the 5 x 2 split
}

// Forward DFT of R values in registers (exp(-2 pi i k n / R)).
template <int R>
struct Dft;
template <>
struct Dft<2> {
  static __device__ __forceinline__ void go(float2 (&v)[2]) {
    const float2 a = v[0];
    v[0] = c_add(a, v[1]);
    v[1] = c_sub(a, v[1]);
  }
};
template <>
struct Dft<3> {
  static __device__ __forceinline__ void go(float2 (&v)[3]) {
    const float2 t = c_add(v[1], v[2]), e = c_sub(v[1], v[2]);
    const float2 u = make_float2(v[0].x - 0.5f * t.x, v[0].y - 0.5f * t.y);
    const float2 d = make_float2(0.86602540378443865f * e.x, 0.86602540378443865f * e.y);
    v[0] = c_add(v[0], t);
    v[1] = c_sub_i(u, d);
    v[2] = c_add_i(u, d);
  }
};
template <>
struct Dft<4> {
  static __device__ __forceinline__ void go(float2 (&v)[4]) {
    const float2 s0 = c_add(v[0], v[2]), d0 = c_sub(v[0], v[2]);
    const float2 s1 = c_add(v[1], v[3]), d1 = c_sub(v[1], v[3]);
    v[0] = c_add(s0, s1);
    v[1] = c_sub_i(d0, d1);
    v[2] = c_sub(s0, s1);
    v[3] = c_add_i(d0, d1);
  }
};
template <>
struct Dft<5> {
  static __device__ __forceinline__ void go(float2 (&v)[5]) {
    constexpr float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;
    constexpr float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;
    const float2 a = c_add(v[1], v[4]), b = c_add(v[2], v[3]);
    const float2 d = c_sub(v[1], v[4]), e = c_sub(v[2], v[3]);
    const float2 p = make_float2(v[0].x + c1 * a.x + c2 * b.x, v[0].y + c1 * a.y + c2 * b.y);
    const float2 q = make_float2(v[0].x + c2 * a.x + c1 * b.x, v[0].y + c2 * a.y + c1 * b.y);
    const float2 f = make_float2(s1 * d.x + s2 * e.x, s1 * d.y + s2 * e.y);
    const float2 g = make_float2(s2 * d.x - s1 * e.x, s2 * d.y - s1 * e.y);
    v[0] = c_add(v[0], c_add(a, b));
    v[1] = c_sub_i(p, f);
    v[4] = c_add_i(p, f);
    v[2] = c_sub_i(q, g);
    v[3] = c_add_i(q, g);
  }
};
// R = R1 R2: R2 transforms of length R1, twiddles, R1 transforms of length
// R2; output k1 + R1 k2.
template <int R1, int R2>
struct DftSplit {
  static __device__ __forceinline__ void go(float2 (&v)[R1 * R2]) {
    constexpr int R = R1 * R2;
    float2 t[R2][R1];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) t[n2][n1] = v[R2 * n1 + n2];
      Dft<R1>::go(t[n2]);
#pragma unroll
      for (int k1 = 1; k1 < R1; k1++)
        if (n2) t[n2][k1] = c_mul(t[n2][k1], fft_root<R>(n2 * k1));
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
      float2 u[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) u[n2] = t[n2][k1];
      Dft<R2>::go(u);
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) v[k1 + R1 * k2] = u[k2];
    }
  }
};
template <>
struct Dft<6> : DftSplit<3, 2> {};
template <>
struct Dft<8> : DftSplit<4, 2> {};
template <>
struct Dft<9> : DftSplit<3, 3> {};
template <>
struct Dft<10> : DftSplit<5, 2> {};

// One pass of radix R over `lines` lines of length N (element k of line l
// at k * ld + l): Ns is the product of the radices already done.  Thread t0
// of nt takes every nt-th butterfly.
// Buffers and twiddles are given as offsets into the block's memory sm, so
// every access compiles to a shared-memory one.
template <int R>
__device__ __forceinline__ void fft_pass(float2 *sm, int from, int to, int N, int Ns,
                                                  int lines, int ld, int tw, int t0, int nt) {
  const int nb = N / R, items = nb * lines, step = nb / Ns;
  const float il = 1.0f / (float)lines, is = 1.0f / (float)Ns;
  for (int it = t0; it < items; it += nt) {
    const int j = fft_div(it, il), l = it - j * lines;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = sm[from + (j + r * nb) * ld + l];
    int q = j, k = 0;
    if (Ns > 1) {
      q = fft_div(j, is);
      k = j - q * Ns;
      const int m = k * step;  // r m < N
#pragma unroll
      for (int r = 1; r < R; r++) v[r] = c_mul(v[r], sm[tw + r * m]);
    }
    Dft<R>::go(v);
    const int o = to + (q * Ns * R + k) * ld + l;
#pragma unroll
    for (int r = 0; r < R; r++) sm[o + r * Ns * ld] = v[r];
  }
}

__device__ __forceinline__ void fft_pass_r(int R, float2 *sm, int from, int to, int N,
                                                    int Ns, int lines, int ld, int tw, int t0,
                                                    int nt) {
  switch (R) {
    case 2: fft_pass<2>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 3: fft_pass<3>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 4: fft_pass<4>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 5: fft_pass<5>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 6: fft_pass<6>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 8: fft_pass<8>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    case 9: fft_pass<9>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
    default: fft_pass<10>(sm, from, to, N, Ns, lines, ld, tw, t0, nt); break;
  }
}

// All passes of one dimension; buffer a holds the data, b is the other
// one.  Returns the buffer of the result (every pass ends synchronised).
__device__ __forceinline__ int fft_lines(const FftDim &d, float2 *sm, int a, int b,
                                                  int lines, int ld, int tw, int t0, int nt) {
  int Ns = 1;
  for (int s = 0; s < d.ns; s++) {
    fft_pass_r(d.radix[s], sm, a, b, d.n, Ns, lines, ld, tw, t0, nt);
    __syncthreads();
    Ns *= d.radix[s];
    const int t = a;
    a = b;
    b = t;
  }
  return a;
}

// z rows 2p and 2p + 1 (transformed as one complex line) into their half
// spectra, [y][kz].
__device__ __forceinline__ void fft_unpack_rows(const FftGrid &g, float2 *sm, int z, int c,
                                                         int t0, int nt) {
  const int items = g.P * g.Kh;
  const float ik = 1.0f / (float)g.Kh;
  for (int it = t0; it < items; it += nt) {
    const int p = fft_div(it, ik), k = it - p * g.Kh;
    const float2 u = sm[z + k * g.ldz + p], w = sm[z + (k ? g.K2 - k : 0) * g.ldz + p];
    sm[c + 2 * p * g.Kh + k] = make_float2(0.5f * (u.x + w.x), 0.5f * (u.y - w.y));
    if (2 * p + 1 < g.K1)
      sm[c + (2 * p + 1) * g.Kh + k] = make_float2(0.5f * (u.y + w.y), 0.5f * (w.x - u.x));
  }
}

// The inverse of fft_unpack_rows on swapped data: half spectra [y][kz]
// (real and imaginary parts swapped) into swapped complex lines.  The
// self-conjugate modes (kz = 0 and the Nyquist mode) are real in a real
// row's spectrum; their imaginary rounding is dropped.
__device__ __forceinline__ void fft_pack_rows(const FftGrid &g, float2 *sm, int c, int z,
                                                       int t0, int nt) {
  const int items = g.P * g.Kh;
  const float ik = 1.0f / (float)g.Kh;
  for (int it = t0; it < items; it += nt) {
    const int p = fft_div(it, ik), k = it - p * g.Kh;
    const float2 sa = sm[c + 2 * p * g.Kh + k];
    const float2 sb = 2 * p + 1 < g.K1 ? sm[c + (2 * p + 1) * g.Kh + k] : make_float2(0.f, 0.f);
    float2 a = make_float2(sa.y, sa.x), b = make_float2(sb.y, sb.x);
    const bool self = k == 0 || 2 * k == g.K2;
    if (self) a.y = b.y = 0.f;
    // a + i b, swapped; its conjugate partner conj(a) + i conj(b)
    sm[z + k * g.ldz + p] = make_float2(a.y + b.x, a.x - b.y);
    if (!self) sm[z + (g.K2 - k) * g.ldz + p] = make_float2(b.x - a.y, a.x + b.y);
  }
}

}  // namespace pmgpu
