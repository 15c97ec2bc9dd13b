// Butterflies and columns of the native FFT passes (ffx.cu, ffxconv.cu).
#pragma once

#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace mrn {

constexpr float kSin3 = 0.866025403784438647f;   // sin(2 pi / 3)
constexpr float kCos51 = 0.309016994374947424f;  // cos(2 pi / 5)
constexpr float kCos52 = -0.809016994374947424f; // cos(4 pi / 5)
constexpr float kSin51 = 0.951056516295153572f;  // sin(2 pi / 5)
constexpr float kSin52 = 0.587785252292473129f;  // sin(4 pi / 5)

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// a w (forward) or a conj(w) (inverse)
template <bool INV>
__device__ __forceinline__ float2 ctw(float2 a, float2 w) {
  return INV ? make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y)
             : make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}

// -i a (forward) or +i a (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// cos and sin of 2 pi k / n at compile time (the Taylor series of an angle
// reduced to [-pi/4, pi/4] by quarter turns)
constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return s;
}
constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int i = 1; i < 14; ++i) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return s;
}
constexpr double kPi = 3.14159265358979323846;
constexpr double root_cs(int k, int n, bool sine) {
  k %= n;
  int quarter = (8 * k + n) / (2 * n);  // nearest multiple of n / 4
  const double x = 2.0 * kPi * (4 * k - quarter * n) / (4.0 * n);
  quarter &= 3;
  const double c = series_cos(x), s = series_sin(x);
  const double cc = quarter == 0 ? c : quarter == 1 ? -s : quarter == 2 ? -c : s;
  const double ss = quarter == 0 ? s : quarter == 1 ? c : quarter == 2 ? -s : -c;
  return sine ? ss : cc;
}
template <int N>
struct Roots {
  float c[N], s[N];
  constexpr Roots() : c(), s() {
    for (int k = 0; k < N; ++k) {
      c[k] = (float)root_cs(k, N, false);
      s[k] = (float)root_cs(k, N, true);
    }
  }
};

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&x)[R]);

// R = A B: B transforms of A points (inputs r, r + B, ..), output u1 of
// transform r turned by e^(-+2 pi i r u1 / R), then A transforms of B points;
// result u1 + A u2.
template <int A, int B, bool INV>
__device__ __forceinline__ void dft_ab(float2 (&x)[A * B]) {
  constexpr int R = A * B;
  constexpr Roots<R> w{};
  float2 a[B][A];
#pragma unroll
  for (int r = 0; r < B; ++r) {
#pragma unroll
    for (int m = 0; m < A; ++m) a[r][m] = x[B * m + r];
    dft<A, INV>(a[r]);
  }
#pragma unroll
  for (int u = 0; u < A; ++u) {
    float2 col[B];
#pragma unroll
    for (int r = 0; r < B; ++r) {
      const int k = r * u;  // below R
      const float2 v = a[r][u];
      if (k == 0) col[r] = v;
      else if (4 * k == R) col[r] = rot<INV>(v);
      else if (2 * k == R) col[r] = make_float2(-v.x, -v.y);
      else col[r] = INV ? make_float2(v.x * w.c[k] - v.y * w.s[k], v.x * w.s[k] + v.y * w.c[k])
                        : make_float2(v.x * w.c[k] + v.y * w.s[k], v.y * w.c[k] - v.x * w.s[k]);
    }
    dft<B, INV>(col);
#pragma unroll
    for (int v = 0; v < B; ++v) x[u + A * v] = col[v];
  }
}

// An odd prime P: with a_k = x_k + x_(P-k), b_k = -+i (x_k - x_(P-k)),
// X_u, X_(P-u) = x_0 + sum_k cos(2 pi k u / P) a_k +- sum_k sin(2 pi k u / P) b_k.
template <int P, bool INV>
__device__ __forceinline__ void dft_prime(float2 (&x)[P]) {
  constexpr int H = (P - 1) / 2;
  constexpr Roots<P> w{};
  float2 a[H], b[H];
  float2 s = x[0];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    a[k] = cadd(x[k + 1], x[P - 1 - k]);
    b[k] = rot<INV>(csub(x[k + 1], x[P - 1 - k]));
    s = cadd(s, a[k]);
  }
#pragma unroll
  for (int u = 1; u <= H; ++u) {
    float2 c = x[0], d = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      const int i = k * u % P;
      c = __ffma2_rn(make_float2(w.c[i], w.c[i]), a[k - 1], c);
      d = k == 1 ? __fmul2_rn(make_float2(w.s[i], w.s[i]), b[0]) : __ffma2_rn(make_float2(w.s[i], w.s[i]), b[k - 1], d);
    }
    x[u] = cadd(c, d);
    x[P - u] = csub(c, d);
  }
  x[0] = s;
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&x)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 a = x[0];
    x[0] = cadd(a, x[1]);
    x[1] = csub(a, x[1]);
  } else if constexpr (R == 3) {
    const float2 s = cadd(x[1], x[2]);
    const float2 m = __ffma2_rn(make_float2(-0.5f, -0.5f), s, x[0]);
    const float2 t = rot<INV>(csub(x[1], x[2]));
    x[0] = cadd(x[0], s);
    x[1] = __ffma2_rn(make_float2(kSin3, kSin3), t, m);
    x[2] = __ffma2_rn(make_float2(-kSin3, -kSin3), t, m);
  } else if constexpr (R == 4) {
    const float2 a0 = cadd(x[0], x[2]), a1 = csub(x[0], x[2]);
    const float2 a2 = cadd(x[1], x[3]), a3 = rot<INV>(csub(x[1], x[3]));
    x[0] = cadd(a0, a2);
    x[2] = csub(a0, a2);
    x[1] = cadd(a1, a3);
    x[3] = csub(a1, a3);
  } else if constexpr (R == 5) {
    const float2 a1 = cadd(x[1], x[4]), b1 = csub(x[1], x[4]);
    const float2 a2 = cadd(x[2], x[3]), b2 = csub(x[2], x[3]);
    const float2 r1 = __ffma2_rn(make_float2(kCos52, kCos52), a2, __ffma2_rn(make_float2(kCos51, kCos51), a1, x[0]));
    const float2 r2 = __ffma2_rn(make_float2(kCos51, kCos51), a2, __ffma2_rn(make_float2(kCos52, kCos52), a1, x[0]));
    const float2 p1 = rot<INV>(__ffma2_rn(make_float2(kSin52, kSin52), b2, __fmul2_rn(make_float2(kSin51, kSin51), b1)));
    const float2 p2 = rot<INV>(__ffma2_rn(make_float2(-kSin51, -kSin51), b2, __fmul2_rn(make_float2(kSin52, kSin52), b1)));
    x[0] = cadd(x[0], cadd(a1, a2));
    x[1] = cadd(r1, p1);
    x[4] = csub(r1, p1);
    x[2] = cadd(r2, p2);
    x[3] = csub(r2, p2);
  } else if constexpr (R == 6) {
    dft_ab<3, 2, INV>(x);
  } else if constexpr (R == 7 || R == 11 || R == 13 || R == 17 || R == 19) {
    dft_prime<R, INV>(x);
  } else if constexpr (R == 14) {
    dft_ab<7, 2, INV>(x);
  } else if constexpr (R == 8) {
    dft_ab<4, 2, INV>(x);
  } else if constexpr (R == 9) {
    dft_ab<3, 3, INV>(x);
  } else if constexpr (R == 10) {
    dft_ab<5, 2, INV>(x);
  } else if constexpr (R == 12) {
    dft_ab<4, 3, INV>(x);
  } else if constexpr (R == 15) {
    dft_ab<5, 3, INV>(x);
  } else if constexpr (R == 16) {
    dft_ab<4, 4, INV>(x);
  } else if constexpr (R == 20) {
    dft_ab<5, 4, INV>(x);
  } else if constexpr (R == 24) {
    dft_ab<6, 4, INV>(x);
  } else {
    static_assert(R == 32, "radix");
    dft_ab<8, 4, INV>(x);
  }
}

// Rows that a first-stage butterfly's R points take in shared memory: an odd
// number, so lanes that run along the axis store without bank conflicts (512 =
// 8 x 8 x 8 from the image: 8-way before).
__host__ __device__ __forceinline__ int ffx_block_rows(int R) { return R | 1; }

// What a pass reads first and writes last.
enum FfxSrc { kFfxGrid = 0, kFfxImage = 1, kFfxSense = 2 };


// The columns of one CTA: where each starts in the grid (-1: no column), its
// image row and coil-map row, the scale and apodization of the earlier axes.
template <int W>
struct FfxCols {
  int64_t base[W];
  int64_t img[W];
  int64_t map[W];
  float a[W];
};

// Columns f0 .. f0 + W - 1 of slice g, by the first W threads. Columns of a
// slice are numbered [coil block][image point of the earlier axes][cell of the
// later axes][coil of the block], without the unused coils of the last block.
// LAST: the last axis, against the image.
template <int W, bool LAST, bool SENSE>
__device__ __forceinline__ void ffx_columns(FfxCols<W>& cols, const SliceGeom& g, const FfxPass& ps, int n, int f0,
                                            int ncols, const float* __restrict__ apod, float scale) {
  const int tid = threadIdx.x;
  if (tid >= W) return;
  const int cb = g.cb, cells = ps.pcols * ps.icells;  // columns of one coil
  const int f = f0 + tid;
  const int kb = f / (cells * cb), nc = min(cb, g.ncoil - kb * cb);
  const int rem = f - kb * cells * cb;
  const int cell = rem / max(nc, 1), cc = rem - cell * nc;
  const int o = cell / ps.icells, i = (cell - o * ps.icells) * cb + cc;
  const int c = kb * cb + cc;
  int64_t base = -1;
  if (f < ncols) {
    const int q0 = o / ps.en1, q1 = o - q0 * ps.en1;
    const int64_t row = (int64_t)q0 * ps.enos1 + q1;
    base = g.grid_off + (kb * g.gos + row * n * ps.icells) * cb + i;
    if (LAST) {
      // the earlier axes' image point o is also the image row
      cols.img[tid] = (SENSE ? g.x_off : g.img_off + (int64_t)c * g.nimg) + (int64_t)o * ps.n_img;
      cols.map[tid] = g.img_off + (int64_t)c * g.nimg + (int64_t)o * ps.n_img;
      float a = scale * g.inv_sqrt_n;
      if (ps.axis == 2) {  // 3D: two earlier axes
        a *= apod[g.apod_off[0] + q0];
        a *= apod[g.apod_off[1] + q1];
      } else {
        a *= apod[g.apod_off[0] + q1];
      }
      cols.a[tid] = a;
    }
  }
  cols.base[tid] = base;
}

}  // namespace mrn
