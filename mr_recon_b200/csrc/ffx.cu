// Native FFT stage of the NUFFT: the d-dimensional C2C transform of the
// plan's oversampled grid as one pass per axis, with the NUFFT's zero padding
// and cropping folded into the passes.
//
// Reference: fourier.py (:470-560) apodizes and pads the image into the
// oversampled grid (centred pad + ifftshift), calls torch.fft.fftn, and on
// the adjoint calls ifftn and crops (norm=None: unnormalised transforms; the
// 1/sqrt(prod N) and the apodization are applied in the first forward / last
// adjoint pass with the same float products as k_pre / k_post).
//
// Layout. The grid is [coil block][cell][cb] (grid_at), so every axis is a
// strided one whose adjacent columns are the coils of a cell and then the
// next cells: 16 adjacent columns are one 128-byte segment of every row. An
// axis that is not transformed yet (forward) or any more (inverse) keeps image
// point q in row q, its other rows unused; a transformed axis is centred, as
// the interpolation addresses it. Both are index maps of the loads and stores.
//
// Passes. Forward: the last axis first, reading the image (x coil map) and
// apodizing it, then the others down to the first; inverse: the first axis
// first, the last one cropping into the image (or back into the grid for the
// SENSE coil combination). Columns exist only for image points of the earlier
// axes, so lines of zero padding are never touched, and rows of padding are
// neither read (forward) nor written (inverse).
//
// A column of n = R0 R1 (R2 ..) points is a Stockham autosort FFT: stage s
// with radix R and L = the product of the earlier radices maps butterfly
// b = k L + j (j < L) to out[k R L + u L + j] = sum_t x[b + t n / R] w^(t j)
// e^(-+2 pi i t u / R), w = e^(-+2 pi i / (L R)). The first stage takes its
// points from global memory into registers and the last one stores from
// registers to global memory, so a two-stage length (radices up to 20: every
// 2-3-5 product up to 225 and most up to 400) crosses shared memory once. The
// passes are bound by HBM in 3D and by latency on L2-resident 2D grids.
// Measured (192^3 image, 240^3 grid, 16 coils): the three forward passes take
// 1.93 ms (7.8 GB through HBM: 62% of the copy bandwidth), the inverse ones
// 1.76; passes over coil planes that crossed shared memory before the first,
// between all and after the last stage took 2.61 and 2.48 ms.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace mrn {

namespace {

constexpr int kFfxThreads = 512;  // most threads of a pass' CTA
constexpr int kFfxMaxRadix = 20;

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
  } else {
    static_assert(R == 20, "radix");
    dft_ab<5, 4, INV>(x);
  }
}

// Geometry of one pass (one axis of one FFT group).
struct FfxPass {
  FfxAxis ax;
  int n_img;        // image points along the axis
  int axis;
  int en1, enos1;   // image and grid size of the second axis when it precedes this one, else 1
  int pcols;        // image points of the earlier axes
  int icells;       // grid cells of the later axes
  int bfast_in, bfast_out;  // lanes of the first / last stage run along the axis, not across columns
};

// What a pass reads first and writes last.
enum FfxSrc { kFfxGrid = 0, kFfxImage = 1, kFfxSense = 2 };

// One pass: a CTA per (slice blockIdx.y, W adjacent columns). Columns of a
// slice are numbered [coil block][image point of the earlier axes][cell of the
// later axes][coil of the block]. Lanes run across columns (one 128-byte
// segment per row for W = 16) except where the other side is the planar image
// or a grid of few coils, whose contiguous direction is the axis itself.
template <bool INV, int SRC, bool TO_IMAGE, int W>
__global__ void __launch_bounds__(kFfxThreads)
k_ffx_pass(const SliceGeom* __restrict__ sl, const int* __restrict__ gsl, FfxPass ps, const float2* __restrict__ twg,
           float2* __restrict__ grid, const float* __restrict__ apod, const float2* __restrict__ src,
           const float2* __restrict__ mps, float scale, float2* __restrict__ out) {
  constexpr bool LAST = SRC != kFfxGrid || TO_IMAGE;  // the last axis, against the image
  constexpr int WS = W + 1;                           // odd column stride: no bank conflicts either way
  extern __shared__ float2 fsm[];
  __shared__ int64_t s_base[W];  // grid offset of the column's first row, -1: no column
  __shared__ int64_t s_img[W];   // image row
  __shared__ int64_t s_map[W];   // coil-map row
  __shared__ float s_a[W];       // scale and apodization of the earlier axes
  const SliceGeom& g = sl[gsl[blockIdx.y]];
  const int cb = g.cb, inner = ps.icells * cb;
  const int per_block = ps.pcols * inner;
  const int ncols = ((g.ncoil + cb - 1) / cb) * per_block;
  const int f0 = blockIdx.x * W;
  if (f0 >= ncols) return;
  const int n = ps.ax.n, tid = threadIdx.x, nt = blockDim.x;
  const int R0 = ps.ax.radix[0], ns = ps.ax.ns;
  const int r0s = R0 + ((ns == 2 && !(R0 & 1)) ? 1 : 0);  // odd row stride of the first stage's blocks
  float2* tw = fsm;
  float2* A = fsm + n;
  float2* B = A + (size_t)(n / R0) * r0s * WS;  // used from three stages on
  for (int i = tid; i < n - 1; i += nt) tw[i] = twg[ps.ax.tw_base + i];
  if (tid < W) {
    const int f = f0 + tid;
    const int kb = f / per_block;
    const int rem = f - kb * per_block;
    const int o = rem / inner, i = rem - o * inner;
    const int c = kb * cb + i % cb;
    int64_t base = -1;
    if (f < ncols && c < g.ncoil) {
      const int q0 = o / ps.en1, q1 = o - q0 * ps.en1;
      const int64_t row = (int64_t)q0 * ps.enos1 + q1;
      base = g.grid_off + (kb * g.gos + row * n * ps.icells) * cb + i;
      if (LAST) {
        // the earlier axes' image point o is also the image row
        s_img[tid] = (SRC == kFfxSense ? g.x_off : g.img_off + (int64_t)c * g.nimg) + (int64_t)o * ps.n_img;
        s_map[tid] = g.img_off + (int64_t)c * g.nimg + (int64_t)o * ps.n_img;
        float a = scale * g.inv_sqrt_n;
        if (ps.axis == 2) {  // 3D: two earlier axes
          a *= apod[g.apod_off[0] + q0];
          a *= apod[g.apod_off[1] + q1];
        } else {
          a *= apod[g.apod_off[0] + q1];
        }
        s_a[tid] = a;
      }
    }
    s_base[tid] = base;
  }
  const int h = ps.n_img / 2, hs = n / 2;
  const int es = inner;  // elements between rows of a column
  const float* al = nullptr;
  if (LAST) al = apod + g.apod_off[ps.axis];
  __syncthreads();

  // first stage: global -> registers -> shared
  auto first = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R;
    for (int idx = tid; idx < nr * W; idx += nt) {
      int b, w;
      if (ps.bfast_in) {
        w = nr == 1 ? idx : (int)__umulhi((unsigned)idx, ps.ax.mag_nr[0]);
        b = idx - w * nr;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = s_base[w];
      float2 x[R];
      if (SRC == kFfxGrid) {
        const float2* gp = grid + base;
#pragma unroll
        for (int t = 0; t < R; ++t) {
          int j = b + t * nr + (INV ? hs : h);
          if (j >= n) j -= n;
          x[t] = make_float2(0.f, 0.f);
          if (base >= 0 && (INV || j < ps.n_img)) x[t] = gp[(int64_t)j * es];
        }
      } else {
        const float2* ip = src + s_img[w];
        const float2* mp = SRC == kFfxSense ? mps + s_map[w] : nullptr;
        const float a0 = s_a[w];
        float2 m[SRC == kFfxSense ? R : 1];
#pragma unroll
        for (int t = 0; t < R; ++t) {
          int q = b + t * nr + h;
          if (q >= n) q -= n;
          const bool on = base >= 0 && q < ps.n_img;
          x[t] = make_float2(0.f, 0.f);
          if (on) x[t] = __ldg(ip + q);
          if (SRC == kFfxSense) {
            m[SRC == kFfxSense ? t : 0] = make_float2(0.f, 0.f);
            if (on) m[SRC == kFfxSense ? t : 0] = __ldg(mp + q);
          }
        }
#pragma unroll
        for (int t = 0; t < R; ++t) {
          int q = b + t * nr + h;
          if (q >= n) q -= n;
          const float a = q < ps.n_img ? a0 * __ldg(al + q) : 0.f;
          float2 v = x[t];
          if (SRC == kFfxSense) {
            const float2 mm = m[SRC == kFfxSense ? t : 0];
            v = make_float2(v.x * mm.x - v.y * mm.y, v.x * mm.y + v.y * mm.x);
          }
          x[t] = make_float2(v.x * a, v.y * a);
        }
      }
      dft<R, INV>(x);
      float2* d = A + b * r0s * WS + w;
#pragma unroll
      for (int u = 0; u < R; ++u) d[u * WS] = x[u];
    }
  };
  // middle stage: shared -> shared
  auto middle = [&](auto rc, const float2* a, float2* d, int s, int L) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R;
    const float2* tws = tw + ps.ax.tw_off[s];
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int k = (int)__umulhi((unsigned)b, ps.ax.mag_l[s]), j = b - k * L;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(b + t * nr) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<INV>(x[t], tws[j * (R - 1) + t - 1]);
      dft<R, INV>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) d[(k * R * L + u * L + j) * WS + w] = x[u];
    }
  };
  // last stage: shared -> registers -> global
  auto last = [&](auto rc, const float2* a, int s, int row_stride) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R;
    const float2* tws = tw + ps.ax.tw_off[s];
    for (int idx = tid; idx < nr * W; idx += nt) {
      int b, w;
      if (ps.bfast_out) {
        w = nr == 1 ? idx : (int)__umulhi((unsigned)idx, ps.ax.mag_nr[s]);
        b = idx - w * nr;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = s_base[w];
      if (base < 0) continue;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(b + t * row_stride) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<INV>(x[t], tws[b * (R - 1) + t - 1]);
      dft<R, INV>(x);
      if (TO_IMAGE) {
        float2* op = out + s_img[w];
        const float a0 = s_a[w];
#pragma unroll
        for (int u = 0; u < R; ++u) {
          int q = u * nr + b + h;
          if (q >= n) q -= n;
          if (q < ps.n_img) {
            const float av = a0 * __ldg(al + q);
            op[q] = make_float2(x[u].x * av, x[u].y * av);
          }
        }
      } else {
        float2* gp = grid + base;
#pragma unroll
        for (int u = 0; u < R; ++u) {
          int j = u * nr + b + (INV ? h : hs);
          if (j >= n) j -= n;
          if (!INV || j < ps.n_img) gp[(int64_t)j * es] = x[u];
        }
      }
    }
  };
#define MRN_FFX_RADIX(R_, CALL)                                                 \
  switch (R_) {                                                                 \
    case 1: { std::integral_constant<int, 1> rc; CALL; } break;                 \
    case 2: { std::integral_constant<int, 2> rc; CALL; } break;                 \
    case 3: { std::integral_constant<int, 3> rc; CALL; } break;                 \
    case 4: { std::integral_constant<int, 4> rc; CALL; } break;                 \
    case 5: { std::integral_constant<int, 5> rc; CALL; } break;                 \
    case 6: { std::integral_constant<int, 6> rc; CALL; } break;                 \
    case 8: { std::integral_constant<int, 8> rc; CALL; } break;                 \
    case 9: { std::integral_constant<int, 9> rc; CALL; } break;                 \
    case 10: { std::integral_constant<int, 10> rc; CALL; } break;               \
    case 12: { std::integral_constant<int, 12> rc; CALL; } break;               \
    case 15: { std::integral_constant<int, 15> rc; CALL; } break;               \
    case 16: { std::integral_constant<int, 16> rc; CALL; } break;               \
    default: { std::integral_constant<int, 20> rc; CALL; } break;               \
  }
  MRN_FFX_RADIX(R0, first(rc))
  __syncthreads();
  int L = R0;
#pragma unroll 1
  for (int s = 1; s + 1 < ns; ++s) {
    const int R = ps.ax.radix[s];
    // radices above 12 come in two-stage lengths or first and last
    switch (R) {
      case 2: middle(std::integral_constant<int, 2>(), A, B, s, L); break;
      case 3: middle(std::integral_constant<int, 3>(), A, B, s, L); break;
      case 4: middle(std::integral_constant<int, 4>(), A, B, s, L); break;
      case 5: middle(std::integral_constant<int, 5>(), A, B, s, L); break;
      case 6: middle(std::integral_constant<int, 6>(), A, B, s, L); break;
      case 8: middle(std::integral_constant<int, 8>(), A, B, s, L); break;
      case 9: middle(std::integral_constant<int, 9>(), A, B, s, L); break;
      case 10: middle(std::integral_constant<int, 10>(), A, B, s, L); break;
      default: middle(std::integral_constant<int, 12>(), A, B, s, L); break;
    }
    __syncthreads();
    float2* t = A;
    A = B;
    B = t;
    L *= R;
  }
  {
    const int R = ps.ax.radix[ns - 1];
    const int rs = ns == 2 ? r0s : n / R;
    MRN_FFX_RADIX(R, last(rc, A, ns - 1, rs))
  }
}

constexpr int kRadices[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 20};
constexpr int kMidMax = 12;  // largest radix of a middle stage

// Radices of n: two stages with the smallest larger radix where one exists,
// else three, else four (first and last up to 20, the middle ones up to 12);
// false if n has a prime factor above 5. The largest radix comes first: the
// first stage's loads are the ones in flight from global memory.
bool ffx_radices(int n, int stages, int cap, std::vector<int>& best) {
  std::vector<int> cur;
  int best_max = 1 << 30;
  auto rec = [&](auto&& self, int m, int left, int most) -> void {
    if (left == 0) {
      if (m == 1 && !cur.empty() && cur[0] < best_max) {
        best_max = cur[0];
        best = cur;
      }
      return;
    }
    for (int r : kRadices)
      if (m % r == 0 && r <= most) {
        cur.push_back(r);
        self(self, m / r, left - 1, r);
        cur.pop_back();
      }
  };
  rec(rec, n, stages, cap);
  return best_max < (1 << 30);
}

bool ffx_factor(int n, FfxAxis& ax) {
  ax = FfxAxis{};
  ax.n = n;
  if (n < 2 || n > kFfxMaxN) return false;
  std::vector<int> r;
  bool ok = false;
  for (int stages = 2; stages <= kFfxMaxStages && !ok; ++stages) {
    r.clear();
    ok = ffx_radices(n, stages, kFfxMaxRadix, r);
    // the second-largest radix is last, so every middle one is at most 12
    if (ok && stages > 2) {
      std::swap(r[1], r[stages - 1]);
      for (int s = 1; s + 1 < stages; ++s) ok &= r[s] <= kMidMax;
    }
  }
  if (!ok) {
    if (n > 5) return false;
    r = {n, 1};
  }
  ax.ns = (int)r.size();
  for (int s = 0; s < ax.ns; ++s) ax.radix[s] = r[s];
  return true;
}

template <class T>
int upload(T** dst, const std::vector<T>& v) {
  if (*dst) cudaFree(*dst);
  *dst = nullptr;
  if (cudaMalloc(dst, std::max<size_t>(1, v.size()) * sizeof(T)) != cudaSuccess) return MRN_ERR_CUDA;
  if (!v.empty() && cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
    return MRN_ERR_CUDA;
  return MRN_OK;
}

size_t pass_smem(const FfxAxis& ax, int w) {
  const int r0s = ax.radix[0] + ((ax.ns == 2 && !(ax.radix[0] & 1)) ? 1 : 0);
  const size_t a = (size_t)(ax.n / ax.radix[0]) * r0s * (w + 1);
  const size_t b = ax.ns > 2 ? (size_t)ax.n * (w + 1) : 0;
  return ((size_t)ax.n + a + b) * sizeof(float2);
}

// Pass of group q along axis a. SRC / TO_IMAGE as in k_ffx_pass.
template <bool INV, int SRC, bool TO_IMAGE>
int launch_pass(const FfxSet& S, const FfxGrid& G, int q, int a, const float2* src, const float2* mps, float2* out,
                float scale, cudaStream_t st) {
  const int D = G.ndim;
  const FfxGroup& fg = S.grp[q];
  const SliceGeom& g = G.hsl[fg.first_slice];
  FfxPass ps{};
  ps.ax = fg.ax[a];
  ps.n_img = g.n[a];
  ps.axis = a;
  ps.pcols = ps.icells = 1;
  for (int i = 0; i < a; ++i) ps.pcols *= g.n[i];
  for (int i = a + 1; i < D; ++i) ps.icells *= g.nos[i];
  ps.en1 = a == 2 ? g.n[1] : std::max(1, ps.pcols);
  ps.enos1 = a == 2 ? g.nos[1] : 1;
  // The image is planar, so its side runs along the axis. So does the grid
  // side of the last axis with fewer than 8 coils per cell: adjacent columns
  // are then other lines, a whole line apart.
  const bool last_axis = a == D - 1;
  const bool narrow = last_axis && g.cb < 8;
  ps.bfast_in = SRC != kFfxGrid || narrow;
  ps.bfast_out = TO_IMAGE || narrow;
  // W = 16 columns (128-byte rows) while two CTAs' buffers fit an SM; fewer
  // where that leaves SMs without work (2D, few coils).
  const int64_t cols = (int64_t)fg.max_coil * ps.pcols * ps.icells;
  const int64_t total = (int64_t)fg.total_coil * ps.pcols * ps.icells;
  int w = 16;
  while (w > 4 && (pass_smem(ps.ax, w) > 100 * 1024 || total / w < 2 * G.sm_count)) w /= 2;
  const int64_t nb = (cols + w - 1) / w;
  if (cols > 0x7fffffffLL) return MRN_ERR_UNSUPPORTED;
  int most = 1;
  for (int s = 0; s < ps.ax.ns; ++s) most = std::max(most, ps.ax.n / ps.ax.radix[s]);
  const int threads = std::min(kFfxThreads, std::max(32, (most * w + 31) / 32 * 32));
  const size_t smem = pass_smem(ps.ax, w);
  int rc = MRN_OK;
#define MRN_FFX_LAUNCH(WW)                                                                                  \
  do {                                                                                                      \
    auto kern = k_ffx_pass<INV, SRC, TO_IMAGE, WW>;                                                         \
    rc = set_dynamic_smem(kern, smem);                                                                      \
    for (int s0 = 0; rc == MRN_OK && s0 < fg.nsl; s0 += 65535)                                              \
      kern<<<dim3((unsigned)nb, (unsigned)std::min(65535, fg.nsl - s0)), threads, smem, st>>>(              \
          G.dsl, S.d_sl + fg.sl_off + s0, ps, S.d_tw, G.grid, G.apod, src, mps, scale, out);                \
  } while (0)
  if (w == 16) MRN_FFX_LAUNCH(16);
  else if (w == 8) MRN_FFX_LAUNCH(8);
  else MRN_FFX_LAUNCH(4);
#undef MRN_FFX_LAUNCH
  if (rc != MRN_OK) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

FfxGrid plan_grid(mrn_plan* P) {
  return FfxGrid{P->ndim, P->h_slices.data(), P->d_slices, P->d_apod, P->d_grid, P->sm_count};
}

}  // namespace

// Whether every axis of a grid can run the native passes.
bool ffx_can(int ndim, const int* nos) {
  if (ndim != 2 && ndim != 3) return false;
  FfxAxis ax;
  for (int i = 0; i < ndim; ++i)
    if (!ffx_factor(nos[i], ax)) return false;
  return true;
}

// Build the native FFT of a grid buffer: per group spec (grid size), the
// group's slices (those of that grid size, in slice order), its axes' twiddle
// tables and slice list. A group whose slices differ in image size, or with
// an axis that has a prime factor above 5 or more than kFfxMaxN points, is
// not native.
int ffx_build(FfxSet& S, int ndim, const std::vector<SliceGeom>& hsl, const std::vector<FfxGroupSpec>& spec) {
  S.release();
  if ((ndim != 2 && ndim != 3) || hsl.empty()) return MRN_OK;
  const int D = ndim;
  std::vector<float2> tab;
  std::vector<int> sl_ids;
  int nnative = 0;
  for (const FfxGroupSpec& gs : spec) {
    FfxGroup fg{};
    fg.native = true;
    fg.first_slice = -1;
    fg.sl_off = (int)sl_ids.size();
    for (int s = 0; s < (int)hsl.size(); ++s) {
      const SliceGeom& g = hsl[s];
      bool same = true;
      for (int i = 0; i < D; ++i) same &= g.nos[i] == gs.nos[i];
      if (!same) continue;
      if (fg.first_slice < 0) fg.first_slice = s;
      const SliceGeom& g0 = hsl[fg.first_slice];
      for (int i = 0; i < D; ++i) fg.native &= g.n[i] == g0.n[i];
      const int cb = coil_block(g.ncoil), padded = (g.ncoil + cb - 1) / cb * cb;
      fg.max_coil = std::max(fg.max_coil, padded);
      fg.total_coil += padded;
      sl_ids.push_back(s);
      ++fg.nsl;
    }
    if (fg.first_slice < 0) fg.native = false;
    for (int i = 0; i < D; ++i) {
      FfxAxis& ax = fg.ax[i];
      if (!ffx_factor(gs.nos[i], ax)) {
        fg.native = false;
        continue;
      }
      ax.tw_base = (int)tab.size();
      int L = 1, off = 0;
      for (int st = 0; st < ax.ns; ++st) {
        const int R = ax.radix[st], nr = ax.n / R;
        ax.tw_off[st] = off;
        ax.mag_l[st] = L > 1 ? (unsigned)((1ull << 32) / (unsigned long long)L + 1ull) : 0u;
        ax.mag_nr[st] = nr > 1 ? (unsigned)((1ull << 32) / (unsigned long long)nr + 1ull) : 0u;
        for (int j = 0; j < L; ++j)
          for (int t = 1; t < R; ++t) {
            const double ang = -2.0 * M_PI * (double)t * (double)j / (double)(L * R);
            tab.push_back(make_float2((float)std::cos(ang), (float)std::sin(ang)));
          }
        off += L * (R - 1);
        L *= R;
      }
    }
    nnative += fg.native ? 1 : 0;
    S.grp.push_back(fg);
  }
  if (nnative == 0) {
    S.grp.clear();
    return MRN_OK;
  }
  int rc = upload(&S.d_tw, tab);
  if (rc == MRN_OK) rc = upload(&S.d_sl, sl_ids);
  if (rc != MRN_OK) {
    S.release();
    return rc;
  }
  S.ok = true;
  S.all = nnative == (int)spec.size();
  return MRN_OK;
}

int ffx_fwd(const FfxSet& S, const FfxGrid& G, PreMode mode, const float2* src, const float2* mps, float scale,
            cudaStream_t st) {
  for (size_t q = 0; q < S.grp.size(); ++q) {
    if (!S.grp[q].native) continue;
    const int a = G.ndim - 1;
    int rc = mode == kPreSense
                 ? launch_pass<false, kFfxSense, false>(S, G, (int)q, a, src, mps, nullptr, scale, st)
                 : launch_pass<false, kFfxImage, false>(S, G, (int)q, a, src, mps, nullptr, scale, st);
    for (int i = a - 1; i >= 0 && rc == MRN_OK; --i)
      rc = launch_pass<false, kFfxGrid, false>(S, G, (int)q, i, nullptr, nullptr, nullptr, scale, st);
    if (rc != MRN_OK) return rc;
  }
  return MRN_OK;
}

int ffx_inv(const FfxSet& S, const FfxGrid& G, float2* out, float scale, cudaStream_t st) {
  for (size_t q = 0; q < S.grp.size(); ++q) {
    if (!S.grp[q].native) continue;
    int rc = MRN_OK;
    const int a = G.ndim - 1;
    for (int i = 0; i < a && rc == MRN_OK; ++i)
      rc = launch_pass<true, kFfxGrid, false>(S, G, (int)q, i, nullptr, nullptr, nullptr, scale, st);
    if (rc == MRN_OK)
      rc = out ? launch_pass<true, kFfxGrid, true>(S, G, (int)q, a, nullptr, nullptr, out, scale, st)
               : launch_pass<true, kFfxGrid, false>(S, G, (int)q, a, nullptr, nullptr, nullptr, scale, st);
    if (rc != MRN_OK) return rc;
  }
  return MRN_OK;
}

bool ffx_active(const mrn_plan* P) { return P->ffx.ok && P->use_ffx; }

// Per-slice layout: a slice whose group runs the native passes (k_pre / k_post
// leave it alone) has its grid in coil blocks, centred; the others keep coil
// planes in FFT order.
int ffx_refresh(mrn_plan* P) {
  if (P->h_slices.empty() || !P->d_slices) return MRN_OK;
  const int D = P->ndim;
  for (auto& g : P->h_slices) {
    g.native_fft = 0;
    if (P->use_ffx)
      for (const auto& fg : P->ffx.grp) {
        bool same = fg.native;
        for (int i = 0; i < D && same; ++i) same = g.nos[i] == fg.ax[i].n;
        if (same) g.native_fft = 1;
      }
    g.cb = g.native_fft ? coil_block(g.ncoil) : 1;
    for (int i = 0; i < D; ++i) g.hshift[i] = g.native_fft || (P->flags & MRN_PLAN_RAW) ? 0 : g.nos[i] / 2;
  }
  return upload_slices(P) == cudaSuccess ? MRN_OK : MRN_ERR_CUDA;
}

// The plan grid's native FFT (plan creation, after the FFT groups exist).
int ffx_setup(mrn_plan* P) {
  P->ffx.release();
  if (P->flags & MRN_PLAN_RAW) return MRN_OK;
  std::vector<FfxGroupSpec> spec;
  for (const auto& f : P->fft) {
    FfxGroupSpec gs{};
    for (int i = 0; i < kMaxDim; ++i) gs.nos[i] = f.nos[i];
    spec.push_back(gs);
  }
  const int rc = ffx_build(P->ffx, P->ndim, P->h_slices, spec);
  if (rc != MRN_OK) return rc;
  return ffx_refresh(P);
}

// Apodize / pad (plain image or SENSE x * maps) and forward FFT of the grid.
int ffx_forward(mrn_plan* P, PreMode mode, const float2* src, const float2* mps, float scale, cudaStream_t st) {
  return ffx_fwd(P->ffx, plan_grid(P), mode, src, mps, scale, st);
}

// Inverse FFT of the grid; out != nullptr: crop / deapodize into the image
// batch (plain adjoint), else the surviving points stay in the grid.
int ffx_inverse(mrn_plan* P, float2* out, float scale, cudaStream_t st) {
  return ffx_inv(P->ffx, plan_grid(P), out, scale, st);
}

}  // namespace mrn
