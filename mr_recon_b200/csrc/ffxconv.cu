// Native FFT passes for lengths with a prime factor above 19: each axis as a
// chirp convolution (Bluestein 1970): with c[j] = e^(-i pi j^2 / n),
//   X[k] = c[k] sum_j (x[j] c[j]) conj(c[k - j]),
// a circular convolution of any length m >= 2 n - 1, here m = R0 R1 with radices
// up to 32. A pass has the layout, columns and padding of ffx.cu; a column goes
//   global -> x c -> R0-point butterflies -> shared
//   -> twiddles, R1-point butterflies, x filter, inverse R1-point butterflies
//      (the outputs of one are the inputs of the other) -> shared
//   -> twiddles, inverse R0-point butterflies -> x c -> global,
// two crossings of shared memory, with the filter (the FFT of conj(c) over m)
// from a host table in double precision. The inverse transform conjugates on the
// way in and out.
//
// Such grids are most that an image size gives when multiplied by the
// oversampling. cuFFT makes several passes over them, wants separate pad and
// crop kernels and coil planes, and one plan per grid size, so an uneven batch
// ran its slices one after the other. Bound by issue and occupancy (radices of
// 24 and 32 take 128 registers).
#include <algorithm>
#include <complex>

#include "ffx_dft.cuh"

namespace mrn {

namespace {

constexpr int kConvThreads = 256;
constexpr int kConvRadices[] = {10, 12, 15, 16, 20, 24, 32};

#define MRN_CONV_RADIX(R_, CALL)                                    \
  if constexpr (!BIG) {                                             \
    switch (R_) {                                                   \
      case 10: { std::integral_constant<int, 10> rc; CALL; } break; \
      case 12: { std::integral_constant<int, 12> rc; CALL; } break; \
      case 15: { std::integral_constant<int, 15> rc; CALL; } break; \
      case 16: { std::integral_constant<int, 16> rc; CALL; } break; \
      default: { std::integral_constant<int, 20> rc; CALL; } break; \
    }                                                               \
  } else {                                                          \
    switch (R_) {                                                   \
      case 10: { std::integral_constant<int, 10> rc; CALL; } break; \
      case 12: { std::integral_constant<int, 12> rc; CALL; } break; \
      case 15: { std::integral_constant<int, 15> rc; CALL; } break; \
      case 16: { std::integral_constant<int, 16> rc; CALL; } break; \
      case 20: { std::integral_constant<int, 20> rc; CALL; } break; \
      case 24: { std::integral_constant<int, 24> rc; CALL; } break; \
      default: { std::integral_constant<int, 32> rc; CALL; } break; \
    }                                                               \
  }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__host__ __device__ constexpr int odd(int r) { return r | 1; }  // row strides of the exchanges

// BIG: radices 24 and 32 among the passes (128 registers); else at most 20 (85).
template <bool INV, int SRC, bool TO_IMAGE, int W, bool BIG>
__global__ void __launch_bounds__(kConvThreads, BIG ? 2 : 3)
k_ffx_conv(const SliceGeom* __restrict__ sl, const FfxSlice* __restrict__ list, const FfxPass* __restrict__ passes,
           const float2* __restrict__ twg, float2* __restrict__ grid, const float* __restrict__ apod,
           const float2* __restrict__ src, const float2* __restrict__ mps, float scale, float2* __restrict__ out) {
  constexpr bool LAST = SRC != kFfxGrid || TO_IMAGE;
  constexpr int WS = W + 1;
  extern __shared__ float2 fsm[];
  __shared__ FfxCols<W> cols;
  __shared__ FfxPass ps;
  const FfxSlice fs = list[blockIdx.y];
  {
    const int* from = reinterpret_cast<const int*>(passes + fs.pass);
    for (int i = threadIdx.x; i < (int)(sizeof(FfxPass) / sizeof(int)); i += blockDim.x)
      reinterpret_cast<int*>(&ps)[i] = from[i];
  }
  __syncthreads();
  const SliceGeom& g = sl[fs.slice];
  const int ncols = g.ncoil * ps.pcols * ps.icells;
  const int f0 = blockIdx.x * W;
  if (f0 >= ncols) return;
  const int n = ps.ax.n, m = ps.ax.m, R0 = ps.ax.radix[0], R1 = ps.ax.radix[1], tid = threadIdx.x, nt = blockDim.x;
  const int r0s = odd(R0), r1s = odd(R1), es = ps.icells * g.cb;
  float2* tw = fsm;
  float2* A = fsm + m;  // [R1][r0s][WS], then [R0][r1s][WS]
  const float2* chirp = twg + ps.ax.chirp;
  const float2* filter = twg + ps.ax.filter;
  for (int i = tid; i < m; i += nt) tw[i] = twg[ps.ax.tw_base + i];
  ffx_columns<W, LAST, SRC == kFfxSense>(cols, g, ps, n, f0, ncols, apod, scale);
  const int h = ps.n_img / 2, hs = n / 2;
  const float* al = LAST ? apod + g.apod_off[ps.axis] : nullptr;
  __syncthreads();

  // point e = b + t R1 of the column, from global memory
  auto first = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int idx = tid;
    if (idx < R1 * W) {  // R1 <= R0: the CTA has R0 W threads
      int b, w;
      if (SRC != kFfxGrid || ps.narrow) {
        w = (int)__umulhi((unsigned)idx, ps.ax.mag_nr[0]);
        b = idx - w * R1;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = cols.base[w];
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int e = b + t * R1;
        x[t] = make_float2(0.f, 0.f);
        if (2 * t > R) continue;  // e >= (t R1) > m / 2 >= n
        int j = e + (SRC == kFfxGrid && INV ? hs : h);
        if (j >= n) j -= n;
        if (e < n && base >= 0 && ((SRC == kFfxGrid && INV) || j < ps.n_img)) {
          float2 v;
          if (SRC == kFfxGrid) {
            v = grid[base + (int64_t)j * es];
          } else {
            v = __ldg(src + cols.img[w] + j);
            if (SRC == kFfxSense) v = cmul(v, __ldg(mps + cols.map[w] + j));
            const float av = cols.a[w] * __ldg(al + j);
            v = make_float2(v.x * av, v.y * av);
          }
          if (INV) v.y = -v.y;
          x[t] = cmul(v, __ldg(chirp + e));
        }
      }
      dft<R, false>(x);
      float2* d = A + b * r0s * WS + w;
#pragma unroll
      for (int u = 0; u < R; ++u) d[u * WS] = x[u];
    }
  };
  auto middle = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int b = tid / W, w = tid - b * W;
    const bool on = b < R0;
    float2 x[R];
    if (on) {
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = A[(t * r0s + b) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<false>(x[t], tw[t * b]);
      dft<R, false>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) x[u] = cmul(x[u], __ldg(filter + u * R0 + b));
      dft<R, true>(x);
    }
    __syncthreads();  // every input of the buffer is read
    if (on) {
      float2* d = A + b * r1s * WS + w;
#pragma unroll
      for (int u = 0; u < R; ++u) d[u * WS] = x[u];
    }
  };
  auto last = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int idx = tid;
    if (idx < R1 * W) {
      int b, w;
      if (TO_IMAGE || ps.narrow) {
        w = (int)__umulhi((unsigned)idx, ps.ax.mag_nr[0]);
        b = idx - w * R1;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = cols.base[w];
      if (base < 0) return;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = A[(t * r1s + b) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<true>(x[t], tw[t * b]);
      dft<R, true>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        if (2 * u > R) continue;  // past n
        const int e = u * R1 + b;
        int j = e + (INV ? h : hs);
        if (j >= n) j -= n;
        if (e >= n || (INV && j >= ps.n_img)) continue;
        float2 v = cmul(x[u], __ldg(chirp + e));
        if (INV) v.y = -v.y;
        if (TO_IMAGE) {
          const float av = cols.a[w] * __ldg(al + j);
          out[cols.img[w] + j] = make_float2(v.x * av, v.y * av);
        } else {
          grid[base + (int64_t)j * es] = v;
        }
      }
    }
  };
  MRN_CONV_RADIX(R0, first(rc))
  __syncthreads();
  MRN_CONV_RADIX(R1, middle(rc))
  __syncthreads();
  MRN_CONV_RADIX(R0, last(rc))
}

// Discrete Fourier transform of x (length r[0] r[1]) in double precision.
void host_fft(std::vector<std::complex<double>>& x, int r0, int r1) {
  const int n = (int)x.size();
  std::vector<std::complex<double>> root(n), y(n);
  for (int i = 0; i < n; ++i) root[i] = std::polar(1.0, -2.0 * M_PI * i / n);
  for (int i = 0; i < r1; ++i)  // r0-point transforms of x[i + r1 t]
    for (int k = 0; k < r0; ++k) {
      std::complex<double> v = 0.0;
      for (int t = 0; t < r0; ++t) v += x[i + r1 * t] * root[(int64_t)t * k * r1 % n];
      y[i * r0 + k] = v * root[(int64_t)i * k % n];
    }
  for (int k = 0; k < r0; ++k)
    for (int q = 0; q < r1; ++q) {
      std::complex<double> v = 0.0;
      for (int i = 0; i < r1; ++i) v += y[i * r0 + k] * root[(int64_t)i * q * r0 % n];
      x[k + r0 * q] = v;
    }
}

size_t conv_smem(const FfxAxis& ax, int w) {
  const int r0 = ax.radix[0], r1 = ax.radix[1];
  return ((size_t)ax.m + (size_t)std::max(r1 * odd(r0), r0 * odd(r1)) * (w + 1)) * sizeof(float2);
}

}  // namespace

bool ffx_conv_axis(int n, FfxAxis& ax) {
  ax = FfxAxis{};
  ax.n = n;
  if (n < kFfxConvMin) return false;
  double best = 0.0;
  for (int r0 : kConvRadices)
    for (int r1 : kConvRadices) {
      const int m = r0 * r1;
      if (r1 > r0 || m < 2 * n - 1) continue;
      // work, with the threads that idle in the outer butterflies
      const double cost = m * (1.0 + 0.5 * ((double)r0 / r1 - 1.0));
      if (ax.m > 0 && cost >= best) continue;
      best = cost;
      ax.m = m;
      ax.ns = 2;
      ax.radix[0] = r0;
      ax.radix[1] = r1;
    }
  return ax.m > 0;
}

// Roots of unity, chirp and filter of an axis: the chirp's angles are reduced
// exactly (j^2 mod 2n).
void ffx_conv_tables(FfxAxis& ax, std::vector<float2>& tab) {
  const int n = ax.n, m = ax.m;
  ax.mag_nr[0] = (unsigned)((1ull << 32) / (unsigned long long)ax.radix[1] + 1ull);
  ax.tw_base = (int)tab.size();
  for (int k = 0; k < m; ++k) {
    const std::complex<double> w = std::polar(1.0, -2.0 * M_PI * k / m);
    tab.push_back(make_float2((float)w.real(), (float)w.imag()));
  }
  std::vector<std::complex<double>> f(m, 0.0);
  ax.chirp = (int)tab.size();
  for (int j = 0; j < n; ++j) {
    const std::complex<double> c = std::polar(1.0, -M_PI * (double)((int64_t)j * j % (2 * n)) / n);
    tab.push_back(make_float2((float)c.real(), (float)c.imag()));
    f[j] = std::conj(c);
    if (j > 0) f[m - j] = std::conj(c);
  }
  host_fft(f, ax.radix[0], ax.radix[1]);
  ax.filter = (int)tab.size();
  for (int k = 0; k < m; ++k) tab.push_back(make_float2((float)(f[k].real() / m), (float)(f[k].imag() / m)));
}

// 8 columns, fewer where that leaves SMs without work.
void ffx_conv_shape(FfxStep& st, const std::vector<FfxPass>& passes, int64_t total_cols, int sm_count) {
  st.w = 8;
  while (st.w > 2 && total_cols / st.w < 2 * (int64_t)sm_count) st.w /= 2;
  int most = 1;
  for (const auto& p : passes) {
    st.smem = std::max(st.smem, conv_smem(p.ax, st.w));
    most = std::max(most, p.ax.radix[0]);
  }
  st.big = most > 20;
  st.threads = (most * st.w + 31) / 32 * 32;
}

int launch_ffx_conv(const FfxSet& S, const FfxGrid& G, const FfxStep& step, bool inv, int source, bool to_image,
                    const float2* src, const float2* mps, float2* out, float scale, cudaStream_t st) {
  const int64_t nb = (step.max_cols + step.w - 1) / step.w;
  if (step.max_cols > 0x7fffffffLL) return MRN_ERR_UNSUPPORTED;
  int rc = MRN_OK;
#define MRN_CONV_LAUNCH_B(II, SS, TT, WW, BB)                                                                     \
  do {                                                                                                      \
    auto kern = k_ffx_conv<II, SS, TT, WW, BB>;                                                                 \
    rc = set_dynamic_smem(kern, step.smem);                                                                 \
    for (int s0 = 0; rc == MRN_OK && s0 < step.nsl; s0 += 65535)                                            \
      kern<<<dim3((unsigned)nb, (unsigned)std::min(65535, step.nsl - s0)), step.threads, step.smem, st>>>(  \
          G.dsl, S.d_list + step.first + s0, S.d_pass, S.d_tw, G.grid, G.apod, src, mps, scale, out);       \
  } while (0)
#define MRN_CONV_LAUNCH(II, SS, TT, WW) \
  if (step.big) MRN_CONV_LAUNCH_B(II, SS, TT, WW, true); else MRN_CONV_LAUNCH_B(II, SS, TT, WW, false)
#define MRN_CONV_W(II, SS, TT)                       \
  if (step.w == 8) { MRN_CONV_LAUNCH(II, SS, TT, 8); }   \
  else if (step.w == 4) { MRN_CONV_LAUNCH(II, SS, TT, 4); } \
  else { MRN_CONV_LAUNCH(II, SS, TT, 2); }
  if (inv) {
    if (to_image) { MRN_CONV_W(true, kFfxGrid, true); }
    else { MRN_CONV_W(true, kFfxGrid, false); }
  } else if (source == kFfxGrid) { MRN_CONV_W(false, kFfxGrid, false); }
  else if (source == kFfxImage) { MRN_CONV_W(false, kFfxImage, false); }
  else { MRN_CONV_W(false, kFfxSense, false); }
#undef MRN_CONV_W
#undef MRN_CONV_LAUNCH
#undef MRN_CONV_LAUNCH_B
  if (rc != MRN_OK) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

}  // namespace mrn
