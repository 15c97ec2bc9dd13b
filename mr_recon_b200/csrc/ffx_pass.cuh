// The direct pass of the native FFT (ffx.cu, ffxprime.cu).
#pragma once

#include "ffx_dft.cuh"

namespace mrn {

constexpr int kFfxThreads = 512;  // most threads of a pass' CTA

// One pass: a CTA per (slice of the list blockIdx.y, W adjacent columns); with
// LIST the slices have passes of their own, one launch for all of a plan's
// grid sizes. Lanes run across columns (one 128-byte
// segment per row for W = 16) except where the other side is the planar image
// or a grid of few coils, whose contiguous direction is the axis itself.
template <bool INV, int SRC, bool TO_IMAGE, int W, bool LIST, bool PRIMES>
__global__ void __launch_bounds__(kFfxThreads)
k_ffx_pass(const SliceGeom* __restrict__ sl, const FfxSlice* __restrict__ list, const FfxPass* __restrict__ passes,
           const __grid_constant__ FfxPass ps0, const float2* __restrict__ twg,
           float2* __restrict__ grid, const float* __restrict__ apod, const float2* __restrict__ src,
           const float2* __restrict__ mps, float scale, float2* __restrict__ out) {
  constexpr bool LAST = SRC != kFfxGrid || TO_IMAGE;  // the last axis, against the image
  constexpr int WS = W + 1;                           // odd column stride: no bank conflicts either way
  extern __shared__ float2 fsm[];
  __shared__ FfxCols<W> cols;
  __shared__ FfxPass s_ps;
  const FfxSlice fs = LIST ? list[blockIdx.y] : FfxSlice{0, 0};
  if (LIST) {
    const int* from = reinterpret_cast<const int*>(passes + fs.pass);
    for (int i = threadIdx.x; i < (int)(sizeof(FfxPass) / sizeof(int)); i += blockDim.x)
      reinterpret_cast<int*>(&s_ps)[i] = from[i];
    __syncthreads();
  }
  const FfxPass& ps = LIST ? s_ps : ps0;
  const SliceGeom& g = sl[LIST ? fs.slice : list[blockIdx.y].slice];
  const int cb = g.cb, inner = ps.icells * cb;
  const int ncols = g.ncoil * ps.pcols * ps.icells;
  const int f0 = blockIdx.x * W;
  if (f0 >= ncols) return;
  const int n = ps.ax.n, tid = threadIdx.x, nt = blockDim.x;
  const int R0 = ps.ax.radix[0], ns = ps.ax.ns;
  const int r0s = ffx_block_rows(R0);  // odd row stride of the first stage's blocks
  float2* tw = fsm;
  float2* A = fsm + n;
  float2* B = A + (size_t)(n / R0) * r0s * WS;  // used from three stages on
  for (int i = tid; i < n - 1; i += nt) tw[i] = twg[ps.ax.tw_base + i];
  ffx_columns<W, LAST, SRC == kFfxSense>(cols, g, ps, n, f0, ncols, apod, scale);
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
      if (SRC != kFfxGrid || ps.narrow) {
        w = nr == 1 ? idx : (int)__umulhi((unsigned)idx, ps.ax.mag_nr[0]);
        b = idx - w * nr;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = cols.base[w];
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
        const float2* ip = src + cols.img[w];
        const float2* mp = SRC == kFfxSense ? mps + cols.map[w] : nullptr;
        const float a0 = cols.a[w];
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
  auto middle = [&](auto rc, const float2* a, float2* d, int s, int L, int rs) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R;
    const int tstep = nr / L * rs;  // rs: rows of a block of L points
    const float2* tws = tw + ps.ax.tw_off[s];
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int k = (int)__umulhi((unsigned)b, ps.ax.mag_l[s]), j = b - k * L;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(k * rs + j + t * tstep) * WS + w];
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
      if (TO_IMAGE || ps.narrow) {
        w = nr == 1 ? idx : (int)__umulhi((unsigned)idx, ps.ax.mag_nr[s]);
        b = idx - w * nr;
      } else {
        b = idx / W;
        w = idx - b * W;
      }
      const int64_t base = cols.base[w];
      if (base < 0) continue;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(b + t * row_stride) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<INV>(x[t], tws[b * (R - 1) + t - 1]);
      dft<R, INV>(x);
      if (TO_IMAGE) {
        float2* op = out + cols.img[w];
        const float a0 = cols.a[w];
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
#define MRN_FFX_CASE(N, CALL) case N: { std::integral_constant<int, N> rc; CALL; } break;
#define MRN_FFX_RADIX(R_, CALL)                                                            \
  if constexpr (PRIMES) {                                                                  \
    switch (R_) {                                                                          \
      MRN_FFX_CASE(2, CALL) MRN_FFX_CASE(3, CALL) MRN_FFX_CASE(4, CALL) MRN_FFX_CASE(5, CALL) \
      MRN_FFX_CASE(6, CALL) MRN_FFX_CASE(7, CALL) MRN_FFX_CASE(8, CALL) MRN_FFX_CASE(9, CALL) \
      MRN_FFX_CASE(10, CALL) MRN_FFX_CASE(11, CALL) MRN_FFX_CASE(12, CALL) MRN_FFX_CASE(13, CALL) \
      MRN_FFX_CASE(14, CALL) MRN_FFX_CASE(15, CALL) MRN_FFX_CASE(16, CALL) MRN_FFX_CASE(17, CALL) \
      MRN_FFX_CASE(19, CALL)                                                               \
      default: { std::integral_constant<int, 20> rc; CALL; } break;                        \
    }                                                                                      \
  } else {                                                                                 \
    switch (R_) {                                                                          \
      MRN_FFX_CASE(1, CALL) MRN_FFX_CASE(2, CALL) MRN_FFX_CASE(3, CALL) MRN_FFX_CASE(4, CALL) \
      MRN_FFX_CASE(5, CALL) MRN_FFX_CASE(6, CALL) MRN_FFX_CASE(8, CALL) MRN_FFX_CASE(9, CALL) \
      MRN_FFX_CASE(10, CALL) MRN_FFX_CASE(12, CALL) MRN_FFX_CASE(15, CALL) MRN_FFX_CASE(16, CALL) \
      default: { std::integral_constant<int, 20> rc; CALL; } break;                        \
    }                                                                                      \
  }
  MRN_FFX_RADIX(R0, first(rc))
  __syncthreads();
  int L = R0;
#pragma unroll 1
  for (int s = 1; s + 1 < ns; ++s) {
    const int R = ps.ax.radix[s];
    // radices above 12 come in two-stage lengths or first and last
    switch (R) {
      case 2: middle(std::integral_constant<int, 2>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 3: middle(std::integral_constant<int, 3>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 4: middle(std::integral_constant<int, 4>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 5: middle(std::integral_constant<int, 5>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 6: middle(std::integral_constant<int, 6>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 7:
        if constexpr (PRIMES) middle(std::integral_constant<int, 7>(), A, B, s, L, s == 1 ? r0s : L);
        break;
      case 11:
        if constexpr (PRIMES) middle(std::integral_constant<int, 11>(), A, B, s, L, s == 1 ? r0s : L);
        break;
      case 8: middle(std::integral_constant<int, 8>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 9: middle(std::integral_constant<int, 9>(), A, B, s, L, s == 1 ? r0s : L); break;
      case 10: middle(std::integral_constant<int, 10>(), A, B, s, L, s == 1 ? r0s : L); break;
      default: middle(std::integral_constant<int, 12>(), A, B, s, L, s == 1 ? r0s : L); break;
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

#undef MRN_FFX_RADIX
#undef MRN_FFX_CASE

// One step of a transform: its slices' passes in one launch.
template <bool INV, int SRC, bool TO_IMAGE, int W, bool LIST, bool PRIMES>
int launch_ffx_pass(const FfxSet& S, const FfxGrid& G, const FfxStep& step, const float2* src, const float2* mps,
                    float2* out, float scale, cudaStream_t st) {
  const unsigned nb = (unsigned)((step.max_cols + W - 1) / W);
  auto kern = k_ffx_pass<INV, SRC, TO_IMAGE, W, LIST, PRIMES>;
  const int rc = set_dynamic_smem(kern, step.smem);
  if (rc != MRN_OK) return rc;
  // image and coil map take 94 registers a thread: above 320 threads one CTA
  // would hold the SM alone
  const int threads = SRC == kFfxSense && step.threads > 320 ? 256 : step.threads;
  for (int s0 = 0; s0 < step.nsl; s0 += 65535)
    kern<<<dim3(nb, (unsigned)std::min(65535, step.nsl - s0)), threads, step.smem, st>>>(
        G.dsl, S.d_list + step.first + s0, S.d_pass, step.pass, S.d_tw, G.grid, G.apod, src, mps, scale, out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

}  // namespace mrn
