// Toeplitz (FFT-only) normal operator A^H A of the NUFFT: the kernel K is the
// centred FFT of the point-spread function on a padded grid (normally twice
// the image size), and
//   normal(x)_c = crop(IFFT(K * FFT(pad(x_c))))           (plain, per image)
//   normal(x)   = sum_c conj(S_c) crop(IFFT(K * FFT(pad(S_c x))))   (SENSE)
// with centred orthonormal FFTs (ifftshift -> fftn -> fftshift) and the
// centred pad / crop of PadLast.
//
// Reference: NUFFT.normal_toeplitz (fourier.py:302-352), the Toeplitz branch
// of sense_linop.normal (linops.py:1249-1308) and calc_teoplitz_kernels
// (fourier.py:552-582), which pad, FFT, multiply, inverse-FFT and crop with
// separate torch passes (and for SENSE an einsum over coils). Here the pad,
// the coil-map product and both shifts are index maps of one pre kernel:
// padded FFT storage cell s (per dimension) holds centred cell
// p = (s + np//2) mod np, i.e. image cell q = p - (np - n)/2; the kernel is
// reordered to storage order once, with the orthonormal scaling 1/prod(np) of
// the two FFTs folded in; the crop, conj(coil-map) sum, lambda x and
// Re<x, out> are one post kernel. cuFFT does the two batched transforms.
//
// 2D and 3D slices whose padded sizes have direct radices (ffx.cu) skip all of
// that but the last kernel: the native passes pad and crop, the turning pass
// (ffxturn.cu) does the first axis both ways with the product in between, and
// the grid holds coil blocks with the kernel in centred order. Only image rows
// cross memory, a quarter (2D) of the traffic of the padded grids.
// Each slice takes its form by its own padded sizes, so its bits do not depend
// on the other slices of the plan.
// Measured (256^2 image, 512^2 grid, 32 coils, SENSE normal): 143 us, cuFFT
// with separate pad, product and crop 160.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace mrn {

// per slice: padded grid geometry of the Toeplitz operator
struct ToepGeom {
  int n[kMaxDim];    // image size (1 for unused dims)
  int np[kMaxDim];   // padded (FFT) size
  int off[kMaxDim];  // (np - n) / 2, the centred pad offset
  int ncoil;
  int native;        // by the native passes: grid in coil blocks, kernel in centred order
  int64_t gp;        // prod(np)
  int64_t grid_off;  // complex offset of the slice's block in the Toeplitz grid ([C][np...] for cuFFT)
  int64_t kern_off;  // complex offset of the slice's kernel (scaled)
  int64_t img_off;   // image layout [C][N...] offset (plain mode input/output, SENSE maps)
  int64_t x_off;     // one-image-per-slice offset (SENSE x / out)
  int64_t nimg;      // prod(n)
  int64_t prow_off;  // first padded row (all dims but the last, all coils) of the cuFFT slices'
  int64_t irow_off;  // first image row, all coils, of the cuFFT slices'
};

struct ToepState {
  std::vector<ToepGeom> h;  // every slice
  ToepGeom* d = nullptr;
  float2* grid = nullptr;  // padded grids
  float2* kern = nullptr;  // kernels, scaled by 1 / prod(np)
  int64_t n_kern = 0;
  bool use_ffx = false;  // the plan's MRN_OPT_NATIVE_FFT when the state was built
  // every slice on its padded grid, as the native passes and the coil sum read it
  std::vector<SliceGeom> hsl;
  SliceGeom* dsl = nullptr;
  float* ones = nullptr;  // their apodization
  // slices by the native passes
  FfxSet ffx;
  FfxTurnSet turn;
  // slices by cuFFT, one batched plan per padded size
  std::vector<ToepGeom> hc;
  ToepGeom* dc = nullptr;
  int64_t n_prow = 0, n_irow = 0;  // their padded rows and image rows
  struct Group {
    int np[kMaxDim];
    int64_t grid_off;
    int batch;
    cufftHandle handle;
  };
  std::vector<Group> fft;
};

__device__ __forceinline__ int toep_slice(const ToepGeom* g, int ns, int64_t row, int which) {
  int lo = 0, hi = ns - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int64_t o = which == 0 ? g[mid].prow_off : g[mid].irow_off;
    if (o <= row) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One warp per padded row (all dims but the last) of one coil of one slice:
// grid[c][s] = pad(x_c)[p(s)] (plain) or pad(S_c x)[p(s)] (SENSE).
template <int D>
__global__ void __launch_bounds__(256)
k_toep_pre(const ToepGeom* __restrict__ tg, int ns, const float2* __restrict__ src,
           const float2* __restrict__ mps, float2* __restrict__ grid, int64_t nrows) {
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= nrows) return;
  const ToepGeom& g = tg[toep_slice(tg, ns, row, 0)];
  const int64_t r = row - g.prow_off;
  const int64_t outer = g.gp / g.np[D - 1];
  const int c = (int)(r / outer);
  int64_t o = r - (int64_t)c * outer;
  const int64_t orow = o;
  bool valid = true;
  int64_t qlin = 0;
  int st[kMaxDim] = {0, 0, 0};
  for (int i = D - 2; i >= 0; --i) {
    st[i] = (int)(o % g.np[i]);
    o /= g.np[i];
  }
  for (int i = 0; i < D - 1; ++i) {
    int p = st[i] + g.np[i] / 2;
    if (p >= g.np[i]) p -= g.np[i];
    const int q = p - g.off[i];
    valid &= q >= 0 && q < g.n[i];
    qlin = qlin * g.n[i] + q;
  }
  const int nl = g.n[D - 1], npl = g.np[D - 1], offl = g.off[D - 1], hl = npl / 2;
  float2* dst = grid + g.grid_off + (int64_t)c * g.gp + orow * npl;
  if (!valid) {
    for (int j = lane; j < npl; j += 32) dst[j] = make_float2(0.f, 0.f);
    return;
  }
  qlin *= nl;
  const float2* srow = mps ? src + g.x_off + qlin : src + g.img_off + (int64_t)c * g.nimg + qlin;
  const float2* mrow = mps ? mps + g.img_off + (int64_t)c * g.nimg + qlin : nullptr;
#pragma unroll 4
  for (int j = lane; j < npl; j += 32) {
    int p = j + hl;
    if (p >= npl) p -= npl;
    const int q = p - offl;
    float2 v = make_float2(0.f, 0.f);
    if (q >= 0 && q < nl) {
      v = __ldg(srow + q);
      if (mrow) {
        const float2 m = __ldg(mrow + q);
        v = make_float2(v.x * m.x - v.y * m.y, v.x * m.y + v.y * m.x);
      }
    }
    dst[j] = v;
  }
}

// grid[c][s] *= kern[s] for every coil of slice blockIdx.y (storage order).
__global__ void __launch_bounds__(256)
k_toep_mul(const ToepGeom* __restrict__ tg, const float2* __restrict__ kern, float2* __restrict__ grid) {
  const ToepGeom& g = tg[blockIdx.y];
  const int64_t total = (int64_t)g.ncoil * g.gp;
  float2* gs = grid + g.grid_off;
  const float2* ks = kern + g.kern_off;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = e % g.gp;
    const float2 k = __ldg(ks + j);
    const float2 v = gs[e];
    gs[e] = make_float2(v.x * k.x - v.y * k.y, v.x * k.y + v.y * k.x);
  }
}

// Scale a centred kernel (caller layout, per slice [np...]) and reorder that of
// a cuFFT slice into FFT storage order: kern[s] = src[p(s)] * scale.
template <int D>
__global__ void k_toep_kernel(const ToepGeom* __restrict__ tg, int ns, const float2* __restrict__ src,
                              float2* __restrict__ kern, int64_t total) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  int lo = 0, hi = ns - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tg[mid].kern_off <= e) lo = mid; else hi = mid - 1;
  }
  const ToepGeom& g = tg[lo];
  int64_t rem = e - g.kern_off;
  int64_t plin = 0;
  int s[kMaxDim] = {0, 0, 0};
  for (int i = D - 1; i >= 0; --i) {
    s[i] = (int)(rem % g.np[i]);
    rem /= g.np[i];
  }
  for (int i = 0; i < D; ++i) {
    int p = s[i] + g.np[i] / 2;
    if (p >= g.np[i]) p -= g.np[i];
    plin = plin * g.np[i] + p;
  }
  const float2 v = src[g.native ? e : g.kern_off + plin];
  const float sc = 1.0f / (float)g.gp;
  kern[e] = make_float2(v.x * sc, v.y * sc);
}

// Plain output of the cuFFT slices, one warp per image row: out[c][q] = grid[c][s(q)].
template <int D>
__global__ void __launch_bounds__(256)
k_toep_post(const ToepGeom* __restrict__ tg, int ns, const float2* __restrict__ grid, float2* __restrict__ out,
            int64_t nrows) {
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= nrows) return;
  const ToepGeom& g = tg[toep_slice(tg, ns, row, 1)];
  const int64_t r = row - g.irow_off;
  const int64_t outer = g.nimg / g.n[D - 1];
  const int c = (int)(r / outer);
  int64_t o = r - (int64_t)c * outer;
  const int64_t orow = o;
  int q[kMaxDim] = {0, 0, 0};
  for (int i = D - 2; i >= 0; --i) {
    q[i] = (int)(o % g.n[i]);
    o /= g.n[i];
  }
  int64_t slin = 0;
  for (int i = 0; i < D - 1; ++i) {
    int s = q[i] + g.off[i] - g.np[i] / 2;
    if (s < 0) s += g.np[i];
    slin = slin * g.np[i] + s;
  }
  const int nl = g.n[D - 1], npl = g.np[D - 1], sh = g.off[D - 1] - npl / 2;
  const float2* yrow = grid + g.grid_off + (int64_t)c * g.gp + slin * npl;
  float2* orow_p = out + g.img_off + (int64_t)c * g.nimg + orow * nl;
  for (int j = lane; j < nl; j += 32) {
    int s = j + sh;
    if (s < 0) s += npl;
    orow_p[j] = yrow[s];
  }
}

static ToepState* toep(mrn_plan* P) { return static_cast<ToepState*>(P->toep); }

void toep_free(mrn_plan* P) {
  ToepState* T = toep(P);
  if (!T) return;
  for (auto& fg : T->fft)
    if (fg.handle) cufftDestroy(fg.handle);
  if (T->d) cudaFree(T->d);
  if (T->dc) cudaFree(T->dc);
  if (T->grid) cudaFree(T->grid);
  if (T->kern) cudaFree(T->kern);
  if (T->dsl) cudaFree(T->dsl);
  if (T->ones) cudaFree(T->ones);
  T->ffx.release();
  T->turn.release();
  delete T;
  P->toep = nullptr;
}

}  // namespace mrn

using namespace mrn;

#define CKT(x)                                   \
  do {                                           \
    cudaError_t _e = (x);                        \
    if (_e != cudaSuccess) return cuda_fail(_e); \
  } while (0)
#define RK(x)                    \
  do {                           \
    int _r = (x);                \
    if (_r != MRN_OK) return _r; \
  } while (0)

namespace mrn {

// The slices by their form (native: allow the native passes), their grids and
// what transforms them.
static int toep_build(mrn_plan* P, ToepState* T, bool native) {
  const int D = P->ndim;
  T->hsl = P->h_slices;
  std::vector<FfxGroupSpec> spec;
  std::vector<int64_t> kern_off;
  int64_t off = 0;
  int longest = 1;
  for (int s = 0; s < P->nslices; ++s) {
    SliceGeom& g = T->hsl[s];
    ToepGeom& t = T->h[s];
    t.native = native && ffx_direct(D, t.np);
    for (int i = 0; i < kMaxDim; ++i) {
      g.nos[i] = t.np[i];
      g.hshift[i] = 0;
      g.apod_off[i] = 0;
      longest = std::max(longest, t.n[i]);
    }
    g.gos = t.gp;
    g.native_fft = t.native;
    g.cb = t.native ? coil_block(g.ncoil) : 1;
    g.inv_sqrt_n = 1.0f;
    kern_off.push_back(t.kern_off);
    if (!t.native) continue;
    FfxGroupSpec* gs = nullptr;  // slices of one padded and one image size
    for (auto& o : spec) {
      const SliceGeom& f = T->hsl[o.slices[0]];
      bool eq = true;
      for (int i = 0; i < D; ++i) eq &= f.nos[i] == g.nos[i] && f.n[i] == g.n[i];
      if (eq) gs = &o;
    }
    if (gs) gs->slices.push_back(s);
    else spec.push_back(FfxGroupSpec{true, {s}});
    g.grid_off = off;
    off += (int64_t)((g.ncoil + g.cb - 1) / g.cb) * g.cb * t.gp;
  }
  // then the cuFFT slices' planes, the slices of one padded size back to back
  for (int s = 0; s < P->nslices; ++s) {
    const ToepGeom& t = T->h[s];
    if (t.native) continue;
    bool found = false;
    for (const auto& fg : T->fft) found |= std::equal(fg.np, fg.np + kMaxDim, t.np);
    if (found) continue;
    ToepState::Group fg{};
    std::copy(t.np, t.np + kMaxDim, fg.np);
    fg.grid_off = off;
    for (int k = s; k < P->nslices; ++k) {
      ToepGeom& o = T->h[k];
      if (o.native || !std::equal(fg.np, fg.np + kMaxDim, o.np)) continue;
      o.grid_off = T->hsl[k].grid_off = off;
      off += (int64_t)o.ncoil * o.gp;
      fg.batch += o.ncoil;
    }
    T->fft.push_back(fg);
  }
  for (ToepGeom& t : T->h) {
    if (t.native) continue;
    t.prow_off = T->n_prow;
    t.irow_off = T->n_irow;
    T->n_prow += (int64_t)t.ncoil * t.gp / t.np[D - 1];
    T->n_irow += (int64_t)t.ncoil * t.nimg / t.n[D - 1];
    T->hc.push_back(t);
  }
  const std::vector<float> ones(longest, 1.0f);
  const size_t tb = T->h.size() * sizeof(ToepGeom), sb = T->hsl.size() * sizeof(SliceGeom);
  CKT(cudaMalloc(&T->grid, std::max<int64_t>(off, 1) * sizeof(float2)));
  if (!spec.empty()) {
    RK(ffx_build(T->ffx, D, T->hsl, spec, P->sm_count));
    if (!T->ffx.all) return MRN_ERR_UNSUPPORTED;
    RK(ffx_turn_build(T->turn, T->ffx, D, T->hsl, kern_off, P->sm_count));
  }
  CKT(cudaMalloc(&T->d, tb));
  CKT(cudaMalloc(&T->dc, tb));
  CKT(cudaMalloc(&T->dsl, sb));
  CKT(cudaMalloc(&T->ones, longest * sizeof(float)));
  CKT(cudaMalloc(&T->kern, std::max<int64_t>(T->n_kern, 1) * sizeof(float2)));
  CKT(cudaMemcpy(T->d, T->h.data(), tb, cudaMemcpyHostToDevice));
  if (!T->hc.empty()) CKT(cudaMemcpy(T->dc, T->hc.data(), T->hc.size() * sizeof(ToepGeom), cudaMemcpyHostToDevice));
  CKT(cudaMemcpy(T->dsl, T->hsl.data(), sb, cudaMemcpyHostToDevice));
  CKT(cudaMemcpy(T->ones, ones.data(), longest * sizeof(float), cudaMemcpyHostToDevice));
  for (auto& fg : T->fft) {
    int n[kMaxDim];
    for (int i = 0; i < D; ++i) n[i] = fg.np[i];
    if (cufftPlanMany(&fg.handle, D, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_C2C, fg.batch) != CUFFT_SUCCESS) {
      fg.handle = 0;
      return MRN_ERR_CUFFT;
    }
  }
  return MRN_OK;
}

}  // namespace mrn

extern "C" {

int mrn_plan_set_toeplitz(mrn_plan* P, const int* pad_size, const void* kern, void* stream) {
  if (!P || !pad_size || !kern || (P->flags & MRN_PLAN_RAW)) return MRN_ERR_ARG;
  const int D = P->ndim;
  cudaStream_t st = (cudaStream_t)stream;
  for (int s = 0; s < P->nslices; ++s)
    for (int i = 0; i < D; ++i) {
      const int np = pad_size[s * D + i], n = P->h_slices[s].n[i];
      // PadLast pads (np - n) / 2 on both sides: np - n must be even
      if (np < n || ((np - n) & 1)) return MRN_ERR_ARG;
    }
  // same padded sizes and FFT option as before: keep buffers and FFT plans, refresh the kernel
  ToepState* T = toep(P);
  bool same = T != nullptr && T->use_ffx == P->use_ffx;
  if (same)
    for (int s = 0; s < P->nslices && same; ++s)
      for (int i = 0; i < D; ++i) same &= T->h[s].np[i] == pad_size[s * D + i];
  if (!same) {
    CKT(cudaSetDevice(P->device));
    int rc = MRN_OK;
    // without room for the coil blocks (up to 8/5 of the planes) every slice takes cuFFT
    for (int native = P->use_ffx ? 1 : 0; native >= 0; --native) {
      toep_free(P);
      T = new ToepState();
      P->toep = T;
      T->use_ffx = P->use_ffx;
      T->h.resize(P->nslices);
      int64_t koff = 0;
      for (int s = 0; s < P->nslices; ++s) {
        const SliceGeom& g = P->h_slices[s];
        ToepGeom& t = T->h[s];
        int64_t gp = 1;
        for (int i = 0; i < kMaxDim; ++i) {
          t.n[i] = i < D ? g.n[i] : 1;
          t.np[i] = i < D ? pad_size[s * D + i] : 1;
          t.off[i] = (t.np[i] - t.n[i]) / 2;
          gp *= t.np[i];
        }
        t.ncoil = g.ncoil;
        t.gp = gp;
        t.kern_off = koff;
        t.img_off = g.img_off;
        t.x_off = g.x_off;
        t.nimg = g.nimg;
        koff += gp;
      }
      T->n_kern = koff;
      rc = toep_build(P, T, native != 0);
      if (rc == MRN_OK) break;
      toep_free(P);  // nothing half built stays bound
      cudaGetLastError();
    }
    if (rc != MRN_OK) return rc;
  }
  const unsigned nb = (unsigned)((T->n_kern + 255) / 256);
  if (D == 1) k_toep_kernel<1><<<nb, 256, 0, st>>>(T->d, P->nslices, (const float2*)kern, T->kern, T->n_kern);
  else if (D == 2) k_toep_kernel<2><<<nb, 256, 0, st>>>(T->d, P->nslices, (const float2*)kern, T->kern, T->n_kern);
  else k_toep_kernel<3><<<nb, 256, 0, st>>>(T->d, P->nslices, (const float2*)kern, T->kern, T->n_kern);
  CKT(cudaGetLastError());
  return MRN_OK;
}

}  // extern "C"

namespace mrn {

// Per form pre (pad, optional coil-map product) -> FFT -> x K -> inverse FFT, then post.
static int toep_apply(mrn_plan* P, const float2* src, const float2* mps, float2* out, float scale,
                      const float2* xin, float lam, double* pap, int pap_stride, cudaStream_t st) {
  ToepState* T = toep(P);
  if (!T) return MRN_ERR_STATE;
  const int D = P->ndim, nc = (int)T->hc.size();
  if (T->ffx.ok) {
    const FfxGrid G{D, T->hsl.data(), T->dsl, T->ones, T->grid, P->sm_count};
    StageTimer t(P, kStageFft, st);
    RK(ffx_fwd(T->ffx, G, mps ? kPreSense : kPrePlain, src, mps, 1.0f, st, 1));
    RK(ffx_turn(T->turn, G, T->kern, st));
    RK(ffx_inv(T->ffx, G, mps ? nullptr : out, 1.0f, st, 1));
  }
  if (nc > 0) {
    {
      StageTimer t(P, kStagePre, st);
      const unsigned nb = (unsigned)((T->n_prow + 7) / 8);
      if (D == 1) k_toep_pre<1><<<nb, 256, 0, st>>>(T->dc, nc, src, mps, T->grid, T->n_prow);
      else if (D == 2) k_toep_pre<2><<<nb, 256, 0, st>>>(T->dc, nc, src, mps, T->grid, T->n_prow);
      else k_toep_pre<3><<<nb, 256, 0, st>>>(T->dc, nc, src, mps, T->grid, T->n_prow);
      CKT(cudaGetLastError());
    }
    StageTimer t(P, kStageFft, st);
    for (auto& fg : T->fft) {
      if (cufftSetStream(fg.handle, st) != CUFFT_SUCCESS) return MRN_ERR_CUFFT;
      cufftComplex* p = reinterpret_cast<cufftComplex*>(T->grid + fg.grid_off);
      if (cufftExecC2C(fg.handle, p, p, CUFFT_FORWARD) != CUFFT_SUCCESS) return MRN_ERR_CUFFT;
    }
    int64_t most = 1;
    for (const auto& t : T->hc) most = std::max<int64_t>(most, (int64_t)t.ncoil * t.gp);
    const unsigned nb = (unsigned)std::max<int64_t>(1, std::min<int64_t>((most + 255) / 256,
                                                                        (8 * (int64_t)P->sm_count + nc - 1) / nc));
    k_toep_mul<<<dim3(nb, (unsigned)nc), 256, 0, st>>>(T->dc, T->kern, T->grid);
    CKT(cudaGetLastError());
    for (auto& fg : T->fft) {
      cufftComplex* p = reinterpret_cast<cufftComplex*>(T->grid + fg.grid_off);
      if (cufftExecC2C(fg.handle, p, p, CUFFT_INVERSE) != CUFFT_SUCCESS) return MRN_ERR_CUFFT;
    }
  }
  if (!mps && nc == 0) return MRN_OK;  // the native inverse passes wrote the images
  StageTimer t(P, kStagePost, st);
  if (mps)
    return launch_post_sense(P, T->dsl, T->ones, T->grid, mps, out, scale, xin, lam, pap, pap_stride, P->d_sync + 3, st);
  const unsigned nb = (unsigned)((T->n_irow + 7) / 8);
  if (nb == 0) return MRN_OK;
  if (D == 1) k_toep_post<1><<<nb, 256, 0, st>>>(T->dc, nc, T->grid, out, T->n_irow);
  else if (D == 2) k_toep_post<2><<<nb, 256, 0, st>>>(T->dc, nc, T->grid, out, T->n_irow);
  else k_toep_post<3><<<nb, 256, 0, st>>>(T->dc, nc, T->grid, out, T->n_irow);
  CKT(cudaGetLastError());
  return MRN_OK;
}

}  // namespace mrn

extern "C" {

int mrn_toeplitz_normal(mrn_plan* P, const void* img, void* out, void* stream) {
  if (!P || !img || !out) return MRN_ERR_ARG;
  return toep_apply(P, (const float2*)img, nullptr, (float2*)out, 1.0f, nullptr, 0.f, nullptr, 0,
                    (cudaStream_t)stream);
}

int mrn_sense_normal_toeplitz(mrn_plan* P, const void* x, const void* mps, void* out, float out_scale,
                              float lam, double* pap, int pap_stride, void* stream) {
  if (!P || !x || !mps || !out) return MRN_ERR_ARG;
  return toep_apply(P, (const float2*)x, (const float2*)mps, (float2*)out, out_scale, (const float2*)x,
                    lam, pap, pap_stride, (cudaStream_t)stream);
}

}  // extern "C"
