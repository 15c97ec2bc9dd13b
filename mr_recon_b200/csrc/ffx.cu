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
// 1.87 ms (7.8 GB through HBM: 64% of the copy bandwidth), the inverse ones
// 1.60; passes over coil planes that crossed shared memory before the first,
// between all and after the last stage took 2.61 and 2.48 ms.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "ffx_pass.cuh"
#include "internal.cuh"

namespace mrn {

namespace {

constexpr int kFfxMaxRadix = 20;

constexpr int kRadices[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 19, 20};
// Largest radix of a middle stage; no length to 1024 needs one above 10, but without
// the instances for 11 and 12 the passes of 512 points compile to 147 us a
// Toeplitz normal (256^2, 32 coils) against 143.
constexpr int kMidMax = 12;

// Radices of n: two stages with the smallest larger radix where one exists,
// else three, else four (first and last up to 20, the middle ones up to 12);
// false if n
// has a prime factor above 19, or above 5 below kFfxConvMin points. The largest radix comes first: the
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
  int odd = n;
  for (int f : {2, 3, 5})
    while (odd % f == 0) odd /= f;
  if (odd > 1 && n < kFfxConvMin) return false;
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

// Direct radices where the length has them, else a chirp convolution.
bool ffx_axis(int n, FfxAxis& ax) { return ffx_factor(n, ax) || ffx_conv_axis(n, ax); }

// Whether an axis of a plan grid of `points` values, `least` along its shortest
// axis, is worth a native pass beside cuFFT with separate pad and crop. Times:
// forward + adjoint with 64 samples, natively and with cuFFT.
// - products of 2, 3 and 5: always.
// - factors 7 to 19: in two stages (323^2, 16 coils: 85 and 97 us; 132^3, 8
//   coils: 0.55 and 0.72 ms). A third stage at these kernels' 90 registers loses
//   (408^2, 32 coils: 272 and 203 us; 175^3, 8 coils: 2.47 and 1.79 ms) unless the
//   grid is so small that launches dominate (338^2, 1 coil: 55 and 57 us; 1001 x
//   10, 8 coils: 56 and 59).
// - chirp convolutions from 0.7 M points (326^2, 4 coils, 0.43 M: 89 and 83 us;
//   272 x 326, 7, 0.62 M: 92 and 88; 394^2, 4, 0.62 M: 94 and 101; 303^2, 8, 0.73 M:
//   107 and 137; 254^2, 32, 2.1 M: 166 and 298; 146^3, 8: 1.83 and 3.45 ms) and for slabs, a few short
//   launches either way (163 x 10, 3 coils: 61 and 59; 401 x 10: 68 and 51), where
//   the largest prime is above 31: cuFFT is fast on the smaller ones (464 = 16 x
//   29, 32 coils: 446 and 181 us; 217^3, 4 coils: 4.2 and 2.9 ms). Not for prime
//   lengths from 201 to 256: their convolutions of 480 and 512 points take
//   radices 24 and 32, which leave fewer warps an SM (227^2, 32 coils: 157 and
//   137 us; 257^2, 32: 171 and 210).
bool ffx_axis_pays(int n, int64_t points, int least) {
  FfxAxis ax;
  if (ffx_factor(n, ax)) return !ffx_has_primes(ax) || ax.ns == 2 || points < 200000;
  if ((points < 700000 && least > 20) || !ffx_conv_axis(n, ax)) return false;
  int p = 2, m = n;
  while (p * p <= m)
    if (m % p == 0) m /= p;
    else ++p;
  return m > 31 && !(m == n && n > 200 && n <= 256);
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

// Radices with a prime factor above 5: kernels of their own, whose butterflies
// need more registers (in one kernel with the others they took the 2D passes
// of 256^2, 32 coils from 83 to 107 us).
bool has_primes(const FfxAxis& ax) { return ffx_has_primes(ax); }

size_t pass_smem(const FfxAxis& ax, int w) {
  const size_t a = (size_t)(ax.n / ax.radix[0]) * ffx_block_rows(ax.radix[0]) * (w + 1);
  const size_t b = ax.ns > 2 ? (size_t)ax.n * (w + 1) : 0;
  return ((size_t)ax.n + a + b) * sizeof(float2);
}

// W = 16 columns (128-byte rows) while two CTAs' buffers fit an SM; fewer where
// that leaves SMs without work (2D, few coils).
void pass_shape(FfxStep& st, const std::vector<FfxPass>& passes, int64_t total_cols, int sm_count) {
  auto smem = [&](int w) {
    size_t m = 0;
    for (const auto& p : passes) m = std::max(m, pass_smem(p.ax, w));
    return m;
  };
  st.w = 16;
  while (st.w > 4 && (smem(st.w) > 100 * 1024 || total_cols / st.w < 2 * (int64_t)sm_count)) st.w /= 2;
  st.smem = smem(st.w);
  int most = 1;
  for (const auto& p : passes)
    for (int s = 0; s < p.ax.ns; ++s) {
      most = std::max(most, p.ax.n / p.ax.radix[s]);
      st.big |= has_primes(p.ax);
    }
  st.threads = std::min(kFfxThreads, std::max(32, (most * st.w + 31) / 32 * 32));
}

// One step of a transform. SRC / TO_IMAGE as in k_ffx_pass.
template <bool INV, int SRC, bool TO_IMAGE>
int launch_pass(const FfxSet& S, const FfxGrid& G, const FfxStep& step, const float2* src, const float2* mps,
                float2* out, float scale, cudaStream_t st) {
  if (step.conv) return launch_ffx_conv(S, G, step, INV, SRC, TO_IMAGE, src, mps, out, scale, st);
  if (step.max_cols > 0x7fffffffLL) return MRN_ERR_UNSUPPORTED;
  if (step.big) return launch_ffx_primes(S, G, step, INV, SRC, TO_IMAGE, src, mps, out, scale, st);
#define MRN_FFX_W(WW)                                                                                           \
  return step.one_pass ? launch_ffx_pass<INV, SRC, TO_IMAGE, WW, false, false>(S, G, step, src, mps, out, scale, st) \
                       : launch_ffx_pass<INV, SRC, TO_IMAGE, WW, true, false>(S, G, step, src, mps, out, scale, st)
  if (step.w == 16) MRN_FFX_W(16);
  if (step.w == 8) MRN_FFX_W(8);
  MRN_FFX_W(4);
#undef MRN_FFX_W
}

FfxGrid plan_grid(mrn_plan* P) {
  return FfxGrid{P->ndim, P->h_slices.data(), P->d_slices, P->d_apod, P->d_grid, P->sm_count};
}

}  // namespace

bool ffx_has_primes(const FfxAxis& ax) {
  for (int s = 0; s < ax.ns; ++s)
    for (int f : {7, 11, 13, 17, 19})
      if (ax.radix[s] % f == 0) return true;
  return false;
}

// Twiddles of a direct length (n - 1 entries appended to tab) and the index
// constants of its stages, for the radices' order.
void ffx_stage_tables(FfxAxis& ax, std::vector<float2>& tab) {
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

// Whether every axis of a grid has direct radices.
bool ffx_direct(int ndim, const int* nos) {
  if (ndim != 2 && ndim != 3) return false;
  FfxAxis ax;
  for (int i = 0; i < ndim; ++i)
    if (!ffx_factor(nos[i], ax)) return false;
  return true;
}

// Whether a slice of a plan grid runs the native passes: by its own grid and
// coils alone, so that it is transformed the same way (the same bits) whatever
// shares its plan.
bool ffx_pays(int ndim, const int* nos, int ncoil) {
  if (ndim != 2 && ndim != 3) return false;
  int64_t points = ncoil;
  int least = nos[0];
  for (int i = 0; i < ndim; ++i) {
    points *= nos[i];
    least = std::min(least, nos[i]);
  }
  for (int i = 0; i < ndim; ++i)
    if (!ffx_axis_pays(nos[i], points, least)) return false;
  return true;
}

// Build the native FFT of a grid buffer: per native group its axes' plans and
// tables, and per axis the lists of slices that run together. The slices of a
// group have one grid and one image size, and `cb` coils a block of their grids.
int ffx_build(FfxSet& S, int ndim, const std::vector<SliceGeom>& hsl, const std::vector<FfxGroupSpec>& spec,
              int sm_count) {
  S.release();
  if ((ndim != 2 && ndim != 3) || hsl.empty()) return MRN_OK;
  const int D = ndim;
  std::vector<float2> tab;
  int nnative = 0;
  for (const FfxGroupSpec& gs : spec) {
    FfxGroup fg{};
    fg.native = gs.native;
    fg.slices = gs.slices;
    for (int i = 0; i < D && fg.native; ++i) {
      FfxAxis& ax = fg.ax[i];
      if (!ffx_axis(hsl[gs.slices[0]].nos[i], ax)) {
        fg.native = false;
        break;
      }
      // axes of one length share their tables
      const FfxAxis* same = nullptr;
      for (const FfxGroup& o : S.grp)
        for (int k = 0; k < D; ++k)
          if (o.native && o.ax[k].n == ax.n) same = &o.ax[k];
      for (int k = 0; k < i; ++k)
        if (fg.ax[k].n == ax.n) same = &fg.ax[k];
      if (same) {
        ax = *same;
        continue;
      }
      ax.tw_base = (int)tab.size();
      if (ax.m > 0) {
        ffx_conv_tables(ax, tab);
        continue;
      }
      ffx_stage_tables(ax, tab);
    }
    nnative += fg.native ? 1 : 0;
    S.grp.push_back(fg);
  }
  if (nnative == 0) {
    S.grp.clear();
    return MRN_OK;
  }
  std::vector<FfxSlice> list;
  std::vector<FfxPass> passes;
  for (int a = 0; a < D; ++a)
    for (int kind = 0; kind < 3; ++kind) {  // direct radices up to 5, up to 19, chirp convolutions
      FfxStep st{};
      st.axis = a;
      st.conv = kind == 2;
      st.first = (int)list.size();
      const size_t p0 = passes.size();
      int64_t total = 0;
      for (const FfxGroup& fg : S.grp) {
        if (!fg.native || (fg.ax[a].m > 0 ? 2 : (int)has_primes(fg.ax[a])) != kind) continue;
        const SliceGeom& g0 = hsl[fg.slices[0]];
        FfxPass ps{};
        ps.ax = fg.ax[a];
        ps.axis = a;
        ps.n_img = g0.n[a];
        ps.pcols = ps.icells = 1;
        for (int i = 0; i < a; ++i) ps.pcols *= g0.n[i];
        for (int i = a + 1; i < D; ++i) ps.icells *= g0.nos[i];
        ps.en1 = a == 2 ? g0.n[1] : std::max(1, ps.pcols);
        ps.enos1 = a == 2 ? g0.nos[1] : 1;
        for (int narrow = 0; narrow < 2; ++narrow) {  // a group's slices by the width of their coil blocks
          bool used = false;
          ps.narrow = narrow;
          for (int s : fg.slices) {
            const int cb = hsl[s].cb;
            if ((a == D - 1 && cb < 8) != (narrow != 0)) continue;
            used = true;
            list.push_back(FfxSlice{s, (int)passes.size()});
            const int64_t cols = (int64_t)hsl[s].ncoil * ps.pcols * ps.icells;
            st.max_cols = std::max(st.max_cols, cols);
            total += cols;
          }
          if (used) passes.push_back(ps);
        }
      }
      st.nsl = (int)list.size() - st.first;
      if (st.nsl == 0) continue;
      const std::vector<FfxPass> mine(passes.begin() + p0, passes.end());
      st.one_pass = mine.size() == 1;
      st.pass = mine[0];
      if (st.conv) ffx_conv_shape(st, mine, total, sm_count);
      else pass_shape(st, mine, total, sm_count);
      S.step[a].push_back(st);
    }
  int rc = upload(&S.d_tw, tab);
  if (rc == MRN_OK) rc = upload(&S.d_list, list);
  if (rc == MRN_OK) rc = upload(&S.d_pass, passes);
  if (rc != MRN_OK) {
    S.release();
    return rc;
  }
  S.ok = true;
  S.all = nnative == (int)spec.size();
  return MRN_OK;
}

int ffx_fwd(const FfxSet& S, const FfxGrid& G, PreMode mode, const float2* src, const float2* mps, float scale,
            cudaStream_t st, int first_axis) {
  for (int a = G.ndim - 1; a >= first_axis; --a)
    for (const FfxStep& step : S.step[a]) {
      const int rc = a < G.ndim - 1 ? launch_pass<false, kFfxGrid, false>(S, G, step, nullptr, nullptr, nullptr, scale, st)
                     : mode == kPreSense
                         ? launch_pass<false, kFfxSense, false>(S, G, step, src, mps, nullptr, scale, st)
                         : launch_pass<false, kFfxImage, false>(S, G, step, src, mps, nullptr, scale, st);
      if (rc != MRN_OK) return rc;
    }
  return MRN_OK;
}

int ffx_inv(const FfxSet& S, const FfxGrid& G, float2* out, float scale, cudaStream_t st, int first_axis) {
  for (int a = first_axis; a < G.ndim; ++a)
    for (const FfxStep& step : S.step[a]) {
      const int rc = a == G.ndim - 1 && out
                         ? launch_pass<true, kFfxGrid, true>(S, G, step, nullptr, nullptr, out, scale, st)
                         : launch_pass<true, kFfxGrid, false>(S, G, step, nullptr, nullptr, nullptr, scale, st);
      if (rc != MRN_OK) return rc;
    }
  return MRN_OK;
}

bool ffx_active(const mrn_plan* P) { return P->ffx.ok && P->use_ffx; }

// Coils per block of a slice's native grid: coil_block, or (no room for partly
// filled blocks) the widest that the coils fill.
static int native_block(const mrn_plan* P, int ncoil) {
  int cb = coil_block(ncoil);
  while (P->tight_grid && ncoil % cb != 0) cb /= 2;
  return cb;
}

// Lay the slices' grids out in d_grid, group by group: native groups in coil
// blocks, centred, each slice from a multiple of 8 elements on (the
// interpolation copies 16 bytes at a time, and the grids before it may have
// any number of points); the others as coil planes in FFT order, back to back
// for one batched cuFFT call. Returns the elements that takes.
static int64_t place_grids(mrn_plan* P, bool use_native) {
  int64_t off = 0;
  for (size_t q = 0; q < P->fft.size(); ++q) {
    auto& fg = P->fft[q];
    const bool native = use_native && P->ffx.ok && P->ffx.grp[q].native;
    off = (off + 7) / 8 * 8;
    fg.grid_off = off;
    for (int s : fg.slices) {
      SliceGeom& g = P->h_slices[s];
      g.native_fft = native ? 1 : 0;
      g.cb = native ? native_block(P, g.ncoil) : 1;
      for (int i = 0; i < P->ndim; ++i) g.hshift[i] = native ? 0 : g.nos[i] / 2;
      if (native) off = (off + 7) / 8 * 8;
      g.grid_off = off;
      off += (int64_t)((g.ncoil + g.cb - 1) / g.cb) * g.cb * g.gos;
    }
  }
  return off;
}

int ffx_refresh(mrn_plan* P) {
  if (P->fft.empty() || !P->d_slices) return MRN_OK;
  place_grids(P, P->use_ffx);
  return upload_slices(P) == cudaSuccess ? MRN_OK : MRN_ERR_CUDA;
}

// The plan grid's native FFT (plan creation, after the FFT groups exist).
int ffx_setup(mrn_plan* P) {
  P->ffx.release();
  if (P->flags & MRN_PLAN_RAW) return MRN_OK;
  for (SliceGeom& g : P->h_slices) g.cb = native_block(P, g.ncoil);
  std::vector<FfxGroupSpec> spec;
  for (const auto& f : P->fft) spec.push_back(FfxGroupSpec{f.native, f.slices});
  const int rc = ffx_build(P->ffx, P->ndim, P->h_slices, spec, P->sm_count);
  if (rc != MRN_OK) return rc;
  // room for either value of MRN_OPT_NATIVE_FFT
  P->n_igrid = place_grids(P, false);
  P->n_igrid = std::max(P->n_igrid, place_grids(P, true));
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
