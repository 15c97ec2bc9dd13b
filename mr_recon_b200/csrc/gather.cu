// Type-2 interpolation (grid -> samples) straight from a grid in coil blocks
// ([coil block][cell][cb], grid_at): the default path of launch_interp for
// 2D / 3D kernels of 5..8 candidate taps, for the slices whose grids the native
// FFT passes transform, and for one-coil caller grids.
//
// Reference: triton_interp/ungrid.py (_ungrid2d / _ungrid3d, :200-495). Tap
// selection and weights are the reference's: taps j = lo + q, lo = ceil(u -
// W/2), valid iff |(float)j - u| <= W/2 in float32 (kernels.py:268-393),
// weight = prod_d KB(|j_d - u_d| / (W/2)), circular cells.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.cuh"
#include "tile_util.cuh"

namespace mrn {

namespace {

constexpr int kGatherWarps = 8;  // most warps per CTA
constexpr int kGatherChunk = 128;
// CTAs per SM: four (64 registers) for 3D kernels of up to 6 candidate taps,
// two (128) where more taps are in flight per row (3D, 192^3, 16 coils, W 4:
// 3.31 ms with four, 3.52 with three, 3.86 with two; 120^3, 12 coils, W 6:
// 2.55 with four, 2.46 with two; 2D one-coil: 17 us with four, 15 with two).
__host__ __device__ constexpr int gather_occ(int d, int k) { return d == 3 && k <= 6 ? 4 : 2; }

constexpr int gather_stride(int d) { return d == 3 ? 24 : 20; }  // floats of weights kept per sample

// Row pointers step by the outer strides, the KE taps of a row sit at
// compile-time offsets: one 64-bit add per row and one load and one packed
// FMA per tap. w: the axes' weights, 8 floats each.
template <int D, int KE, int CB>
__device__ __forceinline__ float2 gather_fast(const float2* gp, int64_t sx, int64_t sy, const float* __restrict__ w) {
  float wx[KE], wy[KE];
  float2 wz[KE];
#pragma unroll
  for (int c = 0; c < KE; ++c) {
    wx[c] = w[c];
    wy[c] = D == 3 ? w[8 + c] : 0.f;
    const float v = w[8 * (D - 1) + c];
    wz[c] = make_float2(v, v);
  }
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll
  for (int a = 0; a < KE; ++a) {
    float2 pa = make_float2(0.f, 0.f);
    if (D == 2) {
#pragma unroll
      for (int c = 0; c < KE; ++c) pa = __ffma2_rn(wz[c], __ldg(gp + c * CB), pa);
    } else {
      const float2* rp = gp;
#pragma unroll
      for (int b = 0; b < KE; ++b) {
        float2 ra = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < KE; ++c) ra = __ffma2_rn(wz[c], __ldg(rp + c * CB), ra);
        pa = __ffma2_rn(make_float2(wy[b], wy[b]), ra, pa);
        rp += sy;
      }
    }
    acc = __ffma2_rn(make_float2(wx[a], wx[a]), pa, acc);
    gp += sx;
  }
  return acc;
}

// With circular wrap: samples at the grid's edge, or (whole widths, window_taps)
// with a coordinate exactly W/2 from their K-th candidate tap, which the others
// leave out. Out of line, so its index arithmetic is not hoisted into every sample.
template <int D, int K, int CB>
__device__ __noinline__ float2 gather_wrap(const float2* g, int64_t cell, int n0, int n1, int n2, const float* w) {
  float2 acc = make_float2(0.f, 0.f);
  const int nl = D == 3 ? n2 : n1;
  const int sl = (int)(cell % nl);
  const int64_t r = cell / nl;
  const int s1 = D == 3 ? (int)(r % n1) : 0, s0 = D == 3 ? (int)(r / n1) : (int)r;
  const bool last = w[K - 1] != 0.f || w[8 + K - 1] != 0.f || (D == 3 && w[16 + K - 1] != 0.f);
  const int ke = last ? K : K - 1;
#pragma unroll 1
  for (int a = 0; a < ke; ++a) {
    int x = s0 + a;
    if (x >= n0) x -= n0;
    float2 pa = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int b = 0; b < (D == 3 ? ke : 1); ++b) {
      int64_t row = x;
      if (D == 3) {
        int y = s1 + b;
        if (y >= n1) y -= n1;
        row = row * n1 + y;
      }
      const float2* rp = g + row * nl * CB;
      float2 ra = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c == K - 1 && !last) break;
        int z = sl + c;
        if (z >= nl) z -= nl;
        const float v = w[8 * (D - 1) + c];
        ra = __ffma2_rn(make_float2(v, v), __ldg(rp + (int64_t)z * CB), ra);
      }
      if (D == 3) pa = __ffma2_rn(make_float2(w[8 + b], w[8 + b]), ra, pa);
      else pa = ra;
    }
    acc = __ffma2_rn(make_float2(w[a], w[a]), pa, acc);
  }
  return acc;
}

// A CTA takes a run of at most kGatherChunk samples in tile order: it
// evaluates their d K weights into shared memory (one per thread and step),
// then walks the coil blocks, CB lanes per sample, 32 / CB samples per warp.
// The taps are loaded from global memory: the footprints of the CTA's samples
// overlap, so L1 holds one coil block of them and no tile has to be staged,
// which for W 4 moved 8^3 cells per 4^3 tile and for W 6 in 3D did not fit
// shared memory. Bound by the L1 load pipe (two wavefronts per warp load).
template <int D, int K, int CB>
__global__ void __launch_bounds__(kGatherWarps * 32, gather_occ(D, K))
k_interp_gather(const int* __restrict__ slices, const int* __restrict__ first_chunk, int nsl, int chunk,
                const SliceGeom* __restrict__ sl, KBParams kb, const float4* __restrict__ coord,
                const int* __restrict__ perm, const float2* __restrict__ grid, int layout, float2* __restrict__ ksp,
                float scale, RowIO rio) {
  constexpr int SUB = 32 / CB, WS = gather_stride(D);
  extern __shared__ __align__(16) float s_w[];                       // [chunk][WS]
  int64_t* s_cell = reinterpret_cast<int64_t*>(s_w + chunk * WS);    // first tap's cell, ~cell where it wraps
  int* s_p = reinterpret_cast<int*>(s_cell + chunk);                 // point ids
  float2* s_o = reinterpret_cast<float2*>(s_p + chunk);              // results of one coil block, [CB][chunk + 1]
  int k = 0;
  {
    int lo = 0, hi = nsl - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first_chunk[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    k = lo;
  }
  const SliceGeom& g = sl[slices[k]];
  const int ncoil = g.ncoil;
  const int64_t m = g.m, gos = g.gos;
  const int64_t b0 = g.pt_off + (int64_t)((int)blockIdx.x - first_chunk[k]) * chunk;
  const int ns = (int)min((int64_t)chunk, g.pt_off + m - b0);
  int nos[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) nos[i] = g.nos[i];
  for (int j = threadIdx.x; j < ns; j += blockDim.x) {
    const float4 c4 = coord[b0 + j];
    const float u[3] = {c4.x, c4.y, c4.z};
    int64_t cell = 0;
    bool wrap = false;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const int lo = (int)ceilf(__fsub_rn(u[i], kb.radius[i]));
      const int s = wrap_once(lo, nos[i]);
      wrap |= s + K > nos[i] || fabsf(__fsub_rn((float)(lo + K - 1), u[i])) <= kb.radius[i];
      cell = cell * nos[i] + s;
    }
    s_cell[j] = wrap ? ~cell : cell;
    s_p[j] = perm[b0 + j];
  }
  for (int t = threadIdx.x; t < ns * D * K; t += blockDim.x) {
    const int j = t / (D * K), r = t - j * (D * K), i = r / K, q = r - i * K;
    const float4 c4 = coord[b0 + j];
    const float u = i == 0 ? c4.x : (i == 1 ? c4.y : c4.z);
    const float rad = sel3(kb.radius, i);
    const int lo = (int)ceilf(__fsub_rn(u, rad));
    const float adx = fabsf(__fsub_rn((float)(lo + q), u));
    s_w[j * WS + 8 * i + q] = adx <= rad ? kb_tap_fast(adx, sel3(kb.inv_radius, i), kb) : 0.f;
  }
  __syncthreads();
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / CB, coil = lane % CB;
  const int64_t sy = (int64_t)nos[2] * CB;                       // 3D rows
  const int64_t sx = (int64_t)nos[1] * (D == 3 ? nos[2] : 1) * CB;
  const float2* gb = grid + (layout == kInternal ? g.grid_off : g.ugrid_off) + coil;
  float2* kspc = ksp + g.ksp_off - g.pt_off;
  const int os = chunk + 1;
  for (int c0 = 0; c0 < ncoil; c0 += CB, gb += gos * CB) {
    const int c = c0 + coil;
    for (int j = warp * SUB + sub; j < ns; j += nw * SUB) {
      if (c >= ncoil) continue;
      const int64_t cell = s_cell[j];
      const float* w = s_w + j * WS;
      const float2 a = cell < 0 ? gather_wrap<D, K, CB>(gb, ~cell, nos[0], nos[1], nos[2], w)
                                : gather_fast<D, K - 1, CB>(gb + cell * CB, sx, sy, w);
      float2 v = make_float2(a.x * scale, a.y * scale);
      if (rio.on) {
        const int p = s_p[j];
        if (rio.dcf) {
          const float d = rio.dcf[p];
          v = make_float2(v.x * d, v.y * d);
        }
        ksp[g.row_off + (p - g.pt_off) * g.rs + c] = v;
      } else if (CB == 1) {
        kspc[(int64_t)c * m + s_p[j]] = v;
      } else {
        s_o[coil * os + j] = v;
      }
    }
    if (CB > 1 && !rio.on) {
      // lanes on samples: consecutive ones of a tile are mostly consecutive
      // samples of the trajectory, so a store covers runs of a coil's row
      __syncthreads();
      const int nc = min(CB, ncoil - c0);
      for (int q = warp; q < nc; q += nw) {
        float2* dst = kspc + (int64_t)(c0 + q) * m;
        for (int j = lane; j < ns; j += 32) dst[s_p[j]] = s_o[q * os + j];
      }
      __syncthreads();
    }
  }
}

constexpr int kTileWarps = 8;
constexpr int kTileRun = 8;  // samples a warp takes at once

// 2D slices in coil blocks of 8: a CTA per work item (interpolation tile) and
// group of NB blocks. The tile and its halo come into shared memory as [cell][8 NB
// coils] by 16-byte asynchronous copies (a grid row of the region is
// contiguous per block); a cell's row is padded by two coils, which keeps it
// 16-byte aligned and puts the two samples a warp reads at once on any
// cells without more than the two wavefronts their 256 bytes need. From
// there on warps work alone: one takes kTileRun samples, evaluates their 2 K
// weights spread over its lanes, gathers 8 NB coils per sample, and stores
// through a small buffer so that lanes run along the trajectory (8-byte
// values of one coil per lane would each take a sector and a wavefront).
template <int K, int NB>
__global__ void __launch_bounds__(kTileWarps * 32, 4)
k_interp_tile(const Item* __restrict__ items, const SliceGeom* __restrict__ sl, KBParams kb,
              const float4* __restrict__ coord, const int* __restrict__ perm, const float2* __restrict__ grid,
              float2* __restrict__ ksp, float scale, RowIO rio) {
  constexpr int CW = 8 * NB, CS = CW + 2, SUB = 32 / CW, R = kTileRun;
  extern __shared__ __align__(16) unsigned char tsm[];
  float2* region = reinterpret_cast<float2*>(tsm);
  __shared__ __align__(16) float s_w[kTileWarps][R][20];  // row weights at 0, column weights at 8
  __shared__ float2 s_o[kTileWarps][R][CW + 1];
  const Item it = items[blockIdx.x];
  if (it.slice < 0) return;  // padding past the real items
  const SliceGeom& g = sl[it.slice];
  const int ncoil = g.ncoil, c0 = blockIdx.y * CW;
  if (c0 >= ncoil || g.cb != 8) return;  // slices of other blocks: k_interp_gather, k_interp_reg
  const int nc = min(CW, ncoil - c0);
  const int nos0 = g.nos[0], nos1 = g.nos[1];
  const int64_t gos = g.gos, m = g.m;
  const Frame f = frame_of(g, it.tile, 2, false);
  const int ext0 = f.size[0] + K - 1, ext1 = f.size[1] + K - 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int coil = lane % CW, sub = lane / CW;
  int run = warp * R;  // first sample of this warp's run
  float4 c_next = make_float4(0.f, 0.f, 0.f, 0.f);
  int p_next = 0;
  if (lane < R && run < it.count) {
    const int e = it.start + min(run + lane, it.count - 1);
    c_next = coord[e];
    p_next = perm[e];
  }
  {
    const float2* gb = grid + g.grid_off + (int64_t)(c0 / 8) * gos * 8;
    const int nblk = min(NB, (ncoil - c0 + 7) / 8);
    for (int r = warp; r < ext0 * nblk; r += kTileWarps) {
      const int kb8 = r / ext0, x = r - kb8 * ext0;
      int sx = f.org[0] + x;
      if (sx >= nos0) sx -= nos0;
      const float2* src = gb + ((int64_t)kb8 * gos + (int64_t)sx * nos1) * 8;
      float2* dst = region + x * ext1 * CS + kb8 * 8;
      for (int q = lane; q < ext1 * 4; q += 32) {
        int sy = f.org[1] + (q >> 2);
        if (sy >= nos1) sy -= nos1;
        cp_async16(dst + (q >> 2) * CS + (q & 3) * 2, src + (int64_t)sy * 8 + (q & 3) * 2);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();
  float2* kspc = ksp + g.ksp_off + (int64_t)c0 * m - g.pt_off;
  for (; run < it.count; run += kTileWarps * R) {
    const int n = min(R, it.count - run);
    const float4 c4 = c_next;
    const int p = p_next;
    if (lane < R) {
      const int e = it.start + min(run + kTileWarps * R + lane, it.count - 1);
      c_next = coord[e];
      p_next = perm[e];
    }
    __syncwarp();  // the previous run's buffers are read
#pragma unroll
    for (int t0 = 0; t0 < R * 2 * K; t0 += 32) {
      const int t = min(t0 + lane, R * 2 * K - 1);
      const int j = t / (2 * K), r = t - j * (2 * K), i = r >= K ? 1 : 0, q = r - i * K;
      const float ux = __shfl_sync(0xffffffffu, c4.x, j), uy = __shfl_sync(0xffffffffu, c4.y, j);
      const float u = i ? uy : ux, rad = i ? kb.radius[1] : kb.radius[0];
      const int lo = (int)ceilf(__fsub_rn(u, rad));
      const float adx = fabsf(__fsub_rn((float)(lo + q), u));
      s_w[warp][j][8 * i + q] = adx <= rad ? kb_tap_fast(adx, i ? kb.inv_radius[1] : kb.inv_radius[0], kb) : 0.f;
    }
    // cell of the first tap in the region
    const int l0 = wrap_once((int)ceilf(__fsub_rn(c4.x, kb.radius[0])), nos0) - f.org[0];
    const int l1 = wrap_once((int)ceilf(__fsub_rn(c4.y, kb.radius[1])), nos1) - f.org[1];
    const int cell0 = (l0 * ext1 + l1) * CS;
    __syncwarp();
#pragma unroll 1
    for (int j0 = 0; j0 < n; j0 += SUB) {
      const int j = j0 + sub;  // R is a multiple of SUB: past n it repeats a valid sample's coordinates
      const int cell = __shfl_sync(0xffffffffu, cell0, j);
      const float* w = s_w[warp][j];
      const float2* rp = region + cell + coil;
      float2 acc = make_float2(0.f, 0.f);
      // the K-th tap of an axis has weight only when it lies exactly W/2 away (window_taps)
      const bool last = w[K - 1] != 0.f || w[8 + K - 1] != 0.f;
      float2 wl[K];
#pragma unroll
      for (int b = 0; b < K; ++b) wl[b] = make_float2(w[8 + b], w[8 + b]);
      if (!last) {
#pragma unroll
        for (int a = 0; a < K - 1; ++a) {
          float2 ra = make_float2(0.f, 0.f);
#pragma unroll
          for (int b = 0; b < K - 1; ++b) ra = __ffma2_rn(wl[b], rp[b * CS], ra);
          acc = __ffma2_rn(make_float2(w[a], w[a]), ra, acc);
          rp += ext1 * CS;
        }
      } else {
#pragma unroll 1
        for (int a = 0; a < K; ++a) {
          float2 ra = make_float2(0.f, 0.f);
#pragma unroll
          for (int b = 0; b < K; ++b) ra = __ffma2_rn(wl[b], rp[b * CS], ra);
          acc = __ffma2_rn(make_float2(w[a], w[a]), ra, acc);
          rp += ext1 * CS;
        }
      }
      float2 v = make_float2(acc.x * scale, acc.y * scale);
      if (rio.on) {
        const int pj = __shfl_sync(0xffffffffu, p, j);
        if (j < n && coil < nc) {
          if (rio.dcf) {
            const float d = rio.dcf[pj];
            v = make_float2(v.x * d, v.y * d);
          }
          ksp[g.row_off + (pj - g.pt_off) * g.rs + c0 + coil] = v;
        }
      } else {
        s_o[warp][j][coil] = v;
      }
    }
    if (!rio.on) {
      __syncwarp();
      const int j = lane % R;
      const int pj = __shfl_sync(0xffffffffu, p, j);
      if (j < n)
        for (int c = lane / R; c < nc; c += 32 / R) kspc[(int64_t)c * m + pj] = s_o[warp][j][c];
    }
  }
}

}  // namespace

// Slices by coil block, and the CTAs of each: chunks of kGatherChunk samples,
// halved while they would leave SMs idle (never below one round of a
// two-warp CTA). Called with MRN_OPT_NATIVE_FFT at its default.
int gather_setup(mrn_plan* P) {
  P->gather.clear();
  if (P->ndim < 2) return MRN_OK;
  std::vector<int> tab;
  for (int kind = 0; kind < 8; ++kind) {
    mrn_plan::GatherSet gs{};
    const int cb = gs.cb = 1 << (kind & 3);
    gs.native = kind < 4;
    gs.off = (int)tab.size();
    int64_t pts = 0;
    for (int s = 0; s < P->nslices; ++s) {
      const SliceGeom& g = P->h_slices[s];
      if (g.cb != cb || (g.native_fft != 0) != gs.native || g.m == 0) continue;
      tab.push_back(s);
      pts += g.m;
      gs.max_coil = std::max(gs.max_coil, g.ncoil);
      ++gs.nsl;
    }
    if (gs.nsl == 0) continue;
    gs.chunk = kGatherChunk;
    while (gs.chunk > 2 * (32 / cb) && gs.chunk > 32 && pts / gs.chunk < 4 * (int64_t)P->sm_count) gs.chunk /= 2;
    int64_t n = 0;
    for (int k = 0; k < gs.nsl; ++k) {
      const SliceGeom& g = P->h_slices[tab[gs.off + k]];
      tab.push_back((int)n);
      n += (g.m + gs.chunk - 1) / gs.chunk;
    }
    tab.push_back((int)n);
    gs.nchunks = (int)n;
    P->gather.push_back(gs);
  }
  if (tab.empty()) return MRN_OK;
  cudaError_t e = cudaMalloc(&P->d_gather, tab.size() * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(P->d_gather, tab.data(), tab.size() * sizeof(int), cudaMemcpyHostToDevice);
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

// Slices of the plan grid that cuFFT transforms (coil planes, FFT order).
static bool gather_rest(const mrn_plan* P) {
  for (const auto& gs : P->gather)
    if (!gs.native) return true;
  return false;
}

// Some slices' grids are in coil blocks: plan grids of the native passes
// (k_interp_reg takes the other slices), a caller's grid (coil planes) when it
// has one coil.
bool gather_ok(const mrn_plan* P, int layout) {
  if (P->gather.empty() || P->coil_group_req > 0) return false;
  if (layout != kInternal) return P->max_coil == 1;
  return ffx_active(P) && P->gather[0].native && (!gather_rest(P) || interp_reg_ok(P));
}

// Each slice takes the kernel of its own grid. 2D, four slices of 12 to 32 coils,
// 32 k samples each (76 us), with a fifth of 4 coils 90 us, where it sent all to
// k_interp_gather 115; with a fifth that cuFFT transforms 117 to 120, where all
// went to k_interp_reg 113 to 115 (its few CTAs run by themselves); 3D, 64^3 and
// 96^3 with one of 56^3 that cuFFT transforms, 8 coils, 633 and 873.
//
// 2D slices in blocks of 8 coils whose tile regions fit: 256^2, 32 coils,
// 98,304 spiral samples, W 6: 60 us (68 with the tile staged from coil planes)
// against 78 from global memory, whose 906 MB of taps need more L1 than the
// CTAs of an SM have.
static size_t tile_smem(const mrn_plan* P, int nb) {
  const int K = P->kb.itaps;
  return (size_t)(P->tmax_cells[0] + K - 1) * (P->tmax_cells[1] + K - 1) * (8 * nb + 2) * sizeof(float2);
}

static int launch_tile(mrn_plan* P, int max_coil, const float2* grid, float2* ksp, float scale, cudaStream_t st,
                       RowIO rio) {
  const int K = P->kb.itaps, nb = max_coil <= 8 ? 1 : 2;
  const size_t smem = tile_smem(P, nb);
  const dim3 gd((unsigned)P->n_items_interp, (unsigned)((max_coil + 8 * nb - 1) / (8 * nb)));
  int rc = MRN_OK;
#define MRN_TILE(KK, NN)                                                                                    \
  do {                                                                                                      \
    auto kern = k_interp_tile<KK, NN>;                                                                      \
    rc = set_dynamic_smem(kern, smem);                                                                      \
    if (rc == MRN_OK)                                                                                       \
      kern<<<gd, kTileWarps * 32, smem, st>>>(P->d_items_i, P->d_slices, P->kb, P->d_coord_i, P->d_perm_i, grid, \
                                              ksp, scale, rio);                                             \
  } while (0)
#define MRN_TILE_N(KK) if (nb == 2) MRN_TILE(KK, 2); else MRN_TILE(KK, 1)
  if (K == 5) { MRN_TILE_N(5); }
  else if (K == 6) { MRN_TILE_N(6); }
  else if (K == 7) { MRN_TILE_N(7); }
  else { MRN_TILE_N(8); }
#undef MRN_TILE_N
#undef MRN_TILE
  if (rc != MRN_OK) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

int launch_interp_gather(mrn_plan* P, const float2* grid, int layout, float2* ksp, float scale, cudaStream_t st,
                         RowIO rio) {
  const int K = P->kb.itaps;
  for (const auto& gs : P->gather) {
    if (layout == kInternal && !gs.native) continue;
    if (P->ndim == 2 && layout == kInternal && gs.cb == 8 && tile_smem(P, gs.max_coil <= 8 ? 1 : 2) <= 100 * 1024) {
      const int rc = launch_tile(P, gs.max_coil, grid, ksp, scale, st, rio);
      if (rc != MRN_OK) return rc;
      continue;
    }
    const int* sl = P->d_gather + gs.off;
    const int sub = 32 / gs.cb;
    const int warps = std::max(2, std::min(kGatherWarps, gs.chunk / sub));
    const size_t smem = (size_t)gs.chunk * (gather_stride(P->ndim) * sizeof(float) + sizeof(int64_t) + sizeof(int)) +
                        (gs.cb > 1 && !rio.on ? (size_t)gs.cb * (gs.chunk + 1) * sizeof(float2) : 0);
#define MRN_GATHER(DD, KK, CC)                                                                                 \
  k_interp_gather<DD, KK, CC><<<gs.nchunks, warps * 32, smem, st>>>(sl, sl + gs.nsl, gs.nsl, gs.chunk, P->d_slices, \
                                                                 P->kb, P->d_coord_i, P->d_perm_i, grid, layout,  \
                                                                 ksp, scale, rio)
#define MRN_GATHER_C(DD, KK)              \
  if (gs.cb == 8) MRN_GATHER(DD, KK, 8);  \
  else if (gs.cb == 4) MRN_GATHER(DD, KK, 4); \
  else if (gs.cb == 2) MRN_GATHER(DD, KK, 2); \
  else MRN_GATHER(DD, KK, 1)
#define MRN_GATHER_K(DD)                      \
  if (K == 5) { MRN_GATHER_C(DD, 5); }        \
  else if (K == 6) { MRN_GATHER_C(DD, 6); }   \
  else if (K == 7) { MRN_GATHER_C(DD, 7); }   \
  else { MRN_GATHER_C(DD, 8); }
    if (P->ndim == 2) { MRN_GATHER_K(2) }
    else { MRN_GATHER_K(3) }
#undef MRN_GATHER_K
#undef MRN_GATHER_C
#undef MRN_GATHER
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e);
  }
  if (layout == kInternal && gather_rest(P))
    return launch_interp_reg(P, grid, layout, ksp, scale, nullptr, st, rio, true);
  return MRN_OK;
}

}  // namespace mrn
