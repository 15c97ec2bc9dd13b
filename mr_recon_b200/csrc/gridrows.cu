// Type-1 gridding (samples -> oversampled grid) with the tile accumulator in
// registers, from sample-major values: the default 2D and 3D path of
// launch_grid_t for kernels of 5..8 candidate taps per dimension (width
// 4 <= W < 8) and tiles of at most 8 cells per edge.
//
// Reference: triton_interp/grid.py _grid2d / _grid3d (:258-502) launches one
// Triton program per chunk of points and adds every tap of every batch element
// into global memory with an fp32 atomic. Here the samples are binned into
// 8-cell tiles (plan.cu, one "entry" per sample and tile its footprint meets),
// and a CTA accumulates a whole tile without atomics. Tap selection and
// weights are the reference's: taps j = lo + q, lo = ceil(u - W/2), valid iff
// |(float)j - u| <= W/2 in float32 (kernels.py:268-393), weight = prod_d
// KB(|j_d - u_d| / (W/2)), circular cells.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.cuh"
#include "tile_util.cuh"

namespace mrn {

// ---------------------------------------------------------------------------
// A thread keeps 4 (y) x 8 (z) complex cells of one coil in registers (64 of
// at most 128, 16 warps resident; at 85 registers, 24 warps, it spills: 192^3,
// 16 coils 6.2 ms against 5.7): half of the rows of one x-plane in 3D, of the
// tile in 2D. A warp's lanes are coils, then x-planes (3D), then
// in 2D the two halves and, below 16 coils, two entry streams whose tiles are
// added at the end. 3D, 16 coils: 8 warps of two planes and one half each.
//
// Weights along x and y are kept aligned to the tile's 8 cells (zero outside
// the support and the tile): a thread takes its plane's x weight and its four
// rows' y weights with one load each. Along z a footprint has K - 1 = KW taps
// unless u - W/2 is an integer, so its part inside the tile fits a window of
// KW cells starting at z0 in [0, NW), NW = 8 - KW + 1; entries with all K taps
// inside (exact boundary taps, a few per spoke through the k-space centre) use
// all 8 cells. z0 is the same for the whole warp and selects straight-line
// packed FMAs (fma.rn.f32x2: re and im of a cell) on fixed registers. The
// entries of a tile are sorted by it (k_emit_entries), so one branch serves a
// run of entries. (Windows along y too, a thread owning 8 x 8 cells: 12% fewer
// instructions, but 12 warps and 25 code paths, which miss the instruction
// cache: 192^3, 16 coils 6.8 ms, 256^2, 32 coils spiral 140 us.) Bound by issue:
// about 150 warp instructions per entry at half the issue rate, 16 coils.
// Measured, gridding stage with k_rows and the reduction, against the kernels
// that gathered 8-byte values from coil rows: 192^3, 16 coils, 7.68 M kooshball
// samples, W 4 5.7 ms (7.9), 120^3, 12 coils, 1.92 M, W 6 3.0 (4.5), 128^3, 8
// coils, 2.05 M, W 4 1.1 (2.2); 256^2, 32 coils, 98,304 spiral samples, W 6
// 105 us (108), from the rows of a normal operator 87 (109).
//
// Values come as rows, one sample's coils side by side (k_rows, or written so
// by the interpolation of a normal operator): sorting the entries by window
// breaks the trajectory order, which gathers from coil rows depended on, but a
// row is one or two 64-byte pieces wherever it lies. Batches of B entries run
// through a cp.async pipeline: in iteration b the values of batch b+1 and the
// coordinates of batch b+3 are in flight while the weights of batch b+1 are
// evaluated and batch b is accumulated; one barrier per batch. Each entry
// carries masks of its planes and rows with weight, so one ballot per warp and
// 32 entries keeps only those the warp has cells of. No atomics; float32
// accumulation in entry order, so results are the same on every run (split
// tiles write partial tiles that a reduction pass adds in item order).
// ---------------------------------------------------------------------------
namespace {

constexpr int kGTile = 8;
constexpr size_t kGStage = 32 * (kGTile * kGTile / 2 + 1) * sizeof(float2);  // write-back to coil planes

// One entry of a batch: its sample's values and weights, one stride for all.
template <int D, int CW>
struct __align__(16) GEntry {
  float2 v[CW];
  float2 wz[8];                // z window weights (all 8 cells for code NW), each twice
  float wy[8];                 // y weights (2D: x scale), tile-aligned
  float wx[D == 3 ? 8 : 4];    // 3D: x weights x scale, tile-aligned; 2D: unused
};

template <int D, int B, int CW>
struct GSmem {
  GEntry<D, CW> e[2][B];
  float4 c[4][B];       // coordinate ring (a batch stays until its weights are evaluated)
  int pm[4][B];         // sample index ring
  unsigned code[2][B];  // byte 0: z0 or NW, byte 1: x-planes with weight, byte 2: rows with weight
  float2 t[2][B];       // temporal weight
};

template <int D, int CW>
__host__ __device__ constexpr int grid_threads() { return D == 3 ? 16 * CW : (CW == 32 ? 64 : 32); }
template <int D, int CW>
__host__ __device__ constexpr int grid_batch() { return D == 3 ? (CW == 16 ? 128 : (CW == 8 ? 64 : 32)) : 32; }
template <int D, int CW>
__host__ __device__ constexpr int grid_streams() { return D == 2 && CW == 8 ? 2 : 1; }

// The entries of one run (bits of `mask`, of the 32 from h32) accumulated by
// the calling warp.
template <int D, int CW, int B, bool TEMP>
struct RunBody {
  float2 (&acc)[4][kGTile];
  const GSmem<D, B, CW>& s;
  int b2, h32, plane, half, coil, stream;
  unsigned mask;
  __device__ __forceinline__ float2 value(int j) const {
    const GEntry<D, CW>& e = s.e[b2][j];
    float2 v = e.v[coil];
    if (TEMP) {  // times conj(t)
      const float2 t = s.t[b2][j];
      v = make_float2(v.x * t.x + v.y * t.y, v.y * t.x - v.x * t.y);
    }
    if (D == 3) {
      const float w = e.wx[plane];
      v = __fmul2_rn(make_float2(w, w), v);
    }
    return v;
  }
  // acc[r][Z0 + c] += wy[r] wz[c] v over 4 rows x N cells, for two entries
  // (v1 = 0: one) whose loads overlap
  template <int Z0, int N>
  __device__ __forceinline__ void add(int j0, float2 v0, int j1, float2 v1) {
    const float4 y0 = *reinterpret_cast<const float4*>(&s.e[b2][j0].wy[4 * half]);
    const float4 y1 = *reinterpret_cast<const float4*>(&s.e[b2][j1].wy[4 * half]);
    const float ya[4] = {y0.x, y0.y, y0.z, y0.w}, yb[4] = {y1.x, y1.y, y1.z, y1.w};
    float2 za[N], zb[N];
#pragma unroll
    for (int c = 0; c < N; ++c) za[c] = s.e[b2][j0].wz[c];
#pragma unroll
    for (int c = 0; c < N; ++c) zb[c] = s.e[b2][j1].wz[c];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float2 v2 = __fmul2_rn(make_float2(ya[r], ya[r]), v0);
#pragma unroll
      for (int c = 0; c < N; ++c) acc[r][Z0 + c] = __ffma2_rn(za[c], v2, acc[r][Z0 + c]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float2 v2 = __fmul2_rn(make_float2(yb[r], yb[r]), v1);
#pragma unroll
      for (int c = 0; c < N; ++c) acc[r][Z0 + c] = __ffma2_rn(zb[c], v2, acc[r][Z0 + c]);
    }
  }
  template <int Z0, int N>
  __device__ __forceinline__ void add(int j, float2 v) {
    const float4 y4 = *reinterpret_cast<const float4*>(&s.e[b2][j].wy[4 * half]);
    const float y[4] = {y4.x, y4.y, y4.z, y4.w};
    float2 z[N];
#pragma unroll
    for (int c = 0; c < N; ++c) z[c] = s.e[b2][j].wz[c];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float2 v2 = __fmul2_rn(make_float2(y[r], y[r]), v);
#pragma unroll
      for (int c = 0; c < N; ++c) acc[r][Z0 + c] = __ffma2_rn(z[c], v2, acc[r][Z0 + c]);
    }
  }
  template <int Z0, int N>
  __device__ __forceinline__ void run() {
    constexpr int S = grid_streams<D, CW>();
    unsigned mm = mask;
    if (S == 1) {
      if (N <= 6) {
#pragma unroll 1
        while (mm & (mm - 1u)) {
          const int j0 = h32 + __ffs(mm) - 1;
          mm &= mm - 1u;
          const int j1 = h32 + __ffs(mm) - 1;
          mm &= mm - 1u;
          add<Z0, N>(j0, value(j0), j1, value(j1));
        }
      }
#pragma unroll 1
      while (mm) {
        const int j = h32 + __ffs(mm) - 1;
        mm &= mm - 1u;
        add<Z0, N>(j, value(j));
      }
    } else {
      static_assert(S <= 2, "entry streams");
      // the streams take the run's entries in turn
#pragma unroll 1
      while (mm) {
        const int j0 = h32 + __ffs(mm) - 1;
        mm &= mm - 1u;
        const bool on = stream == 0 || mm != 0u;
        const int j = stream == 0 || mm == 0u ? j0 : h32 + __ffs(mm) - 1;
        mm &= mm - 1u;
        const float2 v = value(j);
        add<Z0, N>(j, on ? v : make_float2(0.f, 0.f));
      }
    }
  }
  template <int KW>
  __device__ __forceinline__ void dispatch(int code) {
    constexpr int NW = kGTile - KW + 1;
    if (code == 0) run<0, KW>();
    else if (NW > 1 && code == 1) run<(NW > 1 ? 1 : 0), KW>();
    else if (NW > 2 && code == 2) run<(NW > 2 ? 2 : 0), KW>();
    else if (NW > 3 && code == 3) run<(NW > 3 ? 3 : 0), KW>();
    else if (NW > 4 && code == 4) run<(NW > 4 ? 4 : 0), KW>();
    else run<0, kGTile>();
  }
};

}  // namespace

template <int D, int K, int CW, bool TEMP>
__global__ void __launch_bounds__(grid_threads<D, CW>(), 512 / grid_threads<D, CW>())
k_grid_rows(const Item* __restrict__ items, const SliceGeom* __restrict__ sl, KBParams kb,
            const float4* __restrict__ coord, const int* __restrict__ perm, const float2* __restrict__ rows,
            const float2* __restrict__ temporal, float2* __restrict__ grid, int layout, float scale, int cg,
            SplitOut so) {
  constexpr int T = kGTile, NT = grid_threads<D, CW>(), B = grid_batch<D, CW>(), NWARP = NT / 32;
  constexpr int KW = K - 1, NW = T - KW + 1;
  constexpr int PPW = D == 3 ? 32 / CW : 1, NPG = 8 / PPW;  // 3D: planes per warp, plane groups
  static_assert(K <= T, "taps per dimension");
  extern __shared__ __align__(16) unsigned char g_smem[];
  GSmem<D, B, CW>& s = *reinterpret_cast<GSmem<D, B, CW>*>(g_smem);

  const Item it = items[blockIdx.x];
  if (it.slice < 0) return;  // padding past the real items
  const SliceGeom* gp = sl + it.slice;
  const int ncoil = gp->ncoil;
  const int c0 = blockIdx.y * cg;
  if (c0 >= ncoil) return;
  const int ncg = min(cg, ncoil - c0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int coil = lane % CW;
  const int plane = D == 3 ? (warp % NPG) * PPW + lane / CW : 0;
  const int half = D == 3 ? warp / NPG : (CW == 32 ? warp : (lane / CW) & 1);
  const int stream = grid_streams<D, CW>() > 1 ? lane / (2 * CW) : 0;
  const Frame f = frame_of(*gp, it.tile, D, true);
  const int64_t pt_off = gp->pt_off;
  const int rs = gp->rs;
  const float2* rbase = rows + gp->row_off + c0;
  const int nbatch = (it.count + B - 1) / B;
  auto batch_len = [&](int bi) { return bi < nbatch ? min(B, it.count - bi * B) : 0; };
  auto sync = [&]() {
    if (NWARP == 1) __syncwarp();
    else __syncthreads();
  };

  // coordinates and sample indices of batch bi into ring slot bi % 4
  auto copy_coords = [&](int bi) {
    const int nb = batch_len(bi), r4 = bi & 3;
    for (int t = tid; t < nb; t += NT) {
      cp_async16(&s.c[r4][t], coord + it.start + bi * B + t);
      cp_async4(&s.pm[r4][t], perm + it.start + bi * B + t);
    }
  };
  // sample values, two coils per 16-byte copy (rows of one coil: 8 bytes)
  auto copy_values = [&](int bi) {
    const int nb = batch_len(bi), b2 = bi & 1, r4 = bi & 3;
    if (rs > 1) {
      for (int t = tid; t < nb * (CW / 2); t += NT) {
        const int j = t / (CW / 2), q = 2 * (t - j * (CW / 2));
        if (q < ncg) cp_async16(&s.e[b2][j].v[q], rbase + (int64_t)(s.pm[r4][j] - pt_off) * rs + q);
      }
    } else {
      for (int t = tid; t < nb; t += NT) cp_async8(&s.e[b2][t].v[0], rbase + (s.pm[r4][t] - pt_off));
    }
    if (TEMP)
      for (int t = tid; t < nb; t += NT) cp_async8(&s.t[b2][t], temporal + s.pm[r4][t]);
  };
  // unit (entry j, dimension i): the weights of the K candidate taps, placed on
  // the tile's cells (x, y) or from the window start (z), and the masks / code
  auto weights = [&](int bi) {
    const int nb = batch_len(bi), b2 = bi & 1, r4 = bi & 3;
    for (int t = tid; t < D * B; t += NT) {
      const int i = t / B, j = t - i * B;  // warp-uniform dimension
      if (j >= nb) continue;
      const float4 c4 = s.c[r4][j];
      const float u = i == 0 ? c4.x : (i == 1 ? c4.y : c4.z);
      const float r = sel3(kb.radius, i), ir = sel3(kb.inv_radius, i);
      const int n = sel3(gp->nos, i), size = sel3(f.size, i);
      const int lo = (int)ceilf(__fsub_rn(u, r));
      int st = wrap_once(lo, n) - sel3(f.org, i);  // first tap's cell
      if (st >= size) st -= n;                     // footprint wraps into this tile from the end
      unsigned char* cb = reinterpret_cast<unsigned char*>(&s.code[b2][j]);
      if (i == D - 1) {
        const bool all = fabsf(__fsub_rn((float)(lo + K - 1), u)) <= r && st >= 0 && st + K <= size;
        const int z0 = all ? 0 : min(max(st, 0), size - KW);
        const int nz = all ? T : KW;
        cb[0] = (unsigned char)(all ? NW : z0);
#pragma unroll
        for (int c = 0; c < T; ++c) {
          if (c >= KW && c >= nz) break;
          const int q = z0 + c - st;
          const float adx = fabsf(__fsub_rn((float)(lo + q), u));
          const float w = q >= 0 && q < K && adx <= r ? kb_tap_fast(adx, ir, kb) : 0.f;
          s.e[b2][j].wz[c] = make_float2(w, w);
        }
      } else {
        float* wd = D == 3 && i == 0 ? s.e[b2][j].wx : s.e[b2][j].wy;
        const float sc = i == 0 ? scale : 1.f;
        reinterpret_cast<float4*>(wd)[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<float4*>(wd)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned mask = 0;
#pragma unroll
        for (int q = 0; q < K; ++q) {
          const float adx = fabsf(__fsub_rn((float)(lo + q), u));
          const int cell = st + q;
          if (adx <= r && cell >= 0 && cell < size) {
            wd[cell] = kb_tap_fast(adx, ir, kb) * sc;
            mask |= 1u << cell;
          }
        }
        cb[D == 3 && i == 0 ? 1 : 2] = (unsigned char)mask;
      }
    }
  };

  float2 acc[4][T];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < T; ++b) acc[a][b] = make_float2(0.f, 0.f);

  copy_coords(0);
  copy_coords(1);
  cp_async_commit();
  cp_async_wait<0>();
  sync();
  copy_values(0);
  cp_async_commit();
  copy_coords(2);
  cp_async_commit();
  weights(0);
  for (int bi = 0; bi < nbatch; ++bi) {
    cp_async_wait<1>();  // values of bi and coordinates of bi + 1 have landed (this thread's)
    sync();              // ... everyone's; weights of bi visible; buffers of bi - 1 free
    copy_values(bi + 1);
    cp_async_commit();
    copy_coords(bi + 3);
    cp_async_commit();
    weights(bi + 1);
    const int b2 = bi & 1, nb = batch_len(bi);
#pragma unroll 1
    for (int h32 = 0; h32 < nb; h32 += 32) {
      const unsigned mine = h32 + lane < nb ? s.code[b2][h32 + lane] : 0xffu;
      const int zcode = (int)(mine & 0xffu);
      bool meet = h32 + lane < nb;
      if (D == 3) meet &= ((mine >> (8 + (warp % NPG) * PPW)) & ((1u << PPW) - 1u)) != 0u;
      if (D == 3 || CW == 32) meet &= ((mine >> (16 + 4 * half)) & 15u) != 0u;
      // 3D: windows in the order of all 32 entries, also those the warp skips, so
      // that a cell's order does not depend on which planes share its warp (CW;
      // in 2D MRN_OPT_GRID_LANES fixes it)
      unsigned act = __ballot_sync(0xffffffffu, meet), left = 0xffffffffu;
      while (act) {
        const int code = __shfl_sync(0xffffffffu, zcode, __ffs(D == 3 ? left : act) - 1);
        unsigned same = __ballot_sync(0xffffffffu, zcode == code);
        if (D == 3) left &= ~same;
        same &= act;
        if (D == 3 && !same) continue;
        act &= ~same;
        RunBody<D, CW, B, TEMP> body{acc, s, b2, h32, plane, half, coil, stream, same};
        body.template dispatch<KW>(code);
      }
    }
  }
  cp_async_wait<0>();

  // A sample that is not finite times a weight of zero (rows and planes of the
  // tile outside its footprint, the ends of its window) spoils cells it does
  // not belong to. Such a sum never becomes finite again, so the tile's sums
  // tell (one product a cell); the tile is then added up once more, only where
  // there is weight. Costs 3 us of 101 at 256^2, 32 coils and 0.04 ms of 5.8 at
  // 192^3, 16 coils, for the loop's schedule more than for the products (out of
  // line 0 us, but 0.2 ms in 3D, which spills).
  float2 zero = make_float2(0.f, 0.f);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < T; ++b) zero = __ffma2_rn(acc[a][b], make_float2(0.f, 0.f), zero);
  const bool bad = coil < ncg && !(zero.x == 0.f && zero.y == 0.f);
  if (NWARP == 1 ? __any_sync(0xffffffffu, bad) : __syncthreads_or(bad)) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < T; ++b) acc[a][b] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int bi = 0; bi < nbatch; ++bi) {
      sync();  // the batch before is read
      copy_coords(bi);
      cp_async_commit();
      cp_async_wait<0>();
      sync();
      copy_values(bi);
      cp_async_commit();
      weights(bi);
      cp_async_wait<0>();
      sync();
      const int b2 = bi & 1, nb = batch_len(bi);
#pragma unroll 1
      for (int j = stream; j < nb; j += grid_streams<D, CW>()) {
        const GEntry<D, CW>& e = s.e[b2][j];
        const int zc = (int)(s.code[b2][j] & 0xffu), z0 = zc == NW ? 0 : zc, nz = zc == NW ? T : KW;
        float2 v = e.v[coil];
        if (TEMP) {
          const float2 t = s.t[b2][j];
          v = make_float2(v.x * t.x + v.y * t.y, v.y * t.x - v.x * t.y);
        }
        if (D == 3) {
          const float w = e.wx[plane];
          if (w == 0.f) continue;
          v = __fmul2_rn(make_float2(w, w), v);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float w = e.wy[4 * half + r];
          const float2 v2 = __fmul2_rn(make_float2(w, w), v);
#pragma unroll
          for (int z = 0; z < T; ++z) {
            const int c = z - z0;
            const float2 wz = c >= 0 && c < nz ? e.wz[c] : make_float2(0.f, 0.f);
            if (w != 0.f && wz.x != 0.f) acc[r][z] = __ffma2_rn(wz, v2, acc[r][z]);
          }
        }
      }
    }
  }

  if (grid_streams<D, CW>() > 1) {  // add the streams' tiles
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < T; ++b) {
        acc[a][b].x += __shfl_xor_sync(0xffffffffu, acc[a][b].x, 16);
        acc[a][b].y += __shfl_xor_sync(0xffffffffu, acc[a][b].y, 16);
      }
  }

  const int nosy = sel3(gp->nos, D - 2), nosz = sel3(gp->nos, D - 1);
  const int hsx = layout == kInternal ? gp->hshift[0] : 0;
  const int hsy = layout == kInternal ? sel3(gp->hshift, D - 2) : 0;
  const int hsz = layout == kInternal ? sel3(gp->hshift, D - 1) : 0;
  const int sizey = sel3(f.size, D - 2), sizez = sel3(f.size, D - 1);
  const int orgy = sel3(f.org, D - 2), orgz = sel3(f.org, D - 1);
  const int cb = layout == kInternal ? gp->cb : 1;
  float2* dst = grid + (layout == kInternal ? gp->grid_off : gp->ugrid_off);
  const int64_t gos = gp->gos;
  if (it.split || cb > 1 || ncoil == 1) {
    // lanes are coils: the cells of a partial tile and of a grid in coil
    // blocks hold them side by side
    if (coil >= ncg || (D == 3 && plane >= f.size[0]) || stream != 0) return;
    const int64_t xrow = D == 3 ? (int64_t)wrap_once(f.org[0] + plane - hsx, gp->nos[0]) * nosy : 0;
    float2* part = it.split ? split_slot(so, it.split, c0 + coil, plane * sizey * sizez) : nullptr;
    float2* dc = dst + grid_at(gos, cb, c0 + coil, 0);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int y = 4 * half + r;
      if (y >= sizey) break;
      const int64_t row = (xrow + wrap_once(orgy + y - hsy, nosy)) * nosz;
#pragma unroll
      for (int z = 0; z < T; ++z) {
        if (z >= sizez) break;
        if (it.split) {
          part[(int64_t)(y * sizez + z) * so.cell_stride] = acc[r][z];
        } else {
          dc[(row + wrap_once(orgz + z - hsz, nosz)) * cb] = acc[r][z];
        }
      }
    }
    return;
  }
  // Coil planes: through shared memory, a warp's 32 blocks of 4x8 cells at a
  // time (block stride 33 cells: conflict-free 8-byte stores), so that lanes
  // run over the z-cells of a row.
  constexpr int CS = 4 * T + 1;
  float2* stage = reinterpret_cast<float2*>(g_smem);
#pragma unroll 1
  for (int w = 0; w < NWARP; ++w) {
    sync();  // staging buffer free
    if (warp == w) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int z = 0; z < T; ++z) stage[lane * CS + r * T + z] = acc[r][z];
    }
    sync();
    for (int e = tid; e < 32 * 4 * T; e += NT) {
      const int blk = e >> 5, z = e & 7;  // the block's lane
      const int bc = blk % CW, bp = D == 3 ? (w % NPG) * PPW + blk / CW : 0;
      const int bh = D == 3 ? w / NPG : (CW == 32 ? w : (blk / CW) & 1), y = 4 * bh + ((e >> 3) & 3);
      if (bc >= ncg || y >= sizey || z >= sizez) continue;
      if (D == 3 ? bp >= f.size[0] : blk >= 2 * CW) continue;
      const int64_t xrow = D == 3 ? (int64_t)wrap_once(f.org[0] + bp - hsx, gp->nos[0]) * nosy : 0;
      dst[(int64_t)(c0 + bc) * gos + (xrow + wrap_once(orgy + y - hsy, nosy)) * nosz + wrap_once(orgz + z - hsz, nosz)] =
          stage[blk * CS + (e & 31)];
    }
  }
}

// Sample-major copy of the samples: rows[p][c] = ksp[c][p] (x dcf[p]), row
// stride rs (the coils padded to whole blocks; the padding is left alone).
// 64 samples x 16 coils per CTA through shared memory: reads run along a coil's
// row, writes along the rows, both contiguous.
__global__ void __launch_bounds__(256)
k_rows(const SliceGeom* __restrict__ sl, int ns, const float2* __restrict__ ksp, const float* __restrict__ dcf,
       float2* __restrict__ rows) {
  __shared__ float2 tile[16][65];
  for (int s = blockIdx.z; s < ns; s += gridDim.z) {
    const SliceGeom& g = sl[s];
    const int64_t p0 = (int64_t)blockIdx.x * 64;
    if (p0 >= g.m) continue;
    const int np = (int)min((int64_t)64, g.m - p0);
    for (int c0 = blockIdx.y * 16; c0 < g.ncoil; c0 += gridDim.y * 16) {
      const int nc = min(16, g.ncoil - c0);
      __syncthreads();
      for (int e = threadIdx.x; e < 64 * nc; e += 256) {
        const int c = e >> 6, p = e & 63;
        if (p < np) {
          float2 v = __ldg(ksp + g.ksp_off + (int64_t)(c0 + c) * g.m + p0 + p);
          if (dcf) {
            const float d = __ldg(dcf + g.pt_off + p0 + p);
            v = make_float2(v.x * d, v.y * d);
          }
          tile[c][p] = v;
        }
      }
      __syncthreads();
      for (int e = threadIdx.x; e < np * nc; e += 256) {
        const int p = e / nc, c = e - p * nc;
        rows[g.row_off + (p0 + p) * g.rs + c0 + c] = tile[c][p];
      }
    }
  }
}

int launch_rows(mrn_plan* P, const SliceGeom* slices, int ns, const float2* ksp, const float* dcf, float2* rows,
                cudaStream_t st) {
  int64_t m = 0;
  for (int s = 0; s < ns; ++s) m = std::max(m, P->h_slices[s].m);
  if (m == 0) return MRN_OK;
  const dim3 gd((unsigned)((m + 63) / 64), (unsigned)std::min(65535, (P->max_coil + 15) / 16),
                (unsigned)std::min(65535, ns));
  k_rows<<<gd, 256, 0, st>>>(slices, ns, ksp, dcf, rows);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

// Geometry of the register-tile gridding: equal tap counts 5..8 and tiles of
// K - 1 to 8 cells per edge.
bool code_sort_ok(const mrn_plan* P) {
  if (P->ndim < 2) return false;
  const int K = P->kb.ntaps[0];
  if (K < 5 || K > kGTile) return false;
  for (int i = 0; i < P->ndim; ++i)
    if (P->kb.ntaps[i] != K || P->tmax_gcells[i] > kGTile) return false;
  for (const SliceGeom& g : P->h_slices)
    for (int i = 0; i < P->ndim; ++i)
      if (g.nos[i] / g.gntile[i] < K - 1 || g.nos[i] < K || g.gntile[i] < 2) return false;
  return true;
}

// A footprint of a whole width W has W taps unless it lies exactly W/2 from the
// last of its floor(W) + 1 candidates. For other widths half of the footprints
// of an axis have all candidates, so there the kernels count one more, which
// never has weight. Interpolation, up to W 7 (8 taps a row): 3D, 96^3, 8 coils,
// 1 M samples, W 4.5 / 5.5 / 6.5: 830 / 1510 / 1780 -> 510 / 759 / 1138 us. Gridding
// in 2D up to W 6: 4 coils, 98,304 samples, W 4.5 / 5.5: 59 / 64 -> 56 / 59 us (3D, where
// every window costs four rows of a plane: W 4.5 / 5.5 / 6.5 648 / 893 / 1252 -> 642 / 930
// / 1413, so not there).
// Neither where a grid or a gridding tile is too small.
void window_taps(mrn_plan* P) {
  const int K = P->kb.ntaps[0];
  bool whole = true, room = K < 8, groom = P->ndim == 2 && K < 7;
  for (int i = 0; i < P->ndim; ++i) {
    const double f = P->width[i] - std::floor(P->width[i]);
    whole &= f < 0.01 || f > 0.99;
    for (const SliceGeom& g : P->h_slices) {
      room &= g.nos[i] > K;
      groom &= g.nos[i] / g.gntile[i] >= K;
    }
  }
  P->kb.itaps = !whole && room ? K + 1 : K;
  P->kb.gtaps = !whole && room && groom ? K + 1 : K;
}

// The register-tile gridding applies: tiles of at most 8 cells per edge whose
// entries are sorted by window, and a row buffer unless one coil's
// samples are rows already.
bool grid_rows_ok(const mrn_plan* P) {
  if (!P->reg_grid || P->ndim < 2 || !P->code_sorted) return false;
  if (P->ndim == 2 && !P->warp_grid) return false;
  for (int i = 0; i < P->ndim; ++i)
    if (P->tmax_gcells[i] > kGTile) return false;
  return P->d_rows != nullptr;
}

// Grid from rows (launch_rows, or the rows a normal operator's interpolation
// wrote).
int launch_grid_rows(mrn_plan* P, const float2* rows, const float2* temporal, int layout, float2* grid, float scale,
                     cudaStream_t st) {
  if (P->n_items_grid == 0) return MRN_OK;
  const int D = P->ndim, K = P->kb.gtaps, C = P->max_coil;
  // coil groups: whole blocks, so that a group's part of a row starts on 16 bytes
  int cap = D == 3 ? 16 : 32;
  if (P->coil_group_req > 0) cap = std::min(cap, std::max(8, P->coil_group_req / 8 * 8));
  const int ng = (C + cap - 1) / cap;
  const int cg = C <= 8 ? C : std::min(cap, ((C + ng - 1) / ng + 7) / 8 * 8);
  const int groups = (C + cg - 1) / cg;
  const int lanes = D == 2 ? std::max(cg, P->grid_lanes) : cg;
  const dim3 gdim((unsigned)P->n_items_grid, (unsigned)groups);
  const SplitOut so = split_out(P);
  int rc = MRN_OK;
#define MRN_GR_LAUNCH(DD, KK, CC, TT)                                                                          \
  do {                                                                                                         \
    auto kern = k_grid_rows<DD, KK, CC, TT>;                                                                   \
    const size_t smem = std::max(sizeof(GSmem<DD, grid_batch<DD, CC>(), CC>), kGStage);                        \
    rc = set_dynamic_smem(kern, smem);                                                                         \
    if (rc == MRN_OK)                                                                                          \
      kern<<<gdim, grid_threads<DD, CC>(), smem, st>>>(P->d_items_g, P->d_slices, P->kb, P->d_coord_g,         \
                                                       P->d_perm_g, rows, temporal, grid, layout, scale, cg, so); \
  } while (0)
#define MRN_GR_T(DD, KK, CC) if (temporal) MRN_GR_LAUNCH(DD, KK, CC, true); else MRN_GR_LAUNCH(DD, KK, CC, false)
#define MRN_GR_C(DD, KK, C1, C2, C3)         \
  if (lanes > C2) { MRN_GR_T(DD, KK, C1); }  \
  else if (lanes > C3) { MRN_GR_T(DD, KK, C2); } \
  else { MRN_GR_T(DD, KK, C3); }
#define MRN_GR_K(DD, C1, C2, C3)                     \
  if (K == 5) { MRN_GR_C(DD, 5, C1, C2, C3) }        \
  else if (K == 6) { MRN_GR_C(DD, 6, C1, C2, C3) }   \
  else if (K == 7) { MRN_GR_C(DD, 7, C1, C2, C3) }   \
  else { MRN_GR_C(DD, 8, C1, C2, C3) }
  if (D == 2) { MRN_GR_K(2, 32, 16, 8) }
  else { MRN_GR_K(3, 16, 8, 4) }
#undef MRN_GR_K
#undef MRN_GR_C
#undef MRN_GR_T
#undef MRN_GR_LAUNCH
  if (rc != MRN_OK) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

}  // namespace mrn
